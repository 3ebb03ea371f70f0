"""Sweeps of the kernels that small grids do not reach (B200).

k_chain in its two block counts, both precisions: two and 16 (FP64: eight) slots
of a 60x54x15 grid, each bin's result checked against its equation A x' = x.
k_multi where the vectors of 16 right-hand sides leave a task's factor rows
room in part, or none: fronts of 1,568 rows from a leaf of 1,456 cells, against
sweeps of one right-hand side and SciPy.

Bounds: a value is off by at most 800 roundings of the largest (the longest sums
run over fifty terms per lane, twice a bin, and the factors'); a residual by that
times the operator's norm.  Against SciPy, one rounding per term of sums of up to
n + m positive terms, twice a bin, and as much for the factors.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = {64: 2.0 ** -53, 32: 2.0 ** -24}


def _problem(shape, sets):
    import scipy.sparse as sp
    import torch
    from orbit_b200 import device, synthetic
    met = synthetic.make_met(5, *shape, cmfmc_frac=0.3)
    T = [device.assemble_transport(device.MetDevice(g)) for g in met]
    d = [synthetic.make_species(6 + q, *shape).sink_diag(met) for q in range(sets)]

    def operator(q, t):
        return (sp.identity(T[t].numel() // 7) + 10800.0 * (device.stencil_to_csr(T[t].cpu().numpy(), *shape)
                                                          + sp.diags(d[q][t]))).tocsc()
    return [t for _ in range(sets) for t in T], [torch.as_tensor(v, device="cuda") for q in d for v in q], operator


@pytest.mark.parametrize("bits,slots", [(32, 16), (64, 8)])
def test_counter_kernels_solve_their_bins(bits, slots):
    import torch
    from orbit_b200 import device
    from orbit_b200.symbolic import Symbolic
    shape = (15, 54, 60)
    sym = Symbolic(*shape)
    many = 1.6e9 * 8 / bits  # factor entries of one bin that divide the block counts
    assert 40e6 < 2 * sym.lunz <= many < slots * sym.lunz
    T, d, operator = _problem(shape, 2)
    fb = device.FactorBatch(sym, slots, bits, n_sets=2)
    fb.numeric(T, d)
    x = np.exp(np.random.default_rng(7).normal(size=(slots, sym.N)))
    x = torch.as_tensor(x, device="cuda")
    for n in (2, slots):
        y = x[:n]
        for t in range(8):
            z = fb.chain(y, tau0=t, tau1=t + 1, refine=False)
            if t in (0, 5):
                for o in (0, n - 1):
                    A = operator(o % 2, t)
                    got, rhs = z[o].cpu().numpy(), y[o].cpu().numpy()
                    norm = np.abs(A).sum(axis=1).max()
                    assert np.abs(A @ got - rhs).max() <= 800 * EPS[bits] * norm * np.abs(got).max()
            y = z
        assert torch.equal(fb.chain(x[:n], refine=False), y)  # eight bins in one launch


def _row_tasks(sym, K):
    """(staged at once, in batches, not staged) row tasks of k_multi, medium schedule."""
    n, m, ldn, ldm = (sym.array(a).astype(int) for a in ("n", "m", "ldn", "ldm"))
    smem = max(108 * 1024 // 4, (sym.info["max_front"] + 16) // 4 * 4 * K)
    items = sym.array("sitems").reshape(-1, 4)
    count = [0, 0, 0]
    for s, r0, r1, kind in items[items[:, 3] < 2].tolist():
        if kind == 0:
            stride = (min(r1 - 1, n[s]) + 3) // 4 * 4
            positions = (min(r1, n[s]) + 3) // 4 * 4 + max(0, r1 - max(r0, n[s]))
        else:
            stride = ldn[s] - r0 // 4 * 4 + ldm[s]
            positions = (n[s] + 3) // 4 * 4 - r0 // 4 * 4 + m[s]
        room = smem - (positions + 3) // 4 * 4 * K
        b1 = (r0 + room // max(stride, 4)) // 4 * 4
        count[2 if room < 4 * stride else 1 if b1 < r1 else 0] += 1
    return count


def test_many_right_hand_sides_where_the_rows_do_not_fit():
    import scipy.sparse.linalg as spl
    import torch
    from orbit_b200 import device
    from orbit_b200.symbolic import Symbolic
    shape, leaf, rhs = (8, 14, 27), 1456, 17  # a group of 16 and one of one
    sym = Symbolic(*shape, leaf)
    assert sym.info["max_front"] == 1568 and min(_row_tasks(sym, 16)) > 10
    T, d, operator = _problem(shape, 1)
    fb, one = device.FactorBatch(sym, rhs, 32, n_sets=1), device.FactorBatch(sym, 1, 32)
    fb.numeric(T, d)
    one.numeric(T, d)
    x = np.exp(np.random.default_rng(7).normal(size=(rhs, sym.N)))
    xd = torch.as_tensor(x, device="cuda")
    lu = [spl.splu(operator(0, t)) for t in (0, 1)]
    for trans in (False, True):
        kw = dict(trans=trans, tau0=0, tau1=2, refine=False)
        got = fb.chain(xd, **kw).cpu().numpy()
        for o in range(rhs):
            alone = one.chain(xd[o:o + 1], **kw)[0].cpu().numpy()
            assert np.abs(got[o] - alone).max() <= 800 * EPS[32] * np.abs(alone).max()
            ref = x[o]
            for t in (1, 0) if trans else (0, 1):
                ref = lu[t].solve(ref, trans="T" if trans else "N")
            assert np.abs(got[o] - ref).max() <= 2 * 4 * 1568 * EPS[32] * np.abs(ref).max()
