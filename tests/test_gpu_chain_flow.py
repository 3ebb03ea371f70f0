"""Chained sweeps (B200): the dataflow kernels of small domains, and the
kernels of many right-hand sides on one factor set.

Sweeps of domains too small to fill the GPU run on kernels that hand tagged
values from task to task, with the factor rows staged in shared memory, and
all transposed sweeps on their column-oriented twin.  Checked against SciPy's
sparse solves bin by bin, on grids with odd extents, one row or column blocks
of every remainder, one-cell separators, a periodic grid, and batches in which
sets are shared: each value within a few hundred roundings of the largest (a
sweep is eight solves with about a hundred operations on the longest path from
an input to an output).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = {64: 2.0 ** -53, 32: 2.0 ** -24}


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("shape,leaf,batch,sets,periodic", [
    ((3, 4, 5), 4, 1, 1, False), ((5, 7, 6), 16, 3, 2, False), ((7, 11, 13), 8, 2, 2, False),
    ((6, 17, 19), 40, 5, 2, False), ((9, 23, 29), 64, 1, 1, False), ((5, 9, 16), 24, 2, 2, True),
    ((2, 2, 3), 1, 1, 1, False),
    # groups of 4, 8 and 16 right-hand sides, whole and not
    ((5, 7, 6), 16, 2, 1, False), ((2, 2, 3), 1, 4, 1, False), ((7, 11, 13), 8, 5, 1, False),
    ((5, 9, 16), 24, 8, 1, True), ((9, 23, 29), 64, 9, 1, False), ((8, 21, 26), 100, 17, 1, False),
    ((6, 17, 19), 40, 33, 1, False)])
def test_sweeps_match_sparse_solves(shape, leaf, batch, sets, periodic, precision):
    import scipy.sparse as sp
    import scipy.sparse.linalg as spl
    import torch
    from orbit_b200 import device, synthetic
    from orbit_b200.symbolic import Symbolic
    nz, ny, nx = shape
    met = synthetic.make_met(5, nz, ny, nx, cmfmc_frac=0.3, periodic=periodic)
    mets = [device.MetDevice(g) for g in met]
    T = [device.assemble_transport(m) for m in mets]
    d = [synthetic.make_species(6 + q, nz, ny, nx).sink_diag(met) for q in range(sets)]
    sym = Symbolic(nz, ny, nx, leaf, periodic=periodic)
    fb = device.FactorBatch(sym, batch, precision, n_sets=sets)
    fb.numeric([t for _ in range(sets) for t in T], [torch.as_tensor(v, device="cuda") for q in range(sets) for v in d[q]])
    which = [o % sets for o in range(batch)]
    x = np.exp(np.random.default_rng(7).normal(size=(batch, sym.N)))
    lu = [[spl.splu((sp.identity(sym.N) + 10800.0 * (device.stencil_to_csr(T[t].cpu().numpy(), nz, ny, nx, periodic)
                                                     + sp.diags(d[q][t]))).tocsc()) for t in range(8)]
          for q in range(sets)]
    for trans in (False, True):
        for t0, t1 in ((0, 8), (3, 5)):
            got = fb.chain(torch.as_tensor(x, device="cuda"), trans=trans, tau0=t0, tau1=t1, refine=False).cpu().numpy()
            for o in range(batch):
                ref = x[o].copy()
                for t in (range(t1 - 1, t0 - 1, -1) if trans else range(t0, t1)):
                    ref = lu[which[o]][t].solve(ref, trans="T" if trans else "N")
                assert np.abs(got[o] - ref).max() <= 800 * EPS[precision] * np.abs(ref).max()
