"""Chained sweeps over fronts of thousands of rows (B200).

A leaf that holds the whole domain, or half of it, makes dense fronts whose
gathers take several rounds per thread and whose rows are longer than the
shared-memory stage of the row-oriented dataflow kernel.  Checked against
SciPy's sparse solves.  The operators are M-matrices and the vectors positive,
so that all sums are free of cancellation: two bins of two triangular products
with up to n + m terms each, one rounding per term at most, plus as much again
for the factors.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,leaf,front", [((10, 20, 20), 4096, 4000), ((10, 20, 41), 4000, 4200)])
def test_gathers_of_several_rounds(shape, leaf, front):
    import scipy.sparse as sp
    import scipy.sparse.linalg as spl
    import torch
    from orbit_b200 import device, synthetic
    from orbit_b200.symbolic import Symbolic
    nz, ny, nx = shape
    met = synthetic.make_met(5, nz, ny, nx, cmfmc_frac=0.3)
    T = [device.assemble_transport(device.MetDevice(g)) for g in met]
    d = synthetic.make_species(6, nz, ny, nx).sink_diag(met)
    sym = Symbolic(nz, ny, nx, leaf)
    assert sym.info["max_front"] == front  # more than 30 positions for each of 128 threads
    fb = device.FactorBatch(sym, 1, 64)
    fb.numeric(T, [torch.as_tensor(v, device="cuda") for v in d])
    lu = [spl.splu((sp.identity(sym.N) + 10800.0 * (device.stencil_to_csr(T[t].cpu().numpy(), nz, ny, nx)
                                                    + sp.diags(d[t]))).tocsc()) for t in range(2)]
    x = np.exp(np.random.default_rng(7).normal(size=sym.N))
    for trans in (False, True):
        got = fb.chain(torch.as_tensor(x[None], device="cuda"), trans=trans, tau0=0, tau1=2, refine=False)[0].cpu().numpy()
        ref = x
        for t in (1, 0) if trans else (0, 1):
            ref = lu[t].solve(ref, trans="T" if trans else "N")
        assert np.abs(got - ref).max() <= 2 * 4 * front * 2.0 ** -53 * np.abs(ref).max()
