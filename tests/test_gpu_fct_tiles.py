"""The FCT source's tiles (B200).

k_fct_source computes 16 x 16 cells of a layer per block with halos of one
(ratios), two (faces) and three (field) cells; its edges, remainders and single
rows or columns are checked against the oracle's array form, with and without
the limiter and the lateral-inflow field, for one vector and for several per
block, and where the result overwrites its input.  Tolerance: a few hundred
roundings of the largest value (about fifty operations from input to output).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,n_vec", [((2, 3, 3), 1), ((1, 16, 16), 2), ((3, 17, 15), 5), ((2, 33, 31), 3),
                                         ((2, 2, 40), 1), ((2, 40, 2), 2), ((15, 20, 24), 40)])
@pytest.mark.parametrize("limited", [1, 0])
@pytest.mark.parametrize("ghost", [False, True])
def test_tiles_match_oracle(shape, n_vec, limited, ghost):
    import torch
    from oracle import fct as ofct
    from orbit_b200 import device, synthetic
    nz, ny, nx = shape
    g = synthetic.make_met_bin(np.random.default_rng(3), nz, ny, nx, terrain_amp=4000.0, rho_profile=True)
    md = device.MetDevice(g)
    rng = np.random.default_rng(4)
    c = np.exp(rng.normal(size=(n_vec, md.N)))
    gh = np.exp(rng.normal(size=(n_vec, md.N))) if ghost else None
    got = device.fct_source(md, torch.as_tensor(c, device="cuda"), 10800.0, bool(limited),
                            c_ghost=None if gh is None else torch.as_tensor(gh, device="cuda")).cpu().numpy()
    for v in range(n_vec):
        kw = {} if gh is None else {"c_ghost_flat": gh[v]}
        ref = np.asarray(ofct.fct_source(g, c[v], 10800.0, limited=bool(limited), **kw)).reshape(-1)
        assert np.abs(got[v] - ref).max() <= 400 * 2.0 ** -53 * max(np.abs(ref).max(), 1e-300)


def test_result_over_its_input():
    import ctypes as C
    import torch
    from orbit_b200 import _lib, device, synthetic
    g = synthetic.make_met_bin(np.random.default_rng(5), 3, 19, 35)
    md = device.MetDevice(g)
    c = torch.exp(torch.randn(2, md.N, dtype=torch.float64, device="cuda"))
    ref = device.fct_source(md, c)
    for entry in ("orbit_fct_source", "orbit_fct_source_noalloc"):
        d = c.clone()
        _lib.check(getattr(_lib.lib(), entry)(md.nz, md.ny, md.nx, C.byref(md.struct), 2, _lib.ptr(d), 10800.0, 1,
                                              _lib.ptr(d), torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert torch.equal(d, ref)
