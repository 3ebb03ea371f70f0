"""Transposed sweeps do not depend on the batch (B200).

A column's sum has one order, whatever the chunks (small, medium and large
batches have their own), the lanes per row and the kernel (one right-hand side
per task, or several on one factor set): a receptor alone, in a batch, and on a
factor set that it shares, to the bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [64, 32])
def test_transposed_sweeps_alone_and_in_batches(bits):
    import torch
    from orbit_b200 import device, synthetic
    from orbit_b200.symbolic import Symbolic
    shape = (11, 37, 41)
    met = synthetic.make_met(5, *shape, cmfmc_frac=0.3)
    T = [device.assemble_transport(device.MetDevice(g)) for g in met]
    d = [[torch.as_tensor(v, device="cuda") for v in synthetic.make_species(6 + q, *shape).sink_diag(met)]
         for q in range(2)]
    sym = Symbolic(*shape)
    slots = 63
    # the medium and the large schedule's batches (FP64: from 110 M, both types: from 330 M entries a bin)
    medium = next(b for b in range(1, slots) if b * sym.lunz > 110e6)
    assert 330e6 < slots * sym.lunz and medium * sym.lunz < 330e6
    own = device.FactorBatch(sym, slots, bits, n_sets=2)
    own.numeric(T + T, d[0] + d[1])
    own.map([o % 2 for o in range(slots)])
    one = device.FactorBatch(sym, 17, bits, n_sets=1)
    one.numeric(T, d[0])
    x = torch.exp(torch.randn(slots, sym.N, dtype=torch.float64, device="cuda",
                              generator=torch.Generator(device="cuda").manual_seed(7)))
    for t0, t1 in ((0, 8), (2, 3)):
        kw = dict(trans=True, tau0=t0, tau1=t1, refine=False)
        ref = own.chain(x, **kw)
        assert torch.isfinite(ref).all()
        for n in (1, 2, medium - 1, medium):
            assert torch.equal(own.chain(x[:n], **kw), ref[:n])
        first = x[::2][:17].contiguous()  # those on the first set
        for n in (1, 2, 5, 17):
            assert torch.equal(one.chain(first[:n], **kw), ref[::2][:n])
