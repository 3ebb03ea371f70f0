"""What the dataflow sweeps keep beside a factor handle (B200).

A handle is made with the tagged results, or where its slots are swept together
with the interleaved ones; schedules, and the tagged results of the latter
handles, are made by the launch that first takes them, and counted from then on.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(shape, sets, seed=5):
    import torch
    from orbit_b200 import device, synthetic
    met = synthetic.make_met(seed, *shape, cmfmc_frac=0.3)
    T = [device.assemble_transport(device.MetDevice(g)) for g in met]
    d = [torch.as_tensor(v, device="cuda") for q in range(sets)
         for v in synthetic.make_species(seed + 1 + q, *shape).sink_diag(met)]
    return [t for _ in range(sets) for t in T], d


def _tagged(sym, slots, bits):
    """Bytes of the tagged, or of the interleaved, results of all slots."""
    return 2 * slots * (sym.info["update_len"] + 2 * sym.N) * bits // 8


def test_made_by_the_launches_that_take_them():
    import torch
    from orbit_b200 import device
    from orbit_b200.symbolic import Symbolic
    shape = (6, 10, 12)
    sym = Symbolic(*shape)
    T, d = _inputs(shape, 1)
    fb = device.FactorBatch(sym, 5, 32, n_sets=1)
    fb.numeric(T, d)
    made = fb.bytes()[1]
    x = torch.exp(torch.randn(5, sym.N, dtype=torch.float64, device="cuda"))
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        fb.chain(x, refine=False)
        fb.chain(x, trans=True, refine=False)
        assert fb.bytes()[1] == made  # five slots of one set: the interleaved ones, from the start
        one = fb.chain(x[:1], trans=True, refine=False)
        assert fb.bytes()[1] == made + _tagged(sym, 5, 32)
        assert torch.equal(fb.chain(x[:1], trans=True, refine=False), one)
    own = device.FactorBatch(sym, 1, 32)
    own.numeric(T, d)
    assert torch.equal(own.chain(x[:1], trans=True, refine=False), one)


@pytest.mark.parametrize("bits,slots,sets", [(64, 3, 3), (64, 3, 1), (32, 3, 3), (32, 1, 1), (32, 2, 5)])
def test_other_handles_do_not_grow(bits, slots, sets):
    import torch
    from orbit_b200 import device
    from orbit_b200.symbolic import Symbolic
    shape = (6, 10, 12)
    sym = Symbolic(*shape)
    T, d = _inputs(shape, sets)
    fb = device.FactorBatch(sym, slots, bits, n_sets=sets)
    more = device.FactorBatch(sym, slots + 1, bits, n_sets=sets)
    made = fb.bytes()[1]
    if slots > 1:
        assert more.bytes()[1] - made == 8 * 74 * sym.N + _tagged(sym, 1, bits)
    fb.numeric(T, d)
    x = torch.exp(torch.randn(slots, sym.N, dtype=torch.float64, device="cuda"))
    for n in (1, slots):
        for trans in (False, True):
            assert torch.isfinite(fb.chain(x[:n], trans=trans, refine=False)).all()
    assert fb.bytes()[1] == made


@pytest.mark.parametrize("bits", [32, 64])
def test_first_sweeps_of_two_handles_at_once(bits):
    import torch
    from orbit_b200 import device
    from orbit_b200.symbolic import Symbolic
    shape = (9, 23, 29)
    T, d = _inputs(shape, 1)
    x = torch.exp(torch.randn(1, int(np.prod(shape)), dtype=torch.float64, device="cuda"))
    sym = Symbolic(*shape)  # its transposed schedule is not there yet
    handles = [device.FactorBatch(sym, 1, bits) for _ in range(2)]
    for fb in handles:
        fb.numeric(T, d)
    torch.cuda.synchronize()
    out, gate = [None, None], threading.Barrier(2)

    def sweep(q):
        with torch.cuda.stream(torch.cuda.Stream()):
            gate.wait()
            out[q] = [handles[q].chain(x, trans=t, refine=False) for t in (True, False)]
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=sweep, args=(q,)) for q in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(*out):
        assert torch.equal(a, b)
    ref = device.FactorBatch(Symbolic(*shape), 1, bits)
    ref.numeric(T, d)
    for a, trans in zip(out[0], (True, False)):
        assert torch.equal(ref.chain(x, trans=trans, refine=False), a)


@pytest.mark.parametrize("bits,species,slots", [(32, 3, 8), (32, 1, 8), (64, 2, 3)])
def test_a_served_entry_is_admitted_by_what_it_comes_to_hold(bits, species, slots):
    import torch
    from orbit_b200 import synthetic
    from orbit_b200.serve import _Entry
    from orbit_b200.symbolic import Symbolic
    shape = (6, 10, 12)
    mets = synthetic.make_met(5, *shape, cmfmc_frac=0.3)
    e = _Entry(None, Symbolic(*shape), mets, [synthetic.make_species(6 + q, *shape).sink_diag(mets) for q in range(species)],
               slots, bits)
    e.build()
    x = torch.exp(torch.randn(slots, e.sym.N, dtype=torch.float64, device="cuda"))
    for n in (1, slots):
        for trans in (False, True):
            e.fb.chain(x[:n], trans=trans, refine=False)
    held = sum(e.fb.bytes())
    e.release()
    assert held <= e.bytes <= 1.01 * held
