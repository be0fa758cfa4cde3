"""The batched walk's forms (record lists, index lists, packed near lists,
staged records, launches whose jobs differ in packing): the same state of
every walker and no flags, whichever form a launch takes."""
import ctypes
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _specs():
    from nozomi_b200 import batch
    from nozomi_b200.substrates import axon_bundle
    from nozomi_b200.waveforms import PGDiffWaveform
    out = []
    for i, (axons, N, steps) in enumerate([(6, 3001, 90), (25, 1500, 120), (12, 700, 60)]):
        te = steps * 0.005
        gw = PGDiffWaveform(2 * te / 3, te / 3, te, time_step=0.005)
        out.append(batch.JobSpec(axon_bundle(axons, seed=i), gw, np.eye(3), np.array([1.0, 2.0]), N, seed=i, key=i))
    return out


def _states(specs, tuning, threads, width=None, unpacked=()):
    """Final states in walker order; width: index lists of that many bytes;
    unpacked: jobs whose substrates have no near lists."""
    from nozomi_b200 import batch, engine
    cache = batch.SubstrateCache()
    for sp in specs:
        d = cache.get(sp.key, sp.substrate, sp.D, sp.T2, tuning)
        if width:
            d = engine.DeviceSubstrate(sp.substrate.spheres(), d.nstructures, sp.substrate.L, d.nseg, d.D.cpu().numpy(),
                                       d.T2.cpu().numpy(), near_margin=tuning.near_margin, idx_bytes=width)
            cache.items[next(k for k in cache.items if k[0] == sp.key)] = d
        if sp.key in unpacked:
            d.set_near_margin(None)
    run = batch.BatchRun(specs, tuning=tuning, threads=threads, cache=cache).step()
    out = []
    for i in range(len(specs)):
        st = run.final_state(i)
        o = torch.argsort(st.walker_ids())
        out.append([getattr(st, k)[o].view(torch.int32).cpu().numpy() for k in ("pos", "org", "phi", "comp")])
    return run, out


@pytest.mark.parametrize("threads", [32, 128, 256])
def test_forms_agree(threads):
    from nozomi_b200 import simulate
    specs = _specs()
    base = simulate.Tuning(steps_per_launch=50)
    _, want = _states(specs, dataclasses.replace(base, lists="records"), threads)
    assert all((w[3][:, 3] == 0).all() for w in want)  # no flags
    some = sorted(sp.substrate.spheres().shape[1] for sp in specs)[1]  # staged: two jobs of three
    for margin in (0.5, None):
        for width in (2, 4):
            for stage in (0, some, 12288):
                for unpacked in ((), (1,)):
                    t = dataclasses.replace(base, near_margin=margin, stage=stage)
                    run, got = _states(specs, t, threads, width, unpacked)
                    assert run.packed == {width: margin is not None and not unpacked}
                    for g, w in zip(got, want):
                        for a, b in zip(g, w):
                            np.testing.assert_array_equal(a, b, err_msg=f"{margin} {width} {stage} {unpacked}")


def test_packed_bit_over_unpacked_lists():
    """The bit without packed lists: the full lists are walked, with the same
    result; the bit without index lists is refused."""
    from nozomi_b200 import simulate, batch, _lib as L
    specs = _specs()
    base = simulate.Tuning(steps_per_launch=50)
    _, want = _states(specs, base, 128)
    run = batch.BatchRun(specs, tuning=dataclasses.replace(base, near_margin=None), threads=128)
    run.packed = {2: True}
    run.step()
    for i, w in enumerate(want):
        st = run.final_state(i)
        o = torch.argsort(st.walker_ids())
        for k, b in zip(("pos", "org", "phi", "comp"), w):
            np.testing.assert_array_equal(getattr(st, k)[o].view(torch.int32).cpu().numpy(), b, err_msg=k)
    occ = ctypes.c_int(0)
    assert L.load().nz_batch_occupancy(L.MODE_PHI | L.LIST_PACKED, 128, ctypes.byref(occ)) != 0


def test_record_lists_without_near_lists():
    """Full record lists, of which walkers in the box read no structure ids."""
    from nozomi_b200 import simulate
    specs = _specs()
    base = simulate.Tuning(steps_per_launch=50, lists="records")
    _, want = _states(specs, base, 128)
    for near_free in ((0, 1, 2), (1,)):
        _, got = _states(specs, base, 128, unpacked=near_free)
        for g, w in zip(got, want):
            for a, b in zip(g, w):
                np.testing.assert_array_equal(a, b)
