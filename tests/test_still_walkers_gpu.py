"""Structures without diffusion (D = 0) in the fused walk: a jump of length 0
passes over every sphere beyond the filter's 2 nm, so a walker outside all
spheres ends its step in one iteration, with its decay and without the
iteration-cap flag, whatever the form of the lists.  (Inside a sphere the
quadratic of such a jump has no roots, and the walker stays at the cap.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

STEPS, DT = 25, 0.005
NS, T2 = 4, np.array([20.0, 40.0, 60.0, 80.0, 100.0])


def _scene():
    rng = np.random.default_rng(5)
    S, L, N = 140, (7.0, 6.0, 8.0), 3000
    sph = np.zeros((5, S))
    sph[:3] = rng.uniform(-0.55, 0.55, (3, S)) * np.asarray(L)[:, None]
    sph[3] = rng.uniform(0.2, 0.9, S)
    sph[4] = rng.integers(0, NS, S)
    x = (rng.uniform(-0.5, 0.5, (3, N)) * np.asarray(L)[:, None]).astype(np.float32)
    gap = np.sqrt(((x.T[:, None, :].astype(np.float64) - sph[:3].T[None]) ** 2).sum(-1)) - sph[3]
    return sph, L, torch.from_numpy(x).cuda(), gap


def _walk(sub, x, mode):
    from nozomi_b200 import engine
    N = x.shape[1]
    wk = engine.Walkers.with_counters(x.clone(), x.clone(), phi=torch.zeros((6, N), device="cuda"),
                                      sig=torch.ones(N, device="cuda"))
    wk.label -= 1
    st = engine.FusedState.from_walkers(wk)
    G = torch.full((STEPS,), 0.5, device="cuda")
    engine.walk_fused(sub, st, mode, DT, G, G, 0, STEPS, engine.philox_draws(6))
    st.to_walkers(wk)
    return {k: getattr(wk, k).cpu().numpy() for k in ("spins", "spins0", "phi", "sig", "label", "flags")}


@pytest.mark.parametrize("D", [[0.0] * 5, [2.0, 0.0, 1.0, 0.0, 2.0], [2.0, 2.0, 0.0, 2.0, 0.0], [0.0] * 4 + [1e-12]])
def test_list_forms_agree_without_diffusion(D):
    from nozomi_b200 import engine, _lib as L
    sph, box, x, gap = _scene()
    args = (sph, NS, box, (6, 5, 7), np.array(D), T2)
    for mode in (L.MODE_PHI | L.MODE_SIG, L.MODE_PHI | L.MODE_SIG | L.MODE_TANGENT64):
        want = _walk(engine.DeviceSubstrate(*args, near_margin=0.5, idx_bytes=0), x, mode)
        if max(D) == 0.0:
            far = (gap > 3e-3).all(1)
            assert far.sum() > 100 and not want["flags"][far].any()
            np.testing.assert_allclose(want["sig"][far], np.exp(-STEPS * DT / T2[NS]), rtol=1e-5)
        for idx in (2, 4):
            for margin in (0.5, None):
                got = _walk(engine.DeviceSubstrate(*args, near_margin=margin, idx_bytes=idx), x, mode)
                for k, v in want.items():
                    np.testing.assert_array_equal(got[k], v, err_msg=f"{k} idx {idx} margin {margin}")


def test_batch_without_diffusion():
    from nozomi_b200 import batch, simulate
    from nozomi_b200.substrates import axon_bundle
    from nozomi_b200.waveforms import PGDiffWaveform
    gw = PGDiffWaveform(0.2, 0.1, 0.3, time_step=0.005)
    s = axon_bundle(12, seed=1)
    out = []
    for lists in ("records", "index"):
        spec = batch.JobSpec(s, gw, np.eye(3), np.array([1.0, 2.0]), 4000, seed=3, D=0.0)
        run = batch.BatchRun([spec], tuning=simulate.Tuning(lists=lists, steps_per_launch=30))
        run.prepare().run()
        st = run.final_state(0)
        o = torch.argsort(st.walker_ids())
        out.append((st.comp[:, 3].contiguous().view(torch.int32)[o].cpu().numpy(), st.pos[o].cpu().numpy(),
                    st.phi[o].cpu().numpy()))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a.view(np.int32), b.view(np.int32))
    box = out[1][1][:, 3].view(np.int32) == s.nstructures
    assert (out[1][0][box] != 0).mean() < 0.02  # only walkers within the filter's shell of a surface
