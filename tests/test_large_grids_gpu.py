"""Grids of more than 2^24 cells, where a cell index no longer fits single
precision: walks and seeding against the plain step over the same spheres on
a coarse grid.  The grid only chooses which spheres are looked at, so
positions, origins and labels agree bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

STEPS, DT = 30, 0.005


def _walk(sub, x, key):
    from nozomi_b200 import engine
    wk = engine.Walkers.with_counters(x.clone(), x.clone())
    for s in range(STEPS):
        engine.walk_step(sub, wk, 0, DT, 0.0, 0.0, s, engine.philox_draws(key))
    return wk


def _fused(sub, x, key):
    from nozomi_b200 import engine, _lib as L
    wk = engine.Walkers.with_counters(x.clone(), x.clone(), phi=torch.zeros((6, x.shape[1]), device="cuda"))
    wk.label -= 1
    st = engine.FusedState.from_walkers(wk)
    z = torch.zeros(STEPS, device="cuda")
    engine.walk_fused(sub, st, L.MODE_PHI, DT, z, z, 0, STEPS, engine.philox_draws(key))
    st.to_walkers(wk)
    return wk


def _same(got, want):
    for k in ("spins", "spins0", "flags"):
        np.testing.assert_array_equal(getattr(got, k).cpu().numpy(), getattr(want, k).cpu().numpy(), err_msg=k)


def test_more_than_2_24_cells():
    """A nearly empty box of 300^3 cells, spheres and walkers in its last
    corner, whose cells have the largest indices."""
    from nozomi_b200 import engine
    rng = np.random.default_rng(2)
    L, S, ns, N = (120.0, 120.0, 120.0), 250, 5, 6000
    sph = np.zeros((5, S))
    sph[:3] = rng.uniform(48.0, 61.0, (3, S))
    sph[3] = rng.uniform(0.4, 1.2, S)
    sph[4] = rng.integers(0, ns, S)
    pos = rng.uniform(49.0, 60.0, (3, N))
    pos[:, :3] = 60.0 - 1e-4  # the last cell of all
    x = torch.from_numpy(pos.astype(np.float32)).cuda()
    args = (sph, ns, L)
    D = (np.full(ns + 1, 2.0), np.full(ns + 1, 80.0))
    want = _walk(engine.DeviceSubstrate(*args, (24, 24, 24), *D, idx_bytes=0), x, 8)
    assert 0.2 < (want.label.cpu().numpy() < ns).mean() < 0.8  # walkers in the spheres and among them
    spins, label = engine.seed(engine.DeviceSubstrate(*args, (24, 24, 24), *D), range(ns), 500, key=3)
    for idx in (2, 4, 0):
        sub = engine.DeviceSubstrate(*args, (300, 300, 300), *D, near_margin=0.6, idx_bytes=idx)
        _same(_fused(sub, x, 8), want)
        _same(_walk(sub, x, 8), want)
        got = engine.seed(sub, range(ns), 500, key=3)
        assert torch.equal(got[0], spins) and torch.equal(got[1], label)
