"""The fused walk's collision pass (packed near lists, safe balls, marks from
records, walkers spread over warps) against the plain step on the spheres'
arrays, which is pinned to the oracle and the reference in
test_gpu_parity.py: the same positions, origins and labels, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

STEPS, DT = 40, 0.005


def _plain(sub, x, key, steps=STEPS):
    from nozomi_b200 import engine
    wk = engine.Walkers.with_counters(x.clone(), x.clone())
    d = engine.philox_draws(key)
    for s in range(steps):
        engine.walk_step(sub, wk, 0, DT, 0.0, 0.0, s, d)
    return wk


def _fused(sub, x, key, steps=STEPS):
    from nozomi_b200 import engine, _lib as L
    wk = engine.Walkers(x.clone(), x.clone(), phi=torch.zeros((6, x.shape[1]), device="cuda"),
                        label=torch.full((x.shape[1],), -1, dtype=torch.int32, device="cuda"),
                        flags=torch.zeros(x.shape[1], dtype=torch.int32, device="cuda"))
    st = engine.FusedState.from_walkers(wk)
    z = torch.zeros(steps, device="cuda")
    engine.walk_fused(sub, st, L.MODE_PHI, DT, z, z, 0, steps, engine.philox_draws(key))
    st.to_walkers(wk)
    return wk


def _same(got, want):
    for k in ("spins", "spins0", "flags"):
        np.testing.assert_array_equal(getattr(got, k).cpu().numpy(), getattr(want, k).cpu().numpy(), err_msg=k)


def _spheres(kind, S, L, seed):
    """Overlapping spheres of a few structures; big: some of them of 30-150 um
    whose surfaces cross the box (half precision holds the largest badly);
    small: down to 10 nm; ordered: structures in order of the spheres."""
    rng = np.random.default_rng(seed)
    sph = np.zeros((5, S))
    sph[:3] = rng.uniform(-0.6, 0.6, (3, S)) * np.asarray(L)[:, None]
    sph[3] = {"small": rng.uniform(0.01, 0.3, S)}.get(kind, rng.uniform(0.2, 1.4, S))
    if kind == "big":
        n = max(1, S // 10)
        u = rng.standard_normal((3, n))
        u /= np.linalg.norm(u, axis=0)
        sph[3, :n] = rng.uniform(30.0, 150.0, n)
        sph[:3, :n] = u * (sph[3, :n] + rng.uniform(-2.0, 2.0, n))
    ns = max(1, min(6, S // 2))
    sph[4] = np.sort(np.arange(S) % ns) if kind == "ordered" else rng.integers(0, ns, S)
    return sph, ns


# lists of up to 32, 64 and more entries; one sphere; 32-bit lists; cells much
# larger and much smaller than the spheres
@pytest.mark.parametrize("kind,S,L,nseg,margin,D", [
    ("mixed", 1, (5.0, 5.0, 5.0), (4, 4, 4), 0.5, 2.0),
    ("mixed", 7, (5.0, 6.0, 7.0), (3, 5, 7), 0.3, 2.0),
    ("ordered", 150, (6.0, 6.0, 6.0), (6, 6, 6), 0.5, 2.0),
    ("mixed", 400, (6.0, 5.0, 7.0), (2, 1, 3), 0.9, 2.0),
    ("small", 900, (4.0, 4.0, 4.0), (9, 9, 9), 0.4, 0.5),
    ("big", 60, (8.0, 8.0, 8.0), (8, 8, 8), 0.6, 2.0),
    ("mixed", 300, (12.0, 12.0, 12.0), (40, 40, 40), 0.7, 4.0),
    ("mixed", 120, (6.0, 6.0, 6.0), (6, 6, 6), 0.5, 1e-7),   # jumps too short for the filter
    ("mixed", 120, (6.0, 6.0, 6.0), (6, 6, 6), 0.5, 40.0),   # jumps beyond the near margin
])
def test_list_forms_match_the_array_step(kind, S, L, nseg, margin, D):
    from nozomi_b200 import engine
    sph, ns = _spheres(kind, S, L, S)
    rng = np.random.default_rng(S + 1)
    N = 700
    x = torch.from_numpy((rng.uniform(-0.5, 0.5, (3, N)) * np.asarray(L)[:, None]).astype(np.float32)).cuda()
    args = (sph, ns, L, nseg, np.full(ns + 1, D), np.full(ns + 1, 80.0))
    want = _plain(engine.DeviceSubstrate(*args, idx_bytes=0), x, S)
    for idx in (2, 4, 0):
        for m in (margin, None):
            _same(_fused(engine.DeviceSubstrate(*args, near_margin=m, idx_bytes=idx), x, S), want)
    _same(_fused(engine.DeviceSubstrate(*args, near_margin=margin, near_round=False), x, S), want)


# both sides of every number of walkers a warp, and of a CTA's share
@pytest.mark.parametrize("N", [1, 3, 1250, 1251, 2500, 2501, 5000, 5001, 10001, 20000, 20001])
def test_walkers_spread_over_warps(N):
    from nozomi_b200 import engine
    from nozomi_b200.substrates import axon_bundle, cell_grid
    s = axon_bundle(20, seed=3)
    ns = s.nstructures
    args = (s.spheres(), ns, s.L, cell_grid(s.L, 1.0), np.full(ns + 1, 2.0), np.full(ns + 1, 80.0))
    sub = engine.DeviceSubstrate(*args, near_margin=0.5)
    x, _ = engine.seed(sub, range(ns + 1), N, key=4)
    _same(_fused(sub, x, 9, 12), _plain(engine.DeviceSubstrate(*args, idx_bytes=0), x, 9, 12))


# jumps and margins of hundreds of um: squared distances of spheres within
# reach pass the largest half-precision number
@pytest.mark.parametrize("margin,D", [(90.0, 3e4), (300.0, 1e6)])
def test_long_jumps_match_the_array_step(margin, D):
    from nozomi_b200 import engine
    rng = np.random.default_rng(11)
    S, L, N, ns = 60, (1500.0, 1500.0, 1500.0), 4000, 4
    sph = np.zeros((5, S))
    sph[:3] = rng.uniform(-700.0, 700.0, (3, S))
    sph[3] = rng.uniform(60.0, 98.0, S)
    sph[4] = rng.integers(0, ns, S)
    x = torch.from_numpy(rng.uniform(-750.0, 750.0, (3, N)).astype(np.float32)).cuda()
    args = (sph, ns, L, (3, 3, 3), np.full(ns + 1, D), np.full(ns + 1, 80.0))
    want = _plain(engine.DeviceSubstrate(*args, jump_tol=700.0, idx_bytes=0), x, 5)
    _same(_fused(engine.DeviceSubstrate(*args, jump_tol=700.0, near_margin=margin), x, 5), want)
