"""The plain step's two forms on both sides of the rule that chooses between
them (entries a cell, walkers, directions): the same bits as over the spheres'
arrays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _run(sub, N, ndir, steps=5):
    from nozomi_b200 import engine, _lib as L
    rng = np.random.default_rng(N)
    x = torch.from_numpy((rng.uniform(-0.5, 0.5, (3, N)) * 20.0).astype(np.float32)).cuda()
    d = torch.from_numpy(rng.standard_normal((3, ndir)).astype(np.float32)).cuda()
    wk = engine.Walkers.with_counters(x.clone(), x.clone(), phase=torch.zeros((ndir, N), device="cuda"), diffdir=d)
    for s in range(steps):
        engine.walk_step(sub, wk, L.MODE_PHASE, 0.005, 0.4, 0.2, s, engine.philox_draws(5))
    return {k: getattr(wk, k).cpu().numpy() for k in ("spins", "spins0", "phase", "label", "n_iter", "n_scatter", "flags")}


@pytest.mark.parametrize("N,ndir", [(16384, 8), (16385, 8), (100, 1), (500_001, 2)])
@pytest.mark.parametrize("S", [0, 12, 60, 200])  # 0, 0.5, 2 and 7 entries a cell
def test_forms_by_entries_a_cell(N, ndir, S):
    from nozomi_b200 import engine
    rng = np.random.default_rng(S)
    ns = min(S, 5)
    sph = np.zeros((5, S))
    sph[:3] = rng.uniform(-10.0, 10.0, (3, S))
    sph[3] = 1.5
    sph[4] = np.arange(S) % max(ns, 1)
    args = (sph, ns, (20.0,) * 3, (10, 10, 10), np.full(ns + 1, 2.0), np.full(ns + 1, 80.0))
    got = _run(engine.DeviceSubstrate(*args), N, ndir)
    want = _run(engine.DeviceSubstrate(*args, idx_bytes=0), N, ndir)
    for k in got:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
