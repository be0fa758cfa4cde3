"""The plain step over index lists (several lanes a walker) against the same
step over the spheres' arrays (one lane a walker, the reference's two passes):
the same bits in every output.  The second is pinned to the oracle and the
reference in test_gpu_parity.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _run(sub, N, ndir, D, mode, steps=6, dt=0.005):
    from nozomi_b200 import engine
    rng = np.random.default_rng(N)
    L = np.asarray(sub.L)[:, None]
    x = torch.from_numpy((rng.uniform(-0.5, 0.5, (3, N)) * L).astype(np.float32)).cuda()
    d = rng.standard_normal((3, ndir)).astype(np.float32)
    wk = engine.Walkers.with_counters(x.clone(), x.clone(), phase=torch.zeros((ndir, N), device="cuda"),
                                      diffdir=torch.from_numpy(d).cuda(), sig=torch.ones(N, device="cuda"),
                                      phi=torch.zeros((6, N), device="cuda"))
    draws = engine.philox_draws(11)
    for s in range(steps):
        engine.walk_step(sub, wk, mode, dt, 0.7 - 0.2 * s, 0.3, s, draws)
    torch.cuda.synchronize()
    return {k: getattr(wk, k).cpu().numpy() for k in ("spins", "spins0", "phase", "phi", "sig", "label", "n_iter",
                                                     "n_scatter", "flags")}


# 33 and 65: one walker past a block of eight or four lanes each; 57,000: four
# lanes; cell 6: lists too long for the marks (more than 32 entries a lane);
# D per structure: the first jump is longer than the box's, so the marks do
# not cover it; D = 0: no jump, the iteration cap
@pytest.mark.parametrize("N,ndir,cell,D,idx_bytes", [
    (1, 1, 1.0, "same", 2), (33, 3, 1.0, "same", 2), (65, 30, 0.7, "same", 4), (3001, 7, 6.0, "same", 2),
    (2003, 5, 1.0, "inside faster", 2), (500, 2, 1.0, "zero", 4), (57001, 4, 1.0, "same", 2)])
def test_index_list_step_equals_the_array_step(N, ndir, cell, D, idx_bytes):
    from nozomi_b200 import engine, _lib as L
    from nozomi_b200.substrates import axon_bundle, cell_grid
    s = axon_bundle(30, seed=9)
    ns = s.nstructures
    Dv = np.full(ns + 1, {"same": 2.0, "inside faster": 3.0, "zero": 0.0}[D])
    if D == "inside faster":
        Dv[ns] = 0.5
    args = (s.spheres(), ns, s.L, cell_grid(s.L, cell), Dv, np.full(ns + 1, 80.0))
    mode = L.MODE_PHASE | L.MODE_PHI | L.MODE_SIG
    got = _run(engine.DeviceSubstrate(*args, idx_bytes=idx_bytes), N, ndir, D, mode)
    want = _run(engine.DeviceSubstrate(*args, idx_bytes=0), N, ndir, D, mode)
    for k in got:
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
