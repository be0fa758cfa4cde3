"""nz_substrate.near_items is optional (0: not given): packed near lists are
walked the same without it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_margin_below_single_precision_builds():
    """Such near lists stay unpacked, and the plain step walks beside them."""
    from nozomi_b200 import engine
    sph = np.array([[0.0], [0.0], [0.0], [1.0], [0.0]])
    sub = engine.DeviceSubstrate(sph, 1, (4.0,) * 3, (4, 4, 4), np.full(2, 2.0), np.full(2, 80.0), near_margin=1e-46)
    assert not sub.near_packed and sub.near is not None
    x = torch.zeros((3, 10), device="cuda")
    wk = engine.Walkers.with_counters(x, x.clone())
    engine.walk_step(sub, wk, 0, 0.005, 0.0, 0.0, 0, engine.philox_draws(1))
    assert (wk.label == 0).all()


@pytest.mark.parametrize("S", [1, 2, 3, 4, 301])  # the radii end inside or on a 16-byte line
def test_packed_lists_without_their_length(S):
    from nozomi_b200 import engine, _lib as L
    rng = np.random.default_rng(S)
    box, ns, N, steps = (6.0, 7.0, 5.0), min(S, 5), 2000, 40
    sph = np.zeros((5, S))
    sph[:3] = rng.uniform(-0.5, 0.5, (3, S)) * np.asarray(box)[:, None]
    sph[3] = rng.uniform(0.3, 1.4, S)
    sph[4] = np.arange(S) % ns
    x = torch.from_numpy((rng.uniform(-0.5, 0.5, (3, N)) * np.asarray(box)[:, None]).astype(np.float32)).cuda()
    out = []
    for idx, given in ((0, True), (2, True), (2, False), (4, False)):
        sub = engine.DeviceSubstrate(sph, ns, box, (6, 7, 5), np.full(ns + 1, 2.0), np.full(ns + 1, 80.0),
                                     near_margin=0.5, idx_bytes=idx)
        if not given:
            sub.near_n = 0
            assert sub.near_packed and sub.struct().near_items == 0
        wk = engine.Walkers.with_counters(x.clone(), x.clone(), phi=torch.zeros((6, N), device="cuda"))
        wk.label -= 1
        st = engine.FusedState.from_walkers(wk)
        z = torch.ones(steps, device="cuda")
        engine.walk_fused(sub, st, L.MODE_PHI, 0.005, z, z, 0, steps, engine.philox_draws(2))
        st.to_walkers(wk)
        out.append([getattr(wk, k).cpu().numpy() for k in ("spins", "spins0", "phi", "label", "flags")])
    for got in out[1:]:
        for a, b in zip(got, out[0]):
            np.testing.assert_array_equal(a, b)
