"""The fused walk where every structure has its own D and T2, so that a wrong
label changes jumps and decay: label, signal weight, phase and flags of packed
near lists (safe balls, carried labels) against record lists bit for bit, and
positions, labels and weights against the plain step over the spheres' arrays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

STEPS, DT = 60, 0.005
FIELDS = ("spins", "spins0", "label", "flags", "phi", "sig")


def _start(x):
    from nozomi_b200 import engine
    N = x.shape[1]
    wk = engine.Walkers.with_counters(x.clone(), x.clone(), phi=torch.zeros((6, N), device="cuda"),
                                      sig=torch.ones(N, device="cuda"))
    wk.label -= 1
    return wk


def _fused(sub, x, mode, G):
    from nozomi_b200 import engine
    wk = _start(x)
    st = engine.FusedState.from_walkers(wk)
    for s in range(0, STEPS, 25):  # several launches: the label is carried through the state
        engine.walk_fused(sub, st, mode, DT, G, G, s, min(s + 25, STEPS), engine.philox_draws(9))
    st.to_walkers(wk)
    return {k: getattr(wk, k).cpu().numpy() for k in FIELDS}


@pytest.mark.parametrize("S,ns,r,nseg,margin", [(200, 6, (0.4, 1.3), (6, 6, 6), 0.5), (500, 40, (0.2, 0.8), (9, 4, 7), 0.4),
                                                (60, 3, (1.5, 3.0), (12, 12, 12), 0.8)])
def test_labels_and_weights(S, ns, r, nseg, margin):
    from nozomi_b200 import engine, _lib as L
    rng = np.random.default_rng(S)
    box, N = (7.0, 6.0, 8.0), 3000
    sph = np.zeros((5, S))
    sph[:3] = rng.uniform(-0.55, 0.55, (3, S)) * np.asarray(box)[:, None]
    sph[3] = rng.uniform(*r, S)
    sph[4] = rng.integers(0, ns, S)
    x = torch.from_numpy((rng.uniform(-0.5, 0.5, (3, N)) * np.asarray(box)[:, None]).astype(np.float32)).cuda()
    args = (sph, ns, box, nseg, rng.uniform(0.3, 3.0, ns + 1), rng.uniform(0.5, 3.0, ns + 1))
    G = torch.from_numpy(rng.standard_normal(STEPS).astype(np.float32)).cuda()
    records = engine.DeviceSubstrate(*args, near_margin=margin, idx_bytes=0)
    plain = _start(x)
    arrays = engine.DeviceSubstrate(*args, idx_bytes=0)
    for s in range(STEPS):
        engine.walk_step(arrays, plain, L.MODE_SIG, DT, 0.0, 0.0, s, engine.philox_draws(9))
    for mode in (L.MODE_PHI | L.MODE_SIG, L.MODE_PHI | L.MODE_SIG | L.MODE_TANGENT64):
        want = _fused(records, x, mode, G)
        if not mode & L.MODE_TANGENT64:
            for k in ("spins", "spins0", "label", "flags"):
                np.testing.assert_array_equal(want[k], getattr(plain, k).cpu().numpy(), err_msg=k)
            # one rounding a segment of the walk, at most 100 segments a step
            np.testing.assert_allclose(want["sig"], plain.sig.cpu().numpy(), rtol=100 * STEPS * 2 ** -24)
            assert len(np.unique(want["label"])) > min(ns, 4) - 1 and len(np.unique(want["sig"])) > ns
        for idx in (2, 4):
            for m in (margin, None):
                got = _fused(engine.DeviceSubstrate(*args, near_margin=m, idx_bytes=idx), x, mode, G)
                for k in FIELDS:
                    np.testing.assert_array_equal(got[k], want[k], err_msg=f"{k} {idx} {m} {mode}")
