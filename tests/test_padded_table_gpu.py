"""The padded cell table where its single-precision steps are coarse beside the
spheres, and where many spheres lie around the K-th, against the oracle's
table."""
import numpy as np
import pytest

from oracle import oracle as oz

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _check(sph, L, nseg, K):
    from nozomi_b200 import engine
    sub = engine.DeviceSubstrate(sph, 1, L, nseg, np.ones(2), np.full(2, 80.0))
    k, seg = sub.padded_segments(K)
    assert k == K
    np.testing.assert_array_equal(seg.cpu().numpy().reshape(-1), np.asarray(oz.segments(sph, L, nseg, K)).reshape(-1))


# spheres of 1e3 to 1e8 box lengths whose surfaces cross the box, as flat walls
@pytest.mark.parametrize("S,nseg,K", [(700, (5, 4, 3), 90), (5000, (9, 2, 7), 300), (3000, (1, 1, 1), 1000)])
def test_spheres_far_larger_than_the_box(S, nseg, K):
    rng = np.random.default_rng(S)
    L = np.array([10.0, 9.0, 12.0])
    sph = np.zeros((5, S))
    # along an axis: that axis alone decides the distance from a cell
    u = (np.eye(3)[rng.integers(0, 3, S)] * rng.choice([-1.0, 1.0], S)[:, None]).T
    sph[3] = 10.0 ** rng.uniform(4.0, 9.0, S)
    sph[:3] = u * (sph[3] + rng.uniform(-6.0, 6.0, S))
    small = rng.random(S) < 0.3
    sph[3, small] = rng.uniform(0.2, 1.5, small.sum())
    sph[:3, small] = rng.uniform(-0.5, 0.5, (3, small.sum())) * L[:, None]
    _check(sph, tuple(L), nseg, K)


# candidates around the K-th by the hundred and by the thousand: few large
# cells, and lattices of equal distances
@pytest.mark.parametrize("kind,S,nseg,K", [
    ("random", 30000, (3, 3, 3), 2500), ("random", 30000, (1, 1, 1), 20000), ("random", 9000, (8, 2, 1), 4500),
    ("lattice", 32768, (2, 2, 2), 9000), ("lattice", 32768, (9, 1, 1), 9001), ("equal", 6000, (4, 1, 1), 3000)])
def test_many_spheres_around_the_kth(kind, S, nseg, K):
    rng = np.random.default_rng(S)
    L = (30.0, 30.0, 30.0)
    sph = np.zeros((5, S))
    sph[3] = 0.5
    if kind == "lattice":
        g = np.stack(np.meshgrid(*[np.arange(32)] * 3, indexing="ij"), 0).reshape(3, -1)
        sph[:3] = ((g + 0.5) / 32 - 0.5) * 30.0
    elif kind == "random":
        sph[:3] = rng.uniform(-17.0, 17.0, (3, S))
        sph[3] = rng.uniform(0.2, 1.0, S)
    _check(sph, L, nseg, K)  # equal: every sphere at the centre, ties throughout
