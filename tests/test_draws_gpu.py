"""The walks' draws on the device against the oracle's, bit for bit: the
packed Box-Muller transform (two word pairs side by side, its divisions and
roots without the general operators' range checks) on the word range's ends,
both sides of every mantissa and quadrant boundary, and random words."""
import numpy as np
import pytest

from oracle import oracle as oz

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _edges():
    powers = np.array([1 << k for k in range(32)], np.uint64)
    near = np.concatenate([powers - 1, powers, powers + 1, powers + (powers >> 1), (1 << 32) - powers])
    # u = sqrt(1/2) of every binade: the logarithm's range split
    split = np.array([int(2.0 ** (k + 0.5)) + d for k in range(32) for d in (-1, 0, 1)], np.uint64)
    quads = np.array([(q << 30) + d for q in range(4) for d in (0, 1, 2**29 - 1, 2**29, 2**29 + 1, 2**30 - 1)], np.uint64)
    return np.unique(np.concatenate([near, split]) & 0xFFFFFFFF), np.unique(quads & 0xFFFFFFFF)


@pytest.mark.parametrize("what", ["edges", "random"])
def test_device_box_muller_equals_the_oracle(what):
    from nozomi_b200 import _lib as L
    if what == "edges":
        ua, ub = (g.ravel() for g in np.meshgrid(*_edges(), indexing="ij"))
    else:
        ua, ub = np.random.default_rng(5).integers(0, 1 << 32, (2, 1 << 20), dtype=np.uint64)
    ua, ub = ua.astype(np.uint32), ub.astype(np.uint32)
    roll = ua.size // 3  # the second pair beside an unrelated first one
    words = np.stack([ua, ub, np.roll(ua, roll), np.roll(ub, roll)], axis=1)
    w = torch.from_numpy(np.ascontiguousarray(words).view(np.int32)).cuda()
    out = torch.empty((ua.size, 4), dtype=torch.float32, device="cuda")
    L.check(L.load().nz_probe_box_muller(w.data_ptr(), ua.size, out.data_ptr(), None), "nz_probe_box_muller")
    torch.cuda.synchronize()
    want = oz.box_muller_pairs(ua, ub)
    got = out.cpu().numpy()
    assert np.array_equal(got[:, :2].view(np.uint32), want.view(np.uint32))
    assert np.array_equal(got[:, 2:].view(np.uint32), np.roll(want, roll, axis=0).view(np.uint32))
