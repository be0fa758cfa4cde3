"""Cell and index lists at sphere counts where the sort of long lists changes
its form or what it asks of the device."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

ROOT = Path(__file__).resolve().parents[1]

# In a process of its own: a larger substrate built earlier would leave the
# kernel's shared-memory limit raised.  Ascending, so that no size does that
# for the next.
FRESH = """
import numpy as np
from nozomi_b200 import engine
for S in (384_640, 384_641, 390_000, 393_216, 393_217):
    rng = np.random.default_rng(S)
    sph = np.zeros((5, S))
    sph[:3] = rng.uniform(-20.0, 20.0, (3, S))
    sph[3] = 0.2
    sph[4] = rng.integers(0, 3, S)
    sub = engine.DeviceSubstrate(sph, 3, (40.0,) * 3, (6, 6, 6), np.full(4, 2.0), np.full(4, 80.0), near_margin=0.4)
    perm = sub.perm.cpu().numpy()
    for start, count, items, idx in ((sub.cell_start, sub.cell_count, sub.cell_items, sub.cell_idx),
                                     (*sub.near[:3], sub.near[5])):
        start, count, items, idx = (t.cpu().numpy() for t in (start, count, items, idx))
        for c in (0, 100, 215):
            part = slice(start[c], start[c] + count[c])
            assert count[c] > 128 and (np.diff(items[part]) > 0).all()
            assert np.array_equal(idx[part], np.sort(perm[items[part]]))
print("built")
"""


def test_lists_of_a_fresh_process():
    r = subprocess.run([sys.executable, "-c", FRESH], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "built" in r.stdout, r.stderr[-800:]


# both sides of the bitmap's number of keys; lists of more than 128 entries in
# every cell, and in one cell of many empty ones; a grid of empty cells
@pytest.mark.parametrize("S,nseg,spread", [(1 << 20, 12, 20.0), ((1 << 20) + 1, 12, 20.0), ((1 << 20) + 1, 90, 20.0),
                                           ((1 << 20) + 1, 5, 20.0), ((1 << 20) + 1, 6, 20.0),
                                           (5000, 130, 0.5), (3, 130, 20.0)])
def test_sorted_lists(S, nseg, spread):
    from nozomi_b200 import engine
    rng = np.random.default_rng(S)
    sph = np.zeros((5, S))
    sph[:3] = rng.uniform(-spread, spread, (3, S))
    sph[3] = 0.1
    sph[4] = rng.integers(0, 3, S)
    sub = engine.DeviceSubstrate(sph, 3, (40.0,) * 3, (nseg,) * 3, np.full(4, 2.0), np.full(4, 80.0), jump_tol=0.2)
    n = sub.n_items
    start, count, items, idx = (t.cpu().numpy() for t in (sub.cell_start, sub.cell_count, sub.cell_items[:n],
                                                          sub.cell_idx[:n]))
    assert np.array_equal(start, np.cumsum(count) - count) and count.sum() == n
    inner = np.ones(n, bool)  # entries that follow one of the same cell
    inner[start[count > 0]] = False
    assert (np.diff(items)[inner[1:]] > 0).all()
    idx = idx.astype(np.int64) & (0xFFFF if sub.idx_bytes == 2 else 0xFFFFFFFF)
    assert (np.diff(idx)[inner[1:]] > 0).all()
    cell = np.repeat(np.arange(count.size, dtype=np.int64), count)
    want = cell * S + sub.perm.cpu().numpy()[items]
    assert np.array_equal(np.sort(want), cell * S + idx)


# both sides of each number of lanes a sphere: the counts of all spheres are
# the sums of the counts of short runs of them (pinned to the oracle in
# test_lists_gpu.py), for boxes of one cell to hundreds
@pytest.mark.parametrize("S", [16384, 16385, 524288, 524289])
@pytest.mark.parametrize("nseg", [(1, 1, 1), (5, 3, 40), (61, 60, 59)])
def test_members_by_lanes(S, nseg):
    import ctypes
    from nozomi_b200 import _lib as L
    lib = L.load()
    rng = np.random.default_rng(S)
    box, ncell = (24.0, 25.0, 26.0), nseg[0] * nseg[1] * nseg[2]
    sph = np.zeros((5, S))
    sph[:3] = rng.uniform(-0.6, 0.6, (3, S)) * np.asarray(box)[:, None]
    sph[3] = rng.uniform(0.0, 0.9, S)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731

    def counts(fn, part):
        d = torch.from_numpy(np.ascontiguousarray(part)).cuda()
        c = torch.empty(ncell, dtype=torch.int32, device="cuda")
        L.check(fn(p(d), part.shape[1], *box, *nseg, 0.3, p(c), None), "count")
        return c.cpu().numpy()

    for fn in (lib.nz_cells_count, lib.nz_cells_count_round):
        want = sum(counts(fn, sph[:, i:i + 16000]) for i in range(0, S, 16000))
        np.testing.assert_array_equal(counts(fn, sph), want)
