"""The padded cell table at the sizes where its selection can go wrong,
against the oracle's table (same distances, same order of ties), which is
pinned to the reference's."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as oz

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _spheres(kind, S, L):
    rng = np.random.default_rng(S)
    sph = np.zeros((5, S))
    if kind == "random":
        sph[:3] = rng.uniform(-0.55, 0.55, (3, S)) * np.asarray(L)[:, None]
        sph[3] = rng.uniform(0.2, 1.6, S)
    else:  # a lattice of equal spheres: hundreds of equal distances in a cell
        k = int(np.ceil(S ** (1 / 3)))
        g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), 0).reshape(3, -1)[:, :S]
        sph[:3] = ((g + 0.5) / k - 0.5) * np.asarray(L)[:, None]
        sph[3] = 0.5
    return sph


@pytest.mark.parametrize("kind,S,L,nseg,K", [
    ("random", 300, (6.0, 5.0, 7.0), (4, 3, 5), 300),     # K = S: every sphere in every list
    ("random", 300, (6.0, 5.0, 7.0), (4, 3, 5), 299),
    ("random", 300, (6.0, 5.0, 7.0), (1, 1, 1), 1),
    ("random", 33, (8.0, 8.0, 8.0), (9, 2, 3), 32),       # a row of one full and one short run of cells
    ("random", 5000, (20.0, 20.0, 40.0), (17, 9, 11), 61),
    ("random", 2000, (10.0, 10.0, 10.0), (3, 16, 16), 700),
    ("lattice", 1000, (10.0, 10.0, 10.0), (5, 5, 5), 130),  # ties by the hundred
    ("lattice", 4096, (16.0, 16.0, 16.0), (8, 8, 8), 500),
    ("lattice", 4096, (16.0, 16.0, 16.0), (2, 1, 3), 1999),
])
def test_padded_table_matches_oracle(kind, S, L, nseg, K):
    from nozomi_b200 import engine
    sph = _spheres(kind, S, L)
    sub = engine.DeviceSubstrate(sph, 1, L, nseg, np.ones(2), np.full(2, 80.0))
    k, seg = sub.padded_segments(K)
    want = oz.segments(sph, L, nseg, K)
    assert k == K
    np.testing.assert_array_equal(seg.cpu().numpy().reshape(-1), np.asarray(want).reshape(-1))


@pytest.mark.parametrize("S,L,nseg,order", [
    (1, (4.0, 4.0, 4.0), (2, 2, 2), "ids"), (40, (4.0, 4.0, 4.0), (1, 1, 1), "ids"),
    (31, (6.0, 5.0, 7.0), (3, 2, 4), "shuffled"), (400, (9.0, 9.0, 9.0), (9, 9, 9), "shuffled"),
    (6000, (12.0, 11.0, 13.0), (2, 3, 2), "shuffled"),     # lists of hundreds: the bitmap sort
    (70000, (40.0, 40.0, 40.0), (12, 12, 12), "shuffled"),  # 32-bit index lists
    (3000, (30.0, 30.0, 30.0), (40, 30, 20), "ids")])       # more cells than one scan tile
def test_member_near_and_index_lists(S, L, nseg, order):
    """Member lists against the oracle's; near lists are the members within
    the margin by the box test and the Euclidean one; index lists are the records of the members,
    ascending.  Structures given in order of the spheres, or shuffled (the
    index lists then need their sort)."""
    from nozomi_b200 import engine
    sph = _spheres("random", S, L)
    ns = max(1, min(50, S // 3))
    sph[4] = np.random.default_rng(1).integers(0, ns, S) if order == "shuffled" else np.sort(np.arange(S) % ns)
    sub = engine.DeviceSubstrate(sph, ns, L, nseg, np.ones(ns + 1), np.full(ns + 1, 80.0), near_margin=0.4)
    start, count, items = oz.cells(sph, L, nseg)
    np.testing.assert_array_equal(sub.cell_count.cpu().numpy(), count)
    np.testing.assert_array_equal(sub.cell_start.cpu().numpy(), start)
    np.testing.assert_array_equal(sub.cell_items[:sub.n_items].cpu().numpy(), items)
    perm = sub.perm.cpu().numpy()
    st, ct, it = (t.cpu().numpy() for t in sub.near[:3])
    assert np.array_equal(st, np.concatenate([[0], np.cumsum(ct)[:-1]]))
    cell = np.repeat(np.arange(count.size), count)
    n, m, p = cell % nseg[0], (cell // nseg[0]) % nseg[1], cell // (nseg[0] * nseg[1])
    gap2, box, d = np.zeros(items.size), np.full(items.size, -np.inf), np.asarray(L) / np.asarray(nseg)
    for a, i in enumerate((n, m, p)):
        lo = i * d[a] - L[a] / 2
        off = np.maximum(lo - sph[a, items], sph[a, items] - (lo + d[a]))
        box = np.maximum(box, off - sph[3, items])  # the box test's distance: near lists lie within its window
        gap2 += np.maximum(np.maximum(lo - sph[a, items], 0.0), sph[a, items] - (lo + d[a])) ** 2
    R = sph[3, items] + 0.4
    want_in = (gap2 <= (R + 1e-4 - 1e-9) ** 2) & (box < 0.4 - 1e-9)
    want_out = (gap2 > (R + 1e-4 + 1e-9) ** 2) | (box > 0.4 + 1e-9)
    near = set(zip(np.repeat(np.arange(ct.size), ct).tolist(), it[:ct.sum()].tolist()))
    pairs = list(zip(cell.tolist(), items.tolist()))
    assert near >= {q for q, y in zip(pairs, want_in) if y} and not near & {q for q, y in zip(pairs, want_out) if y}
    for cs, cc, members, idx in ((start, count, items, sub.cell_idx), (st, ct, it, sub.near[5])):
        idx = idx.cpu().numpy().astype(np.int64) & (0xFFFF if sub.idx_bytes == 2 else 0xFFFFFFFF)
        for c in np.flatnonzero(cc)[:: max(1, cc.size // 300)]:
            mem = members[cs[c]:cs[c] + cc[c]]
            assert (np.diff(mem) > 0).all()
            np.testing.assert_array_equal(idx[cs[c]:cs[c] + cc[c]], np.sort(perm[mem]))


# out of place, in place, and out one element before in
@pytest.mark.parametrize("shift", [None, 0, 1])
@pytest.mark.parametrize("n", [1, 9000, 100_003])
def test_scan_in_place_and_overlapping(n, shift):
    from nozomi_b200 import _lib as L
    v = np.random.default_rng(n).integers(0, 9, n).astype(np.int32)
    buf = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    src = buf[(shift or 0):][:n]
    src.copy_(torch.from_numpy(v))
    out = torch.empty(n, dtype=torch.int32, device="cuda") if shift is None else buf[:n]
    total = torch.zeros(1, dtype=torch.int32, device="cuda")
    L.check(L.load().nz_exclusive_scan_i32(ctypes.c_void_p(src.data_ptr()), ctypes.c_void_p(out.data_ptr()), n,
                                           ctypes.c_void_p(total.data_ptr()), None), "nz_exclusive_scan_i32")
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), np.cumsum(v) - v)
    assert int(total.item()) == v.sum()
