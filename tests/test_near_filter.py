"""The fused walk's half-precision near filter restated in NumPy, entry
(pack_entry in csrc/cells.cu) and test (near_bits_packed in
csrc/walk_fused.cu), operation by operation: every sphere whose
r (1 + 5e-5) + tol + 2 nm ball comes within reach of the segment is marked,
for walkers anywhere that the near lists serve.  The bound is the one the
entries' radii are derived for; no slack is added here."""
import numpy as np
import pytest

TOL = np.float32(1e-3)
F, H = np.float32, np.float16


def _fma(a, b, c):  # halves: product and sum in double, one rounding that matters
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(H)


def _up(v):  # __float2half_ru
    h = v.astype(H)
    return np.where(h.astype(np.float64) < v, np.nextafter(h, H(np.inf)), h)


def _pack(c, r, h, M):
    u = F(1.0 / 2048)
    rho = r + TOL
    m = F(h) + F(2) * F(M) + rho
    E = F(1.15) * u * (F(3) * m + F(9) * F(M) + F(4) * rho + F(5.5) * F(M) * F(M) / rho)
    R = (r * F(1.00005) + (TOL + F(2e-3)) + E) * F(1.000001)
    fits = (R <= 100) & (np.abs(c) <= 200).all(0)
    with np.errstate(over="ignore"):
        return np.where(fits, c, 0).astype(H), np.where(fits, _up(np.where(fits, R, 0)), H(np.inf))


def _marked(p, j, jr, c, R):
    """Half-precision test of a segment from p (relative to the cell's centre)
    along jr * j."""
    a = (j * j).sum(0, dtype=F)
    ir = (F(1) / np.sqrt(np.maximum(a, F(1e-30)))).astype(F)
    reach = a * ir * jr
    P, e, ln, grow = p.astype(H), (j * ir).astype(H), reach.astype(H), (F(0.02) * reach).astype(H)
    with np.errstate(over="ignore"):  # far spheres: the square overflows to infinity, not near
        d = P - c
        d2 = _fma(d[0], d[0], _fma(d[1], d[1], d[2] * d[2]))
        de = _fma(d[0], e[0], _fma(d[1], e[1], d[2] * e[2]))
        t = np.minimum(np.maximum(-de, H(0)), ln)
        near2 = _fma(t, _fma(de, np.full_like(de, 2), t), d2)
        ro = R + grow
        return near2 <= ro * ro


@pytest.mark.parametrize("edge", [0.05, 0.5, 2.0, 30.0, 1000.0, 1e4])
@pytest.mark.parametrize("M", [0.004, 0.05, 0.4, 0.9, 8.0, 100.0])
def test_no_sphere_in_reach_is_passed_over(edge, M):
    rng = np.random.default_rng(int(edge * 100 + M * 7919))
    n = 200_000
    side = np.array([edge, edge, edge]) * rng.uniform(0.3, 1.0, 3)
    h = F(0.5 * np.sqrt((side ** 2).sum()))
    # the walker in the cell, on its faces and beyond them by the share of the
    # margin that its reach leaves ((distance + reach) * 1.02 + tol + 2 nm <= M)
    room = (M - 3e-3) / 1.02
    reach = room * rng.choice([0.01, 0.3, 0.7, 1.0], n) * rng.uniform(0.3, 1.0, n)
    out = rng.standard_normal((3, n))
    out *= (room - reach) / np.linalg.norm(out, axis=0) * rng.choice([0.0, 0.5, 1.0], n)
    p = rng.uniform(-0.5, 0.5, (3, n)) * side[:, None]
    push = rng.random((3, n)) < 0.4
    p = np.where(push, np.sign(out) * 0.5 * side[:, None], p) + np.where(push, out, 0.0)
    p = p.astype(F)
    e = rng.standard_normal((3, n))
    axis = rng.random(n) < 0.3  # along an axis: one component holds all of the length
    e[:, axis] = np.eye(3)[rng.integers(0, 3, axis.sum())].T * rng.choice([-1, 1], axis.sum())
    e /= np.linalg.norm(e, axis=0)
    jr = rng.choice([1.0, 0.3, 0.01], n).astype(F)
    j = (e * reach / jr).astype(F)
    keep = (j * j).sum(0, dtype=F) >= 1e-8  # shorter jumps mark every entry
    end = p.astype(np.float64) + j.astype(np.float64) * jr
    # spheres whose ball touches the segment at a random point of it, from outside or holding it
    r = (10.0 ** rng.uniform(-3.0, 2.2, n)).astype(F)
    ball = r.astype(np.float64) * 1.00005 + 1e-3 + 2e-3
    out = rng.standard_normal((3, n))
    t = rng.choice([0.0, 1.0, 0.5], n)
    s = end - p
    mid = (t == 0.5)  # sideways from the segment's middle
    k = (out * s).sum(0) / np.maximum((s * s).sum(0), 1e-300)
    out = np.where(mid, out - k * s, out)
    k = np.sign((out * s).sum(0)) * np.where(t == 1.0, 1.0, -1.0)  # beyond its ends
    out = np.where(mid, out, out * np.where(k == 0, 1.0, k))
    out /= np.linalg.norm(out, axis=0)
    c = p + t * s + out * ball * (1 - 1e-9) * rng.choice([1.0, 1.0, 0.9], n)
    c32 = c.astype(F)
    ch, R = _pack(c32, r, h, M)
    # the centre's own rounding to single may move the ball off the segment
    d = p.astype(np.float64) - c32
    w = np.clip(-(d * s).sum(0) / np.maximum((s * s).sum(0), 1e-300), 0.0, 1.0)
    keep &= np.linalg.norm(d + w * s, axis=0) <= ball
    assert keep.sum() > n // 4
    # what the walk reads past 100 um margins or in cells beyond 1e4 um never comes here
    lost = keep & ~_marked(p, j, jr, ch, R)
    assert not lost.any(), (lost.sum(), r[lost][:5], reach[lost][:5], p[:, lost][:, :3])
