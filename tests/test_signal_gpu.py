"""nz_signal_phi at the sizes where its split over threads, tiles and blocks
can go wrong, against 64-bit sums.

The kernel forms each walker's phase and angle in float32 in the order given
here, so the angles are the same numbers; a float32 sine or cosine is then
within 2^-22 of the true one (two units in the last place of 1), and the sums
are FP64, so a sum of N walkers is within N 2^-22 of the 64-bit sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("N,ndir,nb,scale", [
    (1, 1, 1, 1.0), (2, 3, 1, 1.0), (63, 1, 5, 1.0), (511, 6, 4, 1.0), (513, 30, 4, 1.0), (2003, 97, 4, 1.0),
    (1025, 129, 3, 1.0), (700, 200, 7, 1.0), (100_003, 30, 4, 1.0), (3000, 12, 4, 3.0e3), (1500, 5, 2, 1.0e6)])
def test_signal_sums_match_64_bits(N, ndir, nb, scale):
    """scale: size of the phases, up to angles that need the long argument
    reduction."""
    from nozomi_b200 import engine
    rng = np.random.default_rng(N + ndir)
    phi = np.zeros((6, N), np.float32)
    phi[:3] = rng.normal(0, scale, (3, N))
    phi[3:] = rng.normal(0, 1e-6 * scale, (3, N))
    d = rng.standard_normal((3, ndir))
    d = (d / np.linalg.norm(d, axis=0)).astype(np.float32)
    amps = np.linspace(0.0, 2.5, nb).astype(np.float32)
    x = torch.zeros((3, N), device="cuda")
    st = engine.FusedState.from_walkers(engine.Walkers(x, x.clone(), phi=torch.from_numpy(phi).cuda()))
    out = st.signal(torch.from_numpy(d).cuda().contiguous(), torch.from_numpy(amps).cuda()).cpu().numpy()
    p = phi[:3] - phi[3:]
    want = np.zeros((2, ndir, nb))
    for i in range(ndir):
        ph = (p[0] * d[0, i] + p[1] * d[1, i]) + p[2] * d[2, i]
        for b in range(nb):
            a = (amps[b] * ph).astype(np.float64)
            want[:, i, b] = np.cos(a).sum(), np.sin(a).sum()
    assert np.abs(out - want).max() <= N * 2.0**-22


def test_signal_of_non_finite_phases_is_nan():
    """One NaN and one infinite phase among 600 walkers (two tiles): every sum is NaN."""
    from nozomi_b200 import engine
    phi = np.zeros((6, 600), np.float32)
    phi[0, 3], phi[1, 550] = np.nan, np.inf
    x = torch.zeros((3, 600), device="cuda")
    st = engine.FusedState.from_walkers(engine.Walkers(x, x.clone(), phi=torch.from_numpy(phi).cuda()))
    d = torch.ones((3, 2), device="cuda")
    assert torch.isnan(st.signal(d, torch.ones(2, device="cuda"))).all()


def test_a_walker_adds_the_same_numbers_wherever_it_stands():
    """One walker alone, first and last of a few, and beside one of a large
    angle: its cosine and sine are the same bits each time (sums of two
    float32 numbers are exact in FP64)."""
    from nozomi_b200 import engine
    d = torch.tensor([[1.0], [0.0], [0.0]], device="cuda")
    one = torch.ones(1, device="cuda")

    def sums(v):
        phi = np.zeros((6, len(v)), np.float32)
        phi[0] = v
        x = torch.zeros((3, len(v)), device="cuda")
        st = engine.FusedState.from_walkers(engine.Walkers(x, x.clone(), phi=torch.from_numpy(phi).cuda()))
        return st.signal(d, one).cpu().numpy().ravel()

    rng = np.random.default_rng(3)
    for v in rng.normal(0, 30.0, 40).astype(np.float32):
        alone, zero, big = sums([v]), sums([0.0]), sums([3.0e5])
        np.testing.assert_array_equal(sums([v, 0.0]) - zero, alone)
        np.testing.assert_array_equal(sums([0.0, 0.0, v]) - 2 * zero, alone)
        np.testing.assert_allclose(sums([v, 3.0e5]) - big, alone, rtol=0, atol=1e-15)


def test_signal_of_many_pairs():
    """More (direction, b) pairs than 65,535 blocks hold; the last and a few
    others against 64 bits, with the bound above."""
    from nozomi_b200 import engine
    ndir, nb, N = 70_000, 370, 3
    rng = np.random.default_rng(1)
    phi = np.zeros((6, N), np.float32)
    phi[:3] = rng.normal(0, 1.0, (3, N))
    d = rng.standard_normal((3, ndir)).astype(np.float32)
    amps = np.linspace(0.0, 2.5, nb).astype(np.float32)
    x = torch.zeros((3, N), device="cuda")
    st = engine.FusedState.from_walkers(engine.Walkers(x, x.clone(), phi=torch.from_numpy(phi).cuda()))
    out = st.signal(torch.from_numpy(d).cuda().contiguous(), torch.from_numpy(amps).cuda())
    for i in (0, 1, 33_333, ndir - 1):
        ph = (phi[0] * d[0, i] + phi[1] * d[1, i]) + phi[2] * d[2, i]
        a = (amps[:, None] * ph[None]).astype(np.float64)
        want = np.stack([np.cos(a).sum(1), np.sin(a).sum(1)])
        assert np.abs(out[:, i].cpu().numpy() - want).max() <= N * 2.0**-22
