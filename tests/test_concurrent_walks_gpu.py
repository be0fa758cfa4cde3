"""Small walks on several streams at once, where the walkers a warp depend on
what the other streams have in flight: the same state as alone, also while
another thread captures a graph, and inside a capture."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

STEPS = 60


@pytest.fixture(scope="module")
def scene():
    from nozomi_b200 import engine
    from nozomi_b200.substrates import axon_bundle, cell_grid
    s = axon_bundle(15, seed=2)
    ns = s.nstructures
    sub = engine.DeviceSubstrate(s.spheres(), ns, s.L, cell_grid(s.L, 1.0), np.full(ns + 1, 2.0), np.full(ns + 1, 80.0),
                                 near_margin=0.5)
    return sub, ns, torch.ones(STEPS, device="cuda")


def _start(scene, N, key):
    from nozomi_b200 import engine
    sub, ns, _ = scene
    x, lab = engine.seed(sub, range(ns + 1), N, key=key)
    return engine.FusedState.from_walkers(engine.Walkers(x, x.clone(), phi=torch.zeros((6, N), device="cuda"), label=lab))


def _go(scene, st, key, s0=0, s1=STEPS):
    from nozomi_b200 import engine, _lib as L
    sub, _, G = scene
    engine.walk_fused(sub, st, L.MODE_PHI, 0.005, G, G, s0, s1, engine.philox_draws(key))


def _bits(st):
    return [getattr(st, k).view(torch.int32).cpu().numpy() for k in ("pos", "org", "phi", "comp")]


def _equal(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


# more streams than the library keeps events for; walkers on both sides of the
# numbers that set the walkers a warp
@pytest.mark.parametrize("N", [700, 2003, 5001, 30000])
def test_streams(scene, N):
    want = []
    for k in range(40):
        st = _start(scene, N, k)
        _go(scene, st, k)
        torch.cuda.synchronize()
        want.append(_bits(st))
    states = [_start(scene, N, k) for k in range(40)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(40)]
    for half in ((0, STEPS // 2), (STEPS // 2, STEPS)):
        for k, (st, stream) in enumerate(zip(states, streams)):
            with torch.cuda.stream(stream):
                _go(scene, st, k, *half)
    torch.cuda.synchronize()
    for st, w in zip(states, want):
        _equal(_bits(st), w)


def test_threads(scene):
    want = []
    for k in range(6):
        st = _start(scene, 1500, k)
        _go(scene, st, k)
        want.append(_bits(st))
    got, failed = {}, []
    states = [_start(scene, 1500, k) for k in range(6)]
    torch.cuda.synchronize()

    def work(k):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for s in range(0, STEPS, 10):
                    _go(scene, states[k], k, s, s + 10)
            stream.synchronize()
            got[k] = _bits(states[k])
        except Exception as e:  # reported by the main thread
            failed.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for k in range(6):
        _equal(got[k], want[k])


def test_beside_and_inside_a_capture(scene):
    """A walk launched on another stream while a graph is being captured in
    the global mode neither disturbs the capture nor fails."""
    plain, captured, beside = (_start(scene, 1500, 1) for _ in range(3))
    _go(scene, plain, 1)
    want = _bits(plain)
    failed = []
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):  # something in flight, its event known
        warm = _start(scene, 1500, 2)
        _go(scene, warm, 2)
    torch.cuda.synchronize()

    def work():
        try:
            with torch.cuda.stream(side):
                _go(scene, beside, 1)
        except Exception as e:
            failed.append(e)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="global"):
        _go(scene, captured, 1)
        t = threading.Thread(target=work)
        t.start()
        t.join()
    assert not failed
    torch.cuda.synchronize()
    _equal(_bits(beside), want)
    graph.replay()
    torch.cuda.synchronize()
    _equal(_bits(captured), want)
