"""One handle, several clouds: buffers, lists and graph of one cloud serve the next one.
Chosen sets grow, shrink and grow again; bits against the oracle."""
import ctypes
import functools

import numpy as np
import pytest

import oracle as O
from gpu_util import bits_equal, require_cuda
from ridgedetection_b200 import generators as G

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rdb():
    require_cuda()
    import ridgedetection_b200 as rdb
    return rdb


def _scaled(n, dim, scale, seed):
    """n points of a curve: more chosen points with the scale."""
    P = (G.sine2d if dim == 2 else G.helix3d)(n, seed=seed)
    return np.ascontiguousarray(P * np.float32(scale))


@functools.lru_cache(maxsize=None)
def _ridge(n, dim, scale, seed, r1):
    P = _scaled(n, dim, scale, seed)
    return P, O.ridge_bf(P, r1, 2 * r1)[0]


@pytest.mark.parametrize("n,dim,r1", [(700, 2, 0.2), (6000, 2, 0.1), (66_000, 3, 0.4), (12, 3, 0.3)])
@pytest.mark.parametrize("mode", ["LOOP_GRAPH", "LOOP_HOST"])
def test_one_handle_many_clouds(rdb, n, dim, r1, mode):
    h = rdb.BruteForceRidgeDetection(n, r1, 2 * r1, dim, loop_mode=getattr(rdb, mode))
    counts = set()
    for k, scale in enumerate((1.0, 0.5, 3.0, 0.7, 1.0, 3.1, 0.1)):
        P, want = _ridge(n, dim, scale, 50 + k, r1)
        h.set_points(P)
        h.ridge_detection()
        assert bits_equal(h.chosen_points(), want), scale
        counts.add(h.get_chosen_samples_count())
    assert len(counts) > 1 or n < 100
    h.close()


def test_one_batch_handle_many_batches(rdb):
    b = rdb.BatchedRidgeDetection()
    for k, (sizes, scale) in enumerate([((300, 5000, 900), 1.0), ((4000, 20), 2.0), ((1500,), 0.6),
                                        ((300, 5000, 900, 7000, 2), 3.0)]):
        clouds = [(_scaled(n, 2 + i % 2, scale, 10 * k + i), 0.2, 0.4) for i, n in enumerate(sizes)]
        b.run(*rdb.pack_clouds(clouds))
        for i, (P, r1, r2) in enumerate(clouds):
            assert bits_equal(b.chosen_points(i), O.ridge_bf(P, r1, r2)[0]), (k, i)
    b.close()


def test_steps_on_sets_of_many_sizes(rdb):
    """The per-thread engines of the device steps."""
    torch = require_cuda()
    from ridgedetection_b200 import _lib as L
    lib, st = L.lib(), ctypes.c_void_p(0)
    p = lambda x: ctypes.c_void_p(x.data_ptr())  # noqa: E731
    for n, scale in ((5000, 1.0), (90_000, 1.0), (400, 0.2), (20_000, 4.0), (5000, 1.0)):
        P = _scaled(n, 3, scale, n)
        dP = torch.from_numpy(P).cuda()
        S = torch.zeros_like(dP)
        ns, left, passes = ctypes.c_int64(0), ctypes.c_int64(0), ctypes.c_int64(0)
        L.check(lib.rd_choose(3, p(dP), n, 0.3, p(S), ctypes.byref(ns), st))
        S0 = O.choose(P, 0.3)
        assert bits_equal(S[:ns.value].cpu().numpy(), S0)
        L.check(lib.rd_evolve(3, p(dP), n, p(S), ns.value, 0.3, ctypes.byref(passes), st))
        Se = O.evolve(P, S0, 0.3)[0]
        assert bits_equal(S[:ns.value].cpu().numpy(), Se)
        L.check(lib.rd_decimate(3, p(S), ns.value, 0.6, ctypes.byref(left), st))
        assert bits_equal(S[:left.value].cpu().numpy(), O.decimate(Se, 0.6))


def test_handles_in_several_threads(rdb):
    """Each thread solves clouds of changing sizes with a handle of its own and with the module
    function, beside the others."""
    import threading
    want = {}
    for t in range(4):
        for k in range(3):
            P = _scaled(800 + 900 * t, 2 + t % 2, (1.0, 3.0, 0.6)[k], 7 * t + k)
            want[t, k] = (P, O.ridge_bf(P, 0.2, 0.4)[0])
    bad = []

    def work(t):
        try:
            h = rdb.BruteForceRidgeDetection(800 + 900 * t, 0.2, 0.4, 2 + t % 2)
            for i in range(12):
                P, S = want[t, i % 3]
                h.set_points(P)
                h.ridge_detection()
                if not bits_equal(h.chosen_points(), S) or not bits_equal(rdb.ridge_detection(P, 0.2, 0.4)[0], S):
                    bad.append((t, i))
            h.close()
        except Exception as e:  # noqa: BLE001
            bad.append((t, repr(e)))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not bad
