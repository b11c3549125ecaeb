"""1- and 4-dimensional points against the oracle restatement, bit for bit (the same
clouds meet the reference's own compiled code in test_gpu_dims.py where that is built)."""
import ctypes

import numpy as np
import pytest

import oracle as O
from gpu_util import bits_equal, require_cuda
from test_gpu_dims import CASES, helix4d, line1d

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rdb():
    require_cuda()
    import ridgedetection_b200 as rdb
    return rdb


@pytest.mark.parametrize("name,gen,n,r1,r2", CASES, ids=[c[0] for c in CASES])
def test_brute_force(rdb, name, gen, n, r1, r2):
    P = gen(n, seed=n)
    want = O.ridge_bf(P, r1, r2)[0]
    for lm in (rdb.LOOP_GRAPH, rdb.LOOP_HOST):
        S, st = rdb.ridge_detection(P, r1, r2, loop_mode=lm)
        assert st.err_bits == 0 and bits_equal(S, want)


def test_batch_of_mixed_dimensions(rdb):
    clouds = [(line1d(3000, 1), 0.1, 0.2), (helix4d(2500, 2), 0.2, 0.4),
              (line1d(1200, 3), 0.3, 0.6), (helix4d(4000, 4), 0.15, 0.3)]
    b = rdb.BatchedRidgeDetection()
    b.run(*rdb.pack_clouds(clouds))
    for c, (P, r1, r2) in enumerate(clouds):
        assert bits_equal(b.chosen_points(c), O.ridge_bf(P, r1, r2)[0]), c
    b.close()


@pytest.mark.parametrize("gen,r1,r2", [(helix4d, 0.2, 0.4), (line1d, 0.05, 0.1)])
def test_device_steps(rdb, gen, r1, r2):
    torch = require_cuda()
    from ridgedetection_b200 import _lib as L
    lib = L.lib()
    P = gen(5000, 11)
    n, dim = P.shape
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    dP = torch.from_numpy(P).cuda()
    dS = torch.zeros_like(dP)
    ns, passes, left = ctypes.c_int64(0), ctypes.c_int64(0), ctypes.c_int64(0)
    L.check(lib.rd_choose(dim, p(dP), n, r1, p(dS), ctypes.byref(ns), st))
    S0 = O.choose(P, r1)
    assert bits_equal(dS[:ns.value].cpu().numpy(), S0)
    L.check(lib.rd_evolve(dim, p(dP), n, p(dS), ns.value, r1, ctypes.byref(passes), st))
    Se = O.evolve(P, S0, r1)[0]
    assert bits_equal(dS[:ns.value].cpu().numpy(), Se)
    L.check(lib.rd_decimate(dim, p(dS), ns.value, r2, ctypes.byref(left), st))
    assert bits_equal(dS[:left.value].cpu().numpy(), O.decimate(Se, r2))
