"""Choose (rd_choose) against the oracle, bit for bit, at the edges of its blocks, resolve groups, shared-memory mirror
and rounds (rd/cpu/brute_force/choose.hpp:37-70)."""
import ctypes

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


def _choose(P, r1):
    import torch
    from ridgedetection_b200 import _lib as L
    dP = torch.from_numpy(P).cuda()
    dS = torch.zeros_like(dP)
    ns = ctypes.c_int64(0)
    L.check(L.lib().rd_choose(P.shape[1], ctypes.c_void_p(dP.data_ptr()), P.shape[0], r1,
                              ctypes.c_void_p(dS.data_ptr()), ctypes.byref(ns),
                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return dS[:ns.value].cpu().numpy()


def _cloud(n, dim):
    return np.random.default_rng(n + dim).random((n, dim)).astype(np.float32)


# radii: every point chosen (more than the mirror holds at the larger sizes),
# about half, a few
@pytest.mark.parametrize("r1", [1e-5, 0.02, 0.3])
@pytest.mark.parametrize("dim", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 255, 257, 1024, 1025, 7001])
def test_choose_edges(rdb, n, dim, r1):
    P = _cloud(n, dim)
    assert bits_equal(_choose(P, r1), O.choose(P, r1))


@pytest.mark.parametrize("n", [65_535, 65_536, 90_001])
def test_choose_rounds(rdb, n):
    P = G.helix3d(n, seed=n)
    P[100] = np.nan
    P[200] = np.inf
    assert bits_equal(_choose(P, 0.1), O.choose(P, 0.1))
