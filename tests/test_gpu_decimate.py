"""rd_decimate against the oracle, bit for bit, at the sizes where its path
changes: bit matrices in shared and in global memory, neighbour lists of one CTA
and of a cluster, and sets that end at the minimum-count rule
(rd/cpu/brute_force/decimate.hpp:41-81)."""
import ctypes

import numpy as np
import pytest

import oracle as O
from gpu_util import bits_equal, require_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return require_cuda()


def _decimate(torch, S, r2):
    from ridgedetection_b200 import _lib as L
    d = torch.from_numpy(S.copy()).cuda()
    left = ctypes.c_int64(0)
    L.check(L.lib().rd_decimate(S.shape[1], ctypes.c_void_p(d.data_ptr()), S.shape[0], r2,
                                ctypes.byref(left), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return d[:left.value].cpu().numpy()


# neighbours within r2 on average: few, many, (almost) all: the last ends at the minimum count
@pytest.mark.parametrize("near", [3.0, 12.0, 1e4])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 32, 33, 704, 721, 1500, 4096, 4097, 9001])
def test_decimate_sizes(torch, n, dim, near):
    S = np.random.default_rng(n * dim).random((n, dim)).astype(np.float32)
    r2 = float((near / n / (np.pi if dim == 2 else 4.19)) ** (1.0 / dim))
    if near > 100 and n > 2000:
        pytest.skip("all pairs within r2: the oracle is slow, and no path changes there")
    assert bits_equal(_decimate(torch, S, r2), O.decimate(S, r2))


def test_decimate_nan_inf_duplicates(torch):
    S = np.random.default_rng(1).random((5000, 2)).astype(np.float32)
    S[10] = np.nan
    S[20] = np.inf
    S[30] = -np.inf
    S[100:140] = S[100]
    for n in (300, 2000, 5000):
        assert bits_equal(_decimate(torch, S[:n], 0.03), O.decimate(S[:n], 0.03))


# around the largest set of one CTA's shared memory, and where lists or matrices are taken by
# how dense a sample of the set is
@pytest.mark.parametrize("near", [3.0, 60.0, 1e6])
@pytest.mark.parametrize("n,dim", [(705, 1), (864, 2), (865, 2), (865, 3), (900, 4), (2047, 1), (2048, 4)])
def test_decimate_between_matrices_and_lists(torch, n, dim, near):
    S = np.random.default_rng(n + dim).random((n, dim)).astype(np.float32)
    ball = {1: 2.0, 2: np.pi, 3: 4.19, 4: 4.93}[dim]
    r2 = float((near / n / ball) ** (1.0 / dim))
    assert bits_equal(_decimate(torch, S, r2), O.decimate(S, r2))


def test_solves_that_decimate_large_sets(torch):
    """A solve's own decimations of 900 to 4,096 points, sparse and dense, against the oracle."""
    import ridgedetection_b200 as rdb
    r = np.random.default_rng(3)
    for n, dim, r1, k in ((2500, 2, 0.004, 2.0), (4000, 3, 0.02, 2.0), (2500, 2, 0.004, 30.0), (3000, 1, 1e-5, 2.0)):
        P = r.random((n, dim)).astype(np.float32)
        S, st = rdb.ridge_detection(P, r1, k * r1)
        assert st.err_bits == 0 and bits_equal(S, O.ridge_bf(P, r1, k * r1)[0])
