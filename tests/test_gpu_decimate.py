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
