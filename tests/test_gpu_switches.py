"""Process-wide switches flipped by one thread while another one runs: a run takes
each switch once, when it starts, so its layout, buffers and kernels agree and its
results are the same bits whichever setting it met."""
import threading

import pytest

from gpu_util import bits_equal, require_cuda
from ridgedetection_b200 import generators as G

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rdb():
    require_cuda()
    import ridgedetection_b200 as rdb
    yield rdb
    rdb.set_assign_cull(True)


def test_batches_while_the_cull_switch_flips(rdb):
    clouds = [(G.sine2d(400 + 37 * c, seed=c), 0.15, 0.3) for c in range(24)]
    packed, descs = rdb.pack_clouds(clouds)
    b = rdb.BatchedRidgeDetection()
    want = []
    counts = b.run(packed, descs)
    for c in range(len(clouds)):
        want.append(b.chosen_points(c).copy())
    stop = threading.Event()
    flips = [0]

    def flip():
        while not stop.is_set():
            rdb.set_assign_cull(flips[0] % 2 == 0)
            flips[0] += 1

    t = threading.Thread(target=flip)
    t.start()
    try:
        got = []
        for _ in range(60):
            assert list(b.run(packed, descs)) == list(counts)
            got.append([b.chosen_points(c).copy() for c in range(len(clouds))])
    finally:
        stop.set()
        t.join()
        rdb.set_assign_cull(True)
        b.close()
    assert flips[0] > 60
    for one in got:
        assert all(bits_equal(x, y) for x, y in zip(one, want))
