"""Member lists kept across passes (k_assign_cull's edits, k_merge_fold) against the
all-pairs assignment, which regroups every point in every pass: bit for bit,
where lists are longest, shortest, outgrow their regions, or take more edits than
they hold."""
import numpy as np
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


def _blob(n, dim, sigma, seed):
    return np.random.default_rng(seed).normal(0.0, sigma, (n, dim)).astype(np.float32)


def _steep(n, seed):
    """Density rising steeply along x: chosen points travel and their clusters grow."""
    x = np.random.default_rng(seed).random((n, 2))
    return np.stack([8.0 * x[:, 0] ** 0.2, 0.1 * x[:, 1]], 1).astype(np.float32)


CASES = {
    # lists of more chunks than are looked up at once, folded in segments
    "two_huge": (lambda: _blob(150_000, 2, 0.2, 1), 0.9),
    # a long list below the segment threshold, one row around a chunk's end
    "chunk_end": (lambda: _blob(4 * 224 + 1, 3, 0.01, 2), 0.5),
    # more chosen points than the one-CTA scatter takes, lists of a few points
    "many_keys": (lambda: _blob(6_000, 2, 1.0, 3), 0.02),
    # clusters that grow past the room they were given
    "steep": (lambda: _steep(30_000, 4), 0.35),
    # more edits per key than are taken (early passes of a dense curve)
    "helix": (lambda: G.helix3d(120_000, seed=5), 0.15),
    "line": (lambda: _blob(5_000, 1, 1.0, 6), 0.1),
    "four_dims": (lambda: _blob(20_000, 4, 0.5, 7), 0.4),
}


@pytest.mark.parametrize("name", list(CASES))
def test_lists_match_all_pairs(rdb, name):
    gen, r1 = CASES[name]
    P = gen()
    rdb.set_assign_cull(False)
    try:
        S_ref, st_ref = rdb.ridge_detection(P, r1, 2.0 * r1)
    finally:
        rdb.set_assign_cull(True)
    for mode in (rdb.LOOP_GRAPH, rdb.LOOP_HOST):
        S, st = rdb.ridge_detection(P, r1, 2.0 * r1, loop_mode=mode)
        assert st.err_bits == 0 and st.evolve_passes == st_ref.evolve_passes
        assert bits_equal(S, S_ref)


def test_lists_in_a_batch(rdb):
    clouds = [(gen(), r1, 2.0 * r1) for gen, r1 in CASES.values()]
    packed, descs = rdb.pack_clouds(clouds)
    b = rdb.BatchedRidgeDetection()
    for _ in range(2):   # the second run takes over the first one's buffers
        b.run(packed, descs)
        for c, (P, r1, r2) in enumerate(clouds):
            S, _ = rdb.ridge_detection(P, r1, r2)
            assert bits_equal(b.chosen_points(c), S), c
    b.close()


def _beside(n, k, dim, sigma, seed):
    """k points of a blob away from zero, the rest far apart around it."""
    r = np.random.default_rng(seed)
    P = np.concatenate([r.normal(10.0, sigma, (k, dim)), r.uniform(0.0, 20.0, (n - k, dim))])
    return P[r.permutation(n)].astype(np.float32)


@pytest.mark.parametrize("name,gen,r1", [
    # few chosen points: lists of 16,384 and more are folded in segments and regrouped when edited
    ("few_keys", lambda: G.helix3d(200_000, seed=8), 1.5),
    ("few_keys_2d", lambda: G.sine2d(150_000, seed=9), 1.0),
    ("few_keys_1d", lambda: _blob(100_000, 1, 1.0, 10), 1.0),
    ("few_keys_4d", lambda: _blob(60_000, 4, 0.3, 11), 1.0),
    # many chosen points beside lists around 32,768 and 65,536 members
    ("beside_40k", lambda: _beside(42_000, 40_000, 3, 0.1, 12), 0.5),
    ("beside_70k", lambda: _beside(73_000, 70_000, 2, 0.1, 13), 0.5),
])
def test_long_lists_match_oracle(rdb, name, gen, r1):
    import oracle as O
    P = gen()
    S_ref = O.ridge_bf(P, r1, 2.0 * r1)[0]
    for cull in (True, False):
        rdb.set_assign_cull(cull)
        try:
            S, st = rdb.ridge_detection(P, r1, 2.0 * r1)
        finally:
            rdb.set_assign_cull(True)
        assert st.err_bits == 0 and bits_equal(S, S_ref)


def test_long_lists_in_a_batch(rdb):
    clouds = [(G.helix3d(60_000, seed=14), 1.5, 3.0), (_blob(40_000, 3, 0.2, 15), 0.9, 1.8),
              (G.helix3d(90_000, seed=16), 2.0, 4.0)]
    packed, descs = rdb.pack_clouds(clouds)
    b = rdb.BatchedRidgeDetection()
    b.run(packed, descs)
    for c, (P, r1, r2) in enumerate(clouds):
        S, _ = rdb.ridge_detection(P, r1, r2)
        assert bits_equal(b.chosen_points(c), S), c
    b.close()


@pytest.mark.parametrize("n", [2000, 2049, 2600, 9000])
def test_nearly_all_chosen(rdb, n):
    """Chosen sets around the size from which CTAs scan a cloud of few chunks, alone and beside
    clouds that warps scan."""
    import oracle as O
    P = np.random.default_rng(n).random((n, 3)).astype(np.float32)
    r1 = 0.15 / n
    S, st = rdb.ridge_detection(P, r1, 0.02)
    assert st.err_bits == 0 and bits_equal(S, O.ridge_bf(P, r1, 0.02)[0])
    clouds = [(P, r1, 0.02), (G.helix3d(700, seed=1), 0.2, 0.4), (G.helix3d(90_000, seed=2), 0.2, 0.4)]
    packed, descs = rdb.pack_clouds(clouds)
    b = rdb.BatchedRidgeDetection()
    b.run(packed, descs)
    for c, (Q, q1, q2) in enumerate(clouds):
        assert bits_equal(b.chosen_points(c), rdb.ridge_detection(Q, q1, q2)[0]), c
    b.close()


@pytest.mark.parametrize("batch", [False, True])
def test_lists_that_do_not_fit_the_device(rdb, batch):
    """With room for the points but not for the kept lists the run regroups in every pass:
    same bits, same passes."""
    torch = require_cuda()
    n = 6_000_000
    P = torch.from_numpy(G.helix3d(n, seed=21)).cuda()
    flat = P.reshape(-1)
    descs = [(0, 3_500_000, 3, 0.3, 0.6), (10_500_000, 2_500_000, 3, 0.4, 0.8)]

    def run():
        if batch:
            h = rdb.BatchedRidgeDetection()
            h.run(flat, descs)
            out = [h.chosen_points(0), h.chosen_points(1)], h.stats().evolve_passes
        else:
            h = rdb.BruteForceRidgeDetection(n, 0.3, 0.6, 3)
            h.set_points(P)
            h.ridge_detection()
            out = [h.chosen_points()], h.stats().evolve_passes
        used = free0 - torch.cuda.mem_get_info()[0]
        h.close()
        return out, used

    free0 = 0
    run()   # whatever a first run leaves on the device
    torch.cuda.empty_cache()
    free0 = torch.cuda.mem_get_info()[0]
    (want, passes), used = run()
    lists = 55 * n
    assert used > 3 * lists // 2
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free0 - (used - 2 * lists // 5), dtype=torch.uint8, device="cuda")
    try:
        (got, p), _ = run()
    finally:
        del hold
        torch.cuda.empty_cache()
    assert p == passes and all(bits_equal(x, y) for x, y in zip(got, want))


@pytest.mark.parametrize("extra", [-1, 0, 1])
@pytest.mark.parametrize("rows", [96, 224])
def test_list_chunk_edges(rdb, rows, extra):
    """Lists of whole chunks of the merge (96 rows where several clouds evolve, 224 for one) and
    one row less or more, in a batch and alone, against the oracle."""
    import oracle as O
    clouds = []
    for k in (1, 2, 3):
        n = k * rows + extra
        r = np.random.default_rng(100 * k + rows + extra)
        # two clusters of n points whose chosen points travel, so that members change sides
        x = np.concatenate([r.normal(0.0, 0.12, n), r.normal(0.7, 0.12, n)])
        P = np.stack([x, r.normal(0.0, 0.1, 2 * n)], 1).astype(np.float32)
        clouds.append((P[r.permutation(2 * n)], 0.5, 1.0))
        clouds.append((r.normal(0.0, 0.05, (n, 2)).astype(np.float32), 0.5, 1.0))   # one list
    packed, descs = rdb.pack_clouds(clouds)
    b = rdb.BatchedRidgeDetection()
    b.run(packed, descs)
    for c, (P, r1, r2) in enumerate(clouds):
        want = O.ridge_bf(P, r1, r2)[0]
        assert bits_equal(b.chosen_points(c), want), c
        assert bits_equal(rdb.ridge_detection(P, r1, r2)[0], want), c
    b.close()
