"""Results that reach the host through pinned memory up to a size and by pageable
copies beyond it: the bottom-k of a call around its 1024 entries (every length a prefix
of the longest), and a batch of learned queries around its 64 entries a query."""
import numpy as np
import pytest

import cuda_pf_localization_b200 as pkg
from cuda_pf_localization_b200 import sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 1023, 1024, 1025])
def test_topk_lengths_agree(kernels, k):
    g = np.ascontiguousarray(sim.rooms_grid(3))
    h = kernels.pfgl_create(200, 200, 0.05, 0.0, 0.0, pkg.u8ptr(g), 1 << 15)
    assert h
    try:
        rng = np.random.default_rng(1)
        scan = pkg.render_scans(h, np.array([sim.free_pose(g, rng)], np.float32), seed=3)[0]
        assert kernels.pfgl_generate_yaws(h, 500, 16, 9) == 0
        assert kernels.pfgl_score(h, pkg.fptr(scan), len(scan), 10.0, 2 * np.pi) == 0
        got = []
        for n in (k, 3000):
            pose, caer = np.zeros((n, 3), np.float32), np.zeros(n, np.float32)
            idx = np.zeros(n, np.int32)
            assert kernels.pfgl_topk_ex(h, n, pkg.fptr(pose), pkg.fptr(caer), pkg.iptr(idx)) == n
            got.append((pose[:k], caer[:k], idx[:k]))
        for a, b in zip(*got):
            assert np.array_equal(a, b)
        assert kernels.pfgl_topk_ex(h, k, pkg.fptr(pose), None, None) == k  # outputs are optional
        assert np.array_equal(pose[:k], got[0][0])
    finally:
        kernels.pfgl_destroy(h)


@pytest.mark.parametrize("nq,k", [(128, 63), (128, 64), (128, 65)])
def test_query_batches_agree(kernels, nq, k):
    """One batch (a chunk of 128 queries, room for 128 x 64 entries) against the same
    queries in two calls of half as many."""
    g = np.ascontiguousarray(sim.rooms_grid(3))
    h = kernels.pfgl_create(200, 200, 0.05, 0.0, 0.0, pkg.u8ptr(g), 1 << 16)
    assert h
    try:
        rng = np.random.default_rng(1)
        poses = np.array([sim.free_pose(g, rng) for _ in range(nq)], np.float32)
        scans = pkg.render_scans(h, poses, seed=3)
        got = []
        for cuts in ((0, nq), (0, nq // 2, nq)):
            lp = pkg.LearnedProposal(h, batch=128, seed=5)
            try:
                parts = [lp.localize_batch(scans[a:b], 200, 0, k) for a, b in zip(cuts, cuts[1:])]
                got.append([np.concatenate([p[i] for p in parts]) for i in range(3)])
            finally:
                lp.close()
        for a, b in zip(*got):
            assert np.array_equal(a, b)
    finally:
        kernels.pfgl_destroy(h)
