"""A batch of learned queries leaves its results where the caller wants them: every
output is optional, over several chunks, also where a query's fallback takes its place."""
import numpy as np
import pytest

import cuda_pf_localization_b200 as pkg
from cuda_pf_localization_b200 import sim

pytestmark = pytest.mark.gpu

NQ, S, K = 300, 200, 9   # three chunks of a network of 128 rows


def _batch(kernels, h, scans, tau, fallback, want):
    lp = pkg.LearnedProposal(h, batch=128, seed=5)
    try:
        lp.set_threshold(tau)
        out = [np.full((NQ, K, 3), -7, np.float32), np.full((NQ, K), -7, np.float32),
               np.full((NQ, K), -7, np.int32), np.full(NQ, -7, np.int32)]
        ptr = [f(a) if w else None for f, a, w in
               zip((pkg.fptr, pkg.fptr, pkg.iptr, pkg.iptr), out, want)]
        assert kernels.pfgl_learned_localize_batch(
            lp._h, pkg.fptr(scans), NQ, scans.shape[1], 10.0, 2 * np.pi, S, fallback, K,
            *ptr) == K
        return out
    finally:
        lp.close()


@pytest.mark.parametrize("fallback", [0, 800])
def test_outputs_are_optional(kernels, fallback):
    g = np.ascontiguousarray(sim.rooms_grid(3))
    h = kernels.pfgl_create(200, 200, 0.05, 0.0, 0.0, pkg.u8ptr(g), 1 << 16)
    assert h
    try:
        rng = np.random.default_rng(1)
        poses = np.array([sim.free_pose(g, rng) for _ in range(NQ)], np.float32)
        scans = pkg.render_scans(h, poses, seed=3)
        best = _batch(kernels, h, scans, np.inf, 0, [1, 1, 1, 1])[1][:, 0]
        tau = float(np.median(best))
        full = _batch(kernels, h, scans, tau, fallback, [1, 1, 1, 1])
        if fallback:
            assert {0, 2} <= set(full[3]) and np.sum(full[3] > 0) == np.sum(best > tau)
        else:
            assert np.all(full[3] == 0) and np.array_equal(full[1][:, 0], best)
        assert np.all(np.diff(full[1], axis=1) >= 0)
        for want in ([0, 1, 1, 1], [1, 0, 1, 1], [1, 1, 0, 1], [1, 1, 1, 0], [0, 0, 0, 1],
                     [0, 0, 0, 0]):
            for w, a, b in zip(want, full, _batch(kernels, h, scans, tau, fallback, want)):
                assert np.array_equal(b, a if w else np.full_like(b, -7))
    finally:
        kernels.pfgl_destroy(h)
