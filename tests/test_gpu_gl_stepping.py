"""The shared-memory ray stepping of the CAER scorers against the stepping
through global memory: the same map embedded in one too large for shared
memory gives the same rays, so every CAER is the same to the bit."""
import numpy as np
import pytest

import cuda_pf_localization_b200 as pkg

pytestmark = pytest.mark.gpu
BIG = 820  # 822 x 822 cells do not fit an SM's shared memory
RES = 0.05


def _cells(rng, w, h, walls):
    c = np.zeros((h, w), np.uint8)
    if walls:
        c[0, :] = c[-1, :] = 1
        c[:, 0] = c[:, -1] = 1
    for _ in range(max(1, w * h // 2500)):
        bw, bh = rng.integers(1, max(2, min(20, w // 2, h // 2)), 2)
        x, y = rng.integers(0, w - bw + 1), rng.integers(0, h - bh + 1)
        c[y:y + bh, x:x + bw] = 1
    return c


def _hyps(rng, w, h, n):
    x = np.stack([rng.uniform(0, w * RES, n), rng.uniform(0, h * RES, n),
                  rng.uniform(-np.pi, np.pi, n)], 1).astype(np.float32)
    x[0] = (np.float32(RES) * (w // 2), np.float32(RES) * (h // 2), 0.0)  # cell corner, axis ray
    x[1, 2], x[2, 2], x[3, 2] = 0.0, np.pi / 2, np.nan
    x[4, :2] = (np.nan, 0.1)
    x[5, :2] = (0.1, np.nan)
    x[6, :2] = (-1.0, 0.1)                                                # outside the map
    return np.ascontiguousarray(x)


def _run(lib, cells, hyps, scan, span, k, batch):
    h = lib.pfgl_create(cells.shape[1], cells.shape[0], RES, 0.0, 0.0, pkg.u8ptr(cells), len(hyps))
    assert h, pkg.last_error()
    try:
        n, nr = len(hyps), len(scan)
        caer, best, idx = np.zeros(n, np.float32), np.zeros(k, np.float32), np.zeros(k, np.int32)
        assert lib.pfgl_set_hyps(h, pkg.fptr(hyps.reshape(-1)), n) == 0
        assert lib.pfgl_score(h, pkg.fptr(scan), nr, 6.0, span) == 0
        assert lib.pfgl_get_caer(h, pkg.fptr(caer)) == 0
        out = [caer]
        if batch:  # the pruned scorer (no NaN scores there)
            pose = np.zeros(3 * k, np.float32)
            assert lib.pfgl_localize(h, pkg.fptr(scan), nr, 6.0, span, k, pkg.fptr(pose),
                                     pkg.fptr(best), pkg.iptr(idx)) == k
            out += [best, idx, pose]
        return out
    finally:
        lib.pfgl_destroy(h)


# two blocks an SM, one block an SM (403 x 301, 420 x 420 or many rays), narrow maps
@pytest.mark.parametrize("w,h,walls", [(200, 200, True), (401, 299, True), (420, 420, False),
                                       (37, 511, False), (8, 8, True), (1, 1, False)])
@pytest.mark.parametrize("nrays", [1, 31, 33, 271, 500, 1000])
def test_shared_stepping_equals_global_stepping(kernels, w, h, walls, nrays):
    rng = np.random.default_rng(1000 * w + nrays)
    cells = _cells(rng, w, h, walls)
    big = np.zeros((BIG, BIG), np.uint8)
    big[:h, :w] = cells
    hyps = _hyps(rng, w, h, 1500)
    scan = rng.uniform(0, 6, nrays).astype(np.float32)
    span = float(rng.choice([np.pi, 1.5 * np.pi, 2 * np.pi]))
    # beyond the small map the large one is free, so a ray that leaves either
    # ends at rmax; hypotheses outside the small map but inside the large
    # one's free area are left out
    a = _run(kernels, cells, hyps, scan, span, 10, False)
    b = _run(kernels, big, hyps, scan, span, 10, False)
    same = ~((hyps[:, 0] >= np.float32(w * RES)) | (hyps[:, 1] >= np.float32(h * RES)))
    assert np.array_equal(a[0][same], b[0][same], equal_nan=True)


def test_pruned_shared_stepping_equals_global_stepping(kernels):
    rng = np.random.default_rng(5)
    cells = _cells(rng, 401, 299, True)
    big = np.zeros((BIG, BIG), np.uint8)
    big[:299, :401] = cells
    hyps = np.ascontiguousarray(_hyps(rng, 401, 299, 30_008)[8:])
    scan = rng.uniform(0, 6, 271).astype(np.float32)
    a = _run(kernels, cells, hyps, scan, 4.5, 64, True)
    b = _run(kernels, big, hyps, scan, 4.5, 64, True)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
