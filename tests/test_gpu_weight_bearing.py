"""Weighting by range-bearing observations on the packed path, whose root and
quotient come from one reciprocal root, against the scalar kernel
(pfc_set_weight_kernel 1), which calls the library's: the same bits, also where the
packed root and quotient do not apply."""
import numpy as np
import pytest

from pf_helpers import RawPF, cloud, ours_ll, ours_set_state, ours_weights

pytestmark = pytest.mark.gpu


def _both(kernels, lm, rows, pos, quat, sigma, gate):
    got = []
    for variant in (0, 1):
        pf = RawPF(kernels, len(pos))
        try:
            pf.landmarks(lm)
            assert kernels.pfc_set_weight_kernel(pf.h, variant) == 0
            ours_set_state(pf, pos, quat)
            assert pf.weight(rows, sr=sigma, gate=gate) == 0
            got.append((ours_ll(pf), ours_weights(pf)))
        finally:
            pf.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b, equal_nan=True)


def _rows(rng, lm, nobs, share):
    rows = np.zeros((nobs, 6))
    rows[:, 0] = rng.integers(-1, len(lm) + 1, nobs)  # some ids unknown
    body = lm[np.clip(rows[:, 0].astype(int), 0, len(lm) - 1)] + rng.normal(0, 0.3, (nobs, 3))
    far = np.linalg.norm(body, axis=1)
    rb = rng.random(nobs) < share
    rows[:, 2:5] = np.where(rb[:, None], -body / far[:, None], body)
    rows[rb, 1], rows[rb, 5] = 1, far[rb]
    return rows


# a chunk holds 128 observations, a block 256 particles
@pytest.mark.parametrize("n,nobs", [(1, 1), (257, 5), (4096, 128), (30_001, 129), (100_003, 300)])
@pytest.mark.parametrize("gate,sigma", [(3.0, 0.05), (0.0, 0.3)])
@pytest.mark.parametrize("share", [0.3, 1.0])
def test_packed_equals_scalar(kernels, n, nobs, gate, sigma, share):
    rng = np.random.default_rng(n + nobs)
    lm = rng.uniform([-20, -20, 0], [20, 20, 6], (23, 3)).astype(np.float32)
    pos, quat = cloud(n, 3, centre=(0.0, 0.0, 0.0), pos_std=0.3, rot_std=0.1, yaw=0.0)[:2]
    _both(kernels, lm, _rows(rng, lm, nobs, share), pos, quat, sigma, gate)


@pytest.mark.parametrize("gate", [0.0, 3.0])
def test_packed_equals_scalar_outside_its_range(kernels, gate):
    """Landmarks at, very near and very far from a particle; bearings that are
    zero, huge, infinite or NaN; and ranges whose significand is all ones with a
    product that is a power of two (where 1 / range does not round correctly)."""
    f = np.float32
    y = (np.sqrt(f(3.0)) + np.arange(-8, 9, dtype=f) * f(2.0 ** -23)).astype(f)
    s = (y * y + f(1.0)).astype(f)
    ones = y[np.sqrt(s) == f(2.0 - 2.0 ** -23)]
    assert len(ones)
    at = [0.0, 1e-30, 3e-20, 1e-10, 1.3e-9, 2e-9, 1e-3, 1.0, 1e6, 1e11, 1.5e12, 1e19, 3e38, np.inf,
          np.nan]
    lm = np.array([[v, 0, 0] for v in at] + [[0, v, v] for v in at]
                  + [[1.0, v, 0.0] for v in ones], f)
    bearings = [[-1, 0, 0], [0, 0, 0], [0.6, 0.8, 0], [-2, 0, 0], [1e-30, 1e-42, 0], [1e30, 0, 1],
                [np.inf, 0, 0], [np.nan, 0, 0]]
    rng = np.random.default_rng(2)
    pos = rng.normal(0, 1e-3, (600, 3)).astype(f)
    quat = np.tile(np.array([1, 0, 0, 0], f), (600, 1))
    pos[:300] = 0
    pos[5], pos[7, 1], quat[9], quat[11] = 1e25, np.nan, np.inf, 0
    # each alone: a NaN or infinite term would hide the others
    for k in range(len(lm)):
        for b in bearings:
            rows = np.array([[k, 1, *b, 1.25]])
            _both(kernels, lm, rows, pos, quat, 0.5, gate)
