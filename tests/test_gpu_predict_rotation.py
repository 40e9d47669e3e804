"""Rotation noise of the predict over sizes on both sides of the range in which its
norm, root and quotient come from one reciprocal root (|rotation| >= 2^-29): the
same draws scaled give the same axis, the angle that the scale asks for, and a unit
quaternion; no rotation leaves the attitude as it was."""
import numpy as np
import pytest

from pf_helpers import RawPF, ours_set_state

pytestmark = pytest.mark.gpu

N = 5000


def _turned(kernels, scale):
    pf = RawPF(kernels, N)
    try:
        quat = np.zeros((N, 4), np.float32)
        quat[:, 0] = 1
        ours_set_state(pf, np.zeros((N, 3), np.float32), quat)
        pf.predict([0.1, 0, 0], [1, 0, 0, 0], [0.0] * 3, [scale] * 3)
        pos, quat = pf.snapshot()
        return np.float64(pos).reshape(N, 3), np.float64(quat).reshape(N, 4)
    finally:
        pf.close()


def test_no_rotation_is_identity(kernels):
    pos, quat = _turned(kernels, 0.0)
    assert np.all(quat == [1, 0, 0, 0]) and np.allclose(pos, [0.1, 0, 0], atol=1e-7)


@pytest.mark.parametrize("scale", [1e-10, 1e-9, 1.5e-9, 3e-9, 1e-7, 1e-4, 0.02, 1.0, 40.0, 1e5])
def test_scaled_rotation(kernels, scale):
    # the draws themselves: half the rotation vector at a scale where sin(h) = h in f32
    v = 2.0 * _turned(kernels, 1e-5)[1][:, 1:] / float(np.float32(1e-5)) * float(np.float32(scale))
    quat = _turned(kernels, scale)[1]
    angle = np.linalg.norm(v, axis=1)
    sinc = np.sinc(angle / (2 * np.pi)) / 2
    # draws known to 4 ulp: the angle to 2^-21 of itself, and with it sin and cos
    tol = 2.0 ** -21 * (1 + angle)
    assert np.all(np.abs(np.linalg.norm(quat, axis=1) - 1) <= 2.0 ** -21)
    assert np.all(np.abs(quat[:, 0] - np.cos(angle / 2)) <= tol)
    err = np.abs(quat[:, 1:] - v * sinc[:, None])
    assert np.all(err <= (tol * np.minimum(angle, 1.0))[:, None])
