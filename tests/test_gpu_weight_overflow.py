"""Range-bearing and mixed observations where the rotation's products overflow: the packed
path doubles its coefficients beforehand, which is exact short of that, so landmarks and
poses near the largest floats go through the scalar arithmetic, to the bit."""
import ctypes as C

import numpy as np
import pytest

import cuda_pf_localization_b200 as pkg

from pf_helpers import RawPF, ours_ll, ours_set_state, ours_weights

pytestmark = pytest.mark.gpu

BIG = [3e38, 2e38, 1.6e38, 8e37, 1e31, 1.27e30, 1.2e30, 1e20, np.inf, np.nan, 1e-42]


def _scene(mode, nobs, landmarks, n, wild, seed=1):
    """wild: the landmarks, positions and quaternions that get values of BIG."""
    rng = np.random.default_rng(seed)
    lm = rng.uniform([-20, -20, 0], [20, 20, 6], (landmarks, 3)).astype(np.float32)
    rows = np.zeros((nobs, 6))
    rows[:, 0] = rng.integers(0, landmarks, nobs)
    body = lm[rows[:, 0].astype(int)] + rng.normal(0, 0.3, (nobs, 3))
    far = np.linalg.norm(body, axis=1)
    rb = np.ones(nobs, bool) if mode == "bearing" else np.arange(nobs) % 50 == 7
    rows[:, 2:5] = np.where(rb[:, None], -body / far[:, None], body)
    rows[rb, 1], rows[rb, 5] = 1, far[rb]
    pos = rng.normal(0, 0.3, (n, 3)).astype(np.float32)
    quat = rng.normal(0, 0.4, (n, 4)).astype(np.float32)
    quat /= np.linalg.norm(quat, axis=1, keepdims=True)
    big = np.array(BIG, np.float32)
    if "l" in wild:
        lm[:len(big)] = big[:, None] * rng.choice([-1, 1], (len(big), 3)).astype(np.float32)
    if "p" in wild:
        at = rng.choice(n, 3 * len(big), replace=False)
        pos[at, np.arange(len(at)) % 3] = np.tile(big, 3)
    if "q" in wild:
        at = rng.choice(n, 4 * len(big), replace=False)
        quat[at, np.arange(len(at)) % 4] = np.tile(big, 4)
        with np.errstate(over="ignore"):
            quat[at[::2]] *= np.float32(1e19)
    return lm, rows, pos, quat


@pytest.mark.parametrize("wild", ["l", "p", "q", ""])
@pytest.mark.parametrize("gate,sigma", [(3.0, 0.05), (0.0, 1e20)])
@pytest.mark.parametrize("mode", ["bearing", "mixed"])
def test_packed_equals_scalar_near_overflow(kernels, mode, gate, sigma, wild):
    lm, rows, pos, quat = _scene(mode, 200 if mode == "bearing" else 120, 16, 3001, wild)
    # an observation at a time, then all: one that is not finite hides the others
    for part in [rows[k:k + 1] for k in range(0, 60, 3)] + [rows]:
        if part[0, 1] == 0 and len(part) == 1:
            part = np.concatenate([part, rows[rows[:, 1] == 1][:1] * [0, 1, 1, 1, 1, 1]])
            part[1, 0] = 15  # with a bearing of an ordinary landmark: a mixed chunk
        got = []
        for variant in (0, 1):
            pf = RawPF(kernels, len(pos))
            try:
                pf.landmarks(lm)
                assert kernels.pfc_set_weight_kernel(pf.h, variant) == 0
                ours_set_state(pf, pos, quat)
                assert pf.weight(part, sr=sigma, gate=gate) == 0
                got.append((ours_ll(pf), ours_weights(pf)))
            finally:
                pf.close()
        for a, b in zip(*got):
            assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.parametrize("wild", ["l", "p", "q"])
@pytest.mark.parametrize("mode", ["bearing", "mixed"])
def test_wrong_guess_near_overflow(kernels, mode, wild):
    """The same observations from device memory after a Cartesian cycle, and from the host;
    in the mixed case one of the two chunks has no bearing."""
    import torch
    n = 100_003
    lm, rows, pos, quat = _scene(mode, 256, 24, n, wild)
    if mode == "mixed":
        rows = np.concatenate([rows[rows[:, 1] == 0], rows[rows[:, 1] == 1]])
        rows = np.concatenate([rows[-128:], rows[:-128]])
    cart = rows.copy()
    cart[:, 1] = 0
    odom = pkg.PfcOdom()
    odom.t[:], odom.q[:] = [0.0] * 3, [1.0, 0.0, 0.0, 0.0]
    odom.tstd[:], odom.rstd[:] = [0.0] * 3, [0.0] * 3
    prm = pkg.PfcCycleParams(0.5, 0.2, 3.0, 0.5, 0.0, 0)
    est, got = np.zeros(pkg.PFC_EST_LEN), []
    for device in (True, False):
        pf = RawPF(kernels, n)
        try:
            pf.landmarks(lm)
            for r in (cart, rows):
                ours_set_state(pf, pos, quat)
                if device:
                    d_obs = torch.from_numpy(pkg.cobs_records(r).view(np.uint8).copy()).cuda()
                    torch.cuda.synchronize()
                    rc = kernels.pfc_cycle_device(pf.h, C.byref(odom),
                                                  C.c_void_p(d_obs.data_ptr()), len(r),
                                                  C.byref(prm), pkg.dptr(est))
                else:
                    rc = kernels.pfc_cycle(pf.h, C.byref(odom), pkg.make_cobs(r), len(r),
                                           C.byref(prm), pkg.dptr(est))
                assert rc == 0
            got.append(ours_ll(pf))
        finally:
            pf.close()
    assert np.array_equal(got[0], got[1], equal_nan=True)


def test_batch_near_overflow():
    """Range-bearing observations of a batch whose landmarks near the largest floats fall to
    the gate: weights of the packed and of the scalar arithmetic."""
    sizes = [3000, 7001]
    scenes = [_scene("bearing", 150, 16, 8, "", seed=f) for f in range(2)]
    for lm, *_ in scenes:
        lm[:4] = np.array([3e38, 2e38, 1.6e38, 8e37], np.float32)[:, None] * \
            np.float32([[1, -1, 1], [1, 1, 1], [-1, 1, 1], [1, -1, -1]])
    got = []
    for packed in (1, 0):
        b = pkg.BatchPF(sizes, seeds=[3, 4], obs_cap=4096)
        try:
            b.set_params(sigma_r=0.5, sigma_b=0.2, gate=3.0, ess_ratio=0.0, inject=0.0)
            b.set_landmarks([lm for lm, *_ in scenes])
            tiles = np.full(4, 1024, np.int32)
            assert b.lib.pfc_batch_set_tiles(b.handle, pkg.iptr(tiles), packed) == 0
            b.reinit(np.tile(np.float32([0, 0, 0, 1, 0, 0, 0]), (2, 1)), np.full((2, 3), 0.3),
                     np.full((2, 3), 0.1))
            odom = pkg.PfcOdom()
            odom.t[:], odom.q[:] = [0.0] * 3, [1.0, 0.0, 0.0, 0.0]
            odom.tstd[:], odom.rstd[:] = [0.02] * 3, [0.01] * 3
            b.cycle([odom] * 2, [rows for _, rows, *_ in scenes])
            w = [np.zeros(n, np.float32) for n in sizes]
            for f in range(2):
                assert b.lib.pfc_batch_get_weights(b.handle, f, pkg.fptr(w[f])) == 0
                assert len(np.unique(w[f])) > 100  # not uniform
            got.append(w)
        finally:
            b.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
