"""Weighting with every landmark rotated once per particle against the scalar
kernel (pfc_set_weight_kernel 1), which rotates one per observation: the same
f32 operations in the same order, so the same bits."""
import ctypes as C

import numpy as np
import pytest

import cuda_pf_localization_b200 as pkg

from pf_helpers import RawPF, cloud, ours_ll, ours_set_state, ours_weights

pytestmark = pytest.mark.gpu


def _rows(rng, landmarks, nobs, mode="cart", bad_ids=False):
    lm = rng.uniform([-20, -20, 0], [20, 20, 6], (landmarks, 3)).astype(np.float32)
    rows = np.zeros((nobs, 6))
    rows[:, 0] = rng.integers(0, landmarks, nobs)
    body = lm[rows[:, 0].astype(int)] + rng.normal(0, 0.4, (nobs, 3))
    far = np.linalg.norm(body, axis=1)
    rb = {"cart": np.zeros(nobs, bool), "bearing": np.ones(nobs, bool),
          "mixed": rng.random(nobs) < 0.4}[mode]
    rows[:, 2:5] = np.where(rb[:, None], -body / far[:, None], body)
    rows[rb, 1], rows[rb, 5] = 1, far[rb]
    if bad_ids:
        rows[rng.random(nobs) < 0.2, 0] = landmarks + 3
        rows[rng.random(nobs) < 0.1, 0] = -1
    return lm, rows


# the rule takes this kernel at nobs >= 96, nobs >= 2 * landmarks, landmarks <= 64 and
# n * (nobs - landmarks) >= 16e6; 296 groups of a 256-particle tile: 75 776 particles a round
@pytest.mark.parametrize("landmarks,nobs,n", [
    (1, 96, 168_500), (2, 97, 170_001), (48, 96, 333_400), (64, 256, 83_335), (64, 255, 90_049),
    (31, 249, 75_776), (33, 250, 75_777), (5, 256, 65_536), (64, 128, 262_145), (17, 131, 151_553)])
@pytest.mark.parametrize("gate,sigma,bad", [(3.0, 0.05, False), (0.0, 0.05, True),
                                            (2.5, 0.0437, True), (4.0, 0.771, False)])
def test_marks_equal_scalar(kernels, landmarks, nobs, n, gate, sigma, bad):
    rng = np.random.default_rng(1000 * landmarks + nobs)
    lm, rows = _rows(rng, landmarks, nobs, bad_ids=bad)
    pos, quat = cloud(n, 3, centre=(0.0, 0.0, 0.0), pos_std=0.3, rot_std=0.1, yaw=0.0)[:2]
    pos[7], quat[n - 1] = np.nan, np.inf
    got = []
    for variant in (0, 1):
        pf = RawPF(kernels, n)
        try:
            pf.landmarks(lm)
            assert kernels.pfc_set_weight_kernel(pf.h, variant) == 0
            ours_set_state(pf, pos, quat)
            pf.weight(rows, sr=sigma, gate=gate)
            got.append((ours_ll(pf), ours_weights(pf)))
        finally:
            pf.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b, equal_nan=True)


def test_marks_all_ids_unknown_is_uniform(kernels):
    n = 200_000
    lm, rows = _rows(np.random.default_rng(1), 4, 100)
    rows[:, 0] = 99
    pf = RawPF(kernels, n)
    try:
        pf.landmarks(lm)
        pos, quat = cloud(n, 3)[:2]
        ours_set_state(pf, pos, quat)
        pf.weight(rows)
        assert np.array_equal(ours_ll(pf), np.zeros(n, np.float32))
        w = ours_weights(pf)
        assert np.all(w == w[0]) and abs(w[0] * n - 1) < 1e-5
    finally:
        pf.close()


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("device", [0, 1])
def test_cycles_across_the_rule(kernels, graph, device):
    """Cycles whose observations fall on both sides of the rule (two captured
    graphs), from the host and from device memory, where the library learns
    whether they are all Cartesian from the cycle before."""
    import torch
    n, landmarks = 100_001, 24
    rng = np.random.default_rng(8)
    steps = []
    for nobs, mode in ((256, "cart"), (200, "cart"), (20, "cart"), (256, "cart"), (230, "mixed"),
                       (0, "cart"), (256, "bearing"), (190, "cart"), (256, "cart")):
        lm, rows = _rows(np.random.default_rng(8), landmarks, max(nobs, 1), mode)
        odom = pkg.PfcOdom()
        odom.t[:], odom.q[:] = list(rng.normal(0, 0.02, 3)), [1.0, 0.0, 0.0, 0.0]
        odom.tstd[:], odom.rstd[:] = [0.02] * 3, [0.01] * 3
        rec = pkg.cobs_records(rows)
        steps.append((odom, pkg.make_cobs(rows), nobs,
                      torch.from_numpy(rec.view(np.uint8).copy()).cuda()))
    torch.cuda.synchronize()
    prm = pkg.PfcCycleParams(0.5, 0.2, 3.0, 0.5, 0.01, 0)
    got = []
    for variant in (0, 1):
        pf = RawPF(kernels, n)
        try:
            pf.landmarks(lm)
            assert kernels.pfc_set_weight_kernel(pf.h, variant) == 0
            assert kernels.pfc_set_graph(pf.h, graph) == 0
            pf.reinit([0, 0, 0, 1, 0, 0, 0], [0.3] * 3, [0.1] * 3)
            out = []
            for odom, obs, nobs, d_obs in steps:
                est = np.zeros(pkg.PFC_EST_LEN)
                if device:
                    rc = kernels.pfc_cycle_device(pf.h, C.byref(odom),
                                                  C.c_void_p(d_obs.data_ptr()), nobs, C.byref(prm),
                                                  pkg.dptr(est))
                else:
                    rc = kernels.pfc_cycle(pf.h, C.byref(odom), obs, nobs, C.byref(prm),
                                           pkg.dptr(est))
                assert rc == 0
                out.append(est)
            got.append((np.array(out), *pf.snapshot()))
        finally:
            pf.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
