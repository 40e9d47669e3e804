"""Bounded waits of the weighting that rotates every landmark once: with a limit of no
polls every wait of the kernel runs out at once, the kernel returns, the weights stay
uniform and the call that waits for the result reports the error.  As only that kernel
waits, the same limit tells which calls take it."""
import ctypes as C

import numpy as np
import pytest

import cuda_pf_localization_b200 as pkg

from pf_helpers import RawPF, ours_weights

pytestmark = pytest.mark.gpu


def _rows(landmarks, nobs, mode="cart", seed=3):
    rng = np.random.default_rng(seed)
    lm = rng.uniform([-20, -20, 0], [20, 20, 6], (landmarks, 3)).astype(np.float32)
    rows = np.zeros((nobs, 6))
    rows[:, 0] = rng.integers(0, landmarks, nobs)
    body = lm[rows[:, 0].astype(int)] + rng.normal(0, 0.4, (nobs, 3))
    far = np.linalg.norm(body, axis=1)
    rb = {"cart": np.zeros(nobs, bool), "bearing": np.ones(nobs, bool),
          "one": np.arange(nobs) == nobs // 2}[mode]
    rows[:, 2:5] = np.where(rb[:, None], -body / far[:, None], body)
    rows[rb, 1], rows[rb, 5] = 1, far[rb]
    return lm, rows


def _filter(lib, n, lm):
    pf = RawPF(lib, n, cap_obs=300)
    pf.landmarks(lm)
    _prior(pf)
    return pf


def _prior(pf):
    pf.reinit([0, 0, 0, 1, 0, 0, 0], [0.3] * 3, [0.1] * 3)


def _sums(pf):
    out = np.zeros(14)
    return pf.lib.pfc_est_sums(pf.h, pkg.dptr(out)), out


def _cycle(pf, rows, device=False):
    odom = pkg.PfcOdom()
    odom.t[:], odom.q[:] = [0.02, 0.0, 0.01], [1.0, 0.0, 0.0, 0.0]
    odom.tstd[:], odom.rstd[:] = [0.02] * 3, [0.01] * 3
    prm = pkg.PfcCycleParams(0.5, 0.2, 3.0, 0.5, 0.01, 0)
    est = np.zeros(pkg.PFC_EST_LEN)
    if device:
        import torch
        d_obs = torch.from_numpy(pkg.cobs_records(rows).view(np.uint8).copy()).cuda()
        torch.cuda.synchronize()
        rc = pf.lib.pfc_cycle_device(pf.h, C.byref(odom), C.c_void_p(d_obs.data_ptr()), len(rows),
                                     C.byref(prm), pkg.dptr(est))
    else:
        rc = pf.lib.pfc_cycle(pf.h, C.byref(odom), pkg.make_cobs(rows), len(rows), C.byref(prm),
                              pkg.dptr(est))
    return rc, est


# the rule: a table of 64 landmarks at most, 96 to 256 observations, twice the landmarks
# at least, particles x (observations - landmarks) >= 16e6, all of them Cartesian
@pytest.mark.parametrize("landmarks,nobs,n,mode,taken", [
    (64, 256, 83_334, "cart", True), (64, 256, 83_333, "cart", False),
    (1, 96, 168_422, "cart", True), (1, 96, 168_421, "cart", False),
    (1, 95, 200_000, "cart", False), (48, 96, 333_334, "cart", True),
    (49, 97, 400_000, "cart", False), (65, 256, 200_000, "cart", False),
    (64, 257, 200_000, "cart", False), (64, 256, 100_000, "bearing", False),
    (64, 256, 100_000, "one", False)])
def test_which_calls_wait(kernels, landmarks, nobs, n, mode, taken):
    lm, rows = _rows(landmarks, nobs, mode)
    pf = _filter(kernels, n, lm)
    try:
        assert kernels.pfc_set_wait_test(pf.h, 0) == 0
        assert pf.weight(rows) == 0
        assert _sums(pf)[0] == (-1 if taken else 0)
    finally:
        pf.close()


def test_scalar_weighting_does_not_wait(kernels):
    lm, rows = _rows(64, 256)
    pf = _filter(kernels, 100_000, lm)
    try:
        assert kernels.pfc_set_weight_kernel(pf.h, 1) == 0
        assert kernels.pfc_set_wait_test(pf.h, 0) == 0
        assert pf.weight(rows) == 0
        assert _sums(pf)[0] == 0
    finally:
        pf.close()


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("staged", [0, 1])
def test_a_wait_that_runs_out(kernels, graph, staged):
    n = 100_001
    lm, rows = _rows(24, 256)
    few = rows[:20]

    def run(pf, r):
        if staged:
            assert pf.weight(r) == 0
            return _sums(pf)
        return _cycle(pf, r)

    pf, fresh = _filter(kernels, n, lm), _filter(kernels, n, lm)
    try:
        for f in (pf, fresh):
            assert kernels.pfc_set_graph(f.h, graph) == 0
        assert run(pf, rows)[0] == 0 and run(fresh, rows)[0] == 0
        assert kernels.pfc_set_wait_test(pf.h, 0) == 0
        assert run(pf, rows)[0] == -1
        assert "a device wait timed out" in pkg.last_error()
        assert np.all(ours_weights(pf) == np.float32(1) / np.float32(n))
        assert kernels.pfc_set_wait_test(pf.h, -1) == 0
        assert run(pf, few)[0] == -1 and run(pf, rows)[0] == -1  # until the next pfc_init
        for f in (pf, fresh):
            assert kernels.pfc_init(f.h, n, 42) == 0
            assert kernels.pfc_set_lcg(f.h, 99) == 0
            _prior(f)
        for r in (rows, few, rows):
            (rc, a), (rd, b) = run(pf, r), run(fresh, r)
            assert rc == rd == 0 and np.array_equal(a, b)
        for a, b in zip(pf.snapshot(), fresh.snapshot()):
            assert np.array_equal(a, b)
    finally:
        pf.close()
        fresh.close()


def test_a_lowered_limit_alone_does_not_fire(kernels):
    lm, rows = _rows(64, 256)
    got = []
    for polls in (-1, 1 << 16):
        pf = _filter(kernels, 300_001, lm)
        try:
            assert kernels.pfc_set_wait_test(pf.h, polls) == 0
            rc, est = _cycle(pf, rows)
            assert rc == 0
            got.append((est, *pf.snapshot()))
        finally:
            pf.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


def test_arguments_checked(kernels):
    assert kernels.pfc_set_wait_test(None, 0) == -1
    pf = RawPF(kernels, 1000)
    try:
        assert kernels.pfc_set_wait_test(pf.h, -2) == -1
    finally:
        pf.close()


# Observations in device memory: a cycle takes the kernel when the host's guess is that
# they are Cartesian, which the last call of each history shows.
@pytest.mark.parametrize("history,guess", [
    ("", False), ("c", True), ("m", False), ("cm", False), ("cm" + 8 * "c", False),
    ("cm" + 9 * "c", True), (20 * "c" + "m" + 8 * "c", False), ("m" + 9 * "c", True),
    ("m" + 8 * "c" + "m" + 9 * "c", True), ("mmm" + 9 * "c", True), ("ch", True), ("h", False),
    ("mh" + 9 * "c", True), ("cI", False), ("mIc", True), ("cmI", False)])
def test_guess_follows_the_cycles(kernels, history, guess):
    n = 100_001
    lm, rows = _rows(24, 256)
    one = _rows(24, 256, "one")[1]
    pf = _filter(kernels, n, lm)
    try:
        for step in history:
            if step == "I":
                assert kernels.pfc_init(pf.h, n, 5) == 0
                _prior(pf)
            else:  # Cartesian or mixed from the device, Cartesian from the host
                assert _cycle(pf, one if step == "m" else rows, step != "h")[0] == 0
        assert kernels.pfc_set_wait_test(pf.h, 0) == 0
        assert _cycle(pf, rows, True)[0] == (-1 if guess else 0)
    finally:
        pf.close()


@pytest.mark.parametrize("mode", ["one", "bearing"])
@pytest.mark.parametrize("landmarks,nobs,n,gate", [
    (64, 256, 83_334, 3.0), (1, 96, 168_447, 0.0), (24, 131, 151_553, 2.5), (5, 256, 606_209, 3.0)])
def test_a_wrong_guess_gives_the_same_bits(kernels, mode, landmarks, nobs, n, gate):
    """A Cartesian cycle, then one that is not, in the kernel that guesses (151 552 and
    606 208 particles fill 148 blocks' four tiles once and four times) and in the scalar
    one; unknown ids among the observations, and poses that are not finite."""
    import torch
    lm, cart = _rows(landmarks, nobs)
    other = _rows(landmarks, nobs, mode, seed=4)[1]
    other[::7, 0] = landmarks + 2
    other[3::11, 0] = -1
    rng = np.random.default_rng(2)
    pos = rng.normal(0, 0.3, (n, 3)).astype(np.float32)
    quat = rng.normal(0, 0.1, (n, 4)).astype(np.float32) + np.float32([1, 0, 0, 0])
    pos[7], quat[n - 1] = np.nan, np.inf
    got = []
    for variant in (0, 1):
        pf = _filter(kernels, n, lm)
        try:
            assert kernels.pfc_set_weight_kernel(pf.h, variant) == 0
            assert _cycle(pf, cart, True)[0] == 0
            assert kernels.pfc_set_state(pf.h, pkg.fptr(pos), pkg.fptr(quat), None) == 0
            odom = pkg.PfcOdom()
            odom.t[:], odom.q[:] = [0.0] * 3, [1.0, 0.0, 0.0, 0.0]
            odom.tstd[:], odom.rstd[:] = [0.02] * 3, [0.01] * 3
            prm = pkg.PfcCycleParams(0.5, 0.2, gate, 0.5, 0.01, 0)
            d_obs = torch.from_numpy(pkg.cobs_records(other).view(np.uint8).copy()).cuda()
            torch.cuda.synchronize()
            est, ll = np.zeros(pkg.PFC_EST_LEN), np.zeros(n, np.float32)
            assert kernels.pfc_cycle_device(pf.h, C.byref(odom), C.c_void_p(d_obs.data_ptr()),
                                            nobs, C.byref(prm), pkg.dptr(est)) == 0
            assert kernels.pfc_get_ll(pf.h, pkg.fptr(ll)) == 0
            got.append((est, ll, *pf.snapshot()))
        finally:
            pf.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b, equal_nan=True)
    assert len(np.unique(got[0][1])) > n // 100
