"""Cycle graphs whose injection buckets have been replaced.

The buckets that file the injected draws are allocated anew when a larger ratio
needs more room per tile (64, 116 and 256 draws here).  A handle keeps one
captured graph for each weighting kernel; the one that is not in use when that
happens, and both when it happens in a resample between two cycles, name the
freed buckets and have to be captured again before they are replayed.  Checked
by the count of captures and against direct launches, to the bit."""
import ctypes as C

import numpy as np
import pytest

import cuda_pf_localization_b200 as pkg

from pf_helpers import RawPF

pytestmark = pytest.mark.gpu

N, LANDMARKS = 100_003, 24
# (observations, injection ratio) of a cycle or the ratio of a resample, and the
# graphs captured by then: 64 observations take one weighting kernel, 256 the other
STEPS = [((64, 0.002), 1), ((256, 0.01), 2), ((64, 0.002), 3), ((64, 0.002), 3),
         ((256, 0.01), 3), (0.05, 3), ((256, 0.01), 4), ((64, 0.002), 5), ((64, 0.002), 5),
         ((256, 0.01), 5), ((64, 0.05), 6), ((64, 0.0), 7), ((256, 0.01), 7)]


def _cycles(lib, graph, steps):
    rng = np.random.default_rng(5)
    lm = rng.uniform([-20, -20, 0], [20, 20, 6], (LANDMARKS, 3)).astype(np.float32)
    pf = RawPF(lib, N)
    out, captures = [], []
    try:
        assert lib.pfc_set_graph(pf.h, graph) == 0
        pf.landmarks(lm)
        pf.reinit([0, 0, 0, 1, 0, 0, 0], [0.3] * 3, [0.1] * 3)
        for step in steps:
            if isinstance(step, float):
                pf.resample(step)
                out.append(pf.est_sums())
            else:
                nobs, ratio = step
                rows = np.zeros((nobs, 6))
                rows[:, 0] = np.arange(nobs) % LANDMARKS
                rows[:, 2:5] = lm[rows[:, 0].astype(int)] + rng.normal(0, 0.4, (nobs, 3))
                odom = pkg.PfcOdom()
                odom.t[:], odom.q[:] = list(rng.normal(0, 0.02, 3)), [1.0, 0.0, 0.0, 0.0]
                odom.tstd[:], odom.rstd[:] = [0.02] * 3, [0.01] * 3
                prm = pkg.PfcCycleParams(0.5, 0.2, 3.0, 1.0, ratio, 0)  # resamples always
                est = np.zeros(pkg.PFC_EST_LEN)
                assert lib.pfc_cycle(pf.h, C.byref(odom), pkg.make_cobs(rows), nobs,
                                     C.byref(prm), pkg.dptr(est)) == 0
                assert est[pkg.PFC_EST_RESAMPLED] == 1
                out.append(est)
            out.extend(pf.snapshot())
            captures.append(lib.pfc_graph_captures(pf.h))
    finally:
        pf.close()
    return out, captures


def test_replaced_buckets_are_captured_again(kernels):
    steps = [s for s, _ in STEPS]
    direct, none = _cycles(kernels, 0, steps)
    replayed, captures = _cycles(kernels, 1, steps)
    assert none == [0] * len(STEPS)
    assert captures == [c for _, c in STEPS]
    for a, b in zip(direct, replayed):
        assert np.array_equal(a, b)


def test_cycles_without_injection_keep_their_graph(kernels):
    steps = [(64, 0.0), (256, 0.0), 0.05, (64, 0.0), (256, 0.0)]
    direct, _ = _cycles(kernels, 0, steps)
    replayed, captures = _cycles(kernels, 1, steps)
    assert captures == [1, 2, 2, 2, 2]
    for a, b in zip(direct, replayed):
        assert np.array_equal(a, b)


def test_captures_without_a_handle(kernels):
    assert kernels.pfc_graph_captures(None) == -1
