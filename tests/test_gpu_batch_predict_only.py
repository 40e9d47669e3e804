"""Cycles without observations: the last weighting tile of a filter steps its
generation, so the clouds after several of them equal the single filter's."""
import numpy as np
import pytest

import cuda_pf_localization_b200 as pkg
from pf_helpers import RawPF

pytestmark = pytest.mark.gpu

SIZES = [1, 255, 257, 70_001]


def test_predict_only_cycles_equal_single(kernels):
    seeds = [11, 12, 13, 14]
    prior = [0.5, -1.0, 0.2, 1.0, 0.0, 0.0, 0.0]
    t, q = [0.1, 0.02, 0.0], [0.99875026, 0.0, 0.0, 0.04997917]
    tn, rn = [0.02, 0.02, 0.01], [0.01, 0.01, 0.02]
    odom = pkg.PfcOdom()
    odom.t[:], odom.q[:], odom.tstd[:], odom.rstd[:] = t, q, tn, rn
    b = pkg.BatchPF(SIZES, seeds=np.array(seeds, np.uint32), obs_cap=8)
    nf = len(SIZES)
    b.set_landmarks([np.array([[1.0, 2.0, 0.5]])] * nf)
    b.reinit([np.array(prior)] * nf, np.full((nf, 3), 0.3), np.full((nf, 3), 0.1))
    none = [np.zeros((0, 6))] * nf
    for _ in range(3):
        b.cycle([odom] * nf, none)
    for f in range(nf):
        pf = RawPF(kernels, SIZES[f], seed=seeds[f])
        try:
            pf.reinit(prior, [0.3] * 3, [0.1] * 3)
            for _ in range(3):
                pf.predict(t, q, tn, rn)
            for a, c in zip(b.snapshot(f), pf.snapshot()):
                assert np.array_equal(a, c)
        finally:
            pf.close()
