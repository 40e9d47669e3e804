"""Injection ratios whose draws overflow a tile's bucket, over several tiles and rounds of
draws: every output takes its draws in ascending order, as the FP64 oracle applies them."""
import ctypes as C

import numpy as np
import pytest

import oracle
from pf_helpers import RawPF, cloud, i32p, ours_set_state

pytestmark = pytest.mark.gpu


# tiles of 2048 outputs, rounds of 256 draws: a ragged last tile of one output, rounds
# without a draw on a tile (100 001 particles), the last round of one draw (2570 x 0.1 = 257)
@pytest.mark.parametrize("n,inject", [(2049, 1.0), (2570, 0.1), (2570, 0.5), (6150, 1.0),
                                      (30_000, 0.2), (100_001, 0.5), (70_001, 1.0)])
def test_overflowing_draws(kernels, n, inject):
    pf = RawPF(kernels, n, seed=6)
    try:
        pos, quat = cloud(n, 5)[:2]
        w = np.random.default_rng(n).random(n).astype(np.float32)
        w /= w.sum()
        assert kernels.pfc_record_ancestors(pf.h, 1) == 0
        k = int(np.float32(inject) * np.float32(n))
        for _ in range(2):  # the second with the buffers of the first
            ours_set_state(pf, pos, quat, w)
            before = pf.snapshot()[0].reshape(-1, 3)
            pf.resample(inject)
            lcg1 = C.c_ulonglong()
            assert kernels.pfc_get_lcg(pf.h, C.byref(lcg1)) == 0
            anc = np.zeros(n, np.int32)
            assert kernels.pfc_get_ancestors(pf.h, i32p(anc)) == 0
            expect = oracle.inject_apply(before[anc].reshape(-1).copy(), k, lcg1.value, 0)
            got = pf.snapshot()[0]
            assert np.array_equal(got, expect)
            wd = np.float64(np.float32(1.0) / np.float32(n))
            ref = wd * got.reshape(-1, 3).astype(np.float64).sum(0)
            assert np.allclose(pf.est_sums()[:3], ref, rtol=1e-11, atol=1e-12)
    finally:
        pf.close()
