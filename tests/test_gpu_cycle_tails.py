"""The ends of the cycle's kernels: injection draws chained per output (several on
one output, ratios that fill a tile's bucket and overflow it), and the sums over the
grid at block counts around its groups of 32 lanes, against the FP64 oracle."""
import ctypes as C

import numpy as np
import pytest

import oracle
from pf_helpers import RawPF, cloud, i32p, ours_set_state, ours_weights

pytestmark = pytest.mark.gpu


# 2048 outputs a tile; a bucket holds up to 256 draws, so 0.12 fills one and more
# overflows; on 40 or 7 particles most outputs get several draws
@pytest.mark.parametrize("n,inject", [(7, 1.0), (40, 0.9), (2049, 0.02), (5000, 0.05),
                                      (5000, 0.12), (4096, 0.3), (2048, 1.0), (70_001, 0.01)])
def test_injection_chains(kernels, n, inject):
    pf = RawPF(kernels, n, seed=6)
    try:
        pos, quat = cloud(n, 5)[:2]
        w = np.random.default_rng(n).random(n).astype(np.float32)
        w /= w.sum()
        ours_set_state(pf, pos, quat, w)
        before = pf.snapshot()[0].reshape(-1, 3)
        assert kernels.pfc_record_ancestors(pf.h, 1) == 0
        pf.resample(inject)
        lcg1 = C.c_ulonglong()
        assert kernels.pfc_get_lcg(pf.h, C.byref(lcg1)) == 0
        anc = np.zeros(n, np.int32)
        assert kernels.pfc_get_ancestors(pf.h, i32p(anc)) == 0
        k = int(np.float32(inject) * np.float32(n))
        expect = oracle.inject_apply(before[anc].reshape(-1).copy(), k, lcg1.value, 0)
        got = pf.snapshot()[0]
        assert np.array_equal(got, expect)
        # sums of the jittered cloud: its weights are f32(1/n)
        wd = np.float64(np.float32(1.0) / np.float32(n))
        ref = wd * got.reshape(-1, 3).astype(np.float64).sum(0)
        assert np.allclose(pf.est_sums()[:3], ref, rtol=1e-11, atol=1e-12)
    finally:
        pf.close()


# 1024 particles a block of the estimate passes (up to 296 blocks)
@pytest.mark.parametrize("n", [1, 1023, 1025, 31 * 1024, 33 * 1024 + 1, 255 * 2048, 300_000,
                               303_105, 600_001])
def test_sums_over_the_grid(kernels, n):
    pf = RawPF(kernels, n, seed=6)
    try:
        pos, quat = cloud(n, 5)[:2]
        w = np.random.default_rng(n).random(n).astype(np.float32)
        w = (w / w.sum()).astype(np.float32)
        ours_set_state(pf, pos, quat, w)
        sums = pf.est_sums()
        p, q = pos.reshape(-1, 3).astype(np.float64), quat.reshape(-1, 4).astype(np.float64)
        wd = ours_weights(pf).astype(np.float64)
        m = np.einsum("i,ij,ik->jk", wd, q, q)[np.triu_indices(4)]
        ref = np.concatenate([(wd[:, None] * p).sum(0), m, [(wd ** 2).sum()]])
        assert np.allclose(sums, ref, rtol=1e-11, atol=1e-13)
        mp, mq = sums[:3], np.array([1.0, 0, 0, 0])
        cov = pf.covs(mp, mq)
        d = p - np.float64(np.float32(mp))
        ref = np.einsum("i,ij,ik->jk", wd, d, d)[np.triu_indices(3)]
        assert np.allclose(cov[:6], ref, rtol=1e-11, atol=1e-13)
    finally:
        pf.close()
