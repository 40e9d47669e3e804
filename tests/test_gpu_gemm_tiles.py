"""The GEMM's two tile shapes: a product whose size takes 128 x 256 tiles equals,
bit for bit, the same product taken 128 rows at a time on 128 x 128 tiles (both sum
k in the same order), and both match torch fp32."""
import numpy as np
import pytest
import torch

import cuda_pf_localization_b200 as pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [
    (4096, 1024, 64),     # 128 wide tiles in one round (256 narrow ones in two)
    (2432, 1024, 192),    # 76 wide tiles (152 narrow ones)
    (2304, 1024, 192),    # 144 narrow tiles, one round: stays narrow
    (4864, 1024, 448),    # 152 wide tiles, two rounds
    (9472, 256, 64),      # 148 narrow tiles, one round: stays narrow
    (8192, 768, 320)])    # 192 wide tiles
def test_tile_shapes_agree(kernels, M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    a = torch.randn(M, K, generator=g).bfloat16()
    b = torch.randn(N, K, generator=g).bfloat16()
    ah, bh = a.view(torch.uint16).numpy(), b.view(torch.uint16).numpy()
    d = pkg.learned_gemm(ah, bh)
    for r in {0, 128 * (M // 256), M - 128}:
        rows = pkg.learned_gemm(np.ascontiguousarray(ah[r:r + 128]), bh)
        assert np.array_equal(d[r:r + 128].view(np.uint32), rows.view(np.uint32))
    ref = (a.double() @ b.double().T).numpy()
    # products of bf16 values are exact in f32; only the summation order and its
    # roundings differ: |err| <= K 2^-23 sum |a||b|
    bound = K * 2.0 ** -23 * (a.abs().double() @ b.abs().double().T).numpy()
    assert np.all(np.abs(d - ref) <= bound + 1e-6)
