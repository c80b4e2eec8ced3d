"""The matrix kernels at the edges of their tiles, against float64 torch."""
import numpy as np
import pytest
import torch

from helpers import C
import nvllm_pkg

pytestmark = pytest.mark.gpu


def _product(M, N, K, prec, kernel):
    """Largest error over the bound of a K-term fp32 sum: K 2^-24 times the sum of the magnitudes of its terms."""
    L = nvllm_pkg.sub("lib")
    g = torch.Generator().manual_seed(M * 1000003 + N * 1009 + K)
    A, B = torch.randn(M, K, generator=g), torch.randn(K, N, generator=g)
    if prec == C.PREC_BF16:
        A, B = A.to(torch.bfloat16).float(), B.to(torch.bfloat16).float()
    out, _ = L.op_matmul(A.numpy(), B.numpy(), prec=prec, kernel=kernel)
    ref, mag = A.double() @ B.double(), A.double().abs() @ B.double().abs()
    return float(((torch.from_numpy(out).double() - ref).abs() / (mag * K * 2.0 ** -24 + 1e-30)).max())


@pytest.mark.parametrize("M,N,K", [
    (1, 1, 8), (9, 63, 24), (16, 64, 32), (17, 65, 40),  # 16- and 32-row tiles, columns around one tile, k tails
    (32, 130, 256), (33, 64, 264), (64, 192, 1000),      # the first 64-row tile, two and more k ranges
    (65, 3000, 136), (300, 768, 3072),                   # many tiles in one range; slices up to the buffer's room
])
def test_fp32_tiles(M, N, K):
    assert _product(M, N, K, C.PREC_FP32, 2) <= 1.0


@pytest.mark.parametrize("M,N,K", [
    (2, 1, 8), (3, 15, 72), (5, 17, 264), (8, 16, 64),   # rows, columns and k around one 16 x 64 chunk
    (7, 100, 776), (8, 768, 3072), (2, 2304, 768),       # k ranges on several CTAs
    (4, 9473, 520), (8, 9472, 4544),                     # the first column counts with 32-row tiles
])
def test_bf16_rows_on_mma(M, N, K):
    assert _product(M, N, K, C.PREC_BF16, 1) <= 1.0
