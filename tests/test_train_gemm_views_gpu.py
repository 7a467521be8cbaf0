"""The training GEMM into a column slice of a wider matrix: what lies beside C stays."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("acc", [False, True])
@pytest.mark.parametrize("M,N,K", [(64, 64, 5000), (64, 40, 100), (130, 70, 3000)])  # split K, one chunk, split
def test_beside_c(cuda_ready, M, N, K, acc):
    import torch

    from seqtree_b200.learned import train_gemm_bf16
    g = torch.Generator(device="cuda").manual_seed(K)
    a, b = torch.randn((M, K), device="cuda", generator=g), torch.randn((K, N), device="cuda", generator=g)
    wide = torch.randn((M + 1, N + 23), device="cuda", generator=g)
    before = wide.clone()
    train_gemm_bf16(a, b, wide[:M, 10:10 + N], accumulate=acc)
    torch.cuda.synchronize()
    A, B = a.bfloat16().double(), b.bfloat16().double()
    want = A @ B + (before[:M, 10:10 + N].double() if acc else 0)
    bound = (1e-5 + 1e-8 * K) * (A.abs() @ B.abs()) + 1e-6  # as test_train_gemm_gpu, and C's own rounding
    assert bool(((wide[:M, 10:10 + N].double() - want).abs() <= bound).all())
    before[:M, 10:10 + N] = wide[:M, 10:10 + N]
    assert torch.equal(wide, before)
