"""The warp-tile bf16 GEMM gives the same bits as the 64 x 64 tiled kernel: each
output is one chain of float32 multiply-adds over ascending k either way. The
large product (over 296 tiles) takes the tiled kernel; its first rows, computed
on their own, the warp tiles. Ragged M, N and K, aligned and unaligned pitches,
both transposes, and the epilogue's options."""

import ctypes

import pytest
import torch

from pyqrackising_b200 import _lib
from pyqrackising_b200 import device as D

pytestmark = pytest.mark.gpu


def _gemm(tA, tB, M, N, K, A, lda, B, ldb, beta, C32, C16, ldc, bias, relu):
    _lib.call("pqi_mpnn_gemm", tA, tB, M, N, K, ctypes.c_float(0.5), D._ptr(A), lda, D._ptr(B), ldb,
              ctypes.c_float(beta), D._ptr(C32), D._ptr(C16), ldc, D._ptr(bias), relu, D.stream_ptr())


@pytest.mark.parametrize("tA,tB", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("m,N,K,pad", [(1, 1, 1, 0), (16, 8, 128, 0), (17, 9, 129, 1), (100, 64, 64, 0), (128, 64, 1024, 8),
                                       (64, 1, 333, 0), (5, 64, 1000, 3), (130, 128, 127, 0)])
def test_warp_tiles_match_the_tiled_kernel(tA, tB, m, N, K, pad):
    g = torch.Generator(device="cuda").manual_seed(m * N + K)
    big = 64 * 300
    rA, cA = (K, big) if tA else (big, K)
    rB, cB = (N, K) if tB else (K, N)
    A = torch.randn(rA, cA + pad, generator=g, device="cuda").to(torch.bfloat16)
    B = torch.randn(rB, cB + pad, generator=g, device="cuda").to(torch.bfloat16)
    bias = torch.randn(N, generator=g, device="cuda")
    for beta, use_bias, relu in ((0.0, False, 0), (1.0, True, 1)):
        C = torch.randn(big, N + 2, generator=g, device="cuda")
        small, small16 = C[:m].clone(), torch.zeros(m, N + 2, dtype=torch.bfloat16, device="cuda")
        C16 = torch.zeros(big, N + 2, dtype=torch.bfloat16, device="cuda")
        b = bias if use_bias else None
        _gemm(tA, tB, big, N, K, A, cA + pad, B, cB + pad, beta, C, C16, N + 2, b, relu)
        _gemm(tA, tB, m, N, K, A, cA + pad, B, cB + pad, beta, small, small16, N + 2, b, relu)
        assert torch.equal(C[:m], small) and torch.equal(C16[:m], small16)
