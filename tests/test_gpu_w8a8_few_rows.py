"""GPU parity of the 8-bit tensor-core GEMMs with few rows and few tiles: K split over CTAs (int8 without beta, sums kept
in C until they are scaled), rows below a tile, a last block of K that is not whole.  Integer results are exact."""
import numpy as np
import pytest
import torch

import longhornai_b200 as lb
from cpu_checker import best_checker
from gpu_util import assert_close, assert_same_bits, dev, host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def chk():
    return best_checker()


@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (7, 272, 144), (33, 1040, 1024), (63, 128, 4112), (129, 256, 2048), (257, 528, 512), (600, 128, 1040)])
def test_w8a8(chk, M, N, K):
    rng = np.random.default_rng(M + N + K)
    A = rng.integers(-128, 128, size=(M, K)).astype(np.int8)
    B = rng.integers(-128, 128, size=(K, N)).astype(np.int8)
    sa = rng.uniform(1e-3, 1e-1, M).astype(np.float32)
    sb = rng.uniform(1e-3, 1e-1, N).astype(np.float32)
    dA, dB, da, db = dev(A), dev(B), dev(sa), dev(sb)
    C = torch.full((M, N), float("nan"), device="cuda")         # nothing of C is read where beta is 0
    assert_same_bits(host(lb.gemm_w8a8(dA, dB, da, db, C=C, alpha=0.75)), chk.gemm_w8a8(A, B, sa, sb, alpha=0.75), f"{M}x{N}x{K}")
    C0 = rng.standard_normal((M, N)).astype(np.float32)
    got = lb.gemm_w8a8(dA, dB, da, db, C=dev(C0), alpha=0.75, beta=0.5)
    assert_same_bits(host(got), chk.gemm_w8a8(A, B, sa, sb, C0, alpha=0.75, beta=0.5), f"{M}x{N}x{K} with beta")
    assert lb.default_context().poll() == 0


@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (7, 272, 1040), (40, 1040, 4096), (63, 144, 8192)])
def test_fp8_sums_are_no_further_off_than_sequential_fp32(M, N, K):
    """Fewer than 64 rows: parts of K added in fp32.  With beta the shape-agnostic kernel runs, whose sums are sequential."""
    g = torch.Generator(device="cuda").manual_seed(K)
    A, sa = lb.fp8_quantize_per_tensor(torch.randn(M, K, device="cuda", generator=g))
    B, sb = lb.fp8_quantize_per_tensor(torch.randn(K, N, device="cuda", generator=g) * 0.02)
    one, sa, sb = torch.ones(1, device="cuda"), float(sa), float(sb)
    want = (lb.fp8_dequantize(A, one, 0).double() @ lb.fp8_dequantize(B, one, 0).double()) * (sa * sb)
    err = lambda c: ((c.double() - want).norm() / want.norm()).item()  # noqa: E731
    C = torch.full((M, N), float("nan"), device="cuda")
    got = err(lb.gemm_fp8_e4m3(A, B, sa, sb, C=C))
    sequential = err(lb.gemm_fp8_e4m3(A, B, sa, sb, C=torch.zeros(M, N, device="cuda"), beta=1.0))
    # both hold one rounding of the result (2^-24, about 3e-8 in the 2-norm) at least
    assert got <= max(sequential, 6e-8), (got, sequential)
    assert lb.default_context().poll() == 0
