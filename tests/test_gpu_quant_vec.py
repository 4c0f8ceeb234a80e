"""The vector forms of the quantisers and dequantisers against the scalar kernels, bit for bit: the same numbers at a
misaligned address (which only the scalar kernels take) and at an aligned one.  Ragged tiles, every group size
the vector int4 kernels take, rounding ties, zeros, subnormals, infinities and NaN."""
import numpy as np
import pytest
import torch

import longhornai_b200 as lb

pytestmark = pytest.mark.gpu


def misaligned(t):
    """The same values, contiguous, one element past an aligned address."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    flat[1:] = t.reshape(-1)
    return flat[1:].view(t.shape)


def weights(rows, cols, special):
    rng = np.random.default_rng(rows * 7919 + cols)
    w = (rng.standard_normal((rows, cols)) * rng.choice([1e-3, 1.0, 40.0], size=(1, cols))).astype(np.float32)
    # quotients on or beside a rounding boundary: a column whose largest magnitude makes the scale a power of two
    for lim, c in ((7, 0), (127, 1), (15, 2)):
        k = rng.integers(-2 * lim, 2 * lim + 1, size=rows) * 0.5
        w[:, c] = np.clip(k, -lim, lim).astype(np.float32)
        w[0, c] = lim
        w[1::5, c] = np.nextafter(w[1::5, c], np.float32(100.0))
    w[:, 3] = 0.0
    if special:
        w[:, 4 % cols] *= np.float32(1e-42)                 # subnormal scales
        w[rows // 2, 5 % cols] = np.inf
        w[rows // 3, 6 % cols] = -np.inf
        w[rows // 4, 7 % cols] = np.nan
    return torch.from_numpy(w).cuda()


def same(a, b, what):
    a, b = (x if isinstance(x, tuple) else (x,) for x in (a, b))
    for i, (x, y) in enumerate(zip(a, b)):
        assert x.shape == y.shape and torch.equal(x.view(torch.uint8), y.view(torch.uint8)), f"{what}: output {i}"


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("K,N,G", [(16, 4, 16), (144, 132, 16), (96, 260, 32), (192, 8, 64), (384, 516, 128), (128, 1028, 128)])
def test_int4_groups(K, N, G, special):
    w = weights(K, N, special)
    odd = misaligned(w)
    same(lb.q4_quantize_groupwise(w, G), lb.q4_quantize_groupwise(odd, G), "int4")
    same(lb.q4a_quantize_groupwise(w, G), lb.q4a_quantize_groupwise(odd, G), "asymmetric int4")
    p, s = lb.q4_quantize_groupwise(w, G)
    same(lb.q4_dequantize_groupwise(p, s, G), lb.q4_dequantize_groupwise(misaligned(p), s, G), "int4 back")
    p, s, z = lb.q4a_quantize_groupwise(w, G)
    same(lb.q4a_dequantize_groupwise(p, s, z, G), lb.q4a_dequantize_groupwise(misaligned(p), s, z, G), "asymmetric int4 back")


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("rows,cols", [(1, 8), (17, 132), (129, 260), (300, 8), (5, 8196), (130, 4100)])
def test_int8_and_fp8(rows, cols, special):
    w = weights(max(rows, 2), cols, special)[:rows].contiguous()
    odd = misaligned(w)
    for name, quant in (("int8 columns", lb.q8_quantize_per_col), ("int8 rows", lb.q8_quantize_per_row), ("int8 tensor", lb.q8_quantize_per_tensor),
                        ("fp8 columns", lb.fp8_quantize_per_col), ("fp8 rows", lb.fp8_quantize_per_row), ("fp8 tensor", lb.fp8_quantize_per_tensor)):
        same(quant(w), quant(odd), name)
    for name, quant, back in (("int8 columns", lb.q8_quantize_per_col, lb.q8_dequantize_per_col), ("int8 rows", lb.q8_quantize_per_row, lb.q8_dequantize_per_row)):
        q, s = quant(w)
        same(back(q, s), back(misaligned(q), s), name + " back")
    for mode, quant in ((0, lb.fp8_quantize_per_tensor), (1, lb.fp8_quantize_per_row), (2, lb.fp8_quantize_per_col)):
        q, s = quant(w)
        same(lb.fp8_dequantize(q, s, mode), lb.fp8_dequantize(misaligned(q), s, mode), f"fp8 back {mode}")


def test_every_fp8_code_and_boundary():
    """Finite values beside every rounding boundary of E4M3, scale 1 (largest magnitude 448)."""
    codes = torch.arange(256, dtype=torch.uint8, device="cuda")
    v = lb.fp8_dequantize(codes.view(1, 256), torch.ones(1, device="cuda"), 0).view(-1)
    v = v[torch.isfinite(v)]
    v = torch.sort(v).values
    mid = (v[1:] + v[:-1]) * 0.5
    inf = torch.full_like(mid, float("inf"))
    x = torch.cat([v, mid, torch.nextafter(mid, inf), torch.nextafter(mid, -inf)])
    x = x[: x.numel() // 4 * 4].contiguous()
    x[0] = 448.0
    same(lb.fp8_quantize_per_tensor(x.view(1, -1)), lb.fp8_quantize_per_tensor(misaligned(x.view(1, -1))), "fp8 boundaries")
