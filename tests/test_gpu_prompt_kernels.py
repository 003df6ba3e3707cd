"""-m gpu: the tensor-core kernels of a prompt portion at the sizes where their tiling can go wrong (edges of row and column tiles,
remainders of K, K in several parts, one row, both sides of the 128-row line between the two GEMMs), against 64-bit products.

Bounds.  Products of 16-bit values are exact in the fp32 accumulator; its sums lose at most one unit of 2^-23 of the running sum per
addition of 16 products, K / 16 <= 900 of them: 1e-4 of the result's norm at the worst, 3e-5 with signs that vary (measured 1.2e-5)."""
import ctypes as C

import pytest
import torch

from yalm_b200 import api

pytestmark = pytest.mark.gpu


def L():
    return api.lib()


def ptr(t):
    return C.c_void_p(None if t is None else t.data_ptr())


def i32(*v):
    return [C.c_int(x) for x in v]


def normal(seed, shape, std=1.0, dtype=torch.float32):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return (torch.randn(shape, generator=g, device="cuda") * std).to(dtype)


def rel(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("bf16", [0, 1])
@pytest.mark.parametrize("accumulate", [0, 1])
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (17, 4096, 4096), (128, 128, 64), (33, 1000, 520), (100, 20000, 512), (127, 260, 4104),  # few rows
                                   (129, 128, 64), (256, 256, 64), (257, 100, 4096), (300, 1028, 776), (384, 4096, 1024),             # pairs, one K part
                                   (512, 1024, 4096), (512, 4096, 8192), (300, 516, 2056), (512, 20000, 520)])                        # several K parts / tiles per pair
def test_gemm_tiles(M, N, K, accumulate, bf16):
    dt = torch.bfloat16 if bf16 else torch.float16
    a, w = normal(M + N, (M, K), dtype=dt), normal(K, (N, K), K ** -0.5, dt)
    ldc = (N + 3) // 4 * 4 + 4
    c = torch.full((M, ldc), 7.0, device="cuda")
    c[:, :N] = normal(5, (M, N))
    start, again = c.clone(), c.clone()
    for out in (c, again):
        assert L().yalm_gemm_16(ptr(out), C.c_int(ldc), ptr(a), ptr(w), *i32(M, N, K, accumulate, bf16), C.c_float(0.5), None) == 0
    want = 0.5 * (a.double() @ w.double().T) + (start[:, :N].double() if accumulate else 0.0)
    assert rel(c[:, :N], want) < 3e-5
    assert (c[:, N:] == 7.0).all()       # nothing past the columns
    assert torch.equal(c, again)         # the parts of K are added in a fixed order


@pytest.mark.parametrize("act", [api.ACT_SILU, api.ACT_GELU])
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (17, 2816, 1024), (128, 520, 512), (130, 104, 64), (200, 72, 4096), (300, 2816, 1024), (512, 8192, 2048)])
def test_gemm_glu_tiles(M, N, K, act):
    a, w1, w3 = normal(M, (M, K), dtype=torch.float16), normal(N, (N, K), K ** -0.5, torch.float16), normal(K, (N, K), K ** -0.5, torch.float16)
    w1 *= 4                              # gates out to +-16: both ends of the activations
    h = torch.full((M, N + 8), 7.0, device="cuda", dtype=torch.float16)
    assert L().yalm_gemm_glu_f16(ptr(h), C.c_int(N + 8), ptr(a), ptr(w1), ptr(w3), *i32(M, N, K, act), None) == 0
    g, u = a.double() @ w1.double().T, a.double() @ w3.double().T
    y = g if act == api.ACT_SILU else 2 * 0.797885 * (g + 0.044715 * g ** 3)
    want = g * torch.sigmoid(y) * u
    assert rel(h[:, :N], want) < 5e-4    # one fp16 rounding (2^-11 at most, 2.1e-4 in the norm) over the sums' 3e-5
    assert (h[:, N:] == 7.0).all()


@pytest.mark.parametrize("M,K,ends", [(40, 512, [128, 260, 1000]), (300, 1024, [512, 1028, 2048, 2052]), (512, 4096, [256, 512, 768])])
def test_gemm_segments(M, K, ends):
    S, N = len(ends), ends[-1]
    a, w = normal(M, (S * M, K), dtype=torch.bfloat16), normal(K, (N, K), K ** -0.5, torch.bfloat16)
    c = torch.zeros((M, N), device="cuda")
    assert L().yalm_gemm_16_segments(ptr(c), C.c_int(N), ptr(a), ptr(w), *i32(M, N, K, S), (C.c_int * S)(*ends), C.c_int(1), None) == 0
    at = 0
    for s, end in enumerate(ends):
        assert rel(c[:, at:end], a[s * M:(s + 1) * M].double() @ w[at:end].double().T) < 3e-5
        at = end
