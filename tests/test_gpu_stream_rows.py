"""-m gpu: one-row products as a stream of weights (csrc/stream_rows.cuh) at the edges of its geometry - rows of one 512-byte chunk to the longest
that it takes and one past that, ragged last chunks, several rows side by side, one row per CTA and more than one CTA holds sums for - against 64 bits.
Bound: fp32 sums of n <= 32768 products, 1e-6 of the norm (measured 2e-7), or of the norm that as many
values of unit scale have where the sums of a few rows happen to cancel (inputs and rows are of unit norm per element)."""
import ctypes as C

import pytest
import torch

from yalm_b200 import api

pytestmark = pytest.mark.gpu
TYPES = {"fp32": (torch.float32, api.F32, 4), "fp16": (torch.float16, api.F16, 2), "bf16": (torch.bfloat16, api.BF16, 2), "fp8": (torch.float8_e4m3fn, api.F8E4M3, 1)}
# bytes of a row: within one chunk, at and around 16 chunks (two rows a stage), 32 (a row a stage), 64 and 128 (two, four stages a row)
ROW_BYTES = [16, 496, 512, 528, 1536, 2560, 5504, 8176, 8192, 8208, 16384, 16400, 28672, 32768, 32784, 33808, 65536, 65552]


def p(t):
    return C.c_void_p(None if t is None else t.data_ptr())


def rel(got, want):
    return ((got.double() - want).norm() / want.norm().clamp(min=want.numel() ** 0.5)).item()


def matrix(d, n, dtype):
    w = torch.randn((d, n), device="cuda") * n ** -0.5
    if dtype != "fp8":
        t = w.to(TYPES[dtype][0])
        return t, None, t.double()
    scale = w.abs().amax(dim=1) / 448.0
    t = (w / scale[:, None]).to(TYPES[dtype][0])
    return t, scale, t.float().double() * scale[:, None].double()


@pytest.mark.parametrize("dtype", sorted(TYPES))
@pytest.mark.parametrize("row_bytes", ROW_BYTES)
def test_rows_of_every_length(row_bytes, dtype):
    L, (_, code, size) = api.lib(), TYPES[dtype]
    n = row_bytes // size
    for d in (1, 37, 150, 617, (2 << 20) // row_bytes // 2 * 2 + 38):  # (short rows are streamed from some thousands on)
        torch.manual_seed(row_bytes + d)
        (w, s, plain), x = matrix(d, n, dtype), torch.randn(n, device="cuda")
        out = torch.full((d + 4,), 7.0, device="cuda")
        rc = L.yalm_gemv(p(out), p(x), p(w), p(s), C.c_int(n), C.c_int(d), C.c_int(code), None)
        if n * 4 > 200 * 1024:
            assert rc == -1  # a vector that does not fit into shared memory is refused
            continue
        assert rc == 0 and rel(out[:d], plain @ x.double()) < 1e-6 and (out[d:] == 7.0).all()
        if dtype == "bf16":
            continue
        norm, residual = 1 + 0.1 * torch.randn(n, device="cuda"), torch.randn(d, device="cuda")
        y = x.double() / torch.sqrt((x.double() ** 2).mean() + 1e-5) * norm.double()
        assert L.yalm_lm_head(p(out), p(x), p(norm), p(w), p(s), C.c_int(n), C.c_int(d), C.c_float(1e-5), C.c_int(code), None) == 0
        assert rel(out[:d], plain @ y) < 1e-6
        if d % 2 == 0:
            out[:d] = residual  # in place, as the residual stream is
            assert L.yalm_gemv_residual(p(out), p(out), p(x), p(w), p(s), C.c_int(n), C.c_int(d), C.c_int(code), C.c_int(1), None, None, None) == 0
            assert rel(out[:d], residual.double() + plain @ x.double()) < 1e-6 and (out[d:] == 7.0).all()
        (w3, s3, plain3), hb = matrix(d, n, dtype), torch.full((d + 4,), 7.0, device="cuda")
        assert L.yalm_ffn_glu(p(hb), p(x), p(norm), p(w), p(w3), p(s), p(s3), None, None, C.c_int(n), C.c_int(d), C.c_int(api.ACT_SILU), C.c_float(1e-5), C.c_int(code),
                              C.c_int(0), C.c_int(0), None, None, None, None) == 0
        assert rel(hb[:d], torch.nn.functional.silu(plain @ y) * (plain3 @ y)) < 1e-6 and (hb[d:] == 7.0).all()


@pytest.mark.parametrize("dtype", ["fp16", "fp8"])
@pytest.mark.parametrize("d,n", [(148 * 600 + 5, 64), (148 * 270 + 1, 1024), (3000, 16384)])
def test_more_rows_than_sums_are_held(d, n, dtype):
    L, code = api.lib(), TYPES[dtype][1]
    torch.manual_seed(d)
    (w, s, plain), x = matrix(d, n, dtype), torch.randn(n, device="cuda")
    out = torch.full((d + 4,), 7.0, device="cuda")
    assert L.yalm_gemv(p(out), p(x), p(w), p(s), C.c_int(n), C.c_int(d), C.c_int(code), None) == 0
    assert rel(out[:d], plain @ x.double()) < 1e-6 and (out[d:] == 7.0).all()


def test_what_is_not_finite_stays_in_its_row():
    """Neighbouring rows share stages and chunks."""
    L, d, n = api.lib(), 300, 4104
    torch.manual_seed(1)
    w, x = torch.randn((d, n), device="cuda").half(), torch.randn(n, device="cuda")
    w[7, n - 1], w[8, 0], w[200, 512] = float("inf"), float("nan"), float("inf")
    out = torch.zeros(d, device="cuda")
    assert L.yalm_gemv(p(out), p(x), p(w), None, C.c_int(n), C.c_int(d), C.c_int(api.F16), None) == 0
    bad = torch.zeros(d, dtype=torch.bool, device="cuda")
    bad[[7, 8, 200]] = True
    assert torch.equal(~torch.isfinite(out), bad)


def test_weights_written_just_before():
    """The weights' first bytes are fetched into L2 ahead of the kernel's turn: what is stored until then counts."""
    L, d, n = api.lib(), 4096, 4096
    x, out = torch.randn(n, device="cuda"), torch.empty(d, device="cuda")
    w = torch.zeros((d, n), device="cuda", dtype=torch.float16)
    y = torch.empty(d, device="cuda")
    for i in range(8):
        L.yalm_gemv(p(y), p(x), p(w), None, C.c_int(n), C.c_int(d), C.c_int(api.F16), None)
        w.fill_(float(i + 1))
        L.yalm_gemv(p(out), p(x), p(w), None, C.c_int(n), C.c_int(d), C.c_int(api.F16), None)
        assert rel(out, (i + 1) * x.double().sum() * torch.ones(d, device="cuda", dtype=torch.float64)) < 1e-4  # one sum of 4096 values that cancel


def test_weights_written_by_the_kernel_that_lets_it_begin():
    """The matrix of the second product is the first one's result, in fp32: that kernel lets the next begin, which fetches the matrix's first bytes, before it stores it.
    Every round stores other values over the last one's."""
    L, n, d = api.lib(), 2048, 512                     # 4 MB, two rounds of a CTA's first stages
    f32 = C.c_int(api.F32)
    v, x = torch.randn((9, 64), device="cuda"), torch.randn(n, device="cuda")
    first = torch.randn((n * d, 64), device="cuda")    # 268 MB: its last rows are stored long after the next kernel began
    matrix, out = torch.zeros((d, n), device="cuda"), torch.zeros((9, d), device="cuda")
    assert L.yalm_gemv_streamed(0, api.F32, 64, n * d) == 1 and L.yalm_gemv_streamed(0, api.F32, n, d) == 1
    for i in range(9):
        assert L.yalm_gemv(p(matrix), p(v[i]), p(first), None, C.c_int(64), C.c_int(n * d), f32, None) == 0
        assert L.yalm_gemv(p(out[i]), p(x), p(matrix), None, C.c_int(n), C.c_int(d), f32, None) == 0
    for i in range(9):                                 # fp32 sums of 64, then of 2048 terms
        assert rel(out[i], (first.double() @ v[i].double()).view(d, n) @ x.double()) < 2e-6
