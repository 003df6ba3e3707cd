"""-m gpu: the one-row products at sizes where their rows are dealt out in larger and in smaller tasks (fewer rows than warps, a last round
with few tasks, odd counts of rows), against 64 bits.  Bound: fp32 sums of n <= 11008 products, 1e-6 of the norm (measured 3e-7)."""
import ctypes as C

import pytest
import torch

from yalm_b200 import api

pytestmark = pytest.mark.gpu
TYPES = {"fp32": (torch.float32, api.F32), "fp16": (torch.float16, api.F16), "bf16": (torch.bfloat16, api.BF16), "fp8": (torch.float8_e4m3fn, api.F8E4M3)}


def p(t):
    return C.c_void_p(None if t is None else t.data_ptr())


def stored(w, dtype):
    """A matrix as stored, its row scales (fp8), and its values in 64 bits."""
    if dtype != "fp8":
        t = w.to(TYPES[dtype][0])
        return t, None, t.double()
    scale = w.abs().amax(dim=1) / 448.0
    t = (w / scale[:, None]).to(TYPES[dtype][0])
    return t, scale, t.float().double() * scale[:, None].double()


def rel(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("dtype", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("d,n", [(1, 64), (3, 4096), (2047, 1032), (4096, 4096), (6145, 512), (9473, 256), (14211, 264), (32001, 128)])
def test_rows(d, n, dtype):
    L, (td, code) = api.lib(), TYPES[dtype]
    torch.manual_seed(d)
    w, x, out = torch.randn((d, n), device="cuda").to(td), torch.randn(n, device="cuda"), torch.full((d + 4,), 7.0, device="cuda")
    assert L.yalm_gemv_scaled(p(out), p(x), p(w), C.c_int(n), C.c_int(d), C.c_int(code), C.c_float(0.5), None) == 0
    assert rel(out[:d], 0.5 * (w.double() @ x.double())) < 1e-6 and (out[d:] == 7.0).all()


@pytest.mark.parametrize("d,n", [(1, 64), (3, 4096), (2047, 1040), (4096, 4096), (9473, 256), (14211, 272), (32001, 128)])
def test_rows_fp8(d, n):
    torch.manual_seed(d)
    w, scale, plain = stored(torch.randn((d, n), device="cuda"), "fp8")
    x, out = torch.randn(n, device="cuda"), torch.full((d + 4,), 7.0, device="cuda")
    assert api.lib().yalm_gemv(p(out), p(x), p(w), p(scale), C.c_int(n), C.c_int(d), C.c_int(api.F8E4M3), None) == 0
    assert rel(out[:d], plain @ x.double()) < 1e-6 and (out[d:] == 7.0).all()


@pytest.mark.parametrize("dtype", ["fp32", "fp16", "fp8"])
@pytest.mark.parametrize("dim,hidden", [(64, 32), (1024, 2816), (1600, 5120), (2048, 2050), (4096, 11008), (1024, 14336)])
def test_feed_forward(dim, hidden, dtype):
    L, code = api.lib(), TYPES[dtype][1]
    torch.manual_seed(dim + hidden)
    x, norm = torch.randn(dim, device="cuda"), 1 + 0.1 * torch.randn(dim, device="cuda")
    (w1, s1, p1), (w3, s3, p3) = (stored(torch.randn((hidden, dim), device="cuda") * dim ** -0.5, dtype) for _ in range(2))
    hb = torch.full((hidden + 4,), 7.0, device="cuda")
    assert L.yalm_ffn_glu(p(hb), p(x), p(norm), p(w1), p(w3), p(s1), p(s3), None, None, C.c_int(dim), C.c_int(hidden), C.c_int(api.ACT_SILU), C.c_float(1e-5), C.c_int(code),
                          C.c_int(0), C.c_int(0), None, None, None, None) == 0
    y = x.double() / torch.sqrt((x.double() ** 2).mean() + 1e-5) * norm.double()
    want = torch.nn.functional.silu(p1 @ y) * (p3 @ y)
    assert rel(hb[:hidden], want) < 1e-6 and (hb[hidden:] == 7.0).all()
    if hidden % 16 == 0:
        (w2, s2, p2), out = stored(torch.randn((dim, hidden), device="cuda") * hidden ** -0.5, dtype), torch.full((dim + 4,), 7.0, device="cuda")
        assert L.yalm_gemv_residual(p(out), p(x), p(hb), p(w2), p(s2), C.c_int(hidden), C.c_int(dim), C.c_int(code), C.c_int(1), None, None, None) == 0
        assert rel(out[:dim], x.double() + p2 @ hb[:hidden].double()) < 1e-6 and (out[dim:] == 7.0).all()


def test_refused_length_leaves_no_error():
    """An input that does not fit into shared memory is refused, and the next call runs."""
    L, n = api.lib(), 65536
    w, x, out = torch.randn((4, 64), device="cuda"), torch.randn(n, device="cuda"), torch.zeros(4, device="cuda")
    for refused in (lambda: L.yalm_gemv_scaled(p(out), p(x), p(w), C.c_int(n), C.c_int(4), C.c_int(api.F32), C.c_float(1.0), None),
                    lambda: L.yalm_gemv_residual(p(out), None, p(x), p(w), None, C.c_int(n), C.c_int(4), C.c_int(api.F32), C.c_int(1), None, None, None),
                    lambda: L.yalm_ffn_glu(p(out), p(x), p(x), p(w), p(w), None, None, None, None, C.c_int(n), C.c_int(4), C.c_int(api.ACT_SILU), C.c_float(1e-5),
                                           C.c_int(api.F32), C.c_int(0), C.c_int(0), None, None, None, None)):
        assert refused() == -1     # YALM_EINVAL, before anything is launched
        assert L.yalm_gemv_scaled(p(out), p(x), p(w), C.c_int(64), C.c_int(4), C.c_int(api.F32), C.c_float(1.0), None) == 0
        assert rel(out, w.double() @ x[:64].double()) < 1e-6
