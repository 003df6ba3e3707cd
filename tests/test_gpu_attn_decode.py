"""-m gpu: yalm_attn_decode over every head size and group it has a kernel for, at the edges of its splits (one row, one short of and one
past a batch of rows for every warp, several splits, the last with few rows), against the softmax in 64 bits.

Bound: fp32 sums of a few thousand terms, the exponential's 2 units: 1e-6 of the norm (measured 3e-7)."""
import ctypes as C

import pytest
import torch

from yalm_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [128, 64, 32, 16])
@pytest.mark.parametrize("G", [1, 2, 4, 8])
@pytest.mark.parametrize("n_kv", [1, 3, 5, 8, 25])   # (5, 25: KV heads x splits odd on 148 multiprocessors)
def test_attn_decode_splits(hd, G, n_kv):
    L, H, ring = api.lib(), G * n_kv, 5000
    gen = torch.Generator(device="cuda")
    gen.manual_seed(hd + G)
    k, v = (torch.randn((n_kv, ring, hd), generator=gen, device="cuda").half() for _ in range(2))
    q = torch.randn((H, hd), generator=gen, device="cuda")
    work = torch.zeros(L.yalm_attn_workspace_bytes(H, n_kv, hd), device="cuda", dtype=torch.uint8)
    out = torch.empty((H, hd), device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    for rows in (1, 2, 63, 64, 65, 127, 129, 511, 513, 1000, 2049, ring):
        kk, vv = k.clone(), v.clone()
        kk[:, rows:], vv[:, rows:] = float("nan"), float("nan")
        ctl = torch.tensor([0, rows - 1, 0, rows - 1, rows, 0, 0, 0], device="cuda", dtype=torch.int32)
        assert L.yalm_attn_decode(p(out), p(kk), p(vv), p(q), p(work), H, n_kv, hd, ring, p(ctl), None) == 0   # the same workspace throughout
        w = torch.softmax(torch.einsum("ghd,gtd->ght", q.view(n_kv, G, hd).double(), k[:, :rows].double()) * hd ** -0.5, dim=-1)
        want = torch.einsum("ght,gtd->ghd", w, v[:, :rows].double()).reshape(H, hd)
        assert ((out.double() - want).norm() / want.norm()).item() < 1e-6, rows


@pytest.mark.parametrize("ring,n_kv", [(16, 8), (64, 8), (65, 8), (1100, 8), (1200, 8), (16384, 8), (16400, 8), (8484, 14), (8500, 14), (900, 15)])
def test_attn_decode_rings(ring, n_kv):
    """Four heads of 128 a kv head: rings with room for one split, a few, up to one a multiprocessor and more, and both sides of the lines from which two CTAs share
    a multiprocessor again (128 K rows of up to 8 kv heads, 116 K of up to 14); full and nearly empty.  Bound as above."""
    L, G, hd = api.lib(), 4, 128
    gen = torch.Generator(device="cuda")
    gen.manual_seed(ring)
    k, v = (torch.randn((n_kv, ring, hd), generator=gen, device="cuda").half() for _ in range(2))
    q = torch.randn((n_kv * G, hd), generator=gen, device="cuda")
    work = torch.zeros(L.yalm_attn_workspace_bytes(n_kv * G, n_kv, hd), device="cuda", dtype=torch.uint8)
    out = torch.empty_like(q)
    p = lambda t: C.c_void_p(t.data_ptr())
    for rows in (1, ring // 2 + 1, ring):
        ctl = torch.tensor([0, rows - 1, 0, rows - 1, rows, 0, 0, 0], device="cuda", dtype=torch.int32)
        assert L.yalm_attn_decode(p(out), p(k), p(v), p(q), p(work), n_kv * G, n_kv, hd, ring, p(ctl), None) == 0
        w = torch.softmax(torch.einsum("ghd,gtd->ght", q.view(n_kv, G, hd).double(), k[:, :rows].double()) * hd ** -0.5, dim=-1)
        want = torch.einsum("ght,gtd->ghd", w, v[:, :rows].double()).reshape(n_kv * G, hd)
        assert ((out.double() - want).norm() / want.norm()).item() < 1e-6, rows


@pytest.mark.parametrize("hd,size", [(64, 8.0), (16, 4.0)])
@pytest.mark.parametrize("rows", [40, 300, 3000])
def test_attn_decode_large_scores(hd, size, rows):
    """Scores of about 100 that divide exactly by sqrt(head size): their differences are exact, so what is left is the exponential's unit and the
    sums (4e-7 of the norm); a score rounded after a scaling by log2(e) would be off by 100 * 2^-24 of its weight."""
    L, G, n_kv = api.lib(), 4, 2
    gen = torch.Generator(device="cuda")
    gen.manual_seed(hd + rows)
    step = torch.randint(0, 33, (n_kv, rows), generator=gen, device="cuda") / 8.0
    k, v = torch.zeros((n_kv, rows, hd), device="cuda"), torch.randn((n_kv, rows, hd), generator=gen, device="cuda").half()
    k[:, :, 0], k[:, :, 1] = 1.0, step
    q = torch.zeros((n_kv * G, hd), device="cuda")
    q[:, 0], q[:, 1] = 100.0 * size + torch.arange(n_kv * G, device="cuda") * size, size      # scores 100 + head + step
    k = k.half()
    work = torch.zeros(L.yalm_attn_workspace_bytes(n_kv * G, n_kv, hd), device="cuda", dtype=torch.uint8)
    out = torch.empty_like(q)
    ctl = torch.tensor([0, rows - 1, 0, rows - 1, rows, 0, 0, 0], device="cuda", dtype=torch.int32)
    p = lambda t: C.c_void_p(t.data_ptr())
    assert L.yalm_attn_decode(p(out), p(k), p(v), p(q), p(work), n_kv * G, n_kv, hd, rows, p(ctl), None) == 0
    w = torch.softmax(step.double(), dim=-1)
    want = torch.einsum("gt,gtd->gd", w, v.double()).repeat_interleave(G, 0)
    assert ((out.double() - want).norm() / want.norm()).item() < 4e-7


def test_captured_calls_replay():
    """Kernels launched chained under stream capture, behind a memset node (the entry without a workspace), each other and a copy: a replay on
    other inputs gives what the calls give one by one."""
    L, H, G, hd, n, rows = api.lib(), 32, 8, 128, 40, 900
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    rnd = lambda *s: torch.randn(s, generator=gen, device="cuda")
    k, v = rnd(G, rows, hd).half(), rnd(G, rows, hd).half()
    q, q16 = torch.empty((H, hd), device="cuda"), torch.empty((n, H, hd), device="cuda", dtype=torch.float16)
    w = (rnd(512, H * hd) * 0.02).half()
    work = torch.zeros(L.yalm_attn_workspace_bytes(H, G, hd), device="cuda", dtype=torch.uint8)
    ctl = torch.tensor([0, rows - 1, 0, rows - 1, rows, 0, 0, 0], device="cuda", dtype=torch.int32)
    outs = [torch.empty((H, hd), device="cuda"), torch.empty((H, hd), device="cuda"), torch.empty((n, H, hd), device="cuda", dtype=torch.float16),
            torch.empty((n, 512), device="cuda")]
    copy = torch.empty_like(outs[3])
    p, i = lambda t: C.c_void_p(t.data_ptr()), lambda *a: [C.c_int(x) for x in a]

    def calls():
        s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        rc = [L.yalm_attn_decode_static(p(outs[0]), p(k), p(v), p(q), *i(H, G, hd, rows), p(ctl), s),
              L.yalm_attn_decode(p(outs[1]), p(k), p(v), p(q), p(work), *i(H, G, hd, rows), p(ctl), s),
              L.yalm_attn_prefill(p(outs[2]), p(q16), p(k), p(v), *i(n, rows - n, H, G, hd, rows), s),
              L.yalm_gemm_f16(p(outs[3]), C.c_int(512), p(outs[2]), p(w), *i(n, 512, H * hd, 0), s)]
        copy.copy_(outs[3])
        rc.append(L.yalm_gemm_f16(p(outs[3]), C.c_int(512), p(outs[2]), p(w), *i(n, 512, H * hd, 1), s))
        assert rc == [0] * 5

    q.copy_(rnd(H, hd)), q16.copy_(rnd(n, H, hd))
    calls()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="thread_local"):
        calls()
    for _ in range(3):
        q.copy_(rnd(H, hd)), q16.copy_(rnd(n, H, hd))
        for o in outs:
            o.fill_(float("nan"))
        graph.replay()
        got = [o.clone() for o in outs] + [copy.clone()]
        calls()
        assert all(torch.equal(a, b) for a, b in zip(got, outs + [copy])) and got[3].isfinite().all()


@pytest.mark.parametrize("heads,kv_heads,hd", [(5, 5, 7), (3, 1, 20), (6, 2, 48), (9, 3, 64), (9, 3, 72), (12, 4, 128), (3, 1, 136)])
def test_generic_shapes(heads, kv_heads, hd):
    """Pieces of 64 values of a key and 16 rows of values, their remainders, and rows that are not 16-byte aligned.  fp32 sums of hd and kv_len terms of about 1,
    exponentials of scores of about 1: 2e-6 of the norm (measured 3e-7)."""
    L, T = api.lib(), 304
    for kv_len in (1, 15, 16, 17, 256, 257, 300):
        for off in (0, 1):
            torch.manual_seed(kv_len + hd)
            kb, vb = (torch.randn(kv_heads * T * hd + 1, device="cuda").half()[off:off + kv_heads * T * hd] for _ in range(2))
            q, out, att = torch.randn(heads * hd, device="cuda"), torch.zeros(heads * hd, device="cuda"), torch.zeros((heads, T), device="cuda")
            ptr = [C.c_void_p(t.data_ptr()) for t in (out, att, kb, vb, q)]
            assert L.yalm_attn_generic(*ptr, heads, kv_heads, hd, T, kv_len, None, None) == 0
            k, v = (t.double().view(kv_heads, T, hd)[:, :kv_len].repeat_interleave(heads // kv_heads, 0) for t in (kb, vb))
            w = torch.softmax(torch.einsum("hd,htd->ht", q.double().view(heads, hd), k) / hd ** 0.5, 1)
            want = torch.einsum("ht,htd->hd", w, v).flatten()
            assert (out.double() - want).norm() < 2e-6 * want.norm() and (att[:, :kv_len].double() - w).norm() < 2e-6 * w.norm()
