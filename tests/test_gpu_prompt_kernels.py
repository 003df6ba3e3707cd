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


def attend(q, k, v, seen, scale, sink=None):
    """q (n, H, dk), k (G, T, dk), v (Gv, T, dv), seen (n, T); 64 bits, head by head."""
    H, G = q.shape[1], k.shape[0]
    out = []
    for h in range(H):
        g = h // (H // G)
        s = (q[:, h].double() @ k[g].double().T * scale).masked_fill(~seen, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[h].double().expand(len(s), 1)], dim=1)
        p = torch.softmax(s, dim=-1)[:, :k.shape[1]]
        out.append(p @ v[g % v.shape[0]].double())
    return torch.stack(out, dim=1)


@pytest.mark.parametrize("hd", [128, 64, 32])
@pytest.mark.parametrize("n,pos0,H,G", [(1, 0, 4, 1), (2, 127, 8, 8), (7, 397, 32, 8), (129, 0, 8, 8), (33, 5000, 8, 8), (300, 77, 64, 8), (512, 511, 12, 2), (512, 0, 32, 8),
                                        (260, 3000, 3, 1), (33, 1100, 4, 2)])
def test_causal_attention_tiles(n, pos0, H, G, hd):
    """Rows that fill a tile in part, both tiles, several CTAs; one key tile to many, in one part and in several; 3 query heads per
    kv head.  Slots past the portion hold NaN.  P is rounded to fp16 (2^-11) and so is the result: 5e-4 of the norm."""
    ring = pos0 + n + 3
    q = normal(n, (n, H, hd), dtype=torch.float16)
    k, v = (normal(s + pos0, (G, ring, hd), dtype=torch.float16) for s in (1, 2))
    k[:, pos0 + n:], v[:, pos0 + n:] = float("nan"), float("nan")
    store = torch.full((n * H * hd + 8,), 7.0, device="cuda", dtype=torch.float16)
    for shift in (0, 2):                                           # 16-byte aligned rows, and rows that are not
        out = store[shift: shift + n * H * hd]
        assert L().yalm_attn_prefill(ptr(out), ptr(q), ptr(k), ptr(v), *i32(n, pos0, H, G, hd, ring), None) == 0
        i = torch.arange(n, device="cuda")[:, None] + pos0
        seen = torch.arange(pos0 + n, device="cuda")[None] <= i
        assert rel(out.view(n, H, hd), attend(q, k[:, :pos0 + n], v[:, :pos0 + n], seen, hd ** -0.5)) < 5e-4
        assert (store[shift + n * H * hd:] == 7.0).all()


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("n,pos0,H,G", [(5, 100, 8, 2), (5, 128, 8, 2), (5, 381, 8, 2), (5, 400, 8, 2), (5, 515, 8, 2), (5, 1020, 8, 2), (5, 1030, 8, 2),  # 1, 2, 4, 5, 8, 9 key tiles
                                        (512, 0, 37, 37), (512, 0, 38, 38), (511, 70, 38, 38), (505, 0, 32, 8), (100, 0, 75, 75), (509, 0, 152, 19), (160, 4000, 64, 8), (150, 3900, 64, 8), (300, 4200, 64, 8), (16, 300, 128, 1), (3, 300, 256, 1), (40, 200, 20, 4)])
def test_causal_attention_single_tiles_and_pairs(n, pos0, H, G, hd):
    """Key tiles that leave the odd group of softmax warps none or one less, and both sides of the lines for cluster parts; as many row tiles as SMs
    (148 of them: one a CTA) and more (two a CTA); groups of query heads that fill a tile, exceed it or do not divide it; ragged last tiles of results that leave as boxes; enough key tiles for
    warps that rescale, and one less.  Bound as above."""
    T = pos0 + n
    q, k, v = normal(n, (n, H, hd), dtype=torch.float16), normal(1, (G, T, hd), dtype=torch.float16), normal(2, (G, T, hd), dtype=torch.float16)
    k[:, T // 2] *= 4                    # (accumulators are rescaled late, too)
    k[:, 3 * T // 4] *= 8
    out = torch.full((n + 200, H, hd), 7.0, device="cuda", dtype=torch.float16)
    assert L().yalm_attn_prefill(ptr(out), ptr(q), ptr(k), ptr(v), *i32(n, pos0, H, G, hd, T), None) == 0
    seen = torch.arange(T, device="cuda")[None] <= torch.arange(n, device="cuda")[:, None] + pos0
    assert rel(out[:n], attend(q, k, v, seen, hd ** -0.5)) < 5e-4
    assert (out[n:] == 7.0).all()


def test_causal_attention_far_maxima():
    """A row's largest score in its last tiles, 2^40 above the first: the accumulator is rescaled, in every part."""
    n, pos0, H, G, hd = 40, 1500, 8, 2, 128
    q, k, v = normal(1, (n, H, hd), dtype=torch.float16), normal(2, (G, pos0 + n, hd), dtype=torch.float16), normal(3, (G, pos0 + n, hd), dtype=torch.float16)
    for at, size in ((100, 1.0), (700, 2.0), (1400, 3.0), (1500, 4.0)):
        k[:, at] = q[0].view(G, H // G, hd)[:, 0] * size
    out = torch.empty((n, H, hd), device="cuda", dtype=torch.float16)
    assert L().yalm_attn_prefill(ptr(out), ptr(q), ptr(k), ptr(v), *i32(n, pos0, H, G, hd, pos0 + n), None) == 0
    seen = torch.arange(pos0 + n, device="cuda")[None] <= torch.arange(n, device="cuda")[:, None] + pos0
    assert rel(out, attend(q, k, v, seen, hd ** -0.5)) < 5e-4


@pytest.mark.parametrize("bf16", [0, 1])
@pytest.mark.parametrize("n,pos0,H,G,hd", [(40, 200, 8, 2, 128), (60, 1500, 8, 8, 64), (200, 700, 32, 8, 128), (33, 4000, 4, 4, 128)])
def test_attention_rows_of_one_late_key(n, pos0, H, G, hd, bf16):
    """Every row is dominated by one key near its end, whose score lies 2^7.3 .. 2^7.97 above those of a key in 64 before it and far above all
    others.  The weight of a row's largest score is 1 and takes no rounding, so with one value row for all keys the result is that row: to
    the last bit in fp16, and in the fp32 rows over bf16 weights to what the rounding (2^-9) of the at most two weights of 2^-7.3 in its own
    tile and of the sums adds (4e-5)."""
    T, late = pos0 + n, pos0 - 3
    dt = torch.bfloat16 if bf16 else torch.float16
    grow = (1 + torch.arange(n * H, device="cuda").remainder(13) / 128.0).view(n, H)           # exact in both types, as are the keys
    q, k = torch.zeros((n, H, hd), device="cuda"), torch.zeros((G, T, hd), device="cuda")
    to_log2 = 1.0 if bf16 else hd ** 0.5 * 0.6931471805599453                                # score in powers of two = q . k / to_log2
    q[:, :, 0], q[:, :, 1] = grow, 1.0
    k[:, :, 1] = -40.0 * to_log2                                                               # all others
    k[:, 5:late:64, 1] = 0.0
    k[:, late, 0], k[:, late, 1] = 7.3125 * to_log2, 0.0
    k, v = k.to(dt), normal(hd, (G, 1, hd), dtype=dt).expand(G, T, hd).contiguous()
    want = v[:, 0].repeat_interleave(H // G, 0).float().expand(n, H, hd)
    if bf16:
        out = torch.empty((n, H, hd), device="cuda")
        assert L().yalm_attn_window_pool_mma(ptr(out), C.c_int(H * hd), ptr(q), C.c_int(H * hd), ptr(k), ptr(v), None, None, *i32(n, H, G, hd, hd, T, 0, 0, 0),
                                             C.c_float(0.6931471805599453), C.c_int(pos0), None, None) == 0
        assert ((out - want).abs() <= 4e-5 * want.abs()).all()
    else:
        out = torch.empty((n, H, hd), device="cuda", dtype=dt)
        assert L().yalm_attn_prefill(ptr(out), ptr(q.to(dt)), ptr(k), ptr(v), *i32(n, pos0, H, G, hd, T), None) == 0
        assert torch.equal(out.float(), want)


@pytest.mark.parametrize("bf16", [0, 1])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("n,pos0,at", [(20, 4000, 3900), (20, 4000, 5), (40, 2000, 1100), (512, 0, 300)])
def test_attention_not_finite_in_one_part(n, pos0, at, bad, bf16):
    """A key of one kv head that is not a number, or infinite, in any part of the keys: the rows of its query heads that see it are NaN (an
    infinite score takes itself away), and no others."""
    H, G, hd, T, dt = 8, 4, 128, pos0 + n, torch.bfloat16 if bf16 else torch.float16
    q = normal(n, (n, H, hd), dtype=dt)
    k, v = normal(1, (G, T, hd), dtype=dt), normal(2, (G, T, hd), dtype=dt)
    q[:, :, 0], k[1, at] = 1.0, 0.0                    # (scores of the key: + infinity or NaN, not a sum of both signs)
    k[1, at, 0] = bad
    if bf16:
        out = torch.empty((n, H, hd), device="cuda")
        assert L().yalm_attn_window_pool_mma(ptr(out), C.c_int(H * hd), ptr(q.float()), C.c_int(H * hd), ptr(k), ptr(v), None, None,
                                             *i32(n, H, G, hd, hd, T, 0, 0, 0), C.c_float(hd ** -0.5), C.c_int(pos0), None, None) == 0
    else:
        out = torch.empty((n, H, hd), device="cuda", dtype=dt)
        assert L().yalm_attn_prefill(ptr(out), ptr(q), ptr(k), ptr(v), *i32(n, pos0, H, G, hd, T), None) == 0
    hit = torch.zeros((n, H), dtype=torch.bool, device="cuda")
    hit[max(0, at - pos0):, 2:4] = True
    assert out[hit].isnan().all() and out[~hit].isfinite().all()


@pytest.mark.parametrize("dk,dv", [(128, 128), (64, 64), (64, 128), (128, 64), (64, 32), (128, 32)])
@pytest.mark.parametrize("n,pos0,H,G,Gv,window,pool,ring", [
    (32, 0, 8, 2, 2, 128, 64, 640), (512, 3584, 16, 4, 4, 1024, 64, 1536), (100, 777, 8, 2, 1, 500, 64, 1012), (257, 5000, 8, 8, 4, 300, 1, 557),
    (300, 4000, 8, 2, 2, 128, 8, 700), (40, 9000, 16, 4, 4, 130, 16, 170), (64, 300, 6, 2, 2, 0, 0, 400), (90, 1000, 4, 4, 4, 200, 0, 289),
    (33, 2000, 8, 2, 2, 1500, 64, 2100),
    # a tile a CTA while these all run at once, two a CTA beyond: 80, 148, 152 (kv heads of a tile and a half each), 200, 256 tiles of 128 rows
    (300, 600, 32, 8, 8, 128, 64, 640), (460, 0, 37, 37, 37, 200, 0, 500), (190, 333, 76, 76, 19, 300, 64, 900), (513, 100, 40, 40, 40, 130, 16, 700), (512, 700, 64, 8, 8, 300, 64, 1000)])
def test_window_attention_tiles(n, pos0, H, G, Gv, window, pool, ring, dk, dv):
    """Windows that wrap in the ring, rings that are no multiple of a tile, keys in as many parts as there are, pooled blocks in one tile and in many (as blocks of one
    position too), value heads that several key heads share, sinks, a scale of either sign, positions from a control block.  Slots that
    hold no position are NaN.  Queries, pooled means and weights are rounded to bf16 (2^-9): 4e-3 of the norm."""
    q = normal(n, (n, H, dk))
    first = max(0, pos0 - window + 1) if window else 0
    j = torch.arange(first, pos0 + n, device="cuda")
    k, v = torch.full((G, ring, dk), float("nan"), device="cuda").bfloat16(), torch.full((Gv, ring, dv), float("nan"), device="cuda").bfloat16()
    k[:, j % ring], v[:, j % ring] = normal(3, (G, len(j), dk), dtype=torch.bfloat16), normal(4, (Gv, len(j), dv), dtype=torch.bfloat16)
    blocks = max(1, (pos0 + n) // pool) if pool else 0
    kp, vp = (normal(5, (G, blocks, dk), pool ** -0.5), normal(6, (Gv, blocks, dv), pool ** -0.5)) if pool else (None, None)
    sink = normal(7, (H,)) if pos0 % 2 == 0 else None
    i = torch.arange(n, device="cuda")[:, None] + pos0
    seen = (j[None] <= i) & ((i - j[None] < window) if window else True)
    keys, values = k[:, j % ring].float(), v[:, j % ring].float()
    if pool:
        keys, values = torch.cat([keys, kp], dim=1), torch.cat([values, vp], dim=1)
        seen = torch.cat([seen, torch.arange(blocks, device="cuda")[None] * pool + pool - 1 <= i - window], dim=1)
    ctl = torch.tensor([0, pos0, 0, 0, 0, 0, 0, 0], device="cuda", dtype=torch.int32)
    for scale, use_ctl, pad in ((dk ** -0.5, False, 0), (-0.05, True, 2)):
        ldo = H * dv + pad
        out = torch.full((n, ldo), 7.0, device="cuda")
        assert L().yalm_attn_window_pool_mma_sink(ptr(out), C.c_int(ldo), ptr(q), C.c_int(H * dk), ptr(k), ptr(v), ptr(kp), ptr(vp),
                                                  *i32(n, H, G, dk, dv, ring, blocks, window, pool), C.c_float(scale), C.c_int(-1 if use_ctl else pos0),
                                                  ptr(ctl if use_ctl else None), ptr(sink), C.c_int(Gv), None) == 0
        assert rel(out[:, :H * dv].reshape(n, H, dv), attend(q, keys, values, seen, scale, sink)) < 4e-3
        assert (out[:, H * dv:] == 7.0).all()
