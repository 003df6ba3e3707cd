"""-m gpu: batched prefill / perplexity — the tcgen05 GEMM against numpy, and Model::forward_batch
against its oracle, the reference's token loop (src/main.cpp:91-97, 174-184): same per-position next-token probabilities,
same last-position logits (max |delta| <= 2e-2), same KV rows (fp16, +-1 ulp: the GEMM sums in a
different order), same greedy continuation, perplexity equal to 1e-3 relative."""
import math

import numpy as np
import pytest

from conftest import LOGIT_TOL, golden_case
from yalm_b200 import api
from yalm_b200 import yalm_file as yf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (1, 8, 8), (200, 320, 512), (512, 1024, 4096), (130, 64, 256), (384, 4096, 1024)])
def test_gemm_f16_tcgen05_matches_numpy(M, N, K):
    rng = np.random.default_rng(M * 7 + N)
    a = (rng.standard_normal((M, K)) / np.sqrt(K)).astype(np.float16)
    w = rng.standard_normal((N, K)).astype(np.float16)
    want = a.astype(np.float32) @ w.astype(np.float32).T
    got = api.gemm_cuda(a, w)
    np.testing.assert_allclose(got, want, atol=2e-3, rtol=1e-3)
    c0 = rng.standard_normal((M, N)).astype(np.float32)
    np.testing.assert_allclose(api.gemm_cuda(a, w, c=c0), want + c0, atol=2e-3, rtol=1e-3)     # residual tail: c += a w^T


@pytest.mark.parametrize("act", [api.ACT_SILU, api.ACT_GELU])
@pytest.mark.parametrize("M,N,K", [(128, 128, 256), (77, 520, 512), (256, 1792, 1024)])
def test_gemm_glu_tcgen05_matches_numpy(M, N, K, act):
    rng = np.random.default_rng(N + K)
    a = (rng.standard_normal((M, K)) / np.sqrt(K)).astype(np.float16)
    w1, w3 = rng.standard_normal((N, K)).astype(np.float16), rng.standard_normal((N, K)).astype(np.float16)
    g = a.astype(np.float32) @ w1.astype(np.float32).T
    u = a.astype(np.float32) @ w3.astype(np.float32).T
    if act == api.ACT_SILU:
        want = g / (1.0 + np.exp(-g)) * u
    else:
        want = 0.5 * g * (1.0 + np.tanh(0.797885 * (g + 0.044715 * g ** 3))) * u
    got = api.gemm_cuda(a, w1, w3=w3, act=act).astype(np.float32)
    np.testing.assert_allclose(got, want, atol=3e-3, rtol=2e-3)


def _oracle_walk(oracle, img, ids, context=0):
    """The token loop: per-position probability of the next token, the last logits."""
    om = oracle.OracleModel(img, context)
    probs = []
    for pos in range(len(ids) - 1):
        lg = om.forward(ids[pos], pos, 1)
        probs.append(oracle.sample_prob(lg, ids[pos + 1]))
    last = om.forward(ids[-1], len(ids) - 1, 1).copy()
    return om, np.array(probs), last


@pytest.mark.parametrize("name,chunks", [("tiny-fp16", [41]), ("tiny-fp16", [17, 24]), ("tiny-kv8-fp16", [30, 11]), ("tiny-gelu-clip-fp16", [41])])
def test_forward_batch_matches_token_loop(oracle, name, chunks):
    fx, img = golden_case(name)
    n = sum(chunks)
    ids = [1] + [(i * 37 + 11) % 500 + 3 for i in range(n - 1)]
    om, want_p, want_last = _oracle_walk(oracle, img, ids)
    m = api.Model(img).cuda()
    assert m.batch_capacity() >= max(chunks)
    s = api.InferenceState(m)
    got_p, pos = [], 0
    for c in chunks:
        tg = ids[pos + 1: pos + c + 1] + [0] * (pos + c + 1 - len(ids))        # the very last position has no target
        got_p += s.forward_batch(ids[pos: pos + c], pos, tg).tolist()
        pos += c
    got_p = np.array(got_p[:-1])
    np.testing.assert_allclose(got_p, want_p, rtol=2e-2, atol=1e-6)
    ok = want_p > 1e-30            # a random-init model can put a target below fp32's range: no log-probability there
    if ok.sum() >= 8:
        ppl = lambda p: math.exp(-np.log(p[ok].astype(np.float64)).mean())
        assert abs(ppl(got_p) - ppl(want_p)) / ppl(want_p) < 1e-3
    assert np.abs(s.logits() - want_last).max() < LOGIT_TOL
    # the KV rows the chunk appended == the rows the decode path appends (fp16; the GEMM sums in another order: <= 2 ulp)
    L, H, D, T = m.n_layers, m.n_kv_heads, m.head_dim, m.max_seq_len
    for layer in range(L):
        for which in (4, 5):
            pre = s.read(which, n * H * D, np.uint16, layer).view(np.float16).astype(np.float32)
            ref = (om.kc if which == 4 else om.vc)[layer][:n].reshape(-1).view(np.float16).astype(np.float32)
            assert np.abs(pre - ref).max() <= 4e-3 * max(1.0, np.abs(ref).max())
    # decode continues from the prefilled cache: same greedy tokens as the oracle continuing its loop
    want_t = []
    lg = want_last
    for i in range(12):
        t = int(np.argmax(lg))
        want_t.append(t)
        lg = om.forward(t, n + i, 1)
    first = int(np.argmax(s.logits()))
    assert first == want_t[0]
    assert s.generate_greedy(first, n, 11) == want_t[1:]
    s.close()
    m.close()


def test_forward_batch_head_dim_128_long_prompt(oracle):
    """Mistral attention geometry, 600-token prompt = one full 512 chunk + a ragged one; the later chunk attends over the
    rows the first one appended."""
    arch = yf.Arch(1024, 2048, 128, 2, 8, 2, 512, 4096, 1000000.0, name="prefill-hd128")
    img = bytes(yf.random_model(arch, "fp16", seed=6))
    ids = [1] + [(i * 131 + 7) % 509 + 3 for i in range(599)]
    om, want_p, want_last = _oracle_walk(oracle, img, ids)
    m = api.Model(img).cuda()
    s = api.InferenceState(m)
    cap = m.batch_capacity()
    got_p, pos = [], 0
    while pos < len(ids):
        c = min(cap, len(ids) - pos)
        tg = ids[pos + 1: pos + c + 1] + [0] * (pos + c + 1 - len(ids))
        got_p += s.forward_batch(ids[pos: pos + c], pos, tg).tolist()
        pos += c
    got_p = np.array(got_p[:-1])
    ppl = lambda p: math.exp(-np.log(p.astype(np.float64)).mean())
    assert abs(ppl(got_p) - ppl(want_p)) / ppl(want_p) < 1e-3
    np.testing.assert_allclose(got_p, want_p, rtol=3e-2, atol=1e-6)
    assert np.abs(s.logits() - want_last).max() < LOGIT_TOL
    s.close()
    m.close()


def test_forward_batch_refuses_what_it_cannot_do():
    _, moe = golden_case("tiny-moe-fp16")
    m = api.Model(moe).cuda()
    assert m.batch_capacity() == 0                 # MoE: the caller walks the tokens
    s = api.InferenceState(m)
    with pytest.raises(api.YalmError):
        s.forward_batch([1, 2, 3], 0)
    s.close()
    m.close()
    fx, img = golden_case("tiny-fp16")
    m = api.Model(img).cuda()
    s = api.InferenceState(m)
    with pytest.raises(api.YalmError):             # would wrap the 64-row ring
        s.forward_batch(list(range(3, 43)), 30)
    s.close()
    m.close()


@pytest.mark.parametrize("hd,heads,kv,dim,rotary,clip,vocab,n,pos0", [
    (32, 8, 8, 256, 32, None, 1000, 129, 0), (64, 8, 2, 512, 32, 0.5, 516, 300, 40), (128, 8, 2, 1024, 128, None, 3000, 512, 7), (128, 4, 4, 1024, 64, 0.7, 132, 511, 1),
    (64, 4, 1, 1024, 64, None, 20000, 260, 100),
    # K in two parts (dim 2048 and more, few columns), a last half tile that is empty, or has some rows
    (64, 4, 1, 2048, 64, None, 516, 260, 40), (64, 4, 1, 2048, 32, 0.5, 516, 511, 3), (128, 4, 2, 4096, 64, 0.7, 132, 300, 5), (32, 8, 8, 4096, 32, None, 516, 129, 0)])
def test_forward_batch_of_many_rows_matches_few(hd, heads, kv, dim, rotary, clip, vocab, n, pos0):
    """A portion of more than 128 rows, whose products rotate, append and score in their own kernels, against the same positions in portions of 100, which
    leave that to kernels of their own: keys and values in fp16 to a unit (2^-10) or the layer's rounding, probabilities to what a unit in 16-bit operands makes of
    them (as against the token loop: 2e-2).  One key part and several, part of a head rotated, clipped values, ragged vocabularies and portions."""
    arch = yf.Arch(dim, 512, hd, 2, heads, kv, vocab, 1024, 10000.0, rotary_dim=rotary, qkv_clip=clip, name="many-rows")
    img = bytes(yf.random_model(arch, "fp16", seed=hd + n))
    m = api.Model(img).cuda()
    ids = [1] + [(i * 131 + 7) % (vocab - 3) + 3 for i in range(pos0 + n)]
    outs = []
    for most in (n, 100):
        s = api.InferenceState(m)
        probs, pos = [], 0
        while pos < pos0 + n:
            c = min(100, pos0 - pos) if pos < pos0 else min(most, pos0 + n - pos)
            probs += s.forward_batch(ids[pos: pos + c], pos, ids[pos + 1: pos + c + 1]).tolist()
            pos += c
        rows = [s.read(which, (pos0 + n) * kv * hd, np.uint16, layer).view(np.float16).astype(np.float32) for layer in range(2) for which in (4, 5)]
        outs.append((np.array(probs), rows, s.logits().copy()))
        s.close()
    (p0, r0, l0), (p1, r1, l1) = outs
    np.testing.assert_allclose(p0, p1, rtol=2e-2, atol=1e-7)
    for layer, (a, b) in enumerate(zip(r0, r1)):
        assert np.abs(a - b).max() <= (2e-3 if layer < 2 else 6e-3) * max(1.0, np.abs(b).max())
    assert np.abs(l0 - l1).max() < LOGIT_TOL
    m.close()


@pytest.mark.parametrize("n,vocab", [(129, 132), (256, 1000), (300, 20004), (511, 516), (512, 20000), (100, 20004)])
@pytest.mark.parametrize("infinite", [False, True])
def test_target_probabilities_against_64_bits(n, vocab, infinite):
    """The probability of every row's target, of vocabularies that end anywhere in a tile of columns, with targets in the first and last columns and out of range (0).
    A layer that adds nothing leaves the embedding, so the head's fp16 operand is known but for roundings of its last bit: some 2e-4 in a logit of size 1 each, and the
    products' sums 3e-5: 1e-3 of a probability.  All columns count alike: without a tile of 64 of 20000 every probability is off by 3e-3.  infinite: columns of -infinity, the
    first 40, tiles as a whole and the last 8, count as nothing."""
    dim = 256
    arch = yf.Arch(dim, 512, 32, 1, 8, 2, vocab, 1024, 10000.0, name="score")
    tensors, hints = {}, {}
    for name, arr, st in yf.random_tensors(arch, "fp16", seed=n + vocab, lm_scale=1.0):
        if ".wo." in name or ".w2." in name:
            arr = np.zeros_like(arr)
        tensors[name], hints[name] = arr, st
    embed, norm, head = (tensors["model.%s.weight" % x] for x in ("embed", "norm", "output"))
    gone = np.zeros(vocab, bool)
    if infinite:
        embed[:, 0] = 1.0                                    # (times a positive weight: -infinity, not a sum of both signs or NaN)
        norm[0] = 1.0
        gone[512:1024] = vocab > 2000
        gone[:40] = gone[-8:] = True
        head[gone, 0] = -np.inf
    m = api.Model(bytes(yf.build_image(tensors, yf.metadata_of(arch, "fp16"), hints))).cuda()
    s = api.InferenceState(m)
    rng = np.random.default_rng(n)
    ids, targets = rng.integers(3, vocab, n).tolist(), rng.integers(0, vocab, n)
    targets[:6] = [0, vocab - 1, vocab // 2, -1, vocab, vocab - 4]
    got = np.array(s.forward_batch(ids, 0, targets.tolist()))
    x = embed[ids].astype(np.float32)
    a = (x / np.sqrt((x.astype(np.float64) ** 2).mean(1, keepdims=True) + arch.norm_eps) * norm).astype(np.float32).astype(np.float16)
    logits = a.astype(np.float64) @ np.where(gone[:, None], 0, head).astype(np.float64).T
    logits[:, gone] = -np.inf
    e = np.exp(logits - logits.max(1, keepdims=True))
    known = (targets >= 0) & (targets < vocab)
    want = np.where(known, e[np.arange(n), np.where(known, targets, 0)] / e.sum(1), 0.0)
    np.testing.assert_allclose(got, want, rtol=1e-3, atol=0)
    s.close()
    m.close()


def test_portion_keeps_no_space_for_what_it_does_not_store():
    """fp32 logits are stored of up to 128 rows: 66 MB of 128256 columns, not the 263 MB of 512 rows.  Other space is under 10 MB here."""
    import torch
    used = []
    for vocab in (512, 128256):                             # (the first loads the kernels)
        arch = yf.Arch(256, 512, 32, 1, 8, 2, vocab, 1024, 10000.0, tied=True, name="space")
        m = api.Model(bytes(yf.random_model(arch, "fp16", seed=1))).cuda()
        s = api.InferenceState(m)
        free = torch.cuda.mem_get_info()[0]
        for n in (40, 130):
            assert np.isfinite(s.forward_batch([3] * n, 0, [4] * n)).all()
        used.append(free - torch.cuda.mem_get_info()[0])
        s.close()
        m.close()
    assert used[1] < 100e6
