"""-m gpu: the whole-token kernel of dense models on one GPU (csrc/decode_token.cuh) at the edges of its geometry - rows of one 512-byte chunk to four
pieces, ragged last chunks, several rows a stage, stages that q, k and v share, one row of x for most CTAs, contexts shorter and longer than the CTAs of a head - against the
oracle's tokens and logits; and on either side of its limits, which kernel runs."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import LOGIT_TOL
from yalm_b200 import api
from yalm_b200 import yalm_file as yf

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def arch(dim, hidden, hd, heads, kv, vocab=600, layers=2, seq=256, **kw):
    return yf.Arch(dim, hidden, hd, layers, heads, kv, vocab, seq, 10000.0, name="token", **kw)


def runs_here(m):
    """Whether a token of this model is decode_token_kernel: it keeps no input vector in shared memory."""
    return m.uses_megakernel() and m.mega_info()["vec_floats"] == 0


# model, weights, whether a token runs here or, where that is faster, on decode_mega_kernel
CASES = {
    # dim: one chunk, 16 rows a stage that straddle q | k | v; hidden: 3 chunks, the last ragged
    "fp16-one-chunk": (arch(256, 640, 32, 8, 4), "fp16", False),
    "fp16-one-chunk-heads-of-64": (arch(256, 640, 64, 4, 1), "fp16", True),
    "fp32-two-chunks": (arch(256, 640, 32, 8, 4), "fp32", True),
    # dim: 5 chunks (one row each for 5 of 8 warps); hidden: 11 chunks, half of one empty; gelu, clip
    "fp16-odd-chunks": (arch(1280, 2752, 32, 8, 2, act_type="gelu", qkv_clip=0.5), "fp16", True),
    # hidden: 3 pieces, two of 15 chunks and one of 13
    "fp16-three-pieces": (arch(1024, 11008, 64, 8, 2), "fp16", True),
    # dim: two pieces under a norm (20 chunks), hidden: four full ones; 8 query heads a KV head
    "fp16-two-pieces-normed": (arch(5120, 16384, 128, 40, 5, layers=1, vocab=200), "fp16", False),
    # dim: 16 chunks, the longest normed row
    "fp16-sixteen-chunks": (arch(4096, 16384, 128, 32, 4, layers=1, vocab=200), "fp16", True),
    # fp32: 16 chunks of dim (two of a warp), 4 pieces of hidden
    "fp32": (arch(2048, 8192, 128, 8, 2, vocab=100, layers=1), "fp32", True),
    # fp8: rows of 2 chunks with scales, hidden 19 chunks in two pieces
    "fp8": (arch(1024, 9728, 64, 16, 4), "fp8", False),
    "fp8-heads-of-128": (arch(1024, 9728, 128, 8, 2), "fp8", True),
    # fp8: 3 chunks, the fewest with shorter heads, and 8, the most
    "fp8-three-chunks": (arch(1536, 3072, 64, 8, 2), "fp8", True),
    "fp8-eight-chunks": (arch(4096, 512, 128, 8, 1, layers=1, vocab=200), "fp8", True),
    # a row or two of x and none of hidden or of the vocabulary for some CTAs
    "fp16-few-rows": (arch(160, 96, 64, 4, 1, vocab=50), "fp16", True),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_tokens_and_logits(oracle, case):
    a, dt, here = CASES[case]
    img = bytes(yf.random_model(a, dt, seed=5))
    prompt, n = [1, 5, 9, 20, 7], 24 if a.dim <= 1280 else 6
    ref = bytes(yf.dequantized_fp32_image(img)) if dt == "fp8" else img
    to, lo = oracle.OracleModel(ref).generate(prompt, n, keep_logits=True)
    m = api.Model(img).cuda()
    assert m.uses_megakernel() and runs_here(m) == here
    s = api.InferenceState(m)
    tg, lg = s.generate(prompt, n, keep_logits=True)
    assert np.abs(lg - lo).max() < LOGIT_TOL and tg == to
    for pos, tok in enumerate(prompt[:-1]):
        s.forward(tok, pos, api.MODE_HYDRATE)
    assert s.generate_greedy(prompt[-1], len(prompt) - 1, n) == to  # arg-max and position on the device
    s.close()
    m.close()


@pytest.mark.parametrize("context", [1, 2, 63, 64, 65, 300])
def test_contexts_around_the_units_of_attention(oracle, context):
    """One position; the stages' edges at 32 channels (64 positions), half of a stage empty; every CTA of a head with units of its own."""
    a = arch(512, 512, 32, 8, 2, vocab=300, layers=1, seq=512)
    img = bytes(yf.random_model(a, "fp16", seed=6))
    ids = [(37 * i + 1) % 300 for i in range(context)]
    to, lo = oracle.OracleModel(img).generate(ids, 3, keep_logits=True)
    m = api.Model(img).cuda()
    assert runs_here(m)
    s = api.InferenceState(m)
    tg, lg = s.generate(ids, 3, keep_logits=True)
    assert np.abs(lg - lo).max() < LOGIT_TOL and tg == to
    s.close()
    m.close()


@pytest.mark.parametrize("dim,hidden,layers", [(512, 20480, 1), (512, 16640, 1), (4608, 512, 1), (64, 96, 2)])
def test_rows_beyond_it_stay_with_the_other_kernel(oracle, dim, hidden, layers):
    """A hidden size of five pieces, and the least that is one; a normed row past the longest; fewer rows of x than CTAs."""
    heads, hd, kv = (2, 32, 1) if dim < 512 else (8, 64, 2)
    a = arch(dim, hidden, hd, heads, kv, layers=layers, vocab=100)
    img = bytes(yf.random_model(a, "fp16", seed=7))
    to, lo = oracle.OracleModel(img).generate([1, 2, 3], 4, keep_logits=True)
    m = api.Model(img).cuda()
    assert m.uses_megakernel() and not runs_here(m)
    s = api.InferenceState(m)
    tg, lg = s.generate([1, 2, 3], 4, keep_logits=True)
    assert np.abs(lg - lo).max() < LOGIT_TOL and tg == to
    s.close()
    m.close()


@pytest.mark.parametrize("name", ["W2_PIPE", "MMA", "STAGES", "DEBUG", "L2_AHEAD", "TUNE", "TRACE"])
def test_settings_of_the_other_kernel_select_it(name, monkeypatch):
    img = bytes(yf.random_model(arch(512, 512, 64, 8, 2, vocab=100, layers=1), "fp16", seed=8))
    for value, here in ((None, True), ("0", False)):
        if value is not None:
            monkeypatch.setenv("YALM_MEGA_" + name, value)
        m = api.Model(img).cuda()
        assert m.uses_megakernel() and runs_here(m) == here
        m.close()


RECORD = """
import ctypes as C, sys
from yalm_b200 import api
from yalm_b200 import yalm_file as yf
m = api.Model(bytes(yf.random_model(yf.Arch(512, 512, 64, 1, 8, 2, 100, 64, 10000.0, name="token"), "fp16", seed=3))).cuda()
assert m.uses_megakernel() and m.mega_info()["vec_floats"] == 0
s = api.InferenceState(m)
s.forward(1, 0)
f = api.lib().yalm_mega_fault_record
f.restype = C.POINTER(C.c_uint)
record = f()
assert record[0] == 0
s.forward(2, 1, api.MODE_HYDRATE)
record[0], record[1], record[2] = 11, 7, 32     # as the kernel leaves it
print("before", flush=True)
s.forward(3, 2) if sys.argv[1] == "forward" else s.generate_greedy(3, 2, 4) if sys.argv[1] == "greedy" else s.mega_profile(3, 2) if sys.argv[1] == "profile" else s.forward_batch([3, 4, 5], 2)
print("after", flush=True)
"""


@pytest.mark.parametrize("call", ["forward", "greedy", "profile", "portion"])
def test_a_recorded_timeout_fails_the_call(call):
    """The record is written by the host, no kernel waits: the call that synchronises next reports it and ends the process, as a CUDA error does."""
    r = subprocess.run([sys.executable, "-c", RECORD, call], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert "before" in r.stdout and "after" not in r.stdout and r.returncode != 0
    assert "decode_token_kernel timed out" in r.stderr and "CTA 7 thread 32" in r.stderr
