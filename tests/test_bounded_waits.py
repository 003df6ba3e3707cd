"""-m "not gpu": what the tensor-core kernels do when a bounded wait ran out (csrc/tcgen.cuh), read from their source - making one run out would take a
broken kernel.  A warp that gave up states no result as complete, and what was to be stored or carried on becomes NaN."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yalm_b200", "csrc")


def source(name):
    return open(os.path.join(CSRC, name)).read()


@pytest.mark.parametrize("name,barrier,count", [("prefill_gemm.cu", r"umma_commit_pair\(acc_full0", 1), ("prefill_gemm.cu", r"umma_commit\(acc_bar\)", 1),
                                                ("prompt_attn.cu", r"umma_commit\(o_full\)", 1)])
def test_results_are_not_complete_after_giving_up(name, barrier, count):
    lines = [line for line in source(name).split("\n") if re.search(barrier, line)]
    assert len(lines) == count and all("!dead" in line for line in lines)


def test_nan_goes_to_results_clusters_and_state():
    gemm, attn, scan = source("prefill_gemm.cu"), source("prompt_attn.cu"), source("chunk_scan.cuh")
    for send in re.finditer(r"st_cluster4\((dst|slot\(buf)", gemm):              # sums for another CTA of the cluster
        assert "if (dead)" in gemm[send.start() - 260: send.start()]
    assert attn.index("if (dead) l =") < attn.index("st.shared::cluster.v2.f32")   # a row's sum: in the result of every part
    assert "if (dead)" in scan[: scan.index("store_pairs<NP>(state")].rsplit("for (int j = 0; j < 4; ++j)", 1)[1]


@pytest.mark.parametrize("name", ["stream_rows.cuh", "decode_token.cuh"])
def test_streams_of_weights(name):
    """A warp that gave up gives no stage back (the stream would fill it again under a copy on its way), its sums are NaN, and the
    warps that issue copies wait for them before they leave."""
    text = source(name)
    back = [line for line in text.split("\n") if re.search(r"mbar_arrive\(empty0", line)]
    assert len(back) == 1 and "!dead" in back[0]
    sums = [line for line in text.split("\n") if re.search(r"\b(part|sums)\[c \* kCap", line)]
    assert sums and all("dead ? NaN" in line for line in sums)
    stream = text[text.index("---- the stream ----" if name == "stream_rows.cuh" else "=== the stream ==="):]
    stream = stream[: stream.index("---- this warp's chunks" if name == "stream_rows.cuh" else "=== the other warps")]
    assert stream.index("return;", stream.rindex(", late)")) and stream.rindex("(full0") > stream.rindex("bulk_")


def test_waits_are_used():
    text = "".join(source(n) for n in ("prefill_gemm.cu", "prompt_attn.cu", "chunk_scan.cuh"))
    for name in re.findall(r"void (mbar_wait\w*)\(", source("tcgen.cuh")):
        assert re.search(r"\b%s\(" % name, text), name


def test_joins_of_the_token_kernels_attention():
    """A sum that gave up is NaN in the join; and the weights of the joins (not of the positions) are expf, as in the kernel of decode_mega.cuh."""
    text = source("decode_token.cuh")
    assert "if (dead) lsum = NaN;" in text and "= dead ? NaN : ls" in text
    joins = text[text.index("the warps' records in order"): text.index("// ---- a product")]
    assert joins.count("expf(") == 2 and "__expf" not in joins


def test_rescaling_warps_wait_for_every_round():
    """A parity tells neighbouring rounds of a barrier apart and no more: a warp that leaves out round 0 of the scores would find the parity of round 1 while round 0 is
    still open."""
    text = source("prompt_attn.cu")
    rescale = text[text.index("---- rescaling:"): text.index("---- softmax: one row per thread")]
    assert rescale.count("wait(s_full0 + 8 * t, (uint32_t)round & 1u)") == 1
    assert rescale.index("wait(s_full0") < rescale.index("if (round > 0)") < rescale.index("wait(f_full0")
