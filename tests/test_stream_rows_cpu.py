"""-m "not gpu": which one-row products are streams of weights (csrc/stream_rows.cuh) and which run on the row kernels (csrc/ops_gemv.cu), and what the stream
asks of L2."""
import os
import re

import pytest

from yalm_b200 import api

BARE, RESIDUAL, GLU, SCALED = range(4)


@pytest.mark.parametrize("product,dtype,d,n,streams", [
    # where the row kernels are faster, back to back and behind other kernels
    (BARE, api.F16, 256, 256, False), (BARE, api.F16, 2048, 128, False), (BARE, api.F8E4M3, 4096, 1024, False), (BARE, api.F8E4M3, 32000, 4096, False),
    (RESIDUAL, api.F16, 128, 128, False), (RESIDUAL, api.F8E4M3, 512, 512, False), (RESIDUAL, api.F32, 64, 64, False),
    (GLU, api.F16, 512, 256, False), (GLU, api.F8E4M3, 1000, 512, False),
    (SCALED, api.F16, 1024, 64, False), (SCALED, api.BF16, 10896, 2048, False), (SCALED, api.F16, 28672, 4096, False), (SCALED, api.F32, 4096, 14336, False),
    # where the stream is
    (BARE, api.F16, 1024, 1024, True), (BARE, api.F16, 32000, 4096, True), (BARE, api.F32, 512, 512, True), (BARE, api.F8E4M3, 2048, 2048, True), (BARE, api.F8E4M3, 32000, 8192, True),
    (RESIDUAL, api.F16, 4096, 14336, True), (RESIDUAL, api.F8E4M3, 1024, 2816, True), (RESIDUAL, api.F32, 256, 256, True), (RESIDUAL, api.F16, 64, 1024, True),
    (GLU, api.F16, 14336, 4096, True), (GLU, api.F8E4M3, 2816, 1024, True), (GLU, api.F32, 512, 256, True),
    # rows too long for it
    (BARE, api.F16, 512, 32776, False), (RESIDUAL, api.F8E4M3, 512, 32784, False), (GLU, api.F32, 512, 16388, False)])
def test_one_row_products_take_the_faster_kernel(product, dtype, d, n, streams):
    assert api.lib().yalm_gemv_streamed(product, dtype, n, d) == streams


def test_one_row_route_arguments():
    f = api.lib().yalm_gemv_streamed
    assert f(4, api.F16, 64, 64) < 0 and f(BARE, 7, 64, 64) < 0 and f(BARE, api.F16, 0, 64) < 0 and f(BARE, api.F16, 64, 0) < 0


def test_weights_go_first_when_l2_needs_room():
    """A copy without the hint puts every weight in the place of keys, values and states that the next token reads again."""
    text = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yalm_b200", "csrc", "stream_rows.cuh")).read()
    copies = re.findall(r'"cp\.async\.bulk[^ ]* ', text)
    assert len(copies) == 2 and all("L2::cache_hint" in c for c in copies)
    assert re.search(r"createpolicy\.fractional\.L2::evict_first\.b64 %0, 1\.0;", text)
