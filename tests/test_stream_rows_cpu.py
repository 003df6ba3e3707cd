"""-m "not gpu": what the stream of one-row products (csrc/stream_rows.cuh) asks of L2."""
import os
import re


def test_weights_go_first_when_l2_needs_room():
    """A copy without the hint puts every weight in the place of keys, values and states that the next token reads again."""
    text = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yalm_b200", "csrc", "stream_rows.cuh")).read()
    copies = re.findall(r'"cp\.async\.bulk[^ ]* ', text)
    assert len(copies) == 2 and all("L2::cache_hint" in c for c in copies)
    assert re.search(r"createpolicy\.fractional\.L2::evict_first\.b64 %0, 1\.0;", text)
