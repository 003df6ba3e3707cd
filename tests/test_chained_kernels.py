"""-m "not gpu": rules that kernels launched chained (csrc/launch.h: launch_chained) keep, read from their source."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yalm_b200", "csrc")


def kernels():
    """(file:name, parameters, body) of every __global__ function that waits for the kernel before it."""
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\([^()]*(?:\([^()]*\)[^()]*)*\)\s*)?(\w+)\s*\(([^{;]*)\)\s*\{", text):
            depth, at = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            body = text[m.end(): at]
            if "chain_wait()" in body or "chain_next()" in body:
                out.append(pytest.param(m.group(2), body, id="%s:%s" % (os.path.basename(path), m.group(1))))
    return out


def test_kernels_are_found():
    assert len(kernels()) >= 8


@pytest.mark.parametrize("params,body", kernels())
def test_waits_before_it_lets_the_next_begin(params, body):
    assert body.count("chain_wait()") == 1 and body.count("chain_next()") == 1 and body.index("chain_wait()") < body.index("chain_next()")


@pytest.mark.parametrize("params,body", kernels())
def test_tensor_memory_is_taken_before_the_next_may_begin(params, body):
    """Else the next kernel could hold columns while it waits for this one, which waits for the columns."""
    if "tmem_alloc" in body:
        between = body[body.index("tmem_alloc"): body.index("chain_next()")]
        assert "__syncthreads()" in between or "cluster_sync()" in between


@pytest.mark.parametrize("params,body", kernels())
def test_promises_nothing_about_its_inputs(params, body):
    """They are still being written when the kernel begins: __restrict__ and non-coherent loads state the contrary."""
    assert "__restrict__" not in params
    assert not re.search(r"__ldg\(|ldg_stream\(|ld\.global\.nc", body)
