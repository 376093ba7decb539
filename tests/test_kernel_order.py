"""Orders in the kernels' source that nothing on the device may be asked to
show, because getting them wrong would hang it."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "rochpcg_b200", "csrc")


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def _kernels(text):
    """(name, body) of every __global__ function."""
    for m in re.finditer(r"__global__ void[^;{]*?(\bk_\w+)\s*\([^{]*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i]


@pytest.mark.parametrize("kernel", ["k_conv16", "k_layer3_tc", "k_layer1_tc", "k_conv16_wgrad"])
def test_dependents_start_after_the_tensor_memory_is_held(kernel):
    """A dependent's allocation that came first would be kept until this kernel ends, which waits for it."""
    body = dict(_kernels(_source("learned.cu")))[kernel]
    alloc = body.index("tmem_alloc(")
    held = body.index("__syncthreads", alloc)
    starts = [m.start() for m in re.finditer(r"pdl_launch_dependents\(|pdl_begin\(", body)]
    assert all(i > held for i in starts)
    if kernel != "k_conv16_wgrad":
        assert len(starts) == 1 and starts[0] < body.index("pdl_wait(")


def test_aligned_cluster_barriers_follow_a_converged_warp():
    """barrier.cluster.*.aligned is undefined where the lanes of a warp arrive apart."""
    text = _source("small_level.cu")
    barriers = [m.start() for m in re.finditer(r'asm volatile\("barrier\.cluster\.\w+\.\w+\.aligned', text)]
    assert len(barriers) == text.count("barrier.cluster") == 2
    assert all(re.search(r"__syncwarp\(\);\s*$", text[:i]) for i in barriers)
