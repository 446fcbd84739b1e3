"""CPU test of the kernels that are launched behind one another, on their source: every thread block waits for the kernel in front of
it before it ends, so that a kernel's completion stands for that of all in front."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jaxrwkv_b200", "csrc")
WAITS = {"wait_for_grid_in_front", "word_behind"}


def functions(source):
    """(name, whether a kernel, body) of every function whose body follows its parameters."""
    source = re.sub(r"//[^\n]*|/\*.*?\*/", " ", source, flags=re.S)
    source = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", " ", source)
    for head in re.finditer(r"(__global__|__device__)([^;{}]*?)\b(\w+)\s*\(([^;{}]*)\)\s*\{", source):
        depth, at = 1, head.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(source[at], 0)
            at += 1
        yield head.group(3), head.group(1) == "__global__", source[head.end():at - 1]


def calls(body, names):
    return [m.start() for m in re.finditer(r"\b(" + "|".join(names) + r")\b\s*(<[^<>;]*>)?\s*\(", body)]


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_no_thread_block_ends_in_front_of_the_wait(path):
    found = list(functions(open(path).read()))
    waits = WAITS | {name for name, kernel, body in found if not kernel and calls(body, WAITS)}
    for name, kernel, body in found:
        if kernel and calls(body, waits):
            assert "return" not in body[:calls(body, waits)[0]], name


def test_the_kernels_are_found():
    names = {name for path in glob.glob(os.path.join(CSRC, "*.cu")) for name, kernel, body in functions(open(path).read())
             if kernel and re.search("wait_for_grid_in_front|word_behind", body)}
    assert {"wkv7_fp32_chain_kernel", "wkv7_fp32_outputs_kernel", "wkv7_fp32_grads_kernel", "wkv7_chain_blocks_kernel", "wkv5_fwd_kernel",
            "wkv6_chunk_bwd_kernel", "wkv4_parameter_grads_kernel"} <= names, names
