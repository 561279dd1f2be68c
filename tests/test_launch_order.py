"""CPU-only: what the sources say about programmatic launches. A kernel's end stands for the end of all kernels before it, so no block may
leave before it has waited for them; the exits that do (a shared-memory layout that does not fit) cannot be brought about in a test."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ember_b200", "csrc")


def _closing(text, at):
    """The place behind the bracket that closes the one at `at`."""
    depth = 0
    while True:
        depth += {"(": 1, "{": 1, ")": -1, "}": -1}.get(text[at], 0)
        at += 1
        if depth == 0:
            return at


def _kernels(text):
    """(name, body) of each __global__ function."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*(?=\()", text):
        at = _closing(text, m.end())
        if text[at:].lstrip().startswith("{"):
            at = text.index("{", at)
            yield m.group(1), text[at:_closing(text, at)]


FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")))


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_no_block_leaves_before_it_has_waited(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    for name, body in _kernels(text):
        if "pdl_wait()" not in body:
            continue
        waited = re.search(r"\n    (?:ptx::)?pdl_wait\(\);", body)  # by every thread, at the top level
        waited = waited.start() if waited else len(body)
        for m in re.finditer(r"\breturn;", body):
            before = body[:m.start()].rstrip()
            assert m.start() > waited or "pdl_wait();" in before[before.rindex("{"):], f"{name}: return before pdl_wait()"


def test_the_kernels_are_found():
    found = {name for path in FILES for name, body in _kernels(re.sub(r"//[^\n]*", "", open(path).read())) if "pdl_wait()" in body}
    assert {"sm100_fwd_kernel", "sm100_bwd_fused_kernel", "dq_finish_kernel", "sm100_gemm_kernel", "sm100_f32_gemm_kernel", "sm100_f32_bwd_kernel",
            "column_sum_kernel", "decode_sm100_kernel", "skinny_gemm_kernel", "narrow_f32_kernel", "split_f32_kernel"} <= found
