"""Kernels that may start before the kernel ahead of them is done read with plain loads: read-only ones (__ldg, ld.global.nc, pointers
to const with __restrict__) are defined for memory that nobody writes while the kernel lives.  A property of the source that no
output shows, so the source is what is looked at."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dlprimitives_b200", "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))
# written by the host when a plan is made, by no kernel
TABLES = re.compile(r"__ldg\((reinterpret_cast<const int4 \*>\(p\.ktab\) \+ i|p\.tap_dydx \+ \w+|tab \+ i)\)")
READ_ONLY = re.compile(r"__ldg\(|ld\.global\.nc|\bconst\s+\w+\s*\*\s*__restrict__")


def code(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


def kernels(text):
    """name -> source of the __global__ functions in a file (each ends at the first line that is a closing brace alone)."""
    return {re.search(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\([^)]*\)", "", m.group(0))).group(1): m.group(0)
            for m in re.finditer(r"__global__.*?\n}\n", text, re.S)}


def never_early(name):
    return set(re.findall(r"launch_pdl\(false, (?:\w+::)*(\w+)", code(name)))


@pytest.mark.parametrize("name", FILES)
def test_plain_loads(name):
    text = code(name)
    if "launch_pdl(" not in text and name.endswith(".cu"):
        return
    for kernel in never_early(name):
        text = text.replace(kernels(text)[kernel], "")
    found = [m.group(0) for m in READ_ONLY.finditer(TABLES.sub("", text))]
    assert not found, found


@pytest.mark.parametrize("name", [f for f in FILES if f.endswith(".cu")])
def test_the_wait_comes_first(name):
    """Plain kernels load nothing ahead of the wait for the kernel before them.  Kernels of several roles wait role by role, but not before
    their tensor memory is theirs: the wait lets the next kernel in, whose blocks take tensor memory and then wait for this one."""
    early = {k: v for k, v in kernels(code(name)).items() if "pdl_wait()" in v}
    if "launch_pdl(" in code(name):
        assert early
    for kernel, text in early.items():
        if "tcgen05.alloc" in text:
            assert text.index("__syncthreads()", text.index("tcgen05.alloc")) < text.index("pdl_wait()"), kernel
        else:
            load = re.search(r"__ldg\(|ld_plain\(|ld_early\(", text)
            assert load is None or text.index("pdl_wait()") < load.start(), kernel


def test_the_kernels_are_found():
    """The scan sees what it is meant to see."""
    seen = {k for f in FILES if f.endswith(".cu") for k in kernels(code(f))}
    assert {"split_finish_kernel", "prepack_kernel", "contraction_tf32x3_kernel", "stream_tf32x3_kernel", "pool_max3s2_kernel", "wtc_output_kernel",
            "depthwise3_reg_kernel", "batchnorm_inference_kernel", "contraction_ffma_kernel"} <= seen
    assert never_early("contraction_ffma.cu") == {"contraction_ffma_kernel"} and never_early("winograd.cu") == {"winograd_f23_kernel"}
