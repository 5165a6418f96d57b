"""Kernels that may be launched while the previous kernel of the stream still runs (they begin with
wait_previous()) must read their inputs by ordinary loads: the non-coherent path (__ldg, or const
__restrict__ kernel parameters) is only defined for data that stays constant while the kernel is
resident. Read from the sources, on the CPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pmf-glm_b200", "csrc")


def _kernels():
    """(file, text) of every __global__ definition, up to its closing brace."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        src = open(os.path.join(CSRC, name)).read()
        for m in re.finditer(r"__global__", src):
            end = src.find("\n}", m.start())
            yield name, src[m.start():end]


OVERLAPPED = [(n, t) for n, t in _kernels() if "wait_previous()" in t]


def test_the_overlapped_kernels_are_found():
    want = ("mhd_step_kernel(", "ct_emf_col_kernel(", "ct_face_col_kernel(", "ct_bcc_col_kernel(", "wavespeed_kernel(")
    assert len(OVERLAPPED) == len(want)
    assert all(any(w in t for _, t in OVERLAPPED) for w in want)


@pytest.mark.parametrize("at", range(len(OVERLAPPED)))
def test_overlapped_kernel_reads_coherently(at):
    name, text = OVERLAPPED[at]
    body = text[text.index("wait_previous()"):]
    assert "__restrict__" not in text and "__ldg" not in text, name
    # the kernel after this one is let in only once the kernel before this one is complete
    assert body.index("wait_previous()") < body.index("overlap_next()")
    assert "overlap_next()" not in text[:text.index("wait_previous()")]


def test_the_column_step_reads_coherently():
    src = open(os.path.join(CSRC, "step_kernel.cuh")).read()
    assert "__ldg" not in src and "ld.global.nc" not in src
