"""The allocation-free entry point's source calls no allocating routine (include/grand_decoder.h
promises that to callers whose memory is spoken for): neither device nor pinned host memory."""
import os
import re

from conftest import ROOT

CALLS = re.compile(r"\b(cudaMalloc\w*|cudaHostAlloc|cudaHostRegister|cudaFree\w*|cuMem\w*|malloc|calloc|realloc|"
                   r"cudaStreamCreate\w*|cudaEventCreate\w*|cudaGraph\w*)\s*\(")


def test_no_allocating_call():
    csrc = os.path.join(ROOT, "library_s_grand_gb300", "csrc")
    for name in ("grand_noalloc.cu", "grand_prep.cuh", "grand_front.cuh"):
        with open(os.path.join(csrc, name), encoding="utf-8") as f:
            code = re.sub(r"//[^\n]*", "", f.read())
        assert not CALLS.findall(code), (name, CALLS.findall(code))
        assert not re.search(r"\bnew\b|std::vector|std::string", code), name
