"""Rules of the kernel sources that no run can show (a violation would hang a GPU, or show only under a rare schedule)."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "rtxntc-library_b200", "csrc")


def _functions_calling(name):
    """(file, function text up to the call) for every call of `name`; a function starts at its __device__ or __global__."""
    found = []
    for file in sorted(os.listdir(CSRC)):
        if not file.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, file)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for call in re.finditer(r"\b%s\(\)\s*;" % name, text):
            start = max(text.rfind("__device__", 0, call.start()), text.rfind("__global__", 0, call.start()))
            found.append((file, text[start:call.start()]))
    return found


@pytest.mark.parametrize("kernels,text", _functions_calling("GridDependencyLaunch"), ids=lambda v: v if "\n" not in v else "")
def test_dependent_launches_are_released_after_the_tensor_memory_is_held(kernels, text):
    """A kernel that the trigger lets start takes tensor memory and waits for this one to end: this CTA must have its own."""
    allocation = text.find("TmemAlloc(")
    assert allocation >= 0, kernels
    assert "__syncthreads();" in text[allocation:], kernels


def test_every_set_up_of_a_decode_kernel_releases_its_dependents():
    assert sorted(file for file, _ in _functions_calling("GridDependencyLaunch")) == \
        ["decode_kernel.cu", "decode_kernel_ref.cu", "decode_kernel_ref.cu"]
