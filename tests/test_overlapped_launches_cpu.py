"""Kernels that are set up while the one before them still runs promise the compiler nothing about memory that it may be writing."""

import re

from tests.conftest import ROOT

CSRC = ROOT / "vllm_rlt_b200" / "csrc"
OVERLAPPED = {"flat_transfer_kernel", "segmented_transfer_kernel", "inline_transfer_kernel", "move_kernel", "push_kernel", "inline_segments_kernel",
              "post_kernel", "finalize_kernel"}


def code(path):
    return re.sub(r"//.*", "", path.read_text())


def test_overlapped_kernels_have_no_restrict_pointers():
    assert "__restrict__" not in code(CSRC / "common.cuh")  # the copy loops that these kernels share
    seen = set()
    for source in sorted(CSRC.glob("*.cu")):
        text = code(source)
        for kernel in re.split(r"__global__", text)[1:]:
            name, parameters = re.search(r"(\w+_kernel)\(([^)]*)\)\s*\{", kernel).groups()
            if "follow_stream();" in kernel:
                seen.add(name)
                assert "__restrict__" not in parameters, f"{source.name}: {name}"
        if "launch_following(" in text:
            for function in re.findall(r"__device__ __forceinline__ [^;{]*\{", text):
                assert "__restrict__" not in function, f"{source.name}: {function}"
    assert seen == OVERLAPPED
