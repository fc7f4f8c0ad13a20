"""Kernels that start beside their predecessor (programmatic launches) read what that predecessor may still be writing: appended
rows, lengths, locations, tables.  The read-only path (``__ldg``, ``ld.global.nc``, ``const __restrict__`` parameters of a kernel)
is for memory that nobody writes during the whole life of the kernel, and nothing keeps such a load behind the wait."""
import os
import re

import pytest

from inference_lib_b200 import _build

SOURCES = [s for s in _build.cabi_sources() if s.endswith((".cu", ".cuh"))]


def _code(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("path", SOURCES, ids=[os.path.basename(s) for s in SOURCES])
def test_no_load_through_the_read_only_path(path):
    assert not re.findall(r"\b__ldg\s*\(|ld\.global\.nc", _code(path))


def test_no_read_only_parameters_of_kernels_launched_beside_their_predecessor():
    code = "\n".join(_code(s) for s in SOURCES)
    launched = set(re.findall(r"launch_kernel\((\w+_kernel)\b", code))
    assert {"append_kernel", "step_plan_kernel", "copy_to_blocks_kernel", "dense_plan_kernel", "fma_attention_kernel"} <= launched
    signatures = dict(re.findall(r"__global__[^;{]*?\b(\w+_kernel)\s*\(([^{]*)\)\s*\{", code))
    assert launched <= set(signatures)
    assert not [name for name in sorted(launched) if "__restrict__" in signatures[name]]
