"""Properties of the kernels' source that no run can show: an order that is wrong may still never meet its deadlock."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "transformers-turboquant_b200", "csrc")


def _kernels():
    """(file, name, body) of every __global__ function."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        with open(os.path.join(CSRC, name)) as fh:
            text = re.sub(r"//[^\n]*", "", fh.read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\([^{;]*\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            yield name, m.group(1), text[m.end():i]


def test_kernels_are_found():
    assert {"expand_kv_kernel", "attention_dense_kernel", "decode_kernel"} <= {k for _, k, _ in _kernels()}


@pytest.mark.parametrize("file,kernel,body", [pytest.param(*k, id=f"{k[0]}:{k[1]}") for k in _kernels()
                                              if "grid_launch_dependents" in k[2] and "tmem_alloc" in k[2]])
def test_tensor_memory_is_taken_before_dependents_start(file, kernel, body):
    # A dependent that takes all of an SM's tensor memory before it waits for this kernel would otherwise hold what a CTA of
    # this kernel still waits for.
    alloc, trigger = body.index("tmem_alloc"), body.index("grid_launch_dependents")
    assert alloc < trigger and "__syncthreads()" in body[alloc:trigger], f"{kernel} in {file}"
