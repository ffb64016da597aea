"""Rules of the kernels that overlap with their neighbours in the stream (programmatic dependent launch), read from the
sources: nothing is let go before the wait, and tensor memory is taken between the wait and the release."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "nano_vllm_jax_b200" / "csrc"


def _kernels():
    """(file, kernel name, body without comments) of every __global__ function."""
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__\s+void\s+(?:__\w+__\s*\([^)]*\)\s*)*(\w+)\s*\([^{;]*\)\s*\{", text):
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            yield path.name, m.group(1), text[m.end():i]


OVERLAPPING = [k for k in _kernels() if "pdl_release()" in k[2]]


@pytest.mark.parametrize("file,name,body", OVERLAPPING, ids=[k[1] for k in OVERLAPPING])
def test_a_kernel_waits_before_it_lets_the_next_one_go(file, name, body):
    assert 0 <= body.find("pdl_wait()") < body.find("pdl_release()")
    alloc = re.search(r"\btmem2?_alloc\(", body)
    if alloc:
        assert body.find("pdl_wait()") < alloc.start() < body.find("pdl_release()")


def test_the_kernels_are_found():
    names = {k[1] for k in OVERLAPPING}
    assert {"prefill_umma2_kernel", "decode_umma_kernel", "decode_cluster_mma_kernel", "append_copy16_kernel"} <= names
    # a kernel that takes tensor memory and does not overlap is launched in plain stream order
    assert {k[1] for k in _kernels() if re.search(r"\btmem2?_alloc\(", k[2])} == {"prefill_umma2_kernel", "decode_umma_kernel",
                                                                                "prefill_umma_kernel"}
