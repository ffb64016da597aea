"""A CTA may end only after the others of its cluster have read its shared memory.  A relaxed arrival at the cluster's barrier orders
none of a thread's earlier loads, so it is taken only where a vote on what they returned has chosen it over a release; and the barrier
follows the last load from another CTA."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "nano_vllm_jax_b200" / "csrc"
SOURCES = {p.name: re.sub(r"//[^\n]*", "", p.read_text()) for p in sorted([*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")])}


def test_a_relaxed_arrival_hangs_on_what_was_loaded():
    assert re.search(r"void cl_arrive\(\) \{ asm volatile\(\"barrier\.cluster\.arrive\.release", SOURCES["cluster.cuh"])
    for name, text in SOURCES.items():
        for m in re.finditer(r"asm volatile\(\"barrier\.cluster\.arrive\.relaxed", text):
            assert re.search(r"if \(__any_sync\(0xffffffffu, odd\)\) cl_arrive\(\);\s*else $", text[:m.start()]), name
        for call in re.findall(r"cl_sync_read\((.*?)\);", text):
            assert call == "odd" and re.search(r"odd \|= cl_not_finite\(", text), name


@pytest.mark.parametrize("name", [n for n, t in SOURCES.items() if n.endswith(".cu") and re.search(r"= .*\bcl_ld[24]\(", t)])
def test_an_arrival_follows_the_last_load_from_another_cta(name):
    behind = SOURCES[name][max(m.end() for m in re.finditer(r"\bcl_ld[24]\(", SOURCES[name])):]
    assert re.search(r"\bcl_(sync_read\(odd\)|sync\(\))", behind) and "cl_sync_relaxed" not in SOURCES[name]
