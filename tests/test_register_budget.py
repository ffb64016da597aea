"""The launch that folds the partials of rows of 9 - 16 tokens waits in place beside the tile kernel: 256 threads of both within an SM's 65536
registers, as the compiler is told in either kernel (registers are given out eight per thread at a time)."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "nano_vllm_jax_b200" / "csrc"


def test_the_fold_fits_beside_the_tile_kernel():
    sources = {p.name: p.read_text() for p in [*CSRC.glob("*.cu"), *CSRC.glob("*.cuh")]}
    constants = {m[0]: int(m[1]) for t in sources.values() for m in re.findall(r"(\w+Regs) = (\d+)", t)}

    def cap(file, kernel):
        found = re.search(r"__global__ void __maxnreg__\((\w+)\)\s*" + kernel + r"\(", sources[file])
        assert found, f"{kernel} has no register limit"
        return constants.get(found[1]) or int(found[1])

    regs = [cap("paged_decode_umma_query_rows.cu", "decode_umma_kernel"), cap("paged_decode_umma.cu", "decode_umma_merge_kernel")]
    assert 256 * sum(-(-r // 8) * 8 for r in regs) <= 65536
