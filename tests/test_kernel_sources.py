"""Rules of the kernel sources that a run on one GPU does not show when they are broken."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parent.parent / "csrc" / "kernels"
SOURCES = sorted(KERNELS.glob("*.cu"))


def _code(path):
    """The source without comments."""
    s = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    return re.sub(r"//[^\n]*", "", s)


def _kernels(code):
    """Bodies of the __global__ functions."""
    for m in re.finditer(r"__global__", code):
        at = code.index("{", code.index(")", m.end()))
        depth, i = 0, at
        while True:
            depth += {"{": 1, "}": -1}.get(code[i], 0)
            if depth == 0:
                break
            i += 1
        yield code[at:i]


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.stem)
def test_dependents_are_released_after_tensor_memory_is_allocated(path):
    """Else a CTA of the next kernel may take the SM's columns and wait for this kernel, which then waits for the columns."""
    for body in _kernels(_code(path)):
        alloc = max(body.find("tmem_alloc("), body.find("tcgen05.alloc"))
        if alloc < 0 or "pdl_trigger()" not in body:
            continue
        trigger = body.index("pdl_trigger()")
        assert alloc < trigger and "__syncthreads()" in body[alloc:trigger]


def test_pair_of_ctas_waits_for_every_commit_on_its_stages():
    """tcgen05.commit arrives on the barriers of both CTAs of a pair; the arrivals of the last round may still be on their way when the work is
    handed out, so the producer waits for each stage once more behind its loop."""
    code = _code(KERNELS / "gemm_pair.cu")
    body = next(b for b in _kernels(code) if "tma_load_2d_pair" in b)
    producer = body[body.index("if (warp == 0)", body.index("cluster_sync_all")):body.index("} else if (warp == 1)")]
    behind = producer[producer.rindex("tma_load_2d_pair"):]
    assert re.search(r"for \(int i = 0; ok && i < a\.stages;.*mbar_wait\(smem_u32\(&bar_empty\[s\]\)", behind, flags=re.S)
