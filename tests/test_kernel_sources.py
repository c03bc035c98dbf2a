"""Rules of the kernel sources that a run on one GPU does not show when they are broken."""
import re
import subprocess
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


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.stem)
def test_kernel_attributes_are_set_on_every_device(path):
    """Attributes belong to a device: a flag or a grid that is kept for the process leaves a second device without its shared memory."""
    code = _code(path)
    assert not re.search(r"static (bool|int) \w+(\[[24]\])? = ", code) or "cudaFuncSetAttribute" not in code


def test_state_per_device(tmp_path):
    """csrc/kernels/per_device.h: made once per device whatever the number of threads, an error is tried again, devices are apart."""
    src = tmp_path / "t.cpp"
    src.write_text("""
        #include "per_device.h"
        #include <atomic>
        #include <thread>
        #include <vector>
        int main() {
          skein::PerDevice v;
          std::atomic<int> made[3] = {};
          std::vector<std::thread> ts;
          std::atomic<int> wrong{0};
          for (int i = 0; i < 32; ++i)
            ts.emplace_back([&, i] { if (v.get(i % 3, [&] { ++made[i % 3]; return 10 + i % 3; }) != 10 + i % 3) ++wrong; });
          for (auto& t : ts) t.join();
          for (int d = 0; d < 3; ++d) if (made[d] != 1) return 1;
          if (wrong) return 2;
          skein::PerDevice e;
          if (e.get(5, [] { return -7; }) != -7 || e.get(5, [] { return 3; }) != 3 || e.get(5, [] { return 4; }) != 3) return 3;
          return e.get(-1, [] { return 1; }) == -4 && e.get(64, [] { return 1; }) == -4 ? 0 : 4;
        }
    """)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", str(KERNELS), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
