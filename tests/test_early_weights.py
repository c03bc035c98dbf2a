"""Which products may begin to fetch their weights before the kernel in front has ended (early_w)."""
import os
import subprocess
from pathlib import Path
from types import SimpleNamespace

import pytest
import torch

from skein_b200 import ops
from skein_b200.models.decoder import Decoder
from skein_b200.ops import fp8
from skein_b200.utils.runtime_config import RuntimeConfig

ROOT = Path(__file__).resolve().parent.parent


class Weight8:
    shape = (16, 8)

    def dequant(self):
        return torch.zeros(16, 8)


@pytest.mark.parametrize("tp,ep,early", [(1, 1, True), (2, 1, False), (1, 2, False)])
def test_one_rank_only(monkeypatch, tp, ep, early):
    """With more ranks the kernel in front waits for peers, and nothing was measured there."""
    seen = []
    for mod, names in ((ops, ("linear", "swiglu_linear", "grouped_linear")), (fp8, ("linear_a16", "grouped_linear_a16"))):
        for n in names:
            monkeypatch.setattr(mod, n, lambda x, *a, **kw: seen.append(kw.get("early_w", False)) or x)
    d = Decoder.__new__(Decoder)
    d.comm, d.comm_moe, d.w = SimpleNamespace(size=tp), SimpleNamespace(size=ep), SimpleNamespace(lm_head=torch.zeros(16, 8))
    x, groups = torch.zeros(4, 8), (torch.tensor([4]), torch.tensor([0, 4]))
    own, copy8 = SimpleNamespace(fp8={}, wqkv=torch.zeros(16, 8)), SimpleNamespace(fp8={"wqkv": Weight8()}, wqkv=None)
    for lw in (own, copy8):
        for kw in ({}, {"swiglu": True}, {"grouped": groups}):
            d._col_linear(x, lw, "wqkv", **kw)
        if tp == 1:
            d._row_parallel(x, lw, "wqkv")
            d._row_parallel(x, lw, "wqkv", groups)
    d.logits(x, SimpleNamespace(is_prefill=False, logit_rows=None))
    assert len(seen) == (11 if tp == 1 else 7) and all(e == early for e in seen)
    # a weight that is expanded for the call is written by the kernel in front
    del seen[:]
    monkeypatch.setattr(Decoder, "_expand_fp8", lambda *a: True)
    d._col_linear(x, copy8, "wqkv")
    assert seen == [False]


def test_switches(tmp_path):
    """csrc/kernels/launch.cuh: early products have a switch of their own, so that no kernel is a programmatic dependent with both off."""
    cuda = next((p for p in (Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")),) if (p / "include" / "cuda_runtime.h").exists()), None)
    if cuda is None:
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text('#include "launch.cuh"\n#include <cstdio>\nint main() { printf("%d %d", skein::pdl_enabled(), skein::early_weights_enabled()); }\n')
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT / "csrc" / "kernels"), "-I", str(cuda / "include"), str(src), "-o", str(exe)], check=True)
    base = {k: v for k, v in os.environ.items() if not k.startswith("SKEIN_")}
    for cfg, want in ((RuntimeConfig(), "0 1"), (RuntimeConfig(early_weights=False), "0 0"), (RuntimeConfig(pdl=True, early_weights=False), "1 0")):
        assert subprocess.run([str(exe)], env={**base, **cfg.to_env()}, capture_output=True, text=True).stdout == want
    assert subprocess.run([str(exe)], env=base, capture_output=True, text=True).stdout == "0 1"
    assert RuntimeConfig.from_toml("[runtime]\nearly_weights = false\n").to_env()["SKEIN_EARLY_WEIGHTS"] == "0"
