"""Prefill attention, two heads of a group per CTA (csrc/kernels/attn_prefill_tc.cu), against the operator's fp32 reference at the edges of its tiles.

Bound per output: the probabilities are rounded to bf16, at most 2^-8 of each, in the weighted sum of the values and in the sum that divides it,
which moves the result by at most 2 * 2^-8 of the weighted sum of the values' magnitudes; the result is rounded to bf16, 2^-8 of it. A tenth more covers
the fp32 scores and exponentials.
"""
import pytest
import torch

from skein_b200 import ops
from skein_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV, D, PAGE = "cuda", 128, 16


# rows of a chunk and tokens cached before it: one row, tiles less one, whole and one more, key tiles that end inside a 16-token step, sequences of all
# lengths in one launch; groups of one, two, three (the last head alone) and seven heads
@pytest.mark.parametrize("new,cached", [([1], [0]), ([127], [1]), ([128], [0]), ([129], [127]), ([300, 1, 40], [0, 515, 128]), ([257], [1000])])
@pytest.mark.parametrize("heads,kv_heads", [(2, 2), (4, 2), (3, 1), (14, 2)])
def test_tiles(new, cached, heads, kv_heads):
    g = torch.Generator(device=DEV).manual_seed(0)
    total = [n + c for n, c in zip(new, cached)]
    blocks = [(t + PAGE - 1) // PAGE for t in total]
    order = torch.randperm(sum(blocks), device=DEV, generator=g).int()
    table = torch.zeros(len(new), max(blocks), dtype=torch.int32, device=DEV)
    for i, b in enumerate(blocks):
        table[i, :b] = order[sum(blocks[:i]):sum(blocks[:i + 1])]
    cache = torch.randn(sum(blocks), 2, kv_heads, PAGE, D, device=DEV, generator=g).bfloat16()
    for i, t in enumerate(total):       # what follows a sequence in its last page was never written
        if t % PAGE:
            cache[table[i, blocks[i] - 1], :, :, t % PAGE:] = float("nan")
    q = torch.randn(sum(new), (heads + 2 * kv_heads) * D, device=DEV, generator=g).bfloat16()
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)        # noqa: E731
    args = (ints([sum(new[:i]) for i in range(len(new))]), ints(new), ints(total))
    y = ops.attn_prefill(q, cache, table, *args, max(new), heads, kv_heads, D)
    torch.cuda.synchronize()
    ops.workspace().check_status()
    clean = cache.nan_to_num().cpu()
    size = clean.clone()
    size[:, 1] = clean[:, 1].abs()
    cpu = [t.cpu() for t in args]
    want, mass = (ref.attn_prefill(q.float().cpu(), c.float(), table.cpu(), *cpu, heads, kv_heads, D) for c in (clean, size))
    bound = 1.1 * (2 * 2.0 ** -8 * mass.float() + 2.0 ** -8 * want.float().abs())
    assert bool(((y.float().cpu() - want.float()).abs() <= bound).all())
