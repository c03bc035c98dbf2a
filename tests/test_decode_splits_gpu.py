"""Splits of decode attention (functional.split_plan, csrc/kernels/attn_decode_mma.cu): sequences shorter than the hint of the step. A sequence takes
as many splits as its own length is worth; one that takes one is, bit for bit, the unsplit result. Others against the operator's fp32 reference, bound as for
prefill attention: probabilities rounded to bf16, at most 2^-8 of each (their sum is not), the result rounded to bf16, and a tenth more for the fp32 sums."""
import pytest
import torch

from skein_b200 import ops
from skein_b200.ops import functional as F
from skein_b200.ops import reference as ref

D, PAGE = 128, 16


def test_rule():
    """No launch of more than two CTAs per SM for the sake of splits, within the scratch, and few pairs of long sequences are split."""
    for B in (*range(1, 70), 128, 512):
        for Hkv, group in ((1, 8), (2, 16), (4, 7), (8, 4), (8, 8), (32, 1)):
            for ctx in (1, 300, 700, 768, 1024, 2048, 4096, 8000, 131072):
                splits, tokens = F.split_plan(B, Hkv, ctx, 148, group)
                pairs = B * Hkv
                assert 1 <= splits <= 16 and (splits == 1 or pairs * splits <= 2 * 148) and pairs * group * splits <= max(148 * 16, pairs * group)
                assert tokens >= 128 and (splits == 1 or ctx >= splits * 128)
    assert F.split_plan(5, 8, 8000, 148, 4)[0] == 7 and F.split_plan(1, 8, 4096, 148, 4)[0] == 16 and F.split_plan(20, 8, 8000, 148, 4)[0] == 1


def _case(lens, Hq, Hkv, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()      # noqa: E731
    nb = (max(lens) + PAGE - 1) // PAGE + 1
    table = torch.randperm(len(lens) * nb, device="cuda", generator=g).int().view(len(lens), nb)
    return r(len(lens), (Hq + 2 * Hkv) * D), r(len(lens) * nb, 2, Hkv, PAGE, D), table, torch.tensor(lens, dtype=torch.int32, device="cuda")


# a padding row, one token, around a tile, just below and above the lengths at which a second split begins (of 128 and of 256 tokens), many splits
LENS = [0, 1, 17, 191, 192, 193, 383, 384, 385, 640, 1000, 2049]


@pytest.mark.gpu
@pytest.mark.parametrize("Hq,Hkv", [(8, 2), (4, 4), (7, 1), (16, 1)])
@pytest.mark.parametrize("lens", [LENS, [100, 200, 3, 380], [2049, 60]])
def test_short_sequences_under_a_long_hint(Hq, Hkv, lens):
    q, kv, table, sl = _case(lens, Hq, Hkv)
    got = ops.attn_decode(q, kv, table, sl, Hq, Hkv, D, ctx_hint=8192)
    whole = ops.attn_decode(q, kv, table, sl, Hq, Hkv, D, splits=1, impl="mma")
    again = ops.attn_decode(q, kv, table, sl, Hq, Hkv, D, ctx_hint=8192)
    torch.cuda.synchronize()
    ops.workspace().check_status()
    splits, tokens = F.split_plan(len(lens), Hkv, 8192, ops.workspace().sm_count, Hq // Hkv)
    assert splits > 1 and torch.equal(got, again)
    for i, n in enumerate(lens):
        if (n + tokens // 2) // tokens < 2:
            assert torch.equal(got[i], whole[i])
    live = [i for i, n in enumerate(lens) if n]
    args = (table[live].cpu(), sl[live].cpu(), Hq, Hkv, D)
    size = kv.float().cpu()
    want = ref.attn_decode(q[live].float().cpu(), size, *args).float()
    size[:, 1] = size[:, 1].abs()
    mass = ref.attn_decode(q[live].float().cpu(), size, *args).float()
    assert bool(((got[live].float().cpu() - want).abs() <= 1.1 * (2.0 ** -8 * mass + 2.0 ** -8 * want.abs())).all())


@pytest.mark.gpu
@pytest.mark.parametrize("lens", [LENS, [100, 200, 3, 380]])
def test_rope_and_append_under_a_long_hint(lens):
    Hq, Hkv = 8, 2
    qkv, kv, table, sl = _case(lens, Hq, Hkv)
    cs = torch.randn(2100, D // 2, 2, device="cuda")
    out, caches = [], []
    for kw in ({"ctx_hint": 8192}, {"splits": 1}):
        c = kv.clone()
        out.append(ops.attn_decode_rope(qkv, sl - 1, table, cs, c, sl, Hq, Hkv, D, **kw))
        caches.append(c)
    torch.cuda.synchronize()
    ops.workspace().check_status()
    assert torch.equal(*caches)
    tokens = F.split_plan(len(lens), Hkv, 8192, ops.workspace().sm_count, Hq // Hkv)[1]
    short = [i for i, n in enumerate(lens) if (n + tokens // 2) // tokens < 2]
    assert torch.equal(out[0][short], out[1][short])
    assert torch.allclose(out[0].float(), out[1].float(), atol=2.0 ** -6 * float(out[1].abs().max()))
