"""Kernels over the rows of a prefill chunk (norm.cu, rope_kv.cu, router.cu) where they change over from the decode-sized forms and at the edges of their
tiles, against the operators' fp32 references. Bounds: results are sums of a few fp32 terms rounded to bf16 (at most 2^-8 of the value), once for the
residual stream, and twice for a normalised value, before and after its scale; a tenth more covers the fp32 sums."""
import pytest
import torch

from skein_b200 import ops
from skein_b200.ops import reference as ref

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _gen():
    return torch.Generator(device=DEV).manual_seed(0)


def _done():
    torch.cuda.synchronize()
    ops.workspace().check_status()


@pytest.mark.parametrize("rows,H", [(295, 264), (296, 8), (296, 264), (300, 4096), (297, 8200), (296, 16384)])
@pytest.mark.parametrize("slots", [None, 0, 1, 2])
def test_norm(rows, H, slots):
    g = _gen()
    res, gamma = torch.randn(rows, H, device=DEV, generator=g).bfloat16(), (1 + 0.1 * torch.randn(H, device=DEV, generator=g)).bfloat16()
    part = idx = wts = None
    total = res.double()
    if slots is not None:
        part = torch.randn(1, rows * max(slots, 1), H, device=DEV, generator=g).bfloat16()
        terms = part[0].double()[:, None]
        if slots:
            idx = torch.randperm(rows * slots, device=DEV, generator=g).view(rows, slots).int()
            idx[::7, 0] = -1                                         # an expert of another rank
            wts = torch.rand(rows, slots, device=DEV, generator=g)
            terms = part[0].double()[idx.clamp(min=0).long()] * (wts * (idx >= 0))[..., None].double()
        total = total + terms.sum(1)
    r, n = ops.reduce_residual_rmsnorm(res, part, gamma, 1e-5, idx, wts)
    r2, _ = ops.reduce_residual_rmsnorm(res, part, None, 1e-5, idx, wts)
    _done()
    assert torch.equal(r, r2)
    assert bool(((r.double() - total).abs() <= 1.1 * 2.0 ** -8 * total.abs() + 2.0 ** -20).all())
    x = r.double()
    want = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5) * gamma.double()
    assert bool(((n.double() - want).abs() <= 2.2 * 2.0 ** -8 * want.abs()).all())


@pytest.mark.parametrize("D,Hq,Hkv", [(128, 5, 1), (64, 4, 2), (48, 3, 3), (16, 2, 1), (24, 2, 1)])      # (24: no 16-byte halves)
def test_rope(D, Hq, Hkv):
    g, T, page = _gen(), 37, 16
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device=DEV, generator=g).bfloat16()
    pos = torch.arange(T, device=DEV, dtype=torch.int32) % 20
    pos[5] = -1
    seq = (torch.arange(T, device=DEV) // 20).int()
    table = torch.randperm(4, device=DEV, generator=g).int().view(2, 2)
    cs = torch.randn(32, D // 2, 2, device=DEV, generator=g)
    cache = torch.zeros(4, 2, Hkv, page, D, dtype=torch.bfloat16, device=DEV)
    live = pos >= 0
    q2, c2 = qkv[live].cpu(), cache.clone().cpu()
    ref.rope_kv_append(q2, pos[live].cpu(), seq[live].cpu(), table.cpu(), cs.cpu(), c2, Hq, Hkv, D)
    before = qkv.clone()
    ops.rope_kv_append(qkv, pos, seq, table, cs, cache, Hq, Hkv, D)
    _done()
    for a, b in ((qkv[live][:, :Hq * D].cpu(), q2[:, :Hq * D]), (cache.cpu(), c2)):
        assert torch.allclose(a.float(), b.float(), rtol=2.0 ** -7, atol=2.0 ** -20)      # a step of bf16
    assert torch.equal(qkv[~live], before[~live])


@pytest.mark.parametrize("T,H,E,k", [(255, 4096, 8, 2), (256, 4096, 8, 2), (257, 96, 5, 3), (300, 512, 64, 8), (600, 40, 8, 1), (4099, 256, 8, 2)])
def test_route(T, H, E, k):
    g = _gen()
    x, wg = torch.randn(T, H, device=DEV, generator=g).bfloat16(), (torch.randn(E, H, device=DEV, generator=g) * H ** -0.5).bfloat16()
    z = x.double() @ wg.double().T
    for first, count in ((0, E), (1, E - 2)):
        ids, w, counts, offsets, row_of, src = ops.route(x, wg, k, first, count)
        _done()
        # a chosen expert's logit is, up to the rounding of both to bf16, at least that of any expert left out
        top, left = z.gather(1, ids.long()), z.scatter(1, ids.long(), float("-inf"))
        assert bool((top.min(1).values >= left.max(1).values - 2.0 ** -7 * z.abs().max(1).values).all())
        assert k == 1 or bool((ids.sort(1).values.diff(dim=1) > 0).all())
        assert torch.allclose(w.double(), torch.softmax(top.bfloat16().double(), -1), atol=2.0 ** -7)
        want = [t.to(DEV) for t in ref.router_plan(ids.cpu(), E, first, count)]
        n = int(want[1][E])
        assert torch.equal(counts, want[0]) and torch.equal(offsets, want[1]) and torch.equal(row_of.view(-1), want[2].view(-1))
        assert torch.equal(src[:n], want[3][:n])
        again = ops.router_plan(ids, E, first, count)
        _done()
        assert torch.equal(again[0], want[0]) and torch.equal(again[2].view(-1), want[2].view(-1))


# both sides of the line between a CTA per token and head and one per token: enough tokens, head sizes whose pairs do not divide the threads, heads that leave
# threads idle, more heads than fit at once, no 16-byte halves
@pytest.mark.parametrize("T,D,Hq,Hkv", [(1285, 128, 5, 1), (1286, 128, 5, 1), (2250, 64, 2, 1), (1500, 48, 4, 1), (260, 16, 33, 1), (300, 128, 28, 4), (9000, 16, 2, 1),
                                        (1300, 24, 5, 1), (190, 64, 40, 4)])
def test_rope_of_many_tokens(T, D, Hq, Hkv):
    g, page, S = _gen(), 16, 3
    per = (T + S - 1) // S
    qkv = torch.randn(T, (Hq + 2 * Hkv) * D, device=DEV, generator=g).bfloat16()
    at = torch.arange(T, device=DEV)
    pos, seq = (at % per).int(), (at // per).int()
    pos[7] = -1
    nb = (per + page - 1) // page
    table = torch.randperm(S * nb, device=DEV, generator=g).int().view(S, nb)
    cs = torch.randn(per, D // 2, 2, device=DEV, generator=g)
    cache = torch.zeros(S * nb, 2, Hkv, page, D, dtype=torch.bfloat16, device=DEV)
    live = pos >= 0
    q2, c2 = qkv[live].cpu(), cache.clone().cpu()
    ref.rope_kv_append(q2, pos[live].cpu(), seq[live].cpu(), table.cpu(), cs.cpu(), c2, Hq, Hkv, D)
    before = qkv.clone()
    ops.rope_kv_append(qkv, pos, seq, table, cs, cache, Hq, Hkv, D)
    _done()
    for a, b in ((qkv[live][:, :Hq * D].cpu(), q2[:, :Hq * D]), (cache.cpu(), c2)):
        # x c - y s in fp32, rounded to bf16 (2^-8 of it) here and there; what cancels is bounded by the two products
        assert bool(((a.float() - b.float()).abs() <= 2.0 ** -7 * b.float().abs() + 2.0 ** -20).all())
    assert torch.equal(qkv[~live], before[~live]) and torch.equal(qkv[:, Hq * D:], before[:, Hq * D:])


# up to four experts: rows of 2048 and less take the tiles from 256 tokens on, longer ones from 512
@pytest.mark.parametrize("T,H,E,k", [(255, 2048, 4, 1), (256, 2048, 4, 2), (300, 4096, 4, 1), (511, 2080, 3, 2), (512, 2080, 3, 2), (520, 8192, 4, 1)])
def test_route_of_few_experts(T, H, E, k):
    test_route(T, H, E, k)
