"""Products that begin to fetch their weights before the kernel in front of them has ended (early_w): bit for bit those that wait, behind kernels that
write their activations, eagerly and captured, cut tiles and whole ones."""
import pytest
import torch

from skein_b200 import ops
from skein_b200.ops import fp8

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows,features,K", [(1, 256, 512), (40, 6144, 4096), (64, 20000, 256)])
@pytest.mark.parametrize("kind", ["plain", "packed", "unit", "e4m3", "groups", "sum"])
def test_behind_a_norm(rows, features, K, kind):
    g = torch.Generator(device=DEV).manual_seed(0)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)        # noqa: E731
    features = features // 128 * 128 if kind == "packed" else features
    res, gamma, w = r(rows, K).bfloat16(), (1 + 0.1 * r(K)).bfloat16(), (r(2 * features if kind in ("unit", "e4m3") else features, K) * K ** -0.5).bfloat16()
    total = r(rows, features)
    if kind == "groups":
        cnt = torch.tensor([rows - rows // 3, 0, rows // 3], dtype=torch.int32, device=DEV)
        off = torch.cat([cnt.new_zeros(1), cnt.cumsum(0).int()])
        w = torch.stack([w, w, -w])
    w = ops.pack_weight(w) if kind == "packed" else fp8.quantize_weight(w) if kind == "e4m3" else w

    def chain(early, x):
        for _ in range(3):
            x, n = ops.reduce_residual_rmsnorm(x, None, gamma, 1e-5)
            y = (ops.swiglu_linear(n, w, early_w=early) if kind == "unit" else fp8.linear_a16(n, w, swiglu=True, early_w=early) if kind == "e4m3" else
                 ops.grouped_linear(n, w, cnt, off, early_w=early) if kind == "groups" else
                 ops.linear(n, w, residual=total, out_f32=True, early_w=early) if kind == "sum" else ops.linear(n, w, early_w=early))
            z = y.bfloat16()
            x = x + z[:, :K] if z.shape[1] >= K else x.index_add(1, torch.arange(z.shape[1], device=DEV), z)
        return y

    want = chain(False, res)
    eager = chain(True, res)
    torch.cuda.synchronize()
    graph, x = torch.cuda.CUDAGraph(), torch.zeros_like(res)
    with torch.cuda.graph(graph):
        got = chain(True, x)
    x.copy_(res)
    graph.replay()
    torch.cuda.synchronize()
    ops.workspace().check_status()
    assert torch.equal(eager, want) and torch.equal(got, want)


@pytest.mark.parametrize("kind", ["plain", "unit", "e4m3"])
def test_budget_starts_when_the_kernel_in_front_has_ended(monkeypatch, kind):
    """A norm that stands waiting for a peer longer than the product's own budget: what is recorded is the peer's flag, not a stage of the product."""
    from skein_b200.ops import functional as F
    make = F._base_params

    def short(*args):
        p = make(*args)
        p.wait_budget_ms = 20
        return p

    monkeypatch.setattr(F, "_base_params", short)
    K, features = 1024, 4096
    x, gamma = torch.randn(8, K, device=DEV).bfloat16(), torch.ones(K, device=DEV).bfloat16()
    w = (torch.randn(2 * features, K, device=DEV) * K ** -0.5).bfloat16()
    q = fp8.quantize_weight(w) if kind == "e4m3" else w
    part = torch.randn(2, 8, K, device=DEV).bfloat16()
    flags, epoch = torch.zeros(2, dtype=torch.int32, device=DEV), torch.ones(1, dtype=torch.int32, device=DEV)
    torch.cuda.synchronize()
    _, n = ops.reduce_residual_rmsnorm(x, part, gamma, 1e-5, flags=flags, epoch=epoch, wait_budget_ms=300)
    if kind == "e4m3":
        fp8.linear_a16(n, q, early_w=True)
    else:
        (ops.swiglu_linear if kind == "unit" else ops.linear)(n, q, early_w=True)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="peer flag"):
        ops.workspace().check_status()
