"""Products with e4m3 weights and bf16 activations (csrc/kernels/gemm_ws.cu) over the token tiles that set the lengths of its rings, against the same product
in 64 bits. Bound per output: with power-of-two block scales the weights are exact in bf16, so it is that of a bf16 product: K * 2^-23 of the sum of the
magnitudes for the fp32 sum, 2^-8 of the result for its rounding; through the gate/up unit as in its derivative, at most 1.1 for SiLU."""
import pytest
import torch

from skein_b200 import ops
from skein_b200.ops import fp8

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one K-block (a converter group without work), a few, more than every ring is long; features that end inside a tile; few tiles (cut into aligned pieces), a tile
# per CTA and more (equal shares)
@pytest.mark.parametrize("features,K", [(128, 128), (200, 384), (384, 4096), (19200, 256), (10240, 2048)])
@pytest.mark.parametrize("rows,tile", [(1, 16), (33, 48), (64, 64), (100, 128)])
@pytest.mark.parametrize("unit", [False, True])
def test_rings(features, K, rows, tile, unit):
    if unit and tile > 64:
        tile = 64
    g = torch.Generator(device=DEV).manual_seed(0)
    x = torch.randn(rows, K, device=DEV, generator=g).bfloat16()
    w = torch.randn(features * (2 if unit else 1), K, device=DEV, generator=g) * K ** -0.5
    w *= torch.exp2(torch.randint(-3, 4, (w.shape[0], 1), device=DEV, generator=g).float())
    q = fp8.quantize_weight(w.bfloat16())
    y = fp8.linear_a16(x, q, swiglu=unit, n_tile=tile)
    torch.cuda.synchronize()
    ops.workspace().check_status()
    xd, wd = x.double(), q.dequant().double()
    total, off = xd @ wd.T, K * 2.0 ** -23 * (xd.abs() @ wd.abs().T)
    if unit:
        (a, u), (ea, eu) = total.chunk(2, dim=1), off.chunk(2, dim=1)
        s = a * torch.sigmoid(a)
        total, off = s * u, (1.1 * ea + 2.0 ** -20 * s.abs()) * (u.abs() + eu) + (s.abs() + 1.1 * ea) * eu
    assert bool(((y.double() - total).abs() <= off + 2.0 ** -8 * (total.abs() + off)).all())
    assert torch.equal(y, fp8.linear_a16(x, q, swiglu=unit, n_tile=tile))


# either side of the lines at which a tile is cut into aligned pieces, taken whole or dealt as equal shares (csrc/kernels/gemm_sched.cuh), features x K at `rows`
# tokens: pieces 7 and 15 K-blocks longer than an equal share, whole tiles 8, 15 and 29 longer, with a small token tile and a large one
@pytest.mark.parametrize("features,K,rows,tile,unit", [(7168, 8192, 16, 16, False), (8192, 28672, 16, 16, False), (8192, 8192, 200, 128, False),
                                                       (7168, 8192, 200, 128, False), (10240, 8192, 16, 16, False), (10240, 8192, 100, 112, False),
                                                       (3584, 8192, 200, 64, True), (10240, 8192, 32, 32, True), (3584, 18944, 160, 64, True)])
def test_cuts(features, K, rows, tile, unit):
    test_rings(features, K, rows, tile, unit)
