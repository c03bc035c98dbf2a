"""Products on pairs of CTAs (csrc/kernels/gemm_pair.cu) against the same product in 64 bits, at the edges of its tiles.

Bound per output: the operands are bf16 and exact, products are exact in fp32, and K of them are added in fp32 in some order, which is off by at most
K * 2^-23 times the sum of their magnitudes (truncating adds included); rounding the sum to bf16 adds 2^-8 of it. SiLU has a slope of at most 1.1
and its exponential and division a few units of fp32, so a gate/up pair's bound follows from those of its two sums.
"""
import pytest
import torch

from skein_b200 import ops
from skein_b200.ops import _lib, functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _sum(x, w):
    """x w^T and the bound on an fp32 sum's error."""
    x, w = x.double(), w.double()
    return x @ w.T, x.shape[1] * 2.0 ** -23 * (x.abs() @ w.abs().T)


def _unit(x, w):
    (g, eg), (u, eu) = (_sum(x, h) for h in w.chunk(2))
    s = g * torch.sigmoid(g)
    return s * u, (1.1 * eg + 2.0 ** -20 * s.abs()) * (u.abs() + eu) + (s.abs() + 1.1 * eg) * eu


def _inputs(rows, features, K, lead=(), seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)        # noqa: E731
    return r(rows, K).bfloat16(), (r(*lead, features, K) * K ** -0.5).bfloat16()


def _close(y, want, bound, bf16=True):
    torch.cuda.synchronize()
    ops.workspace().check_status()
    bound = bound + (2.0 ** -8 * (want.abs() + bound) if bf16 else 2.0 ** -23 * want.abs())
    assert bool(((y.double() - want).abs() <= bound).all())


def _pair_only(monkeypatch):
    """Every product of this test, whatever its rows, has to take the kernel under test."""
    monkeypatch.setattr(F, "pair_gemm_ok", lambda p, rows: True)
    monkeypatch.setattr(_lib.lib(), "skein_gemm_ws", None)


# one row; a tile less one, whole, and one more; features that end inside a CTA's rows; K that ends inside a block; cut tiles (few tiles, long K); several
# rounds; whole rounds behind cut tiles
@pytest.mark.parametrize("rows,features,K", [(1, 256, 256), (255, 512, 512), (256, 256, 512), (257, 384, 1024), (300, 1000, 1032), (96, 264, 4096),
                                             (2304, 2304, 256), (2400, 2048, 1024)])
@pytest.mark.parametrize("unit", [False, True])
@pytest.mark.parametrize("packed", [False, True])
def test_tiles(monkeypatch, rows, features, K, unit, packed):
    _pair_only(monkeypatch)
    if packed and (features % 128 or K % 64):
        features, K = 384, 1024
    x, w = _inputs(rows, features * (2 if unit else 1), K)
    y = (ops.swiglu_linear if unit else ops.linear)(x, ops.pack_weight(w) if packed else w)
    _close(y, *(_unit if unit else _sum)(x, w))


# empty groups, groups of a row, groups that end inside a tile
@pytest.mark.parametrize("counts", [[300, 0, 513, 1], [0, 0, 64, 0], [31, 33, 255, 257]])
@pytest.mark.parametrize("unit", [False, True])
def test_groups(monkeypatch, counts, unit):
    _pair_only(monkeypatch)
    cnt = torch.tensor(counts, dtype=torch.int32, device=DEV)
    off = torch.cat([cnt.new_zeros(1), cnt.cumsum(0).int()])
    x, w = _inputs(sum(counts), 640 * (2 if unit else 1), 512, lead=(len(counts),))
    y = ops.grouped_linear(x, w, cnt, off, swiglu=unit)
    for i, n in enumerate(counts):
        at = slice(int(off[i]), int(off[i]) + n)
        _close(y[at], *(_unit if unit else _sum)(x[at], w[i]))


@pytest.mark.parametrize("rows,features,K", [(300, 2048, 2048), (2304, 2304, 256)])       # cut tiles; whole ones
def test_epilogues(monkeypatch, rows, features, K):
    _pair_only(monkeypatch)
    x, w = _inputs(rows, features, K)
    want, bound = _sum(x, w)
    res = torch.randn(rows, features, device=DEV)
    total = res.clone()
    ops.linear(x, w, out=total, residual=total, out_f32=True)                    # in place
    _close(total, want + res.double(), bound, bf16=False)
    _close(ops.linear(x, w, out_f32=True), want, bound, bf16=False)
    half = res.bfloat16()
    _close(ops.linear(x, w, residual=half), want + half.double(), bound)
    cols = features // 2 + 1
    sq = want.clone()
    sq[:, :cols] = sq[:, :cols].clamp(min=0).square()
    _close(ops.linear(x, w, relu2_cols=cols), sq, (2 * want.abs() + bound + 1) * bound)
    wide = torch.zeros(rows, features + 3, dtype=torch.bfloat16, device=DEV)     # rows that are not a multiple of 4 bytes apart
    _close(ops.linear(x, w, out=wide[:, 1:1 + features]), want, bound)
    assert bool((wide[:, 0] == 0).all()) and bool((wide[:, 1 + features:] == 0).all())
    strided = torch.randn(rows, K + 64, device=DEV).bfloat16()
    _close(ops.linear(strided[:, :K], w), *_sum(strided[:, :K], w))


def test_repeats_are_bitwise_alike(monkeypatch):
    _pair_only(monkeypatch)
    x, w = _inputs(300, 2048, 4096)
    assert torch.equal(ops.linear(x, w), ops.linear(x, w))


@pytest.mark.parametrize("rows,features,K", [(300, 2048, 2048), (2304, 2304, 256), (257, 1000, 1032)])       # cut tiles; whole ones; features inside a CTA's rows
def test_residuals_in_place_and_rows_of_any_pitch(monkeypatch, rows, features, K):
    _pair_only(monkeypatch)
    x, w = _inputs(rows, features, K)
    want, bound = _sum(x, w)
    half = torch.randn(rows, features, device=DEV).bfloat16()
    total = half.clone()
    ops.linear(x, w, out=total, residual=total)
    _close(total, want + half.double(), bound)
    for pitch, first in ((8, 4), (3, 1), (2, 2)):                                # whole 16-byte groups; single values; pairs, that are no groups of four
        for dtype in (torch.float32, torch.bfloat16):
            wide = torch.randn(rows, features + pitch, device=DEV).to(dtype)
            before, cols = wide.clone(), slice(first, first + features)
            ops.linear(x, w, out=wide[:, cols], residual=wide[:, cols], out_f32=dtype == torch.float32, relu2_cols=features // 2 + 3)
            sq = want.clone()
            sq[:, :features // 2 + 3] = sq[:, :features // 2 + 3].clamp(min=0).square()
            _close(wide[:, cols], sq + before[:, cols].double(), (2 * want.abs() + bound + 1) * bound, bf16=dtype == torch.bfloat16)
            wide[:, cols] = before[:, cols]
            assert torch.equal(wide, before)


@pytest.mark.parametrize("rows,features,K", [(1000, 2304, 4096), (2100, 2304, 14336), (1000, 4096, 22528), (300, 512, 2048)])
def test_sums_in_32_bits_are_as_good_as_the_streaming_kernels(monkeypatch, rows, features, K):
    """The tensor core's fp32 sums lose with the length of the chain: outputs kept in 32 bits must not be further off than the kernel that cuts K."""
    x, w = _inputs(rows, features, K)
    want = _sum(x, w)[0]
    monkeypatch.setattr(F, "pair_gemm_ok", lambda p, rows: False)
    off = (ops.linear(x, w, out_f32=True).double() - want).norm()
    _pair_only(monkeypatch)
    y = ops.linear(x, w, out_f32=True)
    res = torch.randn(rows, features, device=DEV)
    total = ops.linear(x, w, out=res.clone(), residual=res, out_f32=True)
    torch.cuda.synchronize()
    ops.workspace().check_status()
    assert (y.double() - want).norm() <= 1.02 * off
    assert torch.equal(total, y + res) and torch.equal(y, ops.linear(x, w, out_f32=True))


def _clamped(x, w, limit, slope):
    """min(g, limit) sigmoid(slope g) (clamp(u, +-limit) + 1): clamping does not widen an error, z sigmoid(slope z) has a slope of at most 1.1 whatever `slope` is."""
    (g, eg), (u, eu) = (_sum(x, h) for h in w.chunk(2))
    g, u = g.clamp(max=limit), u.clamp(-limit, limit) + 1
    s = g * torch.sigmoid(slope * g)
    return s * u, (1.1 * eg + 2.0 ** -20 * s.abs()) * (u.abs() + eu) + (s.abs() + 1.1 * eg) * eu + 2.0 ** -22 * s.abs()


# cut tiles and whole ones; limits that clamp many values and few
@pytest.mark.parametrize("rows,features,K", [(300, 512, 2048), (2304, 2304, 256)])
@pytest.mark.parametrize("limit,slope", [(0.5, 1.702), (7.0, 1.0)])
def test_clamped_unit(monkeypatch, rows, features, K, limit, slope):
    _pair_only(monkeypatch)
    x, w = _inputs(rows, 2 * features, K)
    _close(ops.swiglu_linear(x, w, glu=(limit, slope)), *_clamped(x, w, limit, slope))
    cnt = torch.tensor([rows - 40, 0, 40], dtype=torch.int32, device=DEV)
    off = torch.cat([cnt.new_zeros(1), cnt.cumsum(0).int()])
    stack = torch.stack([w, w, -w])
    y = ops.grouped_linear(x, stack, cnt, off, swiglu=True, glu=(limit, slope))
    for i, at in ((0, slice(0, rows - 40)), (2, slice(rows - 40, rows))):
        _close(y[at], *_clamped(x[at], stack[i], limit, slope))


# an average that sends the product to the pairs, whatever the groups are: one with all rows, most of them empty, tiny ones beside a large one
@pytest.mark.parametrize("counts", [[2048, 0, 0, 0, 0, 0, 0, 0], [0, 0, 1, 1990, 0, 57, 0, 0], [3, 700, 5, 0, 650, 1, 689, 0]])
@pytest.mark.parametrize("unit", [False, True])
def test_uneven_groups_by_their_average(monkeypatch, counts, unit):
    monkeypatch.setattr(_lib.lib(), "skein_gemm_ws", None)          # the rule itself has to choose the pairs
    features, K = (512, 512) if unit else (8192, 1536)
    cnt = torch.tensor(counts, dtype=torch.int32, device=DEV)
    off = torch.cat([cnt.new_zeros(1), cnt.cumsum(0).int()])
    x, w = _inputs(sum(counts), features * (2 if unit else 1), K, lead=(8,))
    y = ops.grouped_linear(x, w, cnt, off, swiglu=unit, rows_hint=2048)
    for i, n in enumerate(counts):
        at = slice(int(off[i]), int(off[i]) + n)
        _close(y[at], *(_unit if unit else _sum)(x[at], w[i]))


@pytest.mark.parametrize("rows,kernel", [(191, "skein_gemm_pair"), (192, "skein_gemm_ws"), (256, "skein_gemm_ws"), (257, "skein_gemm_pair"), (4200, "skein_gemm_ws")])
def test_rule_at_its_edges(monkeypatch, rows, kernel):
    """1024 features, K of 4096: the kernel that must not run is not there."""
    monkeypatch.setattr(_lib.lib(), kernel, None)
    x, w = _inputs(rows, 1024, 4096)
    _close(ops.linear(x, w), *_sum(x, w))
