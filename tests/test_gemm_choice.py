"""Which kernel a product of many rows takes (functional.pair_gemm_ok): sizes at which each of the two was measured to be the quicker one."""
from types import SimpleNamespace

import pytest

from skein_b200.ops import functional as F


def _p(F_, K, G=1, unit=False, f32=False, residual=0):
    return SimpleNamespace(F=F_, K=K, G=G, mode=int(unit), out_f32=int(f32), residual=residual)


# served shapes at prefill sizes: projections, experts, heads, the products of parallel layers
@pytest.mark.parametrize("p,rows", [(_p(6144, 4096), 2048), (_p(4096, 4096), 1000), (_p(10240, 8192), 320), (_p(4096, 14336), 512), (_p(4608, 3584), 2600),
                                    (_p(3584, 18944), 2600), (_p(14336, 4096, unit=True), 128), (_p(2048, 2048, unit=True), 96), (_p(14336, 4096, 8, True), 128),
                                    (_p(4096, 14336, 8), 192), (_p(2048, 2048, 8), 400), (_p(64 * 22, 2048, 64), 128), (_p(4096, 22528, f32=True), 1000),
                                    (_p(4096, 8192, f32=True), 4000), (_p(4096, 4096, residual=1), 2048), (_p(1024, 1024), 192)])
def test_pairs(p, rows):
    assert F.pair_gemm_ok(p, rows)


# few rows, short rows of weights, few tiles, small groups, 32-bit outputs whose epilogue is not covered
@pytest.mark.parametrize("p,rows", [(_p(14336, 4096, unit=True), 96), (_p(14336, 4096, 8, True), 96), (_p(512, 1024, 64, True), 128), (_p(1024, 1024, 2, True), 256),
                                    (_p(512, 1024, 64), 512), (_p(2048, 2048, 8), 256), (_p(256, 256, 16), 512), (_p(4096, 1792, 8), 512), (_p(4096, 4096, 2), 512),
                                    (_p(4096, 4096), 192), (_p(8192, 8192), 256), (_p(4096, 14336), 200), (_p(32000, 4096), 192), (_p(256, 256), 4096),
                                    (_p(8192, 512), 3000), (_p(4096, 1024), 4096), (_p(2048, 2048), 1500), (_p(4608, 3584), 1000), (_p(6144, 4096), 512),
                                    (_p(4096, 4096, f32=True), 2048), (_p(2048, 2048, f32=True), 1000), (_p(4096, 512, f32=True), 4096), (_p(128, 4096), 4096)])
def test_streaming(p, rows):
    assert not F.pair_gemm_ok(p, rows)
