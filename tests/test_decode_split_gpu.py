"""How the decode GEMM divides its weight tiles over CTAs: whole tiles, tiles cut between
neighbours, several CTAs per tile. FP32 outputs of the decode kernel against the tiled kernel on the
same operands: both sum the same products in FP32, so they differ by at most 2 * K * 2^-24 of the sum
of magnitudes, which for these operands is below sqrt(K) times the largest result."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _operand(kind, rows, k, gen):
    fp4 = kind == 1
    codes = torch.randint(0, 256, (rows, k // 2 if fp4 else k), dtype=torch.uint8, device=DEV,
                          generator=gen) & (0xFF if fp4 else 0xBF)
    atoms = -(-rows // 128) * -(-k // (64 if fp4 else 128)) * 512
    scales = torch.randint(40 if fp4 else 124, 60 if fp4 else 131, (atoms,), dtype=torch.uint8,
                           device=DEV, generator=gen)
    return codes, scales


# 1, 8, 37, 74, 75 tiles (several CTAs per tile, two, one), 148 and 149, 222 and 297 tiles (one and two
# rounds, the last one empty, nearly empty and half full); K of one and of many 128-byte steps.
@pytest.mark.parametrize("m", [1, 16, 17, 33, 64])
@pytest.mark.parametrize("tiles", [1, 8, 37, 74, 75, 148, 149, 222, 297])
@pytest.mark.parametrize("kind,k", [(0, 128), (0, 1184), (0, 6144), (1, 256), (1, 2112), (1, 9216)])
def test_decode_split(m, tiles, kind, k):
    from sparkinfer_b200._lib import launch

    n = tiles * 128 - 8
    gen = torch.Generator(device=DEV).manual_seed(m * 1000 + tiles + k)
    a, sfa = _operand(kind, m, k, gen)
    b, sfb = _operand(kind, n, k, gen)
    outs = []
    for small in (True, False):
        c = torch.full((m, n), float("nan"), dtype=torch.float32, device=DEV)
        launch.gemm_blockscaled(kind, a, sfa, b, sfb, c, None, m, n, k, small_m=small)
        outs.append(c)
    launch.check_kernel_status(DEV)
    got, ref = outs
    assert not torch.isnan(got).any()
    bound = 2.0 * k * 2.0 ** -24 * k ** 0.5 * float(ref.abs().max())
    assert float((got - ref).abs().max()) <= bound
