"""How the decode GEMM divides its weight tiles over CTAs: whole tiles, tiles cut between
neighbours, several CTAs per tile; one problem and several groups; codes and scales given, or BF16 rows
quantized inside. FP32 outputs against an FP64 product of the dequantized operands."""

from __future__ import annotations

import pytest
import torch

from gpu_util import E2M1_LUT, unswizzle_atoms

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


def dequantized(kind, codes, scales, rows, k):
    """FP64 [rows, k] of MXFP8 (0), NVFP4 (1) or, without scales, plain FP8 operands: exact."""
    if kind == 1:
        lut = torch.tensor(E2M1_LUT, dtype=torch.float64, device=DEV)
        values = torch.stack((lut[(codes & 0xF).int()], lut[(codes >> 4).int()]), dim=-1).view(rows, k)
        scale = unswizzle_atoms(scales, rows, k // 16).view(torch.float8_e4m3fn).double()
        return (values.view(rows, k // 16, 16) * scale[:, :, None]).view(rows, k)
    values = codes.view(torch.float8_e4m3fn).double()
    if scales is None:
        return values
    scale = torch.exp2(unswizzle_atoms(scales, rows, k // 32).double() - 127)
    return (values.view(rows, k // 32, 32) * scale[:, :, None]).view(rows, k)


def assert_fp32_sums(got, ref):
    """FP32 sums of exact products. Seen over the kernels and shapes that use this (MXFP8, K up to
    7168): at most 4.2e-6 of the largest result and 3.2e-6 in the 2-norm (NVFP4 with these scales is
    exact); four times that is allowed. A lost block of 32 elements moves a result by
    about a hundredth of the largest one at these K, a wrong scale byte by half of that or more."""
    assert not torch.isnan(got).any()
    error = got.double() - ref
    assert float(error.abs().max()) <= 1.7e-5 * float(ref.abs().max())
    assert float(error.norm()) <= 1.3e-5 * float(ref.norm())


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
    c = torch.full((m, n), float("nan"), dtype=torch.float32, device=DEV)
    launch.gemm_blockscaled(kind, a, sfa, b, sfb, c, None, m, n, k, small_m=True)
    launch.check_kernel_status(DEV)
    assert_fp32_sums(c, dequantized(kind, a, sfa, m, k) @ dequantized(kind, b, sfb, n, k).T)


# Groups: the tiles of all groups form one list, so a CTA range crosses from one group into the next.
@pytest.mark.parametrize("m,groups,tiles", [(1, 2, 4), (16, 3, 25), (17, 2, 74), (64, 3, 50), (33, 2, 111)])
@pytest.mark.parametrize("kind,k", [(0, 1184), (0, 6144), (1, 2112), (1, 9216)])
def test_decode_split_of_groups(m, groups, tiles, kind, k):
    from sparkinfer_b200._lib import launch

    n = tiles * 128 - 8
    gen = torch.Generator(device=DEV).manual_seed(m * 1000 + tiles + k)
    parts = [(*_operand(kind, m, k, gen), *_operand(kind, n, k, gen)) for _ in range(groups)]
    a, sfa, b, sfb = (torch.cat([p[i].reshape(-1) for p in parts]) for i in range(4))
    c = torch.full((groups, m, n), float("nan"), dtype=torch.float32, device=DEV)
    launch.gemm_blockscaled(kind, a, sfa, b, sfb, c, None, m, n, k, groups=groups, small_m=True)
    launch.check_kernel_status(DEV)
    for got, (a_g, sfa_g, b_g, sfb_g) in zip(c, parts):
        assert_fp32_sums(got, dequantized(kind, a_g, sfa_g, m, k) @ dequantized(kind, b_g, sfb_g, n, k).T)


# Fused activation quantizer: the same split, so the same bytes as the row quantizer and the GEMM on
# its codes (which the tests above hold against FP64).
@pytest.mark.parametrize("m", [1, 8, 9, 16])
@pytest.mark.parametrize("tiles", [1, 37, 75, 149, 222, 297])
@pytest.mark.parametrize("kind,k", [(0, 128), (0, 6144), (1, 256), (1, 9216)])
def test_decode_split_with_fused_quantizer(m, tiles, kind, k):
    from sparkinfer_b200._lib import launch

    n = tiles * 128 - 8
    gen = torch.Generator(device=DEV).manual_seed(m * 1000 + tiles + k)
    x = torch.randn((m, k), device=DEV, generator=gen).to(torch.bfloat16)
    b, sfb = _operand(kind, n, k, gen)
    gs = torch.tensor([300.0], device=DEV) if kind == 1 else None
    codes = torch.zeros((m, k // 2 if kind == 1 else k), dtype=torch.uint8, device=DEV)
    atoms = torch.zeros(-(-k // (64 if kind == 1 else 128)) * 512, dtype=torch.uint8, device=DEV)
    if kind == 1:
        launch.quantize_nvfp4_rows(x, gs, codes, atoms)
    else:
        launch.quantize_mxfp8_rows(x, codes, None, atoms)
    want = torch.full((m, n), float("nan"), dtype=torch.float32, device=DEV)
    got = want.clone()
    launch.gemm_blockscaled(kind, codes, atoms, b, sfb, want, None, m, n, k, small_m=True)
    launch.gemm_smallm_fused_quant(kind, x, gs, b, sfb, got, None, m, n, k)
    launch.check_kernel_status(DEV)
    assert not torch.isnan(got).any()
    assert torch.equal(got, want)
