"""Operands that the kernel launched just before has written, where that kernel releases its dependents
early. Each call is queued behind a busy stream, so that the two grids do overlap, and compared bit for
bit with the same call on an idle device."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
ROUNDS = 6          # other values in the same buffers each time, so that a stale read shows


def _codes(rows, k, gen):
    return torch.randint(0, 256, (rows, k), dtype=torch.uint8, device=DEV, generator=gen) & 0xBF


# The weight in slabs of 128 rows, each by a quantizer launch that releases early. One CTA per tile and
# clusters; 65 rows is the larger activation tile.
@pytest.mark.parametrize("m", [1, 24, 64, 65])
@pytest.mark.parametrize("n,k", [(256, 7168), (1152, 4096), (128 * 150, 512)])
def test_block_fp8_weight_written_just_before(m, n, k):
    from sparkinfer_b200._lib import launch

    gen = torch.Generator(device=DEV).manual_seed(m + n + k)
    a = _codes(m, k, gen)
    sa = torch.rand((m, k // 128), device=DEV, generator=gen) + 0.25
    sb = torch.rand((n // 128, k // 128), device=DEV, generator=gen) + 0.25
    b = torch.zeros((n, k), dtype=torch.uint8, device=DEV)
    sources = [torch.randn((n, k), device=DEV, generator=gen).to(torch.bfloat16) for _ in range(2)]

    def write(source):
        for r in range(0, n, 128):
            launch.quantize_mxfp8_rows(source[r:r + 128], b[r:r + 128], None, None)

    def multiply():
        out = torch.empty((m, n), dtype=torch.float32, device=DEV)
        launch.gemm_block_fp8(a, sa, b, sb, out, None, m, n, k)
        return out

    want = []
    for source in sources:
        write(source)
        torch.cuda.synchronize()
        want.append(multiply())
        torch.cuda.synchronize()
    got = []
    for i in range(ROUNDS):
        torch.cuda._sleep(2_000_000)
        write(sources[i % 2])
        got.append(multiply())
    launch.check_kernel_status(DEV)
    for i, out in enumerate(got):
        assert torch.equal(out, want[i % 2]), i


# The activation scales (FP32, [M, 128] for K = 16384) are the output of the GEMM launched just before,
# and so is the bias, the single row of a GEMM of one activation row. Both releases are early.
@pytest.mark.parametrize("m", [1, 24, 64, 65])
def test_block_fp8_scales_and_bias_written_just_before(m):
    from sparkinfer_b200._lib import launch

    n, k = 1152, 16384
    gen = torch.Generator(device=DEV).manual_seed(m)
    a, b = _codes(m, k, gen), _codes(n, k, gen)
    sb = torch.rand((n // 128, k // 128), device=DEV, generator=gen) + 0.25
    sa = torch.empty((m, k // 128), dtype=torch.float32, device=DEV)
    bias = torch.empty((1, n), dtype=torch.bfloat16, device=DEV)
    small = [_codes(rows, 512, gen) for rows in (m, k // 128, 1, n)]
    ones = [torch.ones((rows, 4), device=DEV) for rows in (m, 1)]
    weight_scales = [torch.rand((rows // 128, 4), device=DEV, generator=gen) for rows in (k // 128, n)]
    alphas = [torch.tensor([v], device=DEV) for v in (1.0, -0.5)]

    def write(alpha):
        launch.gemm_block_fp8(small[2], ones[1], small[3], weight_scales[1], bias, alpha, 1, n, 512)
        launch.gemm_block_fp8(small[0], ones[0], small[1], weight_scales[0], sa, alpha, m, k // 128, 512)

    def multiply():
        out = torch.empty((m, n), dtype=torch.bfloat16, device=DEV)
        launch.gemm_block_fp8(a, sa, b, sb, out, None, m, n, k, bias=bias[0])
        return out

    want = []
    for alpha in alphas:
        write(alpha)
        torch.cuda.synchronize()
        want.append(multiply())
        torch.cuda.synchronize()
    assert not torch.equal(*want)
    got = []
    for i in range(ROUNDS):
        torch.cuda._sleep(2_000_000)
        write(alphas[i % 2])
        got.append(multiply())
    launch.check_kernel_status(DEV)
    for i, out in enumerate(got):
        assert torch.equal(out, want[i % 2]), i


# The same for the bias of the block-scaled decode GEMM, on whole tiles and on tiles cut along K.
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,k", [(1032, 512), (640, 8192)])
def test_decode_bias_written_just_before(n, k, dtype):
    from sparkinfer_b200 import _native
    from sparkinfer_b200._lib import launch

    gen = torch.Generator(device=DEV).manual_seed(n + k)
    m = 7
    tiles, atoms = -(-n // 128), k // 128
    a, b, row = _codes(m, k, gen), _codes(n, k, gen), _codes(1, k, gen)
    sfa = torch.full((atoms * 512,), 127, dtype=torch.uint8, device=DEV)
    sfb = torch.full((tiles * atoms * 512,), 127, dtype=torch.uint8, device=DEV)
    bias = torch.empty((1, n), dtype=dtype, device=DEV)
    alphas = [torch.tensor([v], device=DEV) for v in (1.0, -0.5)]

    def write(alpha):
        launch.gemm_blockscaled(_native.KIND_MXFP8, row, sfa, b, sfb, bias, alpha, 1, n, k)

    def multiply():
        out = torch.empty((m, n), dtype=dtype, device=DEV)
        launch.gemm_blockscaled(_native.KIND_MXFP8, a, sfa, b, sfb, out, None, m, n, k, bias=bias[0])
        return out

    want = []
    for alpha in alphas:
        write(alpha)
        torch.cuda.synchronize()
        want.append(multiply())
        torch.cuda.synchronize()
    assert not torch.equal(*want)
    got = []
    for i in range(ROUNDS):
        torch.cuda._sleep(2_000_000)
        write(alphas[i % 2])
        got.append(multiply())
    launch.check_kernel_status(DEV)
    for i, out in enumerate(got):
        assert torch.equal(out, want[i % 2]), i


# The global scale of the NVFP4 row quantizer, one value of the output of the GEMM launched just before.
@pytest.mark.parametrize("m", [1, 100, 129])
def test_global_scale_written_just_before(m):
    from sparkinfer_b200._lib import launch

    k, width = 4096, 512
    gen = torch.Generator(device=DEV).manual_seed(m)
    x = torch.randn((m, k), device=DEV, generator=gen).to(torch.bfloat16)
    row, weight = (torch.full((rows, width), 0x38, dtype=torch.uint8, device=DEV) for rows in (1, 128))
    ones = torch.ones((1, width // 128), device=DEV)
    scale = torch.empty((1, 128), dtype=torch.float32, device=DEV)
    alphas = [torch.tensor([v], device=DEV) for v in (1.0, 0.25)]
    atoms = -(-m // 128) * (k // 64) * 512

    def write(alpha):   # 512 products of 1.0 each
        launch.gemm_block_fp8(row, ones, weight, ones, scale, alpha, 1, 128, width)

    def quantize():
        codes = torch.empty((m, k // 2), dtype=torch.uint8, device=DEV)
        scales = torch.empty(atoms, dtype=torch.uint8, device=DEV)
        launch.quantize_nvfp4_rows(x, scale[0, :1], codes, scales)
        return codes, scales

    want = []
    for alpha in alphas:
        write(alpha)
        torch.cuda.synchronize()
        want.append(quantize())
        torch.cuda.synchronize()
    assert float(scale[0, 0]) == 128.0 and not torch.equal(want[0][1], want[1][1])
    got = []
    for i in range(ROUNDS):
        torch.cuda._sleep(2_000_000)
        write(alphas[i % 2])
        got.append(quantize())
    launch.check_kernel_status(DEV)
    for i, (codes, scales) in enumerate(got):
        assert torch.equal(codes, want[i % 2][0]) and torch.equal(scales, want[i % 2][1]), i
