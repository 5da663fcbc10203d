"""Every kernel the block-FP8 GEMM chooses from, at the sizes where it can go wrong, against an FP64
product of the dequantized operands. Bound: one rounding of the output type plus the error of the FP32
sums, which was at most 3.6e-7 of the largest value (K up to 18432);
SUM_ERROR allows four times that."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 0.0}
SUM_ERROR = 1.5e-6


def _check(m, n, k, dtype, *, bias=False, ldc=None, alpha=None):
    from sparkinfer_b200._lib import launch

    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(m * 7 + n + k)
    a = torch.randint(0, 256, (m, k), dtype=torch.uint8, device=dev, generator=gen) & 0xBF
    b = torch.randint(0, 256, (n, k), dtype=torch.uint8, device=dev, generator=gen) & 0xBF
    sa = torch.rand((m, k // 128), device=dev, generator=gen) + 0.25
    sb = torch.rand((n // 128, k // 128), device=dev, generator=gen) + 0.25
    store = torch.full((m, ldc or n), float("nan"), dtype=dtype, device=dev)
    vec = (torch.randn(n, device=dev, generator=gen) * 64).to(dtype) if bias else None
    scale = torch.tensor([alpha], device=dev) if alpha is not None else None
    launch.gemm_block_fp8(a, sa, b, sb, store, scale, m, n, k, ldc=ldc, bias=vec)
    torch.cuda.synchronize()
    launch.check_kernel_status(dev)
    a_deq = a.view(torch.float8_e4m3fn).double() * sa.double().repeat_interleave(128, dim=1)
    b_deq = (b.view(torch.float8_e4m3fn).double()
             * sb.double().repeat_interleave(128, dim=0).repeat_interleave(128, dim=1))
    ref = a_deq @ b_deq.T * (alpha if alpha is not None else 1.0)
    bound = (EPS[dtype] + SUM_ERROR) * float(ref.abs().max())
    if bias:
        ref = ref + vec.double()
        bound = 2 * (EPS[dtype] + SUM_ERROR) * float(ref.abs().max())
    got = store[:, :n].double()
    assert not torch.isnan(got).any()
    assert float((got - ref).abs().max()) <= bound
    assert bool(torch.isnan(store[:, n:]).all())       # nothing beyond the output columns


# Weight-streaming kernel: every padded row count and its edges; one CTA per tile, clusters of
# two to eight (k-blocks fewer than, equal to and not a multiple of the cluster), more tiles
# than SMs (up to 64 rows; with more, 151 tiles belong to the tiled kernel).
@pytest.mark.parametrize("m", [1, 16, 17, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("n,k", [(128, 128), (1152, 1152), (2176, 896), (4096, 640), (128 * 151, 256)])
def test_few_rows(m, n, k):
    _check(m, n, k, torch.bfloat16)


# The same kernel where its rings come round: 72 k-blocks for each CTA of a cluster of two (operand
# stages, scale slots of eight k-blocks and tensor-memory buffers all several times), 37 k-blocks on one
# CTA (a partial batch of scales behind full ones), and up to three tiles of 13 k-blocks one after the
# other (a tile starts in the middle of every ring). With more than 64 rows there is no shape of the
# last kind: as many tiles as that go to the tiled kernel.
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("m", [1, 16, 17, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("n,k", [(7168, 18432), (9600, 128 * 37), (128 * 300, 128 * 13)])
def test_few_rows_around_the_rings(m, n, k, dtype):
    if m > 64 and n == 128 * 300:
        pytest.skip("runs the tiled kernel")
    _check(m, n, k, dtype)


@pytest.mark.parametrize("m,dtype,kwargs", [
    (5, torch.float32, {}), (40, torch.float32, {"bias": True}), (7, torch.float16, {"bias": True}),
    (9, torch.bfloat16, {"ldc": 1160}), (9, torch.bfloat16, {"ldc": 1157}),
    (100, torch.float16, {"alpha": 0.125}), (100, torch.bfloat16, {"bias": True, "ldc": 1153})])
def test_few_rows_epilogues(m, dtype, kwargs):
    _check(m, 1152, 1152, dtype, **kwargs)


# CTA-pair kernel (M > 128, K >= 3072, no more rounds than the single-CTA kernel): a last row tile
# of one row, of one CTA of the pair and full; N with half a column tile; scale batches of eight
# k-blocks with and without a remainder; more than one tile per pair.
@pytest.mark.parametrize("m,n,k", [(129, 256, 3072), (257, 128, 3200), (384, 384, 3968),
                                   (512, 1152, 4096), (1100, 9600, 3072), (2304, 4352, 3328)])
def test_pair_tiles(m, n, k):
    _check(m, n, k, torch.bfloat16)


@pytest.mark.parametrize("dtype,kwargs", [
    (torch.float32, {}), (torch.float32, {"bias": True}), (torch.float16, {"bias": True}),
    (torch.bfloat16, {"ldc": 1160}), (torch.bfloat16, {"ldc": 1157, "bias": True}),
    (torch.float16, {"alpha": 0.125})])
def test_pair_epilogues(dtype, kwargs):
    _check(390, 1152, 3200, dtype, **kwargs)


# Neighbours of the rule's lines run the single-CTA kernel.
@pytest.mark.parametrize("m,n,k", [(129, 256, 2944), (640, 7168, 3072)])
def test_beside_the_pair_rule(m, n, k):
    _check(m, n, k, torch.bfloat16)
