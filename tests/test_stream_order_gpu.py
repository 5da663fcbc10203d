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
