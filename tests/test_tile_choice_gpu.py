"""The tile an unforced GEMM gets (single-CTA widths 64 to 256, CTA pair with and without split
leftover tiles): FP32 outputs of the unforced call and of every forced tile against an FP64 product of
the dequantized operands."""

from __future__ import annotations

import pytest
import torch

from sparkinfer_b200 import _native
from test_decode_split_gpu import DEV, _operand, assert_fp32_sums, dequantized

pytestmark = pytest.mark.gpu


# Few rows against a wide weight, short and long K, one and several rounds, ragged edges, and
# shapes whose leftover pair tiles are split along K (80, 78 and 75 pair tiles on 74 pairs).
@pytest.mark.parametrize("m,n,k", [
    (65, 640, 512), (81, 37768, 512), (128, 4096, 4096), (129, 2000, 800), (300, 18432, 1024),
    (1100, 920, 7168), (3353, 1280, 1024), (2048, 2560, 2048), (1536, 3328, 1024), (256, 19200, 1024)])
@pytest.mark.parametrize("kind", [_native.KIND_MXFP8, _native.KIND_NVFP4, _native.KIND_FP8])
@pytest.mark.parametrize("groups", [1, 2])
def test_tiles_agree(kind, m, n, k, groups):
    from sparkinfer_b200._lib import launch

    if groups == 2 and m > 1000:
        pytest.skip("one size of group is enough for the large shapes")
    gen = torch.Generator(device=DEV).manual_seed(m + n + k)
    parts = [(_operand(kind, m, k, gen), _operand(kind, n, k, gen)) for _ in range(groups)]
    a, sfa, b, sfb = (torch.cat([p[i][j].reshape(-1) for p in parts]) for i in (0, 1) for j in (0, 1))
    scales = (None, None) if kind == _native.KIND_FP8 else (sfa, sfb)
    outs = {}
    for block_n in (128, 0, 64, 192, 256, _native.BLOCK_N_PAIR):
        c = torch.full((groups, m, n), float("nan"), dtype=torch.float32, device=DEV)
        launch.gemm_blockscaled(kind, a, scales[0], b, scales[1], c, None, m, n, k, groups=groups,
                                block_n=block_n, small_m=False)
        outs[block_n] = c
    launch.check_kernel_status(DEV)
    for g, ((a_g, sfa_g), (b_g, sfb_g)) in enumerate(parts):
        if kind == _native.KIND_FP8:
            sfa_g = sfb_g = None
        ref = dequantized(kind, a_g, sfa_g, m, k) @ dequantized(kind, b_g, sfb_g, n, k).T
        for c in outs.values():
            assert_fp32_sums(c[g], ref)


# The split of the leftover pair tiles itself, whatever tile the unforced call takes: twice the same
# bytes (the partials are added in a fixed order), and the counters back at zero.
@pytest.mark.parametrize("kind,m,n,k", [
    (_native.KIND_NVFP4, 2048, 2560, 2048), (_native.KIND_MXFP8, 1536, 3328, 1024),
    (_native.KIND_NVFP4, 2000, 2500, 1536), (_native.KIND_FP8, 1792, 2816, 1024),
    (_native.KIND_NVFP4, 256, 19200, 1024)])
def test_split_leftover_tiles_repeat(kind, m, n, k):
    from sparkinfer_b200._lib import launch

    need = _native.load().b12x_b200_gemm_blockscaled_workspace_bytes(
        kind, m, n, k, _native.BLOCK_N_PAIR, 0)
    assert need > 0
    gen = torch.Generator(device=DEV).manual_seed(m + n)
    a, sfa = _operand(kind, m, k, gen)
    b, sfb = _operand(kind, n, k, gen)
    if kind == _native.KIND_FP8:
        sfa = sfb = None
    outs = []
    for _ in range(2):
        c = torch.full((m, n), float("nan"), dtype=torch.float32, device=DEV)
        launch.gemm_blockscaled(kind, a, sfa, b, sfb, c, None, m, n, k, block_n=_native.BLOCK_N_PAIR)
        outs.append(c)
    launch.check_kernel_status(DEV)
    assert torch.equal(outs[0], outs[1])
    assert_fp32_sums(outs[0], dequantized(kind, a, sfa, m, k) @ dequantized(kind, b, sfb, n, k).T)
    assert int(launch.stream_workspace(need, DEV)[:65536].count_nonzero()) == 0


# The plain entry point brings no scratch: 80 pair tiles on 74 pairs are then two whole rounds, and the
# same problem runs single-CTA tiles (first two shapes); with 448 tiles the pair kernel runs unsplit.
@pytest.mark.parametrize("kind,m,n,k", [
    (_native.KIND_MXFP8, 2048, 2560, 4096), (_native.KIND_NVFP4, 2040, 2568, 7168),
    (_native.KIND_NVFP4, 4096, 7168, 4608)])
def test_a_call_without_scratch(kind, m, n, k):
    import ctypes

    from sparkinfer_b200._lib import launch

    lib = _native.load()
    assert lib.b12x_b200_gemm_blockscaled_workspace_bytes(kind, m, n, k, 0, 0) > 0
    gen = torch.Generator(device=DEV).manual_seed(k)
    a, sfa = _operand(kind, m, k, gen)
    b, sfb = _operand(kind, n, k, gen)
    got = torch.full((m, n), float("nan"), dtype=torch.float32, device=DEV)
    status = torch.zeros(4, dtype=torch.int32, device=DEV)
    rc = lib.b12x_b200_gemm_blockscaled(
        kind, a.data_ptr(), sfa.data_ptr(), b.data_ptr(), sfb.data_ptr(), got.data_ptr(),
        _native.DT_FP32, None, m, n, k, n, 0, 0, status.data_ptr(),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    _native.check(rc, "b12x_b200_gemm_blockscaled")
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    assert_fp32_sums(got, dequantized(kind, a, sfa, m, k) @ dequantized(kind, b, sfb, n, k).T)
