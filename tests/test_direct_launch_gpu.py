"""Linears called eagerly go straight to the launcher; whatever listens to operators still gets the
registered custom op. Both routes run the same kernels, so their results are equal bit for bit."""

from __future__ import annotations

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


class Recorder(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.names = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.names.append(str(func))
        return func(*args, **(kwargs or {}))


def _linear(which, k, n=256, dtype=torch.bfloat16):
    from sparkinfer_b200.gemm import mxfp8_linear, tensor_fp8_linear

    gen = torch.Generator(device=DEV).manual_seed(k)
    w = torch.randn((n, k), device=DEV, generator=gen).to(torch.float8_e4m3fn)
    if which == "mxfp8":
        scale = torch.randint(120, 130, (n, k // 32), dtype=torch.uint8, device=DEV, generator=gen)
        packed = mxfp8_linear.pack_weight(w, scale)
        return (lambda x, b: mxfp8_linear.mm(x, packed, bias=b)), dtype
    packed = tensor_fp8_linear.pack_weight(w, torch.full((1,), 0.5, device=DEV))
    return ((lambda x, b: tensor_fp8_linear.mm(x, packed, bias=b, out_dtype=dtype)),
            torch.float8_e4m3fn)


# M on both sides of the decode kernel's range, K inside and at the edge of a 128-element step.
@pytest.mark.parametrize("which", ["mxfp8", "tensor_fp8"])
@pytest.mark.parametrize("m,k", [(1, 256), (5, 288), (64, 352), (65, 160), (300, 512)])
@pytest.mark.parametrize("bias", ["none", "fused", "unfused"])
def test_direct_route_equals_the_custom_op(which, m, k, bias):
    run, source_dtype = _linear(which, k)
    gen = torch.Generator(device=DEV).manual_seed(m)
    x = torch.randn((m, k), device=DEV, generator=gen).to(source_dtype)
    b = None if bias == "none" else torch.randn(256, device=DEV, generator=gen).to(torch.bfloat16)
    if bias == "unfused":
        if which == "tensor_fp8":
            pytest.skip("takes a bias of the output dtype only")
        b = b.float()
    direct = run(x, b)
    with Recorder() as mode:
        listened = run(x, b)
    assert any("b12x" in name for name in mode.names)
    assert direct.shape == (m, 256) and direct.dtype == listened.dtype
    assert torch.equal(direct, listened)
    batched = run(x.view(1, m, k), b)
    assert batched.shape == (1, m, 256) and torch.equal(batched[0], direct)


def test_a_source_that_needs_gradients_keeps_the_op_route():
    run, _ = _linear("mxfp8", 256)
    x = torch.randn((3, 256), device=DEV, dtype=torch.bfloat16)
    plain = run(x, None)
    assert not plain.requires_grad
    tracked = run(x.clone().requires_grad_(), None)
    assert tracked.requires_grad and torch.equal(tracked.detach(), plain)
    with torch.no_grad():
        assert not run(x.clone().requires_grad_(), None).requires_grad


# Ragged K without a padded copy: rows that start on and off a 16-byte boundary, K beside and inside
# a 128-element step, on the decode and the tiled kernels.
@pytest.mark.parametrize("which", ["mxfp8", "tensor_fp8"])
@pytest.mark.parametrize("m,k", [(3, 32), (40, 96), (40, 2080), (100, 160), (300, 1056)])
def test_ragged_k_on_any_alignment(which, m, k):
    run, source_dtype = _linear(which, k)
    gen = torch.Generator(device=DEV).manual_seed(m + k)
    x = torch.randn((m, k), device=DEV, generator=gen).to(source_dtype)
    shifted = torch.empty(m * k + 1, dtype=source_dtype, device=DEV)[1:].view(m, k)
    shifted.copy_(x)
    assert shifted.data_ptr() % 16 != 0
    assert torch.equal(run(x, None), run(shifted, None))


def test_the_switch_and_the_profiler_see_the_op(monkeypatch):
    from sparkinfer_b200._lib import launch
    from sparkinfer_b200.gemm.mxfp8_linear import _kernel

    run, _ = _linear("mxfp8", 288)
    x = torch.randn((5, 288), device=DEV, dtype=torch.bfloat16)
    direct = run(x, None)
    calls = []
    forward = _kernel._forward
    monkeypatch.setattr(_kernel, "_forward", lambda *a, **k: calls.append(k) or forward(*a, **k))
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        profiled = run(x, None)
    assert any("b12x::mxfp8_linear" in event.name for event in prof.events())
    monkeypatch.setattr(launch, "DIRECT_LAUNCH", False)
    switched = run(x, None)
    assert len(calls) == 2
    assert torch.equal(profiled, direct) and torch.equal(switched, direct)


@pytest.mark.parametrize("small", [True, False])
def test_a_refused_weight_pitch_names_its_entry_point(small):
    from sparkinfer_b200 import _native
    from sparkinfer_b200._lib import launch

    a, b = (torch.zeros((rows, 104), dtype=torch.uint8, device=DEV) for rows in (4, 128))
    sf = torch.full((512,), 127, dtype=torch.uint8, device=DEV)
    out = torch.zeros((4, 128), dtype=torch.bfloat16, device=DEV)
    with pytest.raises(_native.NativeLibraryError, match="b12x_b200_gemm_linear"):
        launch.gemm_blockscaled(_native.KIND_MXFP8, a, sf, b, sf, out, None, 4, 128, 96, ldb=104,
                                small_m=small)
