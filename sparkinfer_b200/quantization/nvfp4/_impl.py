"""Host side of the NVFP4 row quantizer: shape plans, output storage, launch validation.

Counterpart of b12x/quantization/nvfp4/_impl.py:32-224. The reference compiles one kernel
per (M, K) and requires both to be multiples of 128; the ahead-of-time kernel here takes
any M >= 1 (it covers the padded scale rows itself) and K % 64 == 0.
"""

from __future__ import annotations

from dataclasses import dataclass
from typing import Callable

import torch

from ..._lib import launch as _launch
from ..._lib.layout import align_up, convert_sf_to_mma_layout

_SF_VEC_SIZE = 16
_K_ALIGN = 64


def _validate_shape(m: int, k: int) -> None:
    if m <= 0 or k <= 0:
        raise ValueError(f"M and K must be positive, got M={m}, K={k}")
    if k % _K_ALIGN != 0:
        raise ValueError(f"K must be a multiple of {_K_ALIGN}, got K={k}")


def _validate_launch_tensor(tensor: torch.Tensor, *, name: str, dtype: torch.dtype,
                            shape: tuple[int, ...], index: int) -> int:
    """Address of the tensor's first byte, after the checks every operand has to pass."""
    if tensor.dtype != dtype:
        raise ValueError(f"{name} must have dtype {dtype}, got {tensor.dtype}")
    if tensor.shape != shape:
        raise ValueError(f"{name} must have shape {shape}, got {tuple(tensor.shape)}")
    if not tensor.is_cuda or tensor.get_device() != index:
        raise ValueError(f"{name} must be on cuda:{max(index, 0)}, got {tensor.device}")
    if not tensor.is_contiguous():
        raise ValueError(f"{name} must be contiguous")
    return tensor.data_ptr()


def _overlaps(a0: int, a_bytes: int, b0: int, b_bytes: int) -> bool:
    return a0 < b0 + b_bytes and b0 < a0 + a_bytes


def scale_storage_numel(m: int, k: int) -> int:
    return align_up(m, 128) * align_up(k // _SF_VEC_SIZE, 4)


@dataclass
class BF16ToFP4TMAOutputs:
    """Packed codes ``(1, M, K/2)`` u8 and flat MMA-layout scale bytes."""

    packed_a_storage: torch.Tensor
    scale_storage: torch.Tensor

    @property
    def packed_a_flat(self) -> torch.Tensor:
        return self.packed_a_storage.view(-1)

    @property
    def scale_flat(self) -> torch.Tensor:
        return self.scale_storage.view(-1)

    @property
    def packed_a_view(self) -> torch.Tensor:
        """``[M, K/2, 1]`` view, the ``A`` operand ``gemm.blockscaled.mm`` expects."""
        return self.packed_a_storage.permute(1, 2, 0)

    def scale_mma_view(self, m: int, k: int) -> torch.Tensor:
        """6-D ``(32, 4, m_tiles, 4, k_tiles, 1)`` view of the scale bytes."""
        return convert_sf_to_mma_layout(self.scale_storage, m, k, 1, _SF_VEC_SIZE)


def allocate_bf16_to_fp4_tma_outputs(m: int, k: int, *,
                                     device: torch.device = torch.device("cuda")) -> BF16ToFP4TMAOutputs:
    _validate_shape(m, k)
    return BF16ToFP4TMAOutputs(
        packed_a_storage=torch.zeros(1, m, k // 2, dtype=torch.uint8, device=device),
        scale_storage=torch.zeros(scale_storage_numel(m, k), dtype=torch.uint8, device=device),
    )


def compile_bf16_to_fp4_tma(m: int, k: int) -> Callable[..., None]:
    """Return ``launch(bf16_input, global_scale, packed_a_flat, scale_flat)`` for (m, k).

    Nothing is compiled at run time; the callable validates its arguments like the
    reference's launcher (dtype, shape, device, contiguity, no overlap) and enqueues the
    kernel on torch's current stream.
    """
    _validate_shape(m, k)
    scale_numel = scale_storage_numel(m, k)
    packed_numel = m * k // 2

    def launch(bf16_input, global_scale, packed_a_flat, scale_flat):
        index = bf16_input.get_device()
        x = _validate_launch_tensor(bf16_input, name="bf16_input", dtype=torch.bfloat16,
                                    shape=(m, k), index=index)
        gs = _validate_launch_tensor(global_scale, name="global_scale", dtype=torch.float32,
                                     shape=(1,), index=index)
        codes = _validate_launch_tensor(packed_a_flat, name="packed_a_flat", dtype=torch.uint8,
                                        shape=(packed_numel,), index=index)
        scales = _validate_launch_tensor(scale_flat, name="scale_flat", dtype=torch.uint8,
                                         shape=(scale_numel,), index=index)
        if _overlaps(codes, packed_numel, scales, scale_numel):
            raise ValueError("packed_a_flat and scale_flat must not overlap")
        if (_overlaps(x, 4 * packed_numel, codes, packed_numel)
                or _overlaps(x, 4 * packed_numel, scales, scale_numel)):
            raise ValueError("bf16_input must not overlap either output")
        if _overlaps(gs, 4, codes, packed_numel) or _overlaps(gs, 4, scales, scale_numel):
            raise ValueError("global_scale must not overlap either output")
        _launch.quantize_nvfp4_rows(bf16_input, global_scale, packed_a_flat, scale_flat)

    return launch


__all__ = ["BF16ToFP4TMAOutputs", "allocate_bf16_to_fp4_tma_outputs", "compile_bf16_to_fp4_tma",
           "scale_storage_numel"]
