"""Performance cases of the block-scaled GEMM path, through its public entry points.

A case is a dict of plain values with an ``"op"`` (which entry points a pass calls) and its
sizes: ``m`` activation rows, ``n`` output features, ``k`` input features. ``listed`` holds the
cases that are always measured, ``draw`` makes more of the same ranges, ``prepare`` builds what a
program holds before the call (weights packed once, plans, scratch, activations on the GPU), ``run``
is one pass, ``work`` the bytes and operations a pass cannot do without, ``tolerance`` how far
another correct implementation may be off.

Ops:

* ``nvfp4``             quantization.nvfp4.run on BF16 rows, then gemm.blockscaled.mm (kept buffers)
* ``fused_mxfp8``       gemm.blockscaled.mm_fused_quant_a (activation quantizer inside the GEMM)
* ``fused_nvfp4``       gemm.blockscaled.mm_fused_quant_a_nvfp4
* ``mxfp8_linear``      gemm.mxfp8_linear.mm on BF16/FP16 rows, with or without bias
* ``block_fp8_linear``  gemm.block_fp8_linear plan / bind once, then run(binding=...)
* ``tensor_fp8_linear`` gemm.tensor_fp8_linear.mm on E4M3 rows, with or without bias
* ``block_fp8``         gemm.blockscaled.mm(block_fp8=True): FP32 scales 1x128 / 128x128
* ``bmm``               gemm.bmm twice: the N-major and the K-major absorb projection of 16 heads
* ``mm``                gemm.blockscaled.mm on operands quantized before, one or more groups
"""

from __future__ import annotations

import math

import torch

from sparkinfer_b200 import gemm
from sparkinfer_b200.gemm import block_fp8_linear, blockscaled, mxfp8_linear, tensor_fp8_linear
from sparkinfer_b200.quantization import mxfp8, nvfp4

# Operand recipes of gemm.blockscaled.mm: (ab_dtype, sf_dtype, sf_vec_size).
RECIPES = {
    "nvfp4": ("float4_e2m1fn", "float8_e4m3fn", 16),
    "mxfp8": ("float8_e4m3fn", "float8_e8m0fnu", 32),
}
DTYPES = {"bfloat16": torch.bfloat16, "float16": torch.float16, "float32": torch.float32}
HEADS = 16                      # gemm.bmm: heads, and (K, N) of its two projections
ABSORB_N_MAJOR = (192, 512)
ABSORB_K_MAJOR = (512, 256)
BMM_TYPES = dict(a_dtype="bfloat16", b_dtype="float8_e4m3fn", sf_dtype="float8_e8m0fnu",
                 c_dtype="bfloat16", sf_vec_size=32)
# No drawn case multiplies more, or holds a larger weight, than the largest listed ones.
MOST_MNK = 4096 * 18432 * 7168
MOST_NK = 57344 * 4096


def listed() -> list[dict]:
    return [
        # One token through an MLP up-projection of a decode step.
        dict(name="nvfp4_decode_m1", op="nvfp4", m=1, n=14336, k=4096, c="bfloat16"),
        # A decode batch against a wide weight (more than the L2 cache holds).
        dict(name="nvfp4_decode_m16_wide", op="nvfp4", m=16, n=57344, k=4096, c="bfloat16"),
        # A few tokens through a small projection, activations quantized inside the GEMM.
        dict(name="fused_mxfp8_m4", op="fused_mxfp8", m=4, n=4096, k=4096),
        # An odd batch through an FP16 linear with a bias; K is not a multiple of the GEMM's step.
        dict(name="mxfp8_linear_m33_bias", op="mxfp8_linear", m=33, n=7168, k=2080, bias=True,
             c="float16"),
        # The absorb projections of one attention layer for a decode batch.
        dict(name="bmm_absorb_m8", op="bmm", m=8),
        # A small GEMM on operands that were quantized before.
        dict(name="nvfp4_mm_m128", op="mm", recipe="nvfp4", m=128, n=4096, k=4096, groups=1,
             c="bfloat16"),
        # A decode batch through the down-projection of a block-FP8 checkpoint.
        dict(name="block_fp8_decode_m24", op="block_fp8", m=24, n=7168, k=18432, c="bfloat16"),
        # A ragged prefill chunk through a bound linear.
        dict(name="block_fp8_linear_m333", op="block_fp8_linear", m=333, n=4096, k=7168,
             bias=False, c="bfloat16"),
        # A short prompt through a per-tensor FP8 linear with a bias.
        dict(name="tensor_fp8_linear_m1000", op="tensor_fp8_linear", m=1000, n=7168, k=4096,
             bias=True, c="bfloat16"),
        # Prefill: rows quantized and multiplied, the three recipes at their large sizes.
        dict(name="mxfp8_linear_m8192", op="mxfp8_linear", m=8192, n=7168, k=7168, bias=False,
             c="bfloat16"),
        dict(name="nvfp4_prefill_m4096", op="nvfp4", m=4096, n=7168, k=18432, c="bfloat16"),
        dict(name="block_fp8_prefill_m4096", op="block_fp8", m=4096, n=18432, k=7168,
             c="bfloat16"),
    ]


def _log_int(rng, low: int, high: int, step: int = 1) -> int:
    value = math.exp(rng.uniform(math.log(low), math.log(high)))
    return max(-(-low // step) * step, int(round(value / step)) * step)


def draw(rng) -> dict:
    op = rng.choice(["nvfp4", "nvfp4", "fused_mxfp8", "fused_nvfp4", "mxfp8_linear",
                     "mxfp8_linear", "block_fp8_linear", "tensor_fp8_linear", "block_fp8",
                     "block_fp8", "bmm", "mm", "mm"])
    if op == "bmm":
        return dict(op=op, m=rng.randint(1, 32))
    while True:
        # K steps that the entry points accept; N down to eight columns where they accept it.
        k = _log_int(rng, 512, 18432, {"nvfp4": 64, "fused_nvfp4": 64, "mxfp8_linear": 32,
                                       "tensor_fp8_linear": 32}.get(op, 128))
        n = _log_int(rng, 512, 57344, rng.choice([128, 128, 8]) if op != "block_fp8" else 128)
        m = _log_int(rng, 1, {"fused_mxfp8": 8, "fused_nvfp4": 16}.get(op, 8192))
        groups = rng.choice([1, 1, 2, 3]) if op == "mm" else 1
        if groups * m * n * k <= MOST_MNK and groups * n * k <= MOST_NK and m * n <= 1 << 27:
            break
    case = dict(op=op, m=m, n=n, k=k)
    if op in ("nvfp4", "fused_nvfp4", "block_fp8"):
        case["c"] = rng.choice(["bfloat16", "bfloat16", "float16"])
    elif op == "mm":
        case.update(recipe=rng.choice(sorted(RECIPES)), groups=groups,
                    c=rng.choice(["bfloat16", "float16", "float32"]))
    elif op != "fused_mxfp8":
        case.update(bias=rng.random() < 0.5, c=rng.choice(["bfloat16", "bfloat16", "float16"]))
    return case


# ----------------------------------------------------------------------------------------
# Inputs
# ----------------------------------------------------------------------------------------
def _randn(gen: torch.Generator, *shape: int, scale: float = 1.0, dtype=torch.bfloat16):
    x = torch.randn(shape, device="cuda", generator=gen, dtype=torch.float32)
    return (x if scale == 1.0 else x.mul_(scale)).to(dtype)


def _nvfp4_rows(x: torch.Tensor):
    """BF16 rows -> (plan, buffers, global scale), the buffers holding the quantized rows."""
    plan = nvfp4.plan(*x.shape)
    buffers = nvfp4.allocate_outputs(plan, device=x.device)
    scale = (448.0 * 6.0 / x.abs().amax().to(torch.float32)).reshape(1)
    nvfp4.run(plan=plan, x=x, global_scale=scale, outputs=buffers)
    return plan, buffers, scale


def _mxfp8_rows(x: torch.Tensor):
    """BF16 rows (K a multiple of 128) -> codes [M, K], row scales [M, K / 32], MMA scale view."""
    m, k = x.shape
    codes = torch.empty((m, k), dtype=torch.float8_e4m3fn, device=x.device)
    rows = torch.empty((m, k // 32), dtype=torch.uint8, device=x.device)
    atoms = torch.full((1, -(-m // 128), -(-k // 128), 32, 4, 4), 127, dtype=torch.uint8,
                       device=x.device)
    mma = atoms.permute(3, 4, 1, 5, 2, 0)
    mxfp8.quantize_rows(x, codes, rows, mma)
    return codes, rows, mma.view(torch.float8_e8m0fnu)


def _block_fp8(x: torch.Tensor, block_rows: int):
    """E4M3 codes and FP32 scales amax / 448 over blocks of block_rows x 128."""
    m, k = x.shape
    pad = -m % block_rows
    blocks = torch.nn.functional.pad(x, (0, 0, 0, pad)).to(torch.float32)
    blocks = blocks.view((m + pad) // block_rows, block_rows, k // 128, 128)
    scale = blocks.abs().amax(dim=(1, 3)).clamp_min_(1e-12) / 448.0
    codes = (blocks / scale[:, None, :, None]).view(m + pad, k)[:m].to(torch.float8_e4m3fn)
    return codes.contiguous(), scale.contiguous()


def _stack(parts: list[torch.Tensor]) -> torch.Tensor:
    """Per-group [rows, cols, 1] views or 6-D scale views -> one operand over [L, ...] storage."""
    if len(parts) == 1:
        return parts[0]
    if parts[0].ndim == 3:
        return torch.stack([p.squeeze(2) for p in parts]).permute(1, 2, 0)
    raw = [p.view(torch.uint8).permute(5, 2, 4, 0, 1, 3)[0].contiguous() for p in parts]
    return torch.stack(raw).permute(3, 4, 1, 5, 2, 0).view(parts[0].dtype)


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device="cuda").manual_seed(seed)
    op, m = case["op"], case["m"]
    state = {"case": dict(case)}
    if op == "bmm":
        for tag, (k, n), n_major in (("n", ABSORB_N_MAJOR, True), ("k", ABSORB_K_MAJOR, False)):
            rows, inner = (k, n) if n_major else (n, k)
            w = _randn(gen, HEADS * rows, inner, scale=0.02)
            codes, scales, _ = _mxfp8_rows(w)
            state["rhs_" + tag] = (codes.view(HEADS, rows, inner),
                                   scales.view(HEADS, rows, inner // 32))
            state["lhs_" + tag] = _randn(gen, HEADS, m, k)
            state["out_" + tag] = torch.empty((HEADS, m, n), dtype=torch.bfloat16, device="cuda")
        return state
    n, k = case["n"], case["k"]
    if op == "mm":
        a, b, alphas = [], [], []
        for _ in range(case["groups"]):
            x, w = _randn(gen, m, k), _randn(gen, n, k, scale=0.02)
            if case["recipe"] == "nvfp4":
                _, qx, sx = _nvfp4_rows(x)
                _, qw, sw = _nvfp4_rows(w)
                a.append((qx.packed_a_view, qx.scale_mma_view(m, k)))
                b.append((qw.packed_a_view, qw.scale_mma_view(n, k)))
                alphas.append(1.0 / (sx * sw))
            else:
                for rows, into in ((x, a), (w, b)):
                    codes, _, mma = _mxfp8_rows(rows)
                    into.append((codes.unsqueeze(2), mma))
        state["lhs"] = tuple(_stack([p[i] for p in a]) for i in range(2))
        state["rhs"] = tuple(_stack([p[i] for p in b]) for i in range(2))
        state["alpha"] = alphas[0] if alphas else None
        return state
    dtype = DTYPES[case.get("c", "bfloat16")]
    if op == "block_fp8":
        a, sfa = _block_fp8(_randn(gen, m, k), 1)
        b, sfb = _block_fp8(_randn(gen, n, k, scale=0.02), 128)
        state.update(lhs=(a.unsqueeze(2), sfa), rhs=(b.unsqueeze(2), sfb),
                     out=torch.empty((m, n, 1), dtype=dtype, device="cuda"))
    elif op in ("nvfp4", "fused_nvfp4"):
        x = _randn(gen, m, k)
        _, qw, sw = _nvfp4_rows(_randn(gen, n, k, scale=0.02))
        plan, buffers, sx = _nvfp4_rows(x)
        state.update(x=x, scale=sx, alpha=1.0 / (sx * sw), plan=plan, buffers=buffers,
                     rhs=(qw.packed_a_view, qw.scale_mma_view(n, k)),
                     out=torch.empty((m, n, 1), dtype=dtype, device="cuda"))
        state["lhs"] = (buffers.packed_a_view, buffers.scale_mma_view(m, k))
    elif op == "fused_mxfp8":
        codes, _, mma = _mxfp8_rows(_randn(gen, n, k, scale=0.02))
        state.update(x=_randn(gen, m, k), rhs=(codes.unsqueeze(2), mma))
    elif op == "mxfp8_linear":
        w = _randn(gen, n, k, scale=0.02)
        wide = torch.nn.functional.pad(w, (0, -k % 128))
        codes, rows, _ = _mxfp8_rows(wide)
        state.update(x=_randn(gen, m, k, dtype=dtype),
                     weight=mxfp8_linear.pack_weight(codes[:, :k].contiguous(),
                                                     rows[:, :k // 32].contiguous()))
    elif op == "block_fp8_linear":
        codes, scale = _block_fp8(_randn(gen, n, k, scale=0.02), 128)
        state.update(x=_randn(gen, m, k, dtype=dtype),
                     weight=block_fp8_linear.pack_weight(codes, scale))
    else:  # tensor_fp8_linear
        w = _randn(gen, n, k, scale=0.02)
        x = _randn(gen, m, k)
        sw, sx = (t.abs().amax().to(torch.float32) / 448.0 for t in (w, x))
        state.update(x=(x.to(torch.float32) / sx).to(torch.float8_e4m3fn),
                     weight=tensor_fp8_linear.pack_weight(
                         (w.to(torch.float32) / sw).to(torch.float8_e4m3fn),
                         (sx * sw).reshape(1)))
    state["bias"] = _randn(gen, n, dtype=dtype) if case.get("bias") else None
    if op == "block_fp8_linear":
        plan = block_fp8_linear.plan(block_fp8_linear.Caps(
            device="cuda", max_tokens=m, in_features=k, out_features=n, output_dtype=dtype))
        spec = plan.scratch_specs()[0]
        state["binding"] = block_fp8_linear.bind(
            plan, scratch=torch.empty(spec.shape, dtype=spec.dtype, device=spec.device),
            source=state["x"], packed_weight=state["weight"], bias=state["bias"],
            output=torch.empty((m, n, 1), dtype=dtype, device="cuda"))
    return state


# ----------------------------------------------------------------------------------------
# One pass
# ----------------------------------------------------------------------------------------
def _mm(state: dict, recipe: str, c: str, out=None) -> torch.Tensor:
    ab_dtype, sf_dtype, vec = RECIPES[recipe]
    return blockscaled.mm(state["lhs"], state["rhs"], out, ab_dtype=ab_dtype, sf_dtype=sf_dtype,
                          sf_vec_size=vec, c_dtype=c, alpha=state["alpha"])


def run(state: dict):
    case = state["case"]
    op = case["op"]
    if op == "nvfp4":
        buffers = state["buffers"]
        nvfp4.run(plan=state["plan"], x=state["x"], global_scale=state["scale"], outputs=buffers)
        out = _mm(state, "nvfp4", case["c"], state["out"])
        return {"out": out, "codes": buffers.packed_a_storage, "scales": buffers.scale_storage}
    if op == "fused_mxfp8":
        return blockscaled.mm_fused_quant_a(state["x"], *state["rhs"])
    if op == "fused_nvfp4":
        return blockscaled.mm_fused_quant_a_nvfp4(state["x"], state["scale"], *state["rhs"],
                                                  alpha=state["alpha"], out=state["out"],
                                                  c_dtype=case["c"])
    if op == "mxfp8_linear":
        return mxfp8_linear.mm(state["x"], state["weight"], bias=state["bias"])
    if op == "block_fp8_linear":
        return block_fp8_linear.run(binding=state["binding"])
    if op == "tensor_fp8_linear":
        return tensor_fp8_linear.mm(state["x"], state["weight"], bias=state["bias"],
                                    out_dtype=DTYPES[case["c"]])
    if op == "block_fp8":
        return blockscaled.mm(state["lhs"], state["rhs"], state["out"], ab_dtype="float8_e4m3fn",
                              sf_dtype="float32", sf_vec_size=128, c_dtype=case["c"],
                              block_fp8=True)
    if op == "bmm":
        return [gemm.bmm(state["lhs_" + tag], state["rhs_" + tag], state["out_" + tag],
                         b_major=tag, sf_axis=tag, **BMM_TYPES) for tag in ("n", "k")]
    return _mm(state, case["recipe"], case["c"])


def work(case: dict) -> dict:
    """Each input read once and each output written once; a product is 2 * M * N * K operations."""
    op, m = case["op"], case["m"]
    if op == "bmm":
        total = {"bytes": 0.0, "flops": 0.0}
        for k, n in (ABSORB_N_MAJOR, ABSORB_K_MAJOR):
            total["bytes"] += HEADS * (m * k * 2 + k * n * (1 + 1 / 32) + m * n * 2)
            total["flops"] += HEADS * 2.0 * m * n * k
        return total
    n, k, groups = case["n"], case["k"], case.get("groups", 1)
    fp4 = "nvfp4" in (case.get("recipe"), op) or op == "fused_nvfp4"
    code = 0.5 + 1 / 16 if fp4 else 1 + 1 / 32        # bytes of an element with its scale
    a = {"mm": code, "block_fp8": 1 + 4 / 128, "tensor_fp8_linear": 1.0,
         "nvfp4": 2 + code}.get(op, 2.0)              # nvfp4: rows read, codes handed back
    b = {"block_fp8": 1 + 4 / (128 * 128), "tensor_fp8_linear": 1.0}.get(op, code)
    out = 4 if case.get("c") == "float32" else 2
    return {"bytes": groups * (m * k * a + n * k * b + m * n * out
                               + (n * 2 if case.get("bias") else 0)),
            "flops": groups * 2.0 * m * n * k}


def tolerance(case: dict) -> dict:
    """Codes and scale bytes of a quantizer are exact. A GEMM's result differs from the same
    product in 64 bits by its output rounding (measured 1.7e-3 to 1.8e-3 for BF16, 2.1e-4 to 2.3e-4
    for FP16) or, with FP32 outputs, by its FP32 sums over K (1.3e-6 at K = 18432); the bounds are
    four times that."""
    return {"rel": {"bfloat16": 7e-3, "float16": 9e-4, "float32": 6e-6}[case.get("c", "bfloat16")]}
