"""GEMM front-end: the replacement for rust-nn's `blas::sgemm` (src/blas.rs:104-186).

``gemm(a, b, ...)`` computes ``act(alpha * A @ B^T + bias) [* act'(aux_in)] [+ residual]`` where
``A`` is logically ``[M, K]`` and ``B`` is logically ``[N, K]``. ``a_mn`` / ``b_mn`` say that the
operand is *stored* transposed (``[K, M]`` / ``[K, N]``); no transposed copy is ever made - the
layout goes into the TMA descriptor and the tensor-core matrix descriptor.

On CUDA tensors this always launches the hand-written tcgen05 kernel (csrc/gemm/gemm_sm100.cu).
On CPU tensors it evaluates the same expression with PyTorch in fp32 (the oracle).
"""
from __future__ import annotations

import ctypes as C
import math

import torch

from .. import _native as nv

ACT = {"none": 0, "relu": 1, "gelu": 2, "silu": 3, "sigmoid": 4, "tanh": 5}
OUT_BF16, OUT_F32, OUT_F32_ATOMIC, OUT_I32 = 0, 1, 2, 3
_NUM_SMS = {}


def _num_sms(device) -> int:
    idx = torch.device(device).index or 0
    if idx not in _NUM_SMS:
        _NUM_SMS[idx] = torch.cuda.get_device_properties(idx).multi_processor_count
    return _NUM_SMS[idx]


def act_ref(x: torch.Tensor, act: str) -> torch.Tensor:
    if act == "relu":
        return torch.relu(x)
    if act == "gelu":
        return torch.nn.functional.gelu(x, approximate="tanh")
    if act == "silu":
        return torch.nn.functional.silu(x)
    if act == "sigmoid":
        return torch.sigmoid(x)
    if act == "tanh":
        return torch.tanh(x)
    return x


def dact_ref(saved: torch.Tensor, act: str) -> torch.Tensor:
    """Derivative of `act` given the saved tensor (pre-activation for gelu/silu, output otherwise)."""
    s = saved.float()
    if act == "relu":
        return (s > 0).float()
    if act == "gelu":
        k0, k1 = 0.7978845608028654, 0.044715
        t = torch.tanh(k0 * (s + k1 * s ** 3))
        return 0.5 * (1 + t) + 0.5 * s * (1 - t * t) * k0 * (1 + 3 * k1 * s * s)
    if act == "silu":
        sg = torch.sigmoid(s)
        return sg * (1 + s * (1 - sg))
    if act == "sigmoid":
        return s * (1 - s)
    if act == "tanh":
        return 1 - s * s
    return torch.ones_like(s)


def gemm_ref(a, b, *, a_mn=False, b_mn=False, bias=None, act="none", residual=None, aux_in=None, dact="none",
             alpha=1.0, out_dtype=None, accumulate_into=None, want_aux=False, row_scale=None, col_scale=None):
    """fp32 PyTorch evaluation of the same expression (used on CPU and as the test oracle)."""
    if out_dtype == torch.int32:          # exact integer accumulation (the igemm contract)
        return (a.to(torch.int64) @ b.to(torch.int64).transpose(-1, -2)).to(torch.int32)
    lowp = a.dtype in (torch.int8, torch.uint8, torch.float8_e4m3fn)
    ft = torch.float64 if lowp else torch.float32
    A = a.to(ft).transpose(-1, -2) if a_mn else a.to(ft)
    B = b.to(ft).transpose(-1, -2) if b_mn else b.to(ft)
    v = (alpha * (A @ B.transpose(-1, -2))).float()
    if row_scale is not None:
        v = v * row_scale.float().reshape(*v.shape[:-1], 1)
    if col_scale is not None:
        v = v * col_scale.float()
    if lowp and out_dtype is None:
        out_dtype = torch.bfloat16
    if bias is not None:
        v = v + (bias.float()[:, None, :] if bias.dim() == 2 else bias.float())   # [batch, N]: one vector per batch
    pre = v
    v = act_ref(v, act)
    if aux_in is not None:
        v = v * dact_ref(aux_in, dact)
    if residual is not None:
        v = v + residual.float()
    if accumulate_into is not None:
        accumulate_into.add_(v.to(accumulate_into.dtype))
        v = accumulate_into
    else:
        v = v.to(out_dtype or a.dtype)
    if want_aux:
        return v, pre.to(torch.bfloat16 if lowp else a.dtype)
    return v


def _readable(t: torch.Tensor) -> bool:
    """Can TMA read this 2-D or 3-D operand where it is (unit inner stride, other strides and base in multiples of 16 bytes)?"""
    q = 16 // t.element_size()
    return (t.stride(-1) == 1 and t.stride(-2) % q == 0 and t.data_ptr() % 16 == 0 and t.stride(-2) >= t.shape[-1]
            and (t.dim() == 2 or t.shape[0] == 1 or t.stride(0) % q == 0))


_OUT_CODE = {None: -1, torch.float32: OUT_F32, torch.int32: OUT_I32}      # any other dtype: bf16


@nv.traced("gemm")
def gemm(a: torch.Tensor, b: torch.Tensor, *, a_mn: bool = False, b_mn: bool = False, bias=None, act: str = "none",
         residual=None, aux_in=None, dact: str = "none", want_aux: bool = False, alpha: float = 1.0,
         out_dtype=None, accumulate_into=None, splits: int = 0, bn: int = 0, alpha_t=None, row_scale=None, col_scale=None,
         out=None, m_valid=None, k_valid=None, _prepare: bool = False):
    """See module docstring. Returns C (and the bf16 pre-activation when ``want_aux``). ``out`` (GPU only): write the
    result into this tensor ([M, N] or [batch, M, N], unit inner stride, dtype of the result) instead of a new one.
    ``m_valid`` / ``k_valid`` (int32 [batch] on the device) make a batched product ragged, as the groups of tokens routed
    to each expert are: row tiles of 128 wholly past ``m_valid[b]`` are skipped (those rows of the result are NOT
    written), and the contraction stops at ``k_valid[b]`` rounded up to 128 (rows up to there must hold finite values).

    8-bit operands (int8 x int8, uint8 x int8, float8_e4m3fn x float8_e4m3fn; both K-major) run on the
    tensor cores' integer / fp8 kinds. ``row_scale`` ([M] or [batch, M] fp32) and ``col_scale`` ([N] fp32)
    dequantise in the epilogue before bias and activation; ``out_dtype=torch.int32`` returns the raw
    accumulators of an integer product (rust-nn `igemm`, src/int8.rs:222-314)."""
    if not a.is_cuda:
        if alpha_t is not None:
            alpha = alpha * float(alpha_t)
        r = gemm_ref(a, b, a_mn=a_mn, b_mn=b_mn, bias=bias, act=act, residual=residual, aux_in=aux_in, dact=dact,
                     alpha=alpha, out_dtype=out_dtype, accumulate_into=accumulate_into, want_aux=want_aux,
                     row_scale=row_scale, col_scale=col_scale)
        # (m_valid / k_valid only skip work whose operands are zero or whose results are never read: nothing to do on CPU)
        if out is not None:
            out.copy_((r[0] if want_aux else r).reshape(out.shape))
            r = (out, r[1]) if want_aux else out
        return r
    if a.dtype == torch.float32 and (a_mn or b_mn) and b.dtype == torch.float32:
        # a transposed fp32 operand that TMA cannot read in place (rows of other than 4 n elements) is transposed by a kernel: one
        # launch, where padding its rows would take two
        from .kernels import transpose_last2
        if a_mn and not _readable(a):
            a, a_mn = transpose_last2(a), False
        if b_mn and not _readable(b):
            b, b_mn = transpose_last2(b), False
    e = nv.entry()
    r = (e.gemm_record if _prepare else e.gemm)(
        a, b, a_mn, b_mn, bias, ACT[act], residual, aux_in, ACT[dact], want_aux, alpha, _OUT_CODE.get(out_dtype, OUT_BF16), accumulate_into,
        splits, bn, alpha_t, row_scale, col_scale, out, m_valid, k_valid)
    if _prepare:
        # a fused kernel runs this product itself: the filled launch record, the tile width, the results and everything the record
        # points at (kept alive by the caller until the launch has been issued)
        rec, bn, res, aux, keep = r
        return nv.GemmArgs.from_buffer_copy(rec), bn, res, aux, keep
    return r
