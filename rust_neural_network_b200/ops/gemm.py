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
GEMM_BF16, GEMM_F32, GEMM_S8S8, GEMM_U8S8, GEMM_E4M3 = 0, 1, 2, 3, 4
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


def _as3d(t: torch.Tensor):
    if t.dim() == 2:
        return t.unsqueeze(0)
    if t.dim() == 3:
        return t
    raise ValueError("gemm operands must be 2-D or 3-D")


def _readable(t: torch.Tensor) -> bool:
    """Can TMA read this 2-D or 3-D operand where it is?"""
    q = 16 // t.element_size()
    return (t.stride(-1) == 1 and t.stride(-2) % q == 0 and t.data_ptr() % 16 == 0 and t.stride(-2) >= t.shape[-1]
            and (t.dim() == 2 or t.shape[0] == 1 or t.stride(0) % q == 0))


def _tma_ready(t: torch.Tensor) -> torch.Tensor:
    """Return `t` (3-D view) or a padded copy such that TMA constraints hold:
    innermost stride 1, other strides multiples of 16 bytes, base 16-byte aligned."""
    if _readable(t):
        return t
    q = 16 // t.element_size()
    inner = (t.shape[-1] + q - 1) // q * q
    buf = torch.zeros(t.shape[0], t.shape[1], inner, dtype=t.dtype, device=t.device)
    buf[..., : t.shape[-1]].copy_(t)
    return buf[..., : t.shape[-1]]


def _operand(t: torch.Tensor):
    """(tensor, batch, rows, columns, row stride, batch stride) of an operand that TMA can read: `t` itself, or the padded
    copy `_tma_ready` makes of it."""
    if t.dim() == 2:
        rows, cols = t.shape
        ld, inner = t.stride()
        if inner == 1 and ld >= cols and ld * t.element_size() % 16 == 0 and t.data_ptr() % 16 == 0:
            return t, 1, rows, cols, ld, rows * ld
    t = _tma_ready(_as3d(t))
    return t, t.shape[0], t.shape[1], t.shape[2], t.stride(1), t.stride(0)


_KINDS = {(torch.bfloat16, torch.bfloat16): GEMM_BF16, (torch.float32, torch.float32): GEMM_F32,
          (torch.int8, torch.int8): GEMM_S8S8, (torch.uint8, torch.int8): GEMM_U8S8,
          (torch.float8_e4m3fn, torch.float8_e4m3fn): GEMM_E4M3}


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
    lib = nv.cuda()
    kind = _KINDS.get((a.dtype, b.dtype))
    if kind is None:
        raise TypeError(f"gemm operands must be bf16 x bf16, fp32 x fp32, int8 x int8, uint8 x int8 or e4m3 x e4m3 (got {a.dtype}, {b.dtype})")
    is_f32 = kind == GEMM_F32
    lowp = kind >= GEMM_S8S8
    if lowp and (a_mn or b_mn):
        raise ValueError("8-bit GEMM operands must be K-major")
    if is_f32 and (a_mn or b_mn):
        # a transposed fp32 operand that TMA cannot read in place (rows of other than 4 n elements) is transposed by a kernel: one
        # launch, where padding its rows would take two
        from .kernels import transpose_last2
        if a_mn and not _readable(a):
            a, a_mn = transpose_last2(a), False
        if b_mn and not _readable(b):
            b, b_mn = transpose_last2(b), False
    squeeze = a.dim() == 2
    a3, batch, ar, ac, lda, stride_a = _operand(a)
    b3, batch_b, br, bc, ldb, stride_b = _operand(b)
    if batch_b != batch:
        raise ValueError("batch mismatch")
    M, K = (ac, ar) if a_mn else (ar, ac)
    N, Kb = (bc, br) if b_mn else (br, bc)
    if K != Kb:
        raise ValueError(f"gemm K mismatch: {K} vs {Kb}")
    dev = a.device
    may_divide = False
    if accumulate_into is not None:
        out = accumulate_into
        if out.dtype != torch.float32 or not out.is_contiguous():
            raise ValueError("accumulate_into must be a contiguous fp32 tensor")
        out_mode = OUT_F32_ATOMIC
    else:
        odt = out_dtype or (torch.float32 if is_f32 else torch.bfloat16)
        if odt == torch.int32:
            if kind not in (GEMM_S8S8, GEMM_U8S8):
                raise TypeError("an int32 result needs integer operands")
            out_mode = OUT_I32
        else:
            out_mode = OUT_F32 if odt == torch.float32 else OUT_BF16
        if out is not None:
            want = torch.int32 if out_mode == OUT_I32 else torch.float32 if out_mode == OUT_F32 else torch.bfloat16
            if out.dtype != want or out.stride(-1) != 1 or out.numel() != batch * M * N:
                raise ValueError("`out` must have the result's dtype, size and a unit inner stride")
            if splits > 1:
                raise ValueError("`out` and split-K do not go together (split-K accumulates into a zeroed fp32 buffer)")
            may_divide = splits == 0
            splits = 1
    # The launcher chooses the tiles (bn = 0) and may divide a sum over the CTAs of a cluster (0 splits). Here: into how many
    # parts that are added in memory an fp32 result's contraction is split, on the tiles that go with it.
    sms = _num_sms(dev)
    one_cta = _prepare or splits == 1 and not may_divide
    if splits == 0:
        splits = 1
        num_kb = -(-K // (32 if is_f32 else 128 if lowp else 64))
        if out_mode in (OUT_F32, OUT_F32_ATOMIC) and num_kb >= (64 if lowp else 16) and act == "none" and aux_in is None and not want_aux:
            row_tiles = -(-M // 128) * batch
            t256 = row_tiles * -(-N // 256)
            # Few tiles and a long K (weight gradients): split-K fills the machine either way, and the wider tile moves
            # a third less operand traffic from L2 per FLOP (measured 167 -> 113 us on 2048 x 512 x 65536).
            if bn:
                sbn = bn
            elif not is_f32 and not lowp and N >= 256 and (t256 >= sms or K >= 16 * 64 * max(1, sms // t256)):
                sbn = 256
            else:
                sbn = 64 if N <= 64 and not is_f32 and not lowp else 128
            tiles = row_tiles * -(-N // sbn)
            if tiles < sms // 2:
                splits = max(1, min(sms // tiles, num_kb // 8))
            if splits > 1 or sbn == 256:
                bn = sbn
    if splits > 1:
        num_kb = -(-K // (32 if is_f32 else 128 if lowp else 64))
        per = -(-num_kb // splits)
        splits = -(-num_kb // per)
    if splits > 1:
        if out_mode == OUT_BF16 or act != "none" or aux_in is not None or want_aux:
            raise ValueError("split-K needs an fp32 output and a linear epilogue")
        out_mode = OUT_F32_ATOMIC
    if out is None:
        shape = (M, N) if squeeze else (batch, M, N)
        odt = torch.int32 if out_mode == OUT_I32 else torch.float32 if out_mode != OUT_BF16 else torch.bfloat16
        out = torch.zeros(shape, dtype=odt, device=dev) if out_mode == OUT_F32_ATOMIC else torch.empty(shape, dtype=odt, device=dev)
    if out.dim() == 2 and batch == 1 and out.shape[0] == M and out.shape[1] == N:
        out3, ldc, out_ptr = out, out.stride(0), out.data_ptr()
        stride_c = M * ldc
    else:
        out3 = out if out.dim() == 3 else out.view(1, M, N) if batch == 1 else out.view(batch, M, N)
        ldc, out_ptr = out3.stride(1), out3.data_ptr()
        stride_c = out3.stride(0) if batch > 1 else M * ldc
    aux = torch.empty((M, N) if squeeze else (batch, M, N), dtype=torch.bfloat16, device=dev) if want_aux else None
    if aux_in is not None:
        aux_in = aux_in.contiguous().view(batch, M, N)
        if aux_in.dtype != torch.bfloat16:
            raise TypeError("aux_in must be bf16")
    if residual is not None:
        residual = residual.reshape(batch, M, N)
        if residual.dtype != torch.bfloat16:
            residual = residual.to(torch.bfloat16)
        if residual.stride(-1) != 1:
            residual = residual.contiguous()
    if bias is not None and bias.dtype not in (torch.float32, torch.bfloat16):
        raise TypeError("bias must be fp32 or bf16")

    if (aux is not None or aux_in is not None) and ldc != N:
        raise ValueError("aux tensors need a dense output (ldc == N)")
    if row_scale is not None:
        row_scale = row_scale.float().contiguous()
        if row_scale.numel() != batch * M:
            raise ValueError("row_scale needs one value per row of A")
    if col_scale is not None:
        col_scale = col_scale.float().contiguous()
        if col_scale.numel() != N:
            raise ValueError("col_scale needs one value per row of B")
    for name, t in (("m_valid", m_valid), ("k_valid", k_valid)):
        if t is not None and (t.dtype != torch.int32 or t.numel() != batch or not t.is_cuda):
            raise ValueError(f"{name} must be an int32 device tensor with one entry per batch")
    if alpha_t is not None and alpha_t.dtype != torch.float32:
        alpha_t = alpha_t.float()
    bias_ptr = bias_f32 = bias_vec_ok = bias_stride = 0
    if bias is not None:
        bias_ptr, bias_f32 = bias.data_ptr(), int(bias.dtype == torch.float32)
        bias_vec_ok = int(bias_ptr % 16 == 0 and N % 4 == 0 and bias.is_contiguous())
        bias_stride = N if bias.dim() == 2 else 0                  # [batch, N] bias: one vector per batch
    res_ptr = ldr = stride_r = res_vec_ok = 0
    if residual is not None:
        res_ptr, ldr, stride_r = residual.data_ptr(), residual.stride(1), residual.stride(0)
        res_vec_ok = int(ldr % 8 == 0 and res_ptr % 16 == 0 and (batch == 1 or stride_r % 8 == 0))
    es_out = 4 if out_mode != OUT_BF16 else 2
    vec_ok = int(ldc * es_out % 16 == 0 and out_ptr % 16 == 0 and (batch == 1 or stride_c * es_out % 16 == 0)
                 and ((aux is None and aux_in is None) or N % 8 == 0))
    rec = nv.GEMM_PACK.pack(
        M, N, K, batch, splits if one_cta or splits > 1 else 0, out_ptr, ldc, stride_c, bias_ptr, bias_f32, bias_vec_ok, bias_stride, res_ptr, ldr, stride_r,
        nv.ptr(aux), nv.ptr(aux_in), nv.f32(alpha), nv.ptr(alpha_t), ACT[act], ACT[dact], out_mode, vec_ok, res_vec_ok,
        nv.ptr(row_scale), nv.ptr(col_scale), nv.status_ptr(dev), nv.ptr(m_valid), nv.ptr(k_valid),
        a3.data_ptr(), lda, stride_a, int(a_mn), b3.data_ptr(), ldb, stride_b, int(b_mn), M, N, K, batch, kind)
    res = out3[0] if (squeeze and out.dim() == 3) else out
    if _prepare:
        # a fused kernel runs this product itself: hand back the filled launch record, the tile width, the results and
        # everything the record points at (kept alive by the caller until the launch has been issued)
        return nv.GemmArgs.from_buffer_copy(rec), bn, res, aux, (a3, b3, bias, residual, aux_in, row_scale, col_scale, m_valid, k_valid, out3)
    rc = lib.b200_gemm_launch(rec, bn, sms, nv.stream_ptr())
    nv.check(rc, "b200_gemm_launch")
    nv.count_launch()
    if accumulate_into is not None:
        res = accumulate_into
    if want_aux:
        return res, aux
    return res
