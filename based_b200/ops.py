"""Torch-facing wrappers of the C-ABI kernels.

Each function validates what only the Python side can know (device, dtype, contiguity of
the innermost dimension), passes raw device pointers, element strides and torch's current
stream to the library, and returns torch tensors.  CUDA tensors only.
"""
from typing import Optional, Tuple

import torch

from torch._C._functorch import is_functorch_wrapped_tensor as _wrapped
from torch.autograd import forward_ad as _forward_ad
from torch.utils._device import DeviceContext as _DeviceContext

from . import _capi
from ._capi import BASED_BF16, BASED_F32, IMPL_AUTO, IMPL_DECODE, IMPL_SIMT, IMPL_TCGEN05  # noqa: F401

EXPANDED_DIM = 273
_IMPLS = {"auto": IMPL_AUTO, "simt": IMPL_SIMT, "tcgen05": IMPL_TCGEN05, "decode": IMPL_DECODE}


def _dt(t: torch.dtype) -> int:
    if t == torch.float32:
        return BASED_F32
    if t == torch.bfloat16:
        return BASED_BF16
    raise TypeError(f"unsupported dtype {t}: the kernels take float32 or bfloat16")


def _need_cuda(*ts):
    """Every op starts here: CUDA tensors only, and no autograd.  The kernels write into fresh buffers through
    raw pointers and register no backward, so under grad mode the result would silently be cut off from the
    graph (the projections before a mixer would get no gradient and nothing would say so)."""
    _capi.native().need_cuda(*ts)


def check_status(reset: bool = True) -> int:
    """Read the tensor-core kernels' status word and raise if a bounded in-kernel wait ever expired (the results
    of that launch are then meaningless).  It synchronises the device, so call it where the caller synchronises
    anyway: after a generation loop, at the end of a timed region."""
    code = _capi.read_status(reset)
    if code != 0:
        raise _capi.BasedLibraryError(f"a bounded wait expired inside a tensor-core kernel (status 0x{code:x}); "
                                      "the outputs of that launch are not valid")
    return code


def _inner_contig(t, name):
    if t.stride(-1) != 1:
        raise ValueError(f"{name}: innermost stride must be 1")


def _rows(t, width):
    """``t [..., width]`` as a ``[M, width]`` view of the same memory (rows one constant stride apart)."""
    if t.shape[-1] != width or t.stride(-1) != 1:
        raise ValueError(f"out must be a [..., {width}] tensor with contiguous rows")
    return flat_rows(t)


def flat_rows(t):
    """``t [..., W]`` as ``[M, W]`` without a copy; raises when its rows are not one constant stride apart."""
    if t.is_contiguous() and t.numel():
        return t if t.dim() == 2 else t.view(-1, t.shape[-1])
    dims = [(n, st) for n, st in zip(t.shape[:-1], t.stride()[:-1]) if n != 1]
    for (_, outer), (n, inner) in zip(dims, dims[1:]):
        if outer != inner * n:
            raise ValueError("rows are not one constant stride apart")
    m = 1
    for n, _ in dims:
        m *= n
    return t.as_strided((m, t.shape[-1]), (dims[-1][1] if dims else t.shape[-1], t.stride(-1)))


def _flat(t, width):
    """``t [..., width]`` for a kernel that takes rows: itself where it is contiguous, else as ``[M, width]`` (a copy where the
    rows are not one stride apart)."""
    return t if t.is_contiguous() else t.reshape(-1, width)


def _row_stride(t, width):
    """Elements between the rows of :func:`_flat`'s result."""
    return width if t.is_contiguous() else t.stride(0)


def _position(pos, like):
    """(device pointer or None, scalar) of a call's first position: an int, or an int32 CUDA tensor with one per row."""
    if torch.is_tensor(pos):
        if pos.dtype != torch.int32 or pos.device != like.device or not pos.is_contiguous():
            raise TypeError("positions must be a contiguous int32 tensor on the inputs' device")
        if pos.numel() < like.shape[0]:
            raise ValueError("positions: one per batch row is needed")
        return pos.data_ptr(), 0
    return None, int(pos)


def _ptr(t):
    return None if t is None else t.data_ptr()


def _stream():
    return torch.cuda.current_stream().cuda_stream


def linattn_prefill(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, *, eps: float = 1e-12,
                    return_state: bool = True, state_dtype: Optional[torch.dtype] = None,
                    out: Optional[torch.Tensor] = None, impl: str = "auto",
                    kv_state: Optional[torch.Tensor] = None, k_state: Optional[torch.Tensor] = None,
                    nseg: Optional[int] = None, scratch: Optional[torch.Tensor] = None,
                    ) -> Tuple[torch.Tensor, Optional[torch.Tensor], Optional[torch.Tensor]]:
    """Causal Taylor linear attention over a whole sequence.

    q, k ``[B, H, L, 16]`` (raw), v ``[B, H, L, dv]``; any batch/head/seq strides (e.g. the
    transposed views LinearAttention.forward makes, linear_attention.py:127-129).
    Returns ``y`` as a ``[B, H, L, dv]`` view of a ``[B, L, H, dv]`` buffer (so the reference's
    ``'b h l d -> b l (h d)'`` rearrange is free), ``kv_state [B, H, 1, dv, 273]`` and
    ``k_state [B, H, 1, 1, 273]`` (linear_attention.py:220-222), or ``None`` for the states
    when ``return_state`` is false.  ``kv_state``/``k_state`` may be given to be filled in place.

    ``nseg`` splits the SEQUENCE into that many segments that run on different SMs (bf16, tensor-core
    kernel only): ``None`` lets the library choose (it splits only when ``B*H`` is below half the SM
    count and ``L >= 1024``), ``1`` never splits.  The split needs a workspace of
    ``based_linattn_prefill_scratch_bytes`` bytes; ``scratch`` (a CUDA uint8/float tensor at least that
    large) may be given to reuse one, else it is taken from torch's caching allocator.
    """
    _need_cuda(q, k, v)
    B, H, L, d = q.shape
    dv = v.shape[-1]
    if k.shape != q.shape or v.shape[:3] != q.shape[:3]:
        raise ValueError("q, k, v shapes disagree")
    if not (q.dtype == k.dtype == v.dtype):
        raise TypeError("q, k, v must share a dtype")
    for t, n in ((q, "q"), (k, "k"), (v, "v")):
        _inner_contig(t, n)
    if out is None:
        out = torch.empty(B, L, H, dv, dtype=q.dtype, device=q.device).permute(0, 2, 1, 3)
    else:
        _inner_contig(out, "out")
    sdt = kv_state.dtype if kv_state is not None else (state_dtype or q.dtype)
    if return_state:
        if kv_state is None:
            kv_state = torch.empty(B, H, 1, dv, EXPANDED_DIM, dtype=sdt, device=q.device)
            k_state = torch.empty(B, H, 1, 1, EXPANDED_DIM, dtype=sdt, device=q.device)
        elif not (kv_state.is_contiguous() and k_state.is_contiguous()):
            raise ValueError("kv_state / k_state must be contiguous")
    if L == 0 or B == 0 or H == 0:  # empty tensors have no device pointer to pass
        if return_state:
            kv_state.zero_()
            k_state.zero_()
        return out, (kv_state if return_state else None), (k_state if return_state else None)
    lib = _capi.lib()
    can_split = q.dtype == torch.bfloat16 and dv <= 112 and impl in ("auto", "tcgen05")
    if nseg is not None and nseg > 1 and not can_split:
        raise ValueError("nseg > 1 needs bf16 inputs, dv <= 112 and the tensor-core kernel")
    if nseg is None:
        nseg = lib.based_linattn_prefill_segments(B, H, L) if can_split else 1
    if nseg > 1:
        need = lib.based_linattn_prefill_scratch_bytes(B, H, L, dv, nseg)
        if scratch is None:
            scratch = torch.empty(max(need, 16), dtype=torch.uint8, device=q.device)
        elif scratch.device != q.device or not scratch.is_contiguous():
            raise ValueError("scratch must be a contiguous tensor on the inputs' device")
        code = _capi.native().linattn_prefill_split(
            q, k, v, out,
            kv_state if return_state else None, k_state if return_state else None,
            B, H, L, d, dv,
            q.stride()[:3], k.stride()[:3],
            v.stride()[:3], out.stride()[:3],
            _dt(sdt), float(eps), int(nseg), scratch, scratch.numel() * scratch.element_size())
        _capi.check(code, "based_linattn_prefill_split")
        return out, (kv_state if return_state else None), (k_state if return_state else None)
    code = _capi.native().linattn_prefill(
        q, k, v, out,
        kv_state if return_state else None, k_state if return_state else None,
        B, H, L, d, dv,
        q.stride()[:3], k.stride()[:3],
        v.stride()[:3], out.stride()[:3],
        _dt(q.dtype), _dt(sdt), float(eps), _IMPLS[impl])
    _capi.check(code, "based_linattn_prefill")
    return out, (kv_state if return_state else None), (k_state if return_state else None)


def linattn_decode(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, kv_state: torch.Tensor,
                   k_state: torch.Tensor, *, eps: float = 1e-12, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """One recurrent step; ``kv_state``/``k_state`` are updated IN PLACE.

    q, k ``[B, H, 1, 16]`` or ``[B, H, 16]`` (raw), v ``[B, H, 1, dv]`` or ``[B, H, dv]``;
    ``kv_state [B, H, 1, dv, 273]``, ``k_state [B, H, 1, 1, 273]`` (fp32 or bf16).
    Returns ``y [B, 1, H*dv]`` in ``q.dtype`` (the layout recurrent_forward hands to out_proj,
    linear_attention.py:251).
    """
    _need_cuda(q, k, v, kv_state, k_state)
    if q.dim() == 4:
        q, k, v = q[:, :, 0], k[:, :, 0], v[:, :, 0]
    B, H, d = q.shape
    dv = v.shape[-1]
    if kv_state.shape != (B, H, 1, dv, EXPANDED_DIM) or k_state.shape != (B, H, 1, 1, EXPANDED_DIM):
        raise ValueError(f"state shapes {tuple(kv_state.shape)}, {tuple(k_state.shape)} do not match B={B} H={H} dv={dv}")
    if not (kv_state.is_contiguous() and k_state.is_contiguous()):
        raise ValueError("kv_state / k_state must be contiguous")
    if kv_state.dtype != k_state.dtype:
        raise TypeError("kv_state and k_state must share a dtype")
    for t, n in ((q, "q"), (k, "k"), (v, "v")):
        _inner_contig(t, n)
    if out is None:
        out = torch.empty(B, 1, H * dv, dtype=q.dtype, device=q.device)
    y = out.view(B, H, dv)
    code = _capi.native().linattn_decode(
        q, k, v, y, kv_state, k_state,
        B, H, d, dv, q.stride()[:2], k.stride()[:2],
        v.stride()[:2], y.stride()[:2],
        _dt(q.dtype), _dt(kv_state.dtype), float(eps))
    _capi.check(code, "based_linattn_decode")
    return out


def swa_prefill(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, window_left: int,
                softmax_scale: Optional[float] = None, *, impl: str = "auto",
                out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Causal sliding-window softmax attention; q, k, v ``[B, L, H, hd]`` (views into a packed
    qkv tensor are fine).  Query i sees keys ``[i - window_left, i]`` (slide_attention.py:97)."""
    _need_cuda(q, k, v)
    B, L, H, hd = q.shape
    if k.shape != q.shape or v.shape != q.shape:
        raise ValueError("q, k, v shapes disagree")
    for t, n in ((q, "q"), (k, "k"), (v, "v")):
        _inner_contig(t, n)
    if out is None:
        out = torch.empty(B, L, H, hd, dtype=q.dtype, device=q.device)
    scale = hd ** -0.5 if softmax_scale is None else float(softmax_scale)
    if out.numel() == 0:
        return out
    code = _capi.native().swa_prefill(
        q, k, v, out, B, L, H, hd,
        q.stride()[:3], k.stride()[:3],
        v.stride()[:3], out.stride()[:3],
        int(window_left), scale, _dt(q.dtype), _IMPLS[impl])
    _capi.check(code, "based_swa_prefill")
    return out


def swa_decode(q: torch.Tensor, k_new: torch.Tensor, v_new: torch.Tensor, kv_cache: torch.Tensor,
               cache_seqlens, window_left: int, softmax_scale: Optional[float] = None, *,
               rotary_cos: Optional[torch.Tensor] = None, rotary_sin: Optional[torch.Tensor] = None,
               out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """One decode step: optional RoPE at the new position, append to ``kv_cache
    [B, maxL, 2, H, hd]`` IN PLACE, attend over the window (slide_attention.py:414-427).
    q, k_new, v_new ``[B, 1, H, hd]``; ``cache_seqlens`` an int or an int32 ``[B]`` CUDA tensor."""
    _need_cuda(q, k_new, v_new, kv_cache)
    B, one, H, hd = q.shape
    assert one == 1
    if not kv_cache.is_contiguous() or kv_cache.shape[0] < B or kv_cache.shape[2:] != (2, H, hd):
        raise ValueError("kv_cache must be contiguous [B, maxL, 2, H, hd]")
    if kv_cache.dtype != q.dtype:
        raise TypeError("kv_cache and q must share a dtype")
    q3, k3, v3 = q[:, 0], k_new[:, 0], v_new[:, 0]
    for t, n in ((q3, "q"), (k3, "k_new"), (v3, "v_new")):
        _inner_contig(t, n)
    if out is None:
        out = torch.empty(B, 1, H, hd, dtype=q.dtype, device=q.device)
    o3 = out[:, 0]
    if torch.is_tensor(cache_seqlens):
        if cache_seqlens.dtype != torch.int32 or not cache_seqlens.is_cuda or not cache_seqlens.is_contiguous():
            raise TypeError("cache_seqlens must be a contiguous int32 CUDA tensor")
        lens_ptr, lens_scalar = cache_seqlens, 0
    else:
        lens_ptr, lens_scalar = None, int(cache_seqlens)
    rdim = 0
    if rotary_cos is not None:
        if rotary_cos.dtype != q.dtype or rotary_sin.dtype != q.dtype:
            raise TypeError("rotary tables must be in the q dtype")
        if not (rotary_cos.is_contiguous() and rotary_sin.is_contiguous()):
            raise ValueError("rotary tables must be contiguous")
        rdim = 2 * rotary_cos.shape[-1]
    scale = hd ** -0.5 if softmax_scale is None else float(softmax_scale)
    code = _capi.native().swa_decode(
        q3, k3, v3, o3, kv_cache, lens_ptr, lens_scalar,
        rotary_cos,
        rotary_sin, rdim,
        B, H, hd, kv_cache.shape[1], q3.stride()[:2], k3.stride()[:2],
        v3.stride()[:2], o3.stride()[:2],
        int(window_left), scale, _dt(q.dtype))
    _capi.check(code, "based_swa_decode")
    return out


def rotary_apply_(x: torch.Tensor, rotary_cos: torch.Tensor, rotary_sin: torch.Tensor, seqlen_offset=0) -> torch.Tensor:
    """In-place non-interleaved RoPE on ``x [B, L, H, hd]`` (a view into packed qkv is fine);
    ``seqlen_offset`` an int or an int32 ``[B]`` CUDA tensor (based/ops/triton/rotary.py:68-105)."""
    _need_cuda(x, rotary_cos, rotary_sin)
    B, L, H, hd = x.shape
    _inner_contig(x, "x")
    if rotary_cos.dtype != x.dtype or rotary_sin.dtype != x.dtype:
        raise TypeError("rotary tables must be in the dtype of x")
    if not (rotary_cos.is_contiguous() and rotary_sin.is_contiguous()):
        raise ValueError("rotary tables must be contiguous")
    if x.numel() == 0:
        return x
    if torch.is_tensor(seqlen_offset):
        if seqlen_offset.dtype != torch.int32 or not seqlen_offset.is_cuda:
            raise TypeError("seqlen_offset tensor must be int32 on CUDA")
        off_ptr, off_scalar = seqlen_offset, 0
        max_pos = None
    else:
        off_ptr, off_scalar = None, int(seqlen_offset)
        if off_scalar + L > rotary_cos.shape[0]:
            raise ValueError("rotary tables are shorter than seqlen_offset + L")
    code = _capi.native().rotary_apply(
        x, B, L, H, hd, x.stride()[:3], rotary_cos, rotary_sin,
        2 * rotary_cos.shape[-1], off_ptr, off_scalar, _dt(x.dtype))
    _capi.check(code, "based_rotary_apply")
    return x


def gated_conv_prefill(u: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None, *,
                       state: Optional[torch.Tensor] = None, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``silu(causal_depthwise_conv(u1) + bias) * u2`` with ``u1, u2`` the halves of ``u [B, L, 2*di]``.

    ``weight [di, k]`` (or ``[di, 1, k]`` as nn.Conv1d stores it), ``bias [di]`` or None, both in one
    dtype (float32 or bfloat16).  ``state [B, di, k]`` (dtype of ``u``), when given, receives the
    last k inputs of the convolution (convolution.py:63-67).  Returns ``v [B, L, di]``.
    """
    _need_cuda(u, weight, bias, state)
    B, L, two_di = u.shape
    di = two_di // 2
    weight = weight.reshape(weight.shape[0], -1)
    k = weight.shape[1]
    if weight.shape[0] != di or two_di != 2 * di:
        raise ValueError("u must be [B, L, 2*di] and weight [di, k]")
    _inner_contig(u, "u")
    weight = weight.contiguous()
    if bias is not None:
        bias = bias.to(weight.dtype).contiguous()
    if out is None:
        out = torch.empty(B, L, di, dtype=u.dtype, device=u.device)
    else:
        _inner_contig(out, "out")
    if state is not None and (state.shape != (B, di, k) or state.dtype != u.dtype or not state.is_contiguous()):
        raise ValueError("state must be a contiguous [B, di, k] tensor of u's dtype")
    if B == 0 or L == 0:
        if state is not None:
            state.zero_()
        return out
    su = u.stride()[:2]
    code = _capi.native().gated_conv_prefill(
        u, u.data_ptr() + di * u.element_size(), out, state, weight, bias, B, L, di, k, su, su, out.stride()[:2],
        _dt(u.dtype), _dt(weight.dtype))
    _capi.check(code, "based_gated_conv_prefill")
    return out


def gated_conv_step(u: torch.Tensor, state: torch.Tensor, weight: torch.Tensor,
                    bias: Optional[torch.Tensor] = None, *, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """One decode step of :func:`gated_conv_prefill`; ``state [B, di, k]`` is updated IN PLACE
    (convolution.py:104-107).  ``u [B, 2*di]`` or ``[B, 1, 2*di]``; returns ``[B, di]``."""
    _need_cuda(u, state, weight, bias)
    if u.dim() == 3:
        u = u[:, 0]
    B, two_di = u.shape
    di = two_di // 2
    weight = weight.reshape(weight.shape[0], -1).contiguous()
    k = weight.shape[1]
    _inner_contig(u, "u")
    if bias is not None:
        bias = bias.to(weight.dtype).contiguous()
    if state.shape != (B, di, k) or state.dtype != u.dtype or not state.is_contiguous():
        raise ValueError("state must be a contiguous [B, di, k] tensor of u's dtype")
    if out is None:
        out = torch.empty(B, di, dtype=u.dtype, device=u.device)
    if B == 0:
        return out
    code = _capi.native().gated_conv_step(
        u, u.data_ptr() + di * u.element_size(), out, state, weight, bias, B, di, k, u.stride(0), u.stride(0), out.stride(0),
        _dt(u.dtype), _dt(weight.dtype))
    _capi.check(code, "based_gated_conv_step")
    return out


def add_rmsnorm(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None,
                residual: Optional[torch.Tensor] = None, *, eps: float = 1e-6, prenorm: bool = False,
                residual_in_fp32: bool = False, round_input: bool = False):
    """``z = x + residual``; ``out = rmsnorm(z) * weight (+ bias)`` in one pass; with ``prenorm`` returns
    ``(out, z)`` like rms_norm_fn (layer_norm.py:926-953).  ``z`` is fp32 when ``residual_in_fp32`` or
    when ``residual`` already is, else x's dtype.  ``round_input`` rounds ``z`` to x's dtype before the
    norm (the unfused ``norm(residual.to(weight.dtype))`` of block.py:134-137).  x ``[..., D]``."""
    _need_cuda(x, weight, bias, residual)
    D = x.shape[-1]
    x2 = _flat(x, D)
    _inner_contig(x2, "x")
    M = x.numel() // D
    res2, sr = None, 0
    if residual is not None:
        if residual.shape != x.shape:
            raise ValueError("residual must have x's shape")
        res2 = _flat(residual, D)
        _inner_contig(res2, "residual")
    res_dtype = torch.float32 if (residual_in_fp32 or (residual is not None and residual.dtype == torch.float32)) else x.dtype
    if res2 is not None:
        if res2.dtype != res_dtype:
            res2 = res2.to(res_dtype)
        sr = _row_stride(res2, D)
    weight = weight.contiguous()
    if bias is not None:
        bias = bias.to(weight.dtype).contiguous()
    out = torch.empty(x.shape, dtype=x.dtype, device=x.device)
    res_out = torch.empty(x.shape, dtype=res_dtype, device=x.device) if prenorm else None
    if M > 0:
        code = _capi.native().add_rmsnorm(
            x2, res2, weight, bias, out, res_out, M, D, _row_stride(x2, D), sr, D, D if prenorm else 0,
            eps, _dt(x.dtype), _dt(res_dtype), _dt(weight.dtype), round_input)
        _capi.check(code, "based_add_rmsnorm")
    return (out, res_out) if prenorm else out


_ACTS = {"silu": 0, "swiglu": 0, "sigmoid": 1, "glu": 1}


def gated_act(y: torch.Tensor, activation: str = "silu", out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``first_half * act(second_half)`` over the last dim of ``y [..., 2F]`` (mlp.py:141-154).  ``out``: a ``[..., F]``
    tensor or column slice to write (rows one constant stride apart)."""
    _need_cuda(y, out)
    F2 = y.shape[-1]
    F = F2 // 2
    y2 = _flat(y, F2)
    _inner_contig(y2, "y")
    M = y.numel() // F2 if F2 else 0
    if out is None:
        out = o2 = torch.empty(*y.shape[:-1], F, dtype=y.dtype, device=y.device)
    else:
        o2 = _rows(out, F)
        out = o2.reshape(*y.shape[:-1], F)
    if M > 0 and F > 0:
        sy = _row_stride(y2, F2)
        code = _capi.native().gated_act(y2, y2.data_ptr() + F * y2.element_size(), o2, M, F, sy, sy, _row_stride(o2, F),
                                        _ACTS[activation], _dt(y.dtype))
        _capi.check(code, "based_gated_act")
    return out


# Where a product goes to decode_linear; beyond, the library GEMM is the better tool.  us a launch in a chain of such launches with
# the weights from HBM, cuBLAS / ours (N x K, rows): 1024 x 1024 4.6 / 2.9 (16), 4.2 / 3.6 (32); 4096 x 1024 4.7 / 3.1, 4.8 / 4.3,
# 4.9 / 6.3 (64); 1024 x 3072 8.6 / 3.5, 7.2 / 5.3; 1792 x 1792 5.2 / 3.6, 5.2 / 5.8; 7168 x 1792 7.4 / 6.9, 7.5 / 8.0, with the gated
# activation 9.9 / 7.0, 9.9 / 8.5; 50280 x 1024 21 / 30.  So: up to 16 rows whatever K; up to 32 for a short K, for few enough
# outputs that every block of the kernel has an SM, and where the gated activation saves a launch (the convolution does not there: a
# BaseConv step of 24 rows, 7168 x 1792, 17.5 with the library, 20.0).
# With the gated activation and one round of blocks, some more.  An MLP whose second product is the library's, library / ours at 33 and 40
# rows (width x hidden): 512 x 1024 9.5 / 6.6, 9.5 / 6.7; 768 x 1536 10.9 / 10.0, 10.9 / 10.1; 1024 x 1024 10.3 / 8.8, 10.3 / 8.8; 1024 x 2048
# 12.3 / 12.4, 12.3 / 12.6, behind a norm 14.4 / 13.2, 14.4 / 13.4.  At 48 rows 1024 x 2048 is 12.4 / 12.6.  Up to 2368 outputs of the product all
# blocks have an SM: at 64 rows 512 x 1024 8.3 / 6.9, 1024 x 1024 10.4 / 9.0.
DECODE_LINEAR_MAX_ROWS, DECODE_LINEAR_MAX_ROWS_GATED, DECODE_LINEAR_MAX_OUTPUTS = 32, (64, 40), 8192


def decode_linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None, *,
                  epilogue: str = "plain", activation: str = "silu", conv_state: Optional[torch.Tensor] = None,
                  conv_weight: Optional[torch.Tensor] = None, conv_bias: Optional[torch.Tensor] = None,
                  out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``x W^T (+ bias)`` for the few rows of a decode step (bf16), with a fused epilogue:
    ``"plain"``; ``"f32"``: plain with an fp32 result; ``"gated"`` -> ``first_half * act(second_half)`` (mlp.py:146-154); ``"conv"`` -> the BaseConv
    decode step on the first half (``conv_state [M, N/2, k]`` updated in place), silu, gate by the second half
    (convolution.py:88-109, :205-211).  x ``[..., K]``; returns ``[..., N]`` or ``[..., N/2]``."""
    rows = None
    if type(x) is NormRows:
        rows, x = x, x.x
    _need_cuda(x, weight, bias, conv_state, conv_weight, conv_bias)
    if x.dtype != torch.bfloat16 or weight.dtype != torch.bfloat16:
        raise TypeError("decode_linear takes bfloat16 activations and weights")
    K = x.shape[-1]
    x2 = x.reshape(-1, K)
    _inner_contig(x2, "x")
    M, N = x2.shape[0], weight.shape[0]
    if weight.shape[1] != K or not weight.is_contiguous():
        raise ValueError("weight must be a contiguous [N, K] tensor")
    epi = {"plain": 0, "gated": 1, "conv": 2, "f32": 3}[epilogue]
    n_out = N // 2 if epi in (1, 2) else N
    dtype = torch.float32 if epi == 3 else torch.bfloat16
    out = torch.empty(M, n_out, dtype=dtype, device=x.device) if out is None else _rows(out, n_out)
    if out.dtype != dtype:
        raise TypeError(f"out must be {dtype}")
    if bias is not None:
        bias = bias.to(torch.bfloat16).contiguous()
    ck, cw_dt = 0, BASED_BF16
    if epi == 2:
        conv_weight = conv_weight.reshape(conv_weight.shape[0], -1).contiguous()
        ck, cw_dt = conv_weight.shape[1], _dt(conv_weight.dtype)
        if conv_bias is not None:
            conv_bias = conv_bias.to(conv_weight.dtype).contiguous()
        if conv_state.shape != (M, n_out, ck) or conv_state.dtype != torch.bfloat16 or not conv_state.is_contiguous():
            raise ValueError("conv_state must be a contiguous bfloat16 [M, N/2, k] tensor")
    if M > 0:
        code = _capi.native().decode_linear_scaled(
            x2, weight, bias, out,
            M, N, K, x2.stride(0), out.stride(0), epi, _ACTS[activation],
            conv_state if epi == 2 else None, conv_weight if epi == 2 else None,
            conv_bias if (epi == 2 and conv_bias is not None) else None, ck, cw_dt,
            rows.ss if rows is not None else None, rows.ss.shape[1] if rows is not None else 0, rows.eps if rows is not None else 0.0)
        _capi.check(code, "based_decode_linear")
    return out.reshape(*x.shape[:-1], n_out)


def decode_beside(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], f32_weight: Optional[torch.Tensor], x_gated: torch.Tensor,
                  fc1_weight: torch.Tensor, fc1_bias: Optional[torch.Tensor], activation: str, out_gated: torch.Tensor):
    """What the mixer and the MLP of a parallel layer do first in a step, in one launch: ``x W^T + b``, with ``f32_weight`` also
    ``x F^T`` in fp32, and the gated activation of ``x_gated W1^T + b1`` written to ``out_gated``.  Returns the first two; None, nothing
    launched, where :func:`decode_linear` would not take one of them or there are more than 32 rows."""
    K, N, F2 = x.shape[-1], weight.shape[0], fc1_weight.shape[0]
    # us apart / in one launch, weights from HBM, 1 and 16 rows (N x K, fp32 columns, F): 2048 x 1024, 0, 2048 5.9 / 4.1, 6.7 / 4.5 (32 rows
    # 8.1 / 5.4); 4096 x 1024, 16, 2048 7.9 / 4.7, 8.9 / 5.2; 512 x 256, 0, 512 4.0 / 2.4, 4.5 / 2.5; 2048 x 2048, 0, 2048 8.2 / 6.3, 9.8 / 7.0.
    # With more blocks than the device holds at once it saves nothing: 3584 x 1792, 0, 3584 10.9 / 11.9, 12.1 / 13.0; 4096 x 2048, 0, 4096
    # 12.3 / 13.0, 13.8 / 14.2; unless it takes the place of three: 7168 x 1792, 32, 3584 14.9 / 12.9, 16.1 / 13.9.
    if f32_weight is None and -(-N // 32) + -(-F2 // 32) > 2 * 148:
        return None
    if (x.numel() > DECODE_LINEAR_MAX_ROWS * K or x_gated.shape[:-1] != x.shape[:-1] or F2 % 16 or not _decode_rows(x, weight)
            or not _decode_rows(x_gated, fc1_weight, gated=True) or not (f32_weight is None or _decode_rows(x, f32_weight))
            or type(x) is not torch.Tensor or type(x_gated) is not torch.Tensor or out_gated.dtype != torch.bfloat16):
        return None
    for b, n in ((bias, N), (fc1_bias, F2)):
        if b is not None and not (type(b) in _PLAIN_TYPES and b.dtype == torch.bfloat16 and b.shape == (n,) and b.is_contiguous() and b.device == x.device):
            return None
    x2, g2, o2 = x.reshape(-1, K), x_gated.reshape(-1, x_gated.shape[-1]), _rows(out_gated, F2 // 2)
    M = x2.shape[0]
    out = torch.empty(*x.shape[:-1], N, dtype=x.dtype, device=x.device)
    f32 = torch.empty(*x.shape[:-1], f32_weight.shape[0], dtype=torch.float32, device=x.device) if f32_weight is not None else None
    code = _capi.native().decode_beside(x2, weight, bias, out, N, K, x2.stride(0), N, f32_weight, f32, f32_weight.shape[0] if f32 is not None else 0, g2,
                                        fc1_weight, fc1_bias, o2, F2, g2.shape[1], g2.stride(0), o2.stride(0), _ACTS[activation], M)
    _capi.check(code, "based_decode_beside")
    return out, f32


class NormRows:
    """Normed rows before their norm's last factor: ``x [..., D]`` bf16 is the stream times the norm's weight,
    ``ss [rows, n]`` sums of the stream's squares over ``n`` parts of a row.  The products of this module take it for a tensor (they apply the
    factor to their sums); nothing else does.  :func:`dense` gives the tensor it stands for."""
    __slots__ = ("x", "ss", "eps")

    def __init__(self, x, ss, eps):
        self.x, self.ss, self.eps = x, ss, eps

    shape = property(lambda self: self.x.shape)
    dtype = property(lambda self: self.x.dtype)
    device = property(lambda self: self.x.device)

    def size(self, *dim):
        return self.x.size(*dim)


def dense(x):
    """``x``, or the normed tensor a :class:`NormRows` stands for."""
    if type(x) is not NormRows:
        return x
    rstd = torch.rsqrt(x.ss.sum(1) / x.x.shape[-1] + x.eps)
    return (x.x.float() * rstd.view(*x.x.shape[:-1], 1)).to(x.x.dtype)


STEP_MAX_ROWS = 16


def step_weight(weight, bias=None) -> bool:
    """True for a weight (and bias) that :func:`decode_linear` and :func:`linear_add_norm` take for a few rows."""
    return (type(weight) in _PLAIN_TYPES and weight.dtype == torch.bfloat16 and weight.dim() == 2 and weight.is_contiguous()
            and weight.shape[1] % 32 == 0 and weight.shape[0] % 8 == 0 and weight.shape[0] <= DECODE_LINEAR_MAX_OUTPUTS
            and weight.data_ptr() % 16 == 0
            and (bias is None or (type(bias) in _PLAIN_TYPES and bias.dtype == torch.bfloat16 and bias.is_contiguous())))


def linear_add_norm(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], residual: torch.Tensor, norm_weight: torch.Tensor,
                    *, eps: float) -> NormRows:
    """``x W^T (+ bias)`` of at most 16 bf16 rows joins the fp32 stream ``residual [..., N]`` IN PLACE, unrounded; returns the
    stream's norm with the weights ``norm_weight``."""
    _need_cuda(x, weight, bias, residual, norm_weight)
    N, K = weight.shape
    M = x.numel() // K
    if x.dtype != torch.bfloat16 or not step_weight(weight, bias) or x.shape[-1] != K or not 0 < M <= STEP_MAX_ROWS:
        raise ValueError("linear_add_norm takes at most 16 bfloat16 rows and a contiguous bfloat16 [N, K] weight")
    if residual.dtype != torch.float32 or not residual.is_contiguous() or residual.shape != (*x.shape[:-1], N):
        raise TypeError("residual must be a contiguous float32 tensor with the product's shape")
    if norm_weight.dtype != torch.bfloat16 or norm_weight.shape != (N,) or not norm_weight.is_contiguous():
        raise TypeError("norm weights must be contiguous bfloat16 [N]")
    x2 = _flat(x, K)
    _inner_contig(x2, "x")
    out = torch.empty(residual.shape, dtype=torch.bfloat16, device=x.device)
    ss = torch.empty(M, N // 8, dtype=torch.float32, device=x.device)
    code = _capi.native().decode_linear_add(x2, weight, bias, M, N, K, _row_stride(x2, K), residual, norm_weight, out, ss)
    _capi.check(code, "based_decode_linear_add")
    return NormRows(out, ss, eps)


def plain_bf16(like: torch.Tensor, *tensors) -> bool:
    """True when all tensors (plain ones or parameters) are contiguous, 16-byte aligned bf16 on ``like``'s device."""
    return all(type(t) in _PLAIN_TYPES and not _wrapped(t) for t in tensors) and _capi.native().plain_bf16(like, *tensors)


def prompt_layer(*args):
    """The products of a prompt's layer in one call (``prompt_layer`` in csrc_host/native.cpp)."""
    out = _capi.native().prompt_layer(*args)
    if type(out) is int:
        _capi.check(out, "prompt_layer")
    return out


_PLAIN_TYPES = (torch.Tensor, torch.nn.Parameter)


def _observed() -> bool:
    """True while a dispatch or function mode (a FLOP counter, ``make_fx``, a logger) watches torch's operators: a product must then be
    one of them.  ``torch.device`` as a context is a function mode too, but only sets the device of new tensors."""
    n = torch._C._len_torch_function_stack()
    return torch._C._len_torch_dispatch_stack() > 0 or (
        n > 0 and any(type(torch._C._get_function_stack_at(i)) is not _DeviceContext for i in range(n)))


def _decode_rows(x: torch.Tensor, weight: torch.Tensor, gated: bool = False) -> bool:
    """True when ``x W^T`` is a decode-step product the library's own kernel should run: a few bf16 rows in a layout it takes, and
    nothing around the call that only a torch operator serves (autograd, autocast, forward mode, function transforms, tracing, modes).
    ``gated``: its epilogue takes the place of the gated activation's launch."""
    if type(x) is NormRows:
        x = x.x
    K = x.shape[-1] if x.dim() else 0
    most = DECODE_LINEAR_MAX_ROWS
    if gated and K <= 1024 and weight.shape[0] <= 2 * 8 * 296:
        most = DECODE_LINEAR_MAX_ROWS_GATED[weight.shape[0] > 2 * 8 * 148]
    if not (0 < x.numel() <= K * most and x.is_cuda and x.dtype == weight.dtype == torch.bfloat16):
        return False
    if type(x) is not torch.Tensor or type(weight) not in _PLAIN_TYPES or weight.dim() != 2 or weight.shape[0] > DECODE_LINEAR_MAX_OUTPUTS:
        return False
    if x.numel() > 16 * K and not (K <= 1024 or (weight.shape[0] <= 8 * 148 and K <= 3072) or (gated and K <= 2048)):
        return False
    return (K % 32 == 0 and weight.shape[1] == K and weight.shape[0] % 8 == 0 and weight.is_contiguous()
            and (x.is_contiguous() or (x.stride(-1) == 1 and all(st % 8 == 0 for st in x.stride()[:-1]))) and _unwatched(x, weight))


def _unwatched(x, weight) -> bool:
    """True when nothing around a product needs it to be a torch operator, and both operands are 16-byte aligned."""
    return (x.device == weight.device and not torch.is_grad_enabled() and not torch.is_autocast_enabled("cuda")
            and _forward_ad._current_level < 0 and torch._C._get_tracing_state() is None
            and not _observed() and not _wrapped(x) and not _wrapped(weight) and x.data_ptr() % 16 == 0 and weight.data_ptr() % 16 == 0)


# From here on a prompt's products go to prompt_linear where that saves a launch: a tile of it has 128 rows (or two times as many), and
# with fewer it computes padding.
PROMPT_MIN_ROWS = 128


def _prompt_rows(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None) -> bool:
    """True when :func:`prompt_linear` takes ``x W^T + b``: a prompt's rows in bf16, one stride apart, and nothing around the call that only
    a torch operator serves."""
    if type(x) is NormRows:
        x = x.x
    K = x.shape[-1] if x.dim() > 1 else 0
    if not (K > 0 and PROMPT_MIN_ROWS * K <= x.numel() < K << 31 and x.is_cuda and x.dtype == weight.dtype == torch.bfloat16):
        return False
    if type(x) is not torch.Tensor or type(weight) not in _PLAIN_TYPES or weight.dim() != 2 or weight.shape[1] != K:
        return False
    if bias is not None and not (type(bias) in _PLAIN_TYPES and bias.dtype == torch.bfloat16 and bias.is_contiguous() and bias.data_ptr() % 16 == 0
                                 and bias.shape == weight.shape[:1] and bias.device == x.device and not _wrapped(bias)):
        return False
    return K % 8 == 0 and weight.shape[0] % 8 == 0 and weight.is_contiguous() and x.is_contiguous() and _unwatched(x, weight)


def prompt_linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None, *, epilogue: str = "plain",
                  activation: str = "silu", out: Optional[torch.Tensor] = None, tile: int = -1) -> torch.Tensor:
    """``x W^T (+ bias)`` for the rows of a prompt (bf16, tensor cores), with a fused epilogue: ``"plain"``, ``"f32"`` (an fp32 result) or
    ``"gated"`` -> ``first_half * act(second_half)`` (mlp.py:146-154; not rounded in between).  x ``[..., K]``, also a :class:`NormRows`;
    ``tile`` chooses the kernel's tile (tests)."""
    rows = None
    if type(x) is NormRows:
        rows, x = x, x.x
    _need_cuda(x, weight, bias, out)
    if x.dtype != torch.bfloat16 or weight.dtype != torch.bfloat16 or (bias is not None and bias.dtype != torch.bfloat16):
        raise TypeError("prompt_linear takes bfloat16 activations, weights and bias")
    K, N = x.shape[-1], weight.shape[0]
    if weight.shape[1] != K or not weight.is_contiguous() or (bias is not None and (bias.numel() != N or not bias.is_contiguous())):
        raise ValueError("weight must be a contiguous [N, K] tensor, bias [N]")
    x2 = _flat(x, K)
    _inner_contig(x2, "x")
    M = x.numel() // K
    epi = {"plain": 0, "gated": 1, "f32": 3}[epilogue]
    n_out = N // 2 if epi == 1 else N
    dtype = torch.float32 if epi == 3 else torch.bfloat16
    shape = (*x.shape[:-1], n_out)
    if out is None:
        out = o2 = torch.empty(shape, dtype=dtype, device=x.device)
        so = n_out
    else:
        if out.dtype != dtype:
            raise TypeError(f"out must be {dtype}")
        o2 = _rows(out, n_out)
        if o2.shape[0] != M:
            raise ValueError("out must have a row for each of x's")
        so, out = o2.stride(0), out if out.shape == shape else o2.reshape(shape)
    if M > 0:
        code = _capi.native().prompt_linear(x2, weight, bias, o2, M, N, K, _row_stride(x2, K), K, so, epi, _ACTS[activation],
                                            None if rows is None else rows.ss, 0 if rows is None else rows.ss.shape[1],
                                            0.0 if rows is None else rows.eps, tile)
        _capi.check(code, "based_prompt_linear")
    return out


def prompt_conv(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], conv_weight: torch.Tensor, *,
                state: Optional[torch.Tensor] = None, tile: int = -1) -> torch.Tensor:
    """``x W^T + bias`` and :func:`gated_conv_prefill` of it in one launch, for the tokens of a prompt: x ``[B, L, K]`` bf16 (or a
    :class:`NormRows`), ``conv_weight [di, 3]`` (or ``[di, 1, 3]``) bf16; ``state [B, di, 3]`` bf16, when given, receives the last three inputs
    of the convolution.  Returns ``[B, L, di]``."""
    rows = None
    if type(x) is NormRows:
        rows, x = x, x.x
    _need_cuda(x, weight, bias, conv_weight, state)
    if x.dtype != torch.bfloat16 or weight.dtype != torch.bfloat16 or (bias is not None and bias.dtype != torch.bfloat16):
        raise TypeError("prompt_conv takes bfloat16 activations, weights and bias")
    B, L, K = x.shape
    N, di = weight.shape[0], weight.shape[0] // 2
    if weight.shape[1] != K or not weight.is_contiguous() or not x.is_contiguous() or (bias is not None and (bias.shape != (N,) or not bias.is_contiguous())):
        raise ValueError("x and weight must be contiguous, bias [N]")
    conv_weight = conv_weight.reshape(conv_weight.shape[0], -1).contiguous()
    if conv_weight.shape != (di, 3) or conv_weight.dtype != torch.bfloat16:
        raise ValueError("prompt_conv takes three bfloat16 taps a channel")
    if state is not None and (state.shape != (B, di, 3) or state.dtype != torch.bfloat16 or not state.is_contiguous()):
        raise ValueError("state must be a contiguous bfloat16 [B, di, 3] tensor")
    out = torch.empty(B, L, di, dtype=torch.bfloat16, device=x.device)
    if out.numel() > 0:
        code = _capi.native().prompt_linear_conv(x, weight, bias, out, B * L, N, K, K, K, L, conv_weight, state,
                                                 None if rows is None else rows.ss, 0 if rows is None else rows.ss.shape[1],
                                                 0.0 if rows is None else rows.eps, tile)
        _capi.check(code, "based_prompt_linear_conv")
    return out


def prompt_add_norm(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], residual: torch.Tensor, norm_weight: torch.Tensor,
                    *, eps: float, tile: int = -1) -> "NormRows":
    """:func:`linear_add_norm` for the rows of a prompt."""
    _need_cuda(x, weight, bias, residual, norm_weight)
    N, K = weight.shape
    if x.dtype != torch.bfloat16 or weight.dtype != torch.bfloat16 or x.shape[-1] != K or not weight.is_contiguous() or (
            bias is not None and (bias.dtype != torch.bfloat16 or bias.shape != (N,) or not bias.is_contiguous())):
        raise TypeError("prompt_add_norm takes bfloat16 rows, a contiguous bfloat16 [N, K] weight and bias [N]")
    if residual.dtype != torch.float32 or not residual.is_contiguous() or residual.shape != (*x.shape[:-1], N):
        raise TypeError("residual must be a contiguous float32 tensor with the product's shape")
    if norm_weight.dtype != torch.bfloat16 or norm_weight.shape != (N,) or not norm_weight.is_contiguous():
        raise TypeError("norm weights must be contiguous bfloat16 [N]")
    x2 = _flat(x, K)
    _inner_contig(x2, "x")
    M = x.numel() // K
    out = torch.empty(residual.shape, dtype=torch.bfloat16, device=x.device)
    ss = torch.empty(M, _capi.lib().based_prompt_linear_sums(M, N, K, tile), dtype=torch.float32, device=x.device)
    if M > 0:
        code = _capi.native().prompt_linear_add(x2, weight, bias, M, N, K, _row_stride(x2, K), K, residual, norm_weight, out, ss, tile)
        _capi.check(code, "based_prompt_linear_add")
    return NormRows(out, ss, eps)


def linear(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``nn.functional.linear`` for the mixers: the decode-step kernel for a few bf16 rows, the prompt kernel for rows that wait for their
    norm's factor, cuBLAS otherwise."""
    if _decode_rows(x, weight) and (bias is None or (type(bias) in _PLAIN_TYPES and bias.dtype == torch.bfloat16
                                                     and bias.shape == weight.shape[:1] and bias.device == x.device)):
        return decode_linear(x, weight, bias)
    if type(x) is NormRows:
        if _prompt_rows(x, weight, bias):
            return prompt_linear(x, weight, bias)
        x = dense(x)
    elif x.dtype is torch.float32 and _split_rows(x, (weight,), bias):
        return linear_split(x, (weight,), bias)
    return torch.nn.functional.linear(x, weight, bias)


def _split_rows(x: torch.Tensor, weights, bias: Optional[torch.Tensor] = None) -> bool:
    """True when :func:`linear_split` takes ``x [W0; W1; ..]^T + b`` and is the faster way: a prompt's rows in fp32, enough of them to fill
    its tiles, and nothing around the call that only a torch operator serves."""
    if type(x) is not torch.Tensor or x.dtype != torch.float32 or not x.is_cuda or x.dim() < 2 or not x.is_contiguous():
        return False
    K = x.shape[-1]
    if K % 8 or x.numel() < PROMPT_MIN_ROWS * K or x.numel() >= K << 31:
        return False
    if any(type(w) not in _PLAIN_TYPES or w.dtype != torch.float32 or w.dim() != 2 or w.shape[1] != K or not w.is_contiguous() for w in weights):
        return False
    N = sum(w.shape[0] for w in weights)
    if N % 4 or not 0 < len(weights) <= 4 or any(w.shape[0] == 0 for w in weights):
        return False
    if x.numel() // K * N < SPLIT_MIN_OUTPUTS or x.numel() * N < SPLIT_MIN_PRODUCTS or N * K > SPLIT_MAX_WEIGHT:
        return False
    if bias is not None and not (type(bias) in _PLAIN_TYPES and bias.dtype == torch.float32 and bias.is_contiguous() and bias.shape == (N,)
                                 and bias.device == x.device and not _wrapped(bias)):
        return False
    if torch.backends.cuda.matmul.fp32_precision not in ("none", "ieee"):   # the caller lets products round: the library's one pass
        return False
    return all(_unwatched(x, w) for w in weights)


# us with the library / linear_split (rows; outputs x K): 256 21 / 25, 512 29 / 25 (1024 x 1024); 1024 21 / 25, 2048 29 / 26.5 (256 x 1024);
# 512 24.5 / 17.6 (2048 x 512); 1024 16 / 16.2 (512 x 512); 2048 9.5 / 12.4, 4096 14.5 / 12.7 (256 x 256).
SPLIT_MIN_OUTPUTS, SPLIT_MIN_PRODUCTS = 1 << 19, 1 << 28
# The call's scratch, 6 bytes an element of the weights and of as many rows as are split at a time, is at most 128 MB with up to
# this many elements of weights (48 MB); a larger matrix (a model's head) stays with the library, which takes none.
SPLIT_MAX_WEIGHT = 1 << 23


def linear_split(x: torch.Tensor, weights, bias: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``x [W0; W1; ..]^T (+ bias)`` in fp32 on the tensor cores, for the rows of a prompt: x ``[..., K]``, up to four weights ``[n, K]``.
    An operand is three bf16 values; what is left out of a product is no more than rounding it once; sums are fp32."""
    _need_cuda(x, *weights, bias)
    K = x.shape[-1]
    if any(t.dtype != torch.float32 for t in (x, *weights)) or any(w.shape[1] != K or not w.is_contiguous() for w in weights) or not 0 < len(weights) <= 4:
        raise TypeError("linear_split takes float32 rows and one to four contiguous float32 [n, K] weights")
    N = sum(w.shape[0] for w in weights)
    if bias is not None and (bias.dtype != torch.float32 or bias.shape != (N,) or not bias.is_contiguous()):
        raise TypeError("bias must be contiguous float32 [N]")
    x2 = _flat(x, K)
    _inner_contig(x2, "x")
    M = x.numel() // K if K else 0
    out = torch.empty(*x.shape[:-1], N, dtype=torch.float32, device=x.device)
    if M > 0:
        scratch = torch.empty(_capi.lib().based_linear_f32_scratch_bytes(M, N, K), dtype=torch.uint8, device=x.device)
        none = 4 - len(weights)
        code = _capi.native().linear_f32(x2, *weights, *[None] * none, *[w.shape[0] for w in weights], *[0] * none, bias, out, M, K,
                                         _row_stride(x2, K), scratch, scratch.numel())
        _capi.check(code, "based_linear_f32")
    return out


def rotary_qkv_cache_(qkv: torch.Tensor, rotary_cos: torch.Tensor, rotary_sin: torch.Tensor,
                      kv_cache: torch.Tensor) -> torch.Tensor:
    """Prompt pass of the sliding-window mixer: whole-head RoPE on q and k of packed ``qkv [B, L, 3, H, hd]`` in
    place, and rotated k plus v written to ``kv_cache[:B, :L]`` (``[*, max_seqlen, 2, H, hd]``) in the same launch
    (slide_attention.py:553-556 and :255-281).  bf16 only; returns ``qkv``."""
    _need_cuda(qkv, rotary_cos, rotary_sin, kv_cache)
    B, L, three, H, hd = qkv.shape
    if three != 3 or qkv.dtype != torch.bfloat16 or kv_cache.dtype != torch.bfloat16:
        raise TypeError("rotary_qkv_cache_ takes a bfloat16 [B, L, 3, H, hd] tensor and a bfloat16 cache")
    _inner_contig(qkv, "qkv")
    if rotary_cos.shape[-1] * 2 != hd or rotary_cos.shape[0] < L or rotary_cos.dtype != torch.bfloat16:
        raise ValueError("rotary tables must be bfloat16 [>= L, hd/2]")
    if not (rotary_cos.is_contiguous() and rotary_sin.is_contiguous()):
        raise ValueError("rotary tables must be contiguous")
    if (kv_cache.shape[0] < B or kv_cache.shape[1] < L or tuple(kv_cache.shape[2:]) != (2, H, hd)
            or kv_cache.stride()[2:] != (H * hd, hd, 1)):
        raise ValueError("kv_cache must be [>= B, >= L, 2, H, hd] with the last three dims contiguous")
    if qkv.numel() == 0:
        return qkv
    code = _capi.native().rotary_qkv_cache(
        qkv, B, L, H, hd, qkv.stride()[:4], rotary_cos, rotary_sin,
        kv_cache, kv_cache.stride()[:2])
    _capi.check(code, "based_rotary_qkv_cache")
    return qkv


def tp_outproj_workspace_bytes(world: int, max_rows: int, n_out: int) -> int:
    """Size of one rank's receive workspace for :func:`tp_outproj_allreduce`."""
    n = _capi.lib().based_tp_outproj_workspace_bytes(int(world), int(max_rows), int(n_out))
    if n == 0:
        raise ValueError("tp_outproj: world must be 1..8, max_rows >= 1 and n_out a multiple of 8")
    return n


def tp_outproj_workspace_init_(ws: torch.Tensor) -> torch.Tensor:
    """Prepare a workspace (zero flags, call counter = 1).  Once, by its owner, before any rank's first call."""
    _need_cuda(ws)
    with torch.cuda.device(ws.device):
        _capi.check(_capi.lib().based_tp_outproj_workspace_init(ws.data_ptr(), ws.numel() * ws.element_size(), _stream()),
                    "based_tp_outproj_workspace_init")
    return ws


def tp_outproj_allreduce(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor], workspace_ptrs, max_rows: int,
                         rank: int, world: int, *, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Row-parallel ``x W^T`` summed over the tensor-parallel ranks (+ bias), one kernel per rank
    (based/ops/fused_dense.py:239-246 as GEMM + all-reduce in one launch).  ``x [..., K_local]`` bf16 with at most
    ``max_rows`` rows, ``weight [N, K_local]`` bf16 contiguous; ``workspace_ptrs`` the device addresses of every rank's
    workspace as mapped in this process.  A collective: every rank calls it with the same shapes."""
    _need_cuda(x, weight, bias)
    if x.dtype != torch.bfloat16 or weight.dtype != torch.bfloat16:
        raise TypeError("tp_outproj_allreduce takes bfloat16 activations and weights")
    K = x.shape[-1]
    x2 = x.reshape(-1, K)
    _inner_contig(x2, "x")
    M, N = x2.shape[0], weight.shape[0]
    if weight.shape[1] != K or not weight.is_contiguous():
        raise ValueError("weight must be a contiguous [N, K] tensor")
    if not 0 < M <= max_rows:
        raise ValueError(f"tp_outproj_allreduce: {M} rows, workspace built for at most {max_rows}")
    if len(workspace_ptrs) != world:
        raise ValueError("one workspace address per rank is needed")
    if bias is not None:
        bias = bias.to(torch.bfloat16).contiguous()
    if out is None:
        out = torch.empty(M, N, dtype=torch.bfloat16, device=x.device)
    o2 = out.reshape(-1, N)
    with torch.cuda.device(x.device):
        code = _capi.lib().based_tp_outproj_allreduce(
            x2.data_ptr(), weight.data_ptr(), bias.data_ptr() if bias is not None else None, o2.data_ptr(), M, N, K,
            x2.stride(0), o2.stride(0), _capi.pointers(workspace_ptrs), int(max_rows), int(rank), int(world), _stream())
    _capi.check(code, "based_tp_outproj_allreduce")
    return out.reshape(*x.shape[:-1], N)


def tp_outproj_allreduce_emulated(xs, weights, bias, workspaces, max_rows: int):
    """All ranks of :func:`tp_outproj_allreduce` inside one cooperative launch on one GPU: ``xs[r] [M, K]``,
    ``weights[r] [N, K]``, ``workspaces[r]`` (prepared uint8 tensors), all on the same device.  Returns the list of the
    ranks' outputs.  For checking the exchange protocol with a single GPU."""
    world = len(xs)
    _need_cuda(*xs, *weights, bias, *workspaces)
    M, K = xs[0].shape
    N = weights[0].shape[0]
    outs = [torch.empty(M, N, dtype=torch.bfloat16, device=xs[0].device) for _ in range(world)]
    if bias is not None:
        bias = bias.to(torch.bfloat16).contiguous()
    with torch.cuda.device(xs[0].device):
        code = _capi.lib().based_tp_outproj_allreduce_emulated(
            _capi.pointers([t.data_ptr() for t in xs]), _capi.pointers([t.data_ptr() for t in weights]),
            bias.data_ptr() if bias is not None else None, _capi.pointers([t.data_ptr() for t in outs]), M, N, K,
            xs[0].stride(0), outs[0].stride(0), _capi.pointers([t.data_ptr() for t in workspaces]), int(max_rows), world,
            _stream())
    _capi.check(code, "based_tp_outproj_allreduce_emulated")
    return outs


# --------------------------------------------------------------------------- stateful mixers of hybrid stacks
# ``pos``: position of a call's first token, an int or an int32 CUDA tensor with one entry per batch row.  A sequence
# that starts (position 0) reads no state, so state tensors need no clearing between sequences.

def linear_f32(x: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    """``x W^T`` with an fp32 result (fp32 accumulation of the operands' products, not rounded to their dtype)."""
    if _decode_rows(x, weight):
        return decode_linear(x, weight, epilogue="f32")
    x = dense(x)
    _need_cuda(x, weight)
    if x.dtype == torch.float32:
        return linear(x, weight)
    y = torch.mm(x.reshape(-1, x.shape[-1]), weight.t(), out_dtype=torch.float32)
    return y.view(*x.shape[:-1], weight.shape[0])


def stream_norm(residual: torch.Tensor, w1: torch.Tensor, w2: Optional[torch.Tensor] = None, *,
                branch: Optional[torch.Tensor] = None, mult: float = 1.0, tokens: Optional[torch.Tensor] = None,
                table: Optional[torch.Tensor] = None, table_norm: Optional[torch.Tensor] = None, eps: float = 1e-6):
    """The norm step of a parallel block: the fp32 stream ``residual [..., D]`` becomes ``residual + mult * branch`` (or,
    with ``tokens``, ``rmsnorm(table[token]) * table_norm``) IN PLACE; returns its RMSNorm scaled by ``w1`` and by ``w2``
    (None without ``w2``), in the weights' dtype."""
    _need_cuda(residual, w1, w2, branch, tokens, table, table_norm)
    D = residual.shape[-1]
    if residual.dtype != torch.float32 or not residual.is_contiguous():
        raise TypeError("residual must be a contiguous float32 tensor")
    M = residual.numel() // D if D else 0
    out1 = torch.empty(residual.shape, dtype=w1.dtype, device=residual.device)
    out2 = torch.empty_like(out1) if w2 is not None else None
    sb = 0
    if branch is not None:
        branch = branch.reshape(-1, D)
        _inner_contig(branch, "branch")
        sb = branch.stride(0)
    V = 0
    if tokens is not None:
        if tokens.dtype != torch.int64 or tokens.numel() != M:
            raise TypeError("tokens must be int64, one per row")
        tokens, V = tokens.contiguous(), table.shape[0]
    for t in (w1, w2, branch, table, table_norm):
        if t is not None and (t.dtype != w1.dtype or (t is not branch and not t.is_contiguous())):
            raise TypeError("weights, table and branch must share a dtype and be contiguous")
    if M > 0:
        code = _capi.native().stream_norm(
            tokens, table, table_norm, V, branch, sb, float(mult), residual,
            w1, w2, out1, out2, M, D, float(eps), _dt(w1.dtype))
        _capi.check(code, "based_stream_norm")
    return out1, out2


def rmsnorm(x: torch.Tensor, weight: torch.Tensor, eps: float) -> torch.Tensor:
    """``x / sqrt(mean(x^2) + eps) * weight`` over the last dim of ``x [..., D]`` (a column slice is fine), contiguous."""
    _need_cuda(x, weight)
    D = x.shape[-1]
    x2 = flat_rows(x) if x.dim() > 1 else x.view(1, D)
    _inner_contig(x2, "x")
    out = torch.empty(x.shape, dtype=x.dtype, device=x.device)
    if weight.dtype != x.dtype:
        raise TypeError("weight must be in x's dtype")
    if out.numel() > 0:
        code = _capi.native().rmsnorm(x2, weight, out, x2.shape[0], D, x2.stride(0), D,
                                         float(eps), _dt(x.dtype))
        _capi.check(code, "based_rmsnorm")
    return out


def short_conv(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None, *,
               ring: Optional[torch.Tensor] = None, pos=0, silu: bool = False) -> torch.Tensor:
    """Depthwise causal convolution ``x [B, L, C]`` by ``weight [C, taps]`` for tokens that start at ``pos``; ``ring
    [B, taps, C]`` carries earlier inputs (position p in slot p mod taps) and is updated.  Contiguous ``[B, L, C]``."""
    _need_cuda(x, weight, bias, ring)
    B, L, C = x.shape
    taps = weight.shape[1]
    _inner_contig(x, "x")
    if weight.shape[0] != C or weight.dtype != x.dtype or not weight.is_contiguous() or (bias is not None and bias.dtype != x.dtype):
        raise ValueError("weight must be a contiguous [C, taps] tensor in x's dtype (bias [C] too)")
    if ring is not None and (ring.shape[0] < B or ring.shape[1:] != (taps, C) or ring.dtype != x.dtype or not ring.is_contiguous()):
        raise ValueError("ring must be a contiguous [>= B, taps, C] tensor in x's dtype")
    y = torch.empty(B, L, C, dtype=x.dtype, device=x.device)
    if y.numel() == 0:
        return y
    off, scalar = _position(pos, x)
    code = _capi.native().short_conv(x, y, ring, weight, bias, B, L, C, taps,
                                        x.stride()[:2], y.stride()[:2], off, scalar,
                                        int(silu), _dt(x.dtype))
    _capi.check(code, "based_short_conv")
    return y


def latent_prepare_(q: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, dim: int, *, z: Optional[torch.Tensor] = None,
                    norm_weight: Optional[torch.Tensor] = None, cache: Optional[torch.Tensor] = None, kv_rank: int = 1,
                    pos=0, eps: float = 1e-6) -> torch.Tensor:
    """Rotate the last dims of every head of ``q [B, L, H, dim + rot]`` IN PLACE and, with ``z [B, L, kv_rank + rot]``,
    append the normed latent and the rotated shared key to ``cache [B, max_len, kv_rank + rot]``.  fp32 tables."""
    _need_cuda(q, cos, sin, z, norm_weight, cache)
    B, L, H, dq = q.shape
    rd = dq - dim
    if not q.is_contiguous() or cos.dtype != torch.float32 or cos.shape[1] * 2 != rd or not (cos.is_contiguous() and sin.is_contiguous()):
        raise ValueError("q must be contiguous and the tables float32 [positions, rot / 2]")
    zs = cs = None
    max_len = 2147483647
    if z is not None:
        _inner_contig(z, "z")
        if z.dtype != q.dtype or cache.dtype != q.dtype or cache.shape[0] < B or cache.shape[2] != kv_rank + rd or cache.stride(2) != 1:
            raise ValueError("cache must be [>= B, max_len, kv_rank + rot] in the inputs' dtype")
        zs, cs, max_len = z.stride()[:2], cache.stride()[:2], cache.shape[1]
    if q.numel() == 0:
        return q
    off, scalar = _position(pos, q)
    code = _capi.native().latent_prepare(z, norm_weight, cache, q, cos, sin,
                                            cos.shape[0], B, L, H, int(kv_rank), rd, int(dim), max_len, zs, cs,
                                            q.stride()[:2], off, scalar, float(eps), _dt(q.dtype))
    _capi.check(code, "based_latent_prepare")
    return q


def split_key_attention(q1, q2, k1, k2, v, scale: float, *, gate: Optional[torch.Tensor] = None, pos=0,
                        out: torch.Tensor) -> torch.Tensor:
    """Causal attention with score ``(q1 . k1 + q2 . k2) * scale`` on CUDA cores (fp32 arithmetic): q1, q2 ``[B, L, H, .]``,
    k1, k2, v ``[B, T, H, .]`` (expand the head dim to share keys), ``gate [B, L, H]`` pre-sigmoid, ``out [B, L, H, dv]``."""
    _need_cuda(q1, q2, k1, k2, v, gate, out)
    B, L, H, d1 = q1.shape
    for t, n in ((q1, "q1"), (q2, "q2"), (k1, "k1"), (k2, "k2"), (v, "v"), (out, "out")):
        _inner_contig(t, n)
        if t.dtype != q1.dtype:
            raise TypeError("all tensors must share a dtype")
    off, scalar = _position(pos, q1)
    if off is None and k1.shape[1] < scalar + L:
        raise ValueError("fewer keys than the last query sees")
    gs = gate.stride()[:2] if gate is not None else None
    if gate is not None:
        _inner_contig(gate, "gate")
    if out.numel() == 0:
        return out
    code = _capi.native().split_key_attention(
        q1, q2, k1, k2, v, gate, out, B, L, H, d1,
        q2.shape[-1], v.shape[-1], q1.stride()[:3], q2.stride()[:3],
        k1.stride()[:3], k2.stride()[:3], v.stride()[:3],
        out.stride()[:3], gs, off, scalar, float(scale), _dt(q1.dtype))
    _capi.check(code, "based_split_key_attention")
    return out


def latent_prefill(q1, q2, k1, k2, v, scale: float, *, gate: Optional[torch.Tensor] = None, pos: int = 0,
                   out: torch.Tensor, impl: str = "auto") -> torch.Tensor:
    """Expanded latent attention over a prompt or portion: q1, q2 ``[B, L, H, .]`` at positions ``pos ..``, per-head keys
    k1 and values v ``[B, T, H, .]``, shared key part k2 ``[B, T, d2]``, ``gate [B, L, H]`` pre-sigmoid -> ``out [B, L, H, dv]``."""
    _need_cuda(q1, q2, k1, k2, v, gate, out)
    B, L, H, d1 = q1.shape
    for t, n in ((q1, "q1"), (q2, "q2"), (k1, "k1"), (k2, "k2"), (v, "v"), (out, "out")):
        _inner_contig(t, n)
        if t.dtype != q1.dtype:
            raise TypeError("all tensors must share a dtype")
    if gate is not None:
        _inner_contig(gate, "gate")
    if out.numel() == 0:
        return out
    code = _capi.native().latent_prefill(
        q1, q2, k1, k2, v, gate, out, B, L, k1.shape[1],
        H, d1, q2.shape[-1], v.shape[-1], q1.stride()[:3], q2.stride()[:3],
        k1.stride()[:3], k2.stride()[:2], v.stride()[:3],
        out.stride()[:3], gate.stride()[:2] if gate is not None else None, int(pos),
        float(scale), _dt(q1.dtype), _IMPLS[impl])
    _capi.check(code, "based_latent_prefill")
    return out


def latent_decode(qa, qr, cache, scale: float, *, gate: Optional[torch.Tensor] = None, pos=0,
                  out: torch.Tensor) -> torch.Tensor:
    """Absorbed latent attention for a few query rows: qa ``[B, L, H, kv_rank]``, qr ``[B, L, H, rot]``, ``cache [B, max_len,
    kv_rank + rot]`` -> gated context ``out [B, L, H, kv_rank]``."""
    _need_cuda(qa, qr, cache, gate, out)
    B, L, H, r = qa.shape
    rd = qr.shape[-1]
    for t, n in ((qa, "qa"), (qr, "qr"), (cache, "cache"), (out, "out")):
        _inner_contig(t, n)
        if t.dtype != qa.dtype:
            raise TypeError("all tensors must share a dtype")
    if cache.shape[0] < B or cache.shape[2] != r + rd:
        raise ValueError("cache must be [>= B, max_len, kv_rank + rot]")
    if gate is not None:
        _inner_contig(gate, "gate")
    if out.numel() == 0:
        return out
    off, scalar = _position(pos, qa)
    lib = _capi.lib()
    need = lib.based_latent_decode_scratch_bytes(B, L, H, r, cache.shape[1])
    scratch = torch.empty(need, dtype=torch.uint8, device=qa.device) if need else None
    code = _capi.native().latent_decode(
        qa, qr, cache, gate, out, scratch, need, B, L, H, r, rd,
        cache.shape[1], qa.stride()[:3], qr.stride()[:3], cache.stride()[:2],
        out.stride()[:3], gate.stride()[:2] if gate is not None else None, off, scalar,
        float(scale), _dt(qa.dtype))
    _capi.check(code, "based_latent_decode")
    return out


def _check_delta(state, B, H, d, dv, *params):
    if state.shape[0] < B or state.shape[1:] != (H, d, dv) or state.dtype != torch.float32 or not state.is_contiguous():
        raise ValueError("state must be a contiguous float32 [>= B, H, d, dv] tensor")
    for t in params:
        if t.dtype != torch.float32 or t.stride(-1) != 1:
            raise TypeError("decay and step-size inputs must be float32")


def delta_prefill(q, k, v, z, a, b, A_log, dt_bias, norm_weight, state, *, pos=0, eps: float = 1e-6,
                  out: torch.Tensor, impl: str = "auto") -> torch.Tensor:
    """Gated delta rule over ``L`` tokens: q, k ``[B, L, Hk, d]``, v, z ``[B, L, H, dv]`` (token-strided views, heads
    contiguous), a, b ``[B, L, H]`` fp32 pre-activations, ``state [B, H, d, dv]`` fp32 updated IN PLACE; ``out [B, L, H * dv]``."""
    _need_cuda(q, k, v, z, a, b, A_log, dt_bias, norm_weight, state, out)
    B, L, Hk, d = q.shape
    H, dv = v.shape[2:]
    _check_delta(state, B, H, d, dv, a, b, A_log, dt_bias)
    for t, w in ((q, d), (k, d), (v, dv), (z, dv)):
        if t.stride(3) != 1 or (t.shape[2] > 1 and t.stride(2) != w) or t.dtype != q.dtype:
            raise ValueError("q, k, v, z: heads must be contiguous inside a token and share a dtype")
    if a.stride()[:2] != b.stride()[:2]:
        raise ValueError("a and b must have the same strides")
    _inner_contig(out, "out")
    off, scalar = _position(pos, q)
    if out.numel() == 0:
        return out
    need = _capi.lib().based_delta_prefill_scratch_bytes(B, L, H, d, dv) if q.dtype == torch.bfloat16 and impl != "simt" else 0
    scratch = torch.empty(need, dtype=torch.uint8, device=q.device) if need else None
    code = _capi.native().delta_prefill(
        q, k, v, z, a, b, A_log, dt_bias,
        norm_weight, state, out, B, L, H, Hk, d, dv, q.stride()[:2],
        k.stride()[:2], v.stride()[:2], z.stride()[:2],
        a.stride()[:2], out.stride()[:2], off, scalar, float(eps), _dt(q.dtype), _IMPLS[impl],
        scratch, need)
    _capi.check(code, "based_delta_prefill")
    return out


def delta_step(x, conv_weight, ring, a, b, A_log, dt_bias, norm_weight, state, kv_heads: int, *, pos, eps: float = 1e-6,
               out: torch.Tensor) -> bool:
    """One token per row in one launch: packed projection ``x [B, q | k | v | z]``, ``ring [B, taps, C]`` and ``state
    [B, H, d, dv]`` updated IN PLACE, ``out [B, H * dv]``.  Returns False, nothing launched, for sizes it does not take."""
    _need_cuda(x, conv_weight, ring, a, b, A_log, dt_bias, norm_weight, state, out)
    B, (_, H, d, dv) = x.shape[0], state.shape
    _check_delta(state, B, H, d, dv, a, b, A_log, dt_bias)
    C, taps = conv_weight.shape
    if C != 2 * kv_heads * d + H * dv or x.shape[1] < C + H * dv or x.stride(1) != 1 or out.stride(1) != 1 or a.stride(0) != b.stride(0):
        raise ValueError("x must be [B, >= 2 kv_heads d + 2 H dv] and conv_weight [2 kv_heads d + H dv, taps]")
    if ring.shape[0] < B or ring.shape[1:] != (taps, C) or ring.dtype != x.dtype or not ring.is_contiguous() or not conv_weight.is_contiguous():
        raise ValueError("ring must be a contiguous [>= B, taps, C] tensor in x's dtype")
    off, scalar = _position(pos, x)
    if B == 0:
        return True
    code = _capi.native().delta_step(
        x, conv_weight, ring, a, b, A_log, dt_bias,
        norm_weight, state, out, B, H, int(kv_heads), d, dv, taps, x.stride(0), a.stride(0),
        out.stride(0), off, scalar, float(eps), _dt(x.dtype))
    if code == _capi.ERR_IMPL:
        return False
    _capi.check(code, "based_delta_step")
    return True


def block_gates(u: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    """Block-diagonal gate products with an fp32 result: ``u [B, L, blocks * n]`` by ``weight [blocks, 2, n, n]`` (r and i
    matrices, stored [out, in]) -> ``[blocks, B * L, 2 n]``."""
    _need_cuda(u, weight)
    nb, _, n, _ = weight.shape
    x, w = u.reshape(-1, nb, n).transpose(0, 1), weight.view(nb, 2 * n, n).transpose(1, 2)
    if u.dtype == torch.float32:
        return torch.bmm(x, w)
    return torch.bmm(x, w, out_dtype=torch.float32)


def rglru(u, y, gates, r_bias, i_bias, lam, state, *, pos=0, out: torch.Tensor) -> torch.Tensor:
    """Real-gated linear recurrent unit: u, y ``[B, L, W]``, ``gates [blocks, B * L, 2 n]`` fp32 (r half, i half),
    ``lam [W]`` fp32, ``state [B, W]`` fp32 updated IN PLACE; ``out [B, L, W] = S * gelu_tanh(y)``."""
    _need_cuda(u, y, gates, r_bias, i_bias, lam, state, out)
    B, L, W = u.shape
    nb, rows, n2 = gates.shape
    if rows != B * L or nb * n2 != 2 * W or gates.dtype != torch.float32 or gates.stride(2) != 1:
        raise ValueError("gates must be float32 [blocks, B * L, 2 * W / blocks]")
    if state.shape[0] < B or state.shape[1] != W or state.dtype != torch.float32 or lam.dtype != torch.float32 or not state.is_contiguous():
        raise ValueError("state must be a contiguous float32 [>= B, W] tensor and lam float32")
    for t, n in ((u, "u"), (y, "y"), (out, "out")):
        _inner_contig(t, n)
    off, scalar = _position(pos, u)
    if out.numel() == 0:
        return out
    code = _capi.native().rglru(
        u, y, gates, r_bias, i_bias, lam, state,
        out, B, L, W, n2 // 2, u.stride()[:2], y.stride()[:2],
        out.stride()[:2], (gates.stride(0), gates.stride(1)), off, scalar, _dt(u.dtype))
    _capi.check(code, "based_rglru")
    return out


# tokens from which the one-pass kernel is used; below it, the gate products and the recurrence are two launches
RGLRU_FUSED_MIN_TOKENS = 8


def rglru_gated(u, y, gate_weight, r_bias, i_bias, lam, state, *, pos=0, out: torch.Tensor) -> torch.Tensor:
    """The recurrent unit with its gate products (``gate_weight`` as in :func:`block_gates`): one pass on the tensor cores
    for bf16 prompts and portions, else :func:`block_gates` and :func:`rglru`."""
    _need_cuda(u, y, gate_weight, r_bias, i_bias, lam, state, out)
    B, L, W = u.shape
    nb, _, n, _ = gate_weight.shape
    if u.dtype == torch.bfloat16 and L >= RGLRU_FUSED_MIN_TOKENS and B > 0:
        if (nb * n != W or not gate_weight.is_contiguous() or gate_weight.dtype != u.dtype or lam.dtype != torch.float32
                or state.dtype != torch.float32 or state.shape[0] < B or state.shape[1] != W or not state.is_contiguous()):
            raise ValueError("gate_weight must be [blocks, 2, n, n] in u's dtype, state [>= B, W] and lam float32, contiguous")
        for t, name in ((u, "u"), (y, "y"), (out, "out")):
            _inner_contig(t, name)
        off, scalar = _position(pos, u)
        code = _capi.native().rglru_gated(
            u, y, gate_weight, r_bias, i_bias, lam,
            state, out, B, L, W, n, u.stride()[:2], y.stride()[:2],
            out.stride()[:2], off, scalar, _dt(u.dtype))
        if code != _capi.ERR_IMPL:
            _capi.check(code, "based_rglru_gated")
            return out
    return rglru(u, y, block_gates(u, gate_weight), r_bias, i_bias, lam, state, pos=pos, out=out)


def rglru_step(x, y, conv_weight, conv_bias, ring, gate_weight, r_bias, i_bias, lam, state, *, pos, out: torch.Tensor) -> bool:
    """One token per row in one launch: ``x, y [B, W]`` column slices of the packed projection through :func:`short_conv`,
    :func:`block_gates` and :func:`rglru`; ``ring [B, taps, W]`` and ``state [B, W]`` are updated IN PLACE, ``out [B, W]``.  Returns
    False, nothing launched, for dtypes, sizes or layouts it does not take."""
    _need_cuda(x, y, conv_weight, conv_bias, ring, gate_weight, r_bias, i_bias, lam, state, out)
    B, W = x.shape
    nb, two, n, n2 = gate_weight.shape
    taps = conv_weight.shape[1]
    if any(t.dtype != torch.bfloat16 for t in (x, y, conv_weight, ring, gate_weight, r_bias, i_bias, out)) or (
            conv_bias is not None and conv_bias.dtype != torch.bfloat16):
        return False
    if (two != 2 or n2 != n or nb * n != W or y.shape != (B, W) or out.shape != (B, W) or conv_weight.shape[0] != W
            or ring.shape[0] < B or ring.shape[1:] != (taps, W) or state.shape[0] < B or state.shape[1] != W
            or state.dtype != torch.float32 or lam.dtype != torch.float32):
        raise ValueError("x, y, out must be [B, W], ring [>= B, taps, W], gate_weight [blocks, 2, n, n], state [>= B, W] and lam float32")
    if not all(t.is_contiguous() for t in (conv_weight, ring, gate_weight, state, r_bias, i_bias, lam)) or (
            conv_bias is not None and not conv_bias.is_contiguous()):
        return False
    for t, name in ((x, "x"), (y, "y"), (out, "out")):
        _inner_contig(t, name)
    off, scalar = _position(pos, x)
    if B == 0:
        return True
    code = _capi.native().rglru_step(x, y, conv_weight, conv_bias, ring, gate_weight, r_bias, i_bias, lam, state, out, B, W, n, taps,
                                     x.stride(0), y.stride(0), out.stride(0), off, scalar)
    if code == _capi.ERR_IMPL:
        return False
    _capi.check(code, "based_rglru_step")
    return True


# --------------------------------------------------------------------------- post-norm stacks

def _strides_bl(t):
    return t.stride()[:2]


def _same_dtype(like, **tensors):
    for name, t in tensors.items():
        if t is not None and (t.dtype != like.dtype or t.stride(-1) != 1):
            raise TypeError(f"{name} must be in the inputs' dtype with an innermost stride of 1")


def stream_embed(residual: torch.Tensor, tokens: torch.Tensor, table: torch.Tensor, scale: float, pos_table: torch.Tensor,
                 pos=0) -> torch.Tensor:
    """Start of a stream: the fp32 ``residual [B, L, D]`` becomes ``table[token] * scale + pos_table[position]`` IN PLACE;
    returns it in the table's dtype (fp32: the stream itself)."""
    _need_cuda(residual, tokens, table, pos_table)
    B, L, D = residual.shape
    if residual.dtype != torch.float32 or not residual.is_contiguous():
        raise TypeError("residual must be a contiguous float32 tensor")
    if tokens.dtype != torch.int64 or tokens.shape != (B, L):
        raise TypeError("tokens must be int64 [B, L]")
    if table.dtype != pos_table.dtype or not (table.is_contiguous() and pos_table.is_contiguous()) or table.shape[1] != D or pos_table.shape[1] != D:
        raise ValueError("table and pos_table must be contiguous [rows, D] of one dtype")
    out = residual if table.dtype == torch.float32 else torch.empty(B, L, D, dtype=table.dtype, device=residual.device)
    off, scalar = _position(pos, residual)
    if residual.numel() > 0:
        tokens = tokens.contiguous()
        code = _capi.native().stream_embed(
            tokens, table, table.shape[0], float(scale), pos_table, pos_table.shape[0],
            residual, None if out is residual else out, B, L, D, off, scalar, _dt(table.dtype))
        _capi.check(code, "based_stream_embed")
    return out


def stream_post_norm(residual: torch.Tensor, branch: torch.Tensor, weight: torch.Tensor, *,
                     out_weight: Optional[torch.Tensor] = None, eps: float = 1e-6) -> torch.Tensor:
    """The norm step of a post-norm block: the fp32 stream ``residual [..., D]`` becomes ``residual + rmsnorm(branch) * weight``
    IN PLACE; returns it in the branch's dtype (fp32: the stream itself), or its RMSNorm scaled by ``out_weight``."""
    _need_cuda(residual, branch, weight, out_weight)
    D = residual.shape[-1]
    if residual.dtype != torch.float32 or not residual.is_contiguous():
        raise TypeError("residual must be a contiguous float32 tensor")
    b2 = flat_rows(branch)
    _same_dtype(branch, branch=branch, weight=weight, out_weight=out_weight)
    M = residual.numel() // D if D else 0
    if b2.shape != (M, D) or weight.shape != (D,) or (out_weight is not None and out_weight.shape != (D,)):
        raise ValueError("branch must have the stream's shape and the weights its width")
    alias = out_weight is None and branch.dtype == torch.float32
    out = residual if alias else torch.empty(residual.shape, dtype=branch.dtype, device=residual.device)
    if M > 0:
        code = _capi.native().stream_post_norm(b2, b2.stride(0), weight, residual, out_weight,
                                                  None if alias else out, M, D, float(eps), _dt(branch.dtype))
        _capi.check(code, "based_stream_post_norm")
    return out


def norm_gate(x: torch.Tensor, weight: torch.Tensor, gate: torch.Tensor, eps: float, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``rmsnorm(x) * weight * sigmoid(gate)`` over the last dim; column slices are fine for all but the weight."""
    _need_cuda(x, weight, gate, out)
    D = x.shape[-1]
    out = torch.empty(x.shape, dtype=x.dtype, device=x.device) if out is None else out
    _same_dtype(x, x=x, weight=weight, gate=gate, out=out)
    x2, g2, o2 = flat_rows(x), flat_rows(gate), flat_rows(out)
    if g2.shape != x2.shape or o2.shape != x2.shape or weight.shape != (D,):
        raise ValueError("gate and out must have x's shape and the weight its width")
    if x2.numel() > 0:
        code = _capi.native().norm_gate(x2, x2.stride(0), weight, g2, g2.stride(0), o2,
                                           o2.stride(0), x2.shape[0], D, float(eps), _dt(x.dtype))
        _capi.check(code, "based_norm_gate")
    return out


def token_gate(z: torch.Tensor, tokens: torch.Tensor, table: torch.Tensor, column: int) -> torch.Tensor:
    """``gelu_tanh(z) * table[token, column : column + n]`` for ``z [..., n]``, contiguous."""
    _need_cuda(z, tokens, table)
    n = z.shape[-1]
    z2 = flat_rows(z)
    _same_dtype(z, z=z, table=table)
    if tokens.dtype != torch.int64 or tokens.numel() != z2.shape[0] or not 0 <= column <= table.shape[1] - n:
        raise ValueError("tokens must be int64, one per row, and the slice inside the table")
    out = torch.empty(z.shape, dtype=z.dtype, device=z.device)
    if out.numel() > 0:
        tokens = tokens.contiguous()
        code = _capi.native().token_gate(z2, z2.stride(0), tokens, table, table.shape[0],
                                            table.stride(0), int(column), out, z2.shape[0], n, _dt(z.dtype))
        _capi.check(code, "based_token_gate")
    return out


# A step's rows; from PROMPT_MIN_ROWS on, a whole tile of rows, there is one launch for prompts, too.  us as four launches / in one, width 1024,
# 64 values, in a graph: clusters of CTAs 64 9.0 / 6.4, 128 9.1 / 6.8, 192 9.4 / 7.5; beyond, on the tensor cores,
# 512 10.0 / 12.6, 1024 11.1 / 12.8, 2048 12.7 / 13.2, 4096 16.4 / 16.3, 6400 21.5 / 22.3, 7168 24.0 / 22.4, 8192 27 / 23, 18944 57 / 48 (other
# widths cross between 4096 and 7168).  A prompt that is not captured is bound by its launches (27 such layers, 130 to 4096 tokens 5.55 to 5.9
# ms / 4.85 to 5.2) or loses less than 1 % of a layer, so there it is one launch at any length; a captured one from TOKEN_SIDE_CAPTURED_ROWS on.
TOKEN_SIDE_MAX_ROWS = 64
TOKEN_SIDE_CAPTURED_ROWS = 7168
TOKEN_SIDE_MAX_WEIGHT = 200_000   # elements of one matrix up to which one cluster per 16 rows beats the separate launches


def _one_launch(M, size) -> bool:
    return (M >= TOKEN_SIDE_CAPTURED_ROWS or (M <= _capi.TOKEN_SIDE_CLUSTER_ROWS and size <= TOKEN_SIDE_MAX_WEIGHT)
            or not torch.cuda.is_current_stream_capturing())


def _prompt_side(residual, x, tokens, gate_weight, proj_weight, table, column, norm_weight) -> bool:
    """True when the kernel of a prompt's token input takes these operands and nothing around its products needs them apart."""
    n, W = gate_weight.shape
    return (n % 8 == 0 and n <= 64 and W % 8 == 0 and x.numel() < W << 31 and column % 8 == 0 and table.dim() == 2 and table.stride(1) == 1 and table.stride(0) % 8 == 0
            and x.is_contiguous() and gate_weight.is_contiguous() and proj_weight.is_contiguous() and proj_weight.shape == (W, n) and norm_weight.is_contiguous()
            and residual.dtype == torch.float32 and residual.is_contiguous() and tokens.dtype == torch.int64
            and all(t.dtype == torch.bfloat16 for t in (gate_weight, proj_weight, table, norm_weight))
            and all(t.data_ptr() % 16 == 0 for t in (residual, table, norm_weight)) and _unwatched(x, gate_weight) and _unwatched(x, proj_weight))


def token_side_step(residual: torch.Tensor, x: torch.Tensor, tokens: torch.Tensor, gate_weight: torch.Tensor, proj_weight: torch.Tensor,
                    table: torch.Tensor, column: int, norm_weight: torch.Tensor, *, out_weight: Optional[torch.Tensor] = None,
                    eps: float = 1e-6) -> Optional[torch.Tensor]:
    """A layer's token input for the rows of a step or of a prompt in one launch: ``x [..., W]`` through ``gate_weight [n, W]``, :func:`token_gate`,
    ``proj_weight [W, n]`` and :func:`stream_post_norm`.  None, nothing launched, for rows, sizes or dtypes it does not take."""
    _need_cuda(residual, x, tokens, gate_weight, proj_weight, table, norm_weight, out_weight)
    n, W = gate_weight.shape
    M = x.numel() // W if W else 0
    if x.dtype != torch.bfloat16 or M <= 0:
        return None
    if M <= TOKEN_SIDE_MAX_ROWS:
        if n * W > TOKEN_SIDE_MAX_WEIGHT:
            return None
    elif not (M >= PROMPT_MIN_ROWS and out_weight is None and _one_launch(M, n * W) and _prompt_side(residual, x, tokens, gate_weight, proj_weight, table, column, norm_weight)):
        return None
    _same_dtype(x, x=x, gate_weight=gate_weight, proj_weight=proj_weight, table=table, norm_weight=norm_weight, out_weight=out_weight)
    x2 = flat_rows(x)
    if residual.dtype != torch.float32 or not residual.is_contiguous() or residual.shape != x.shape:
        raise TypeError("residual must be a contiguous float32 tensor of x's shape")
    if proj_weight.shape != (W, n) or not (gate_weight.is_contiguous() and proj_weight.is_contiguous()):
        raise ValueError("gate_weight must be [n, W] and proj_weight [W, n], contiguous")
    if tokens.dtype != torch.int64 or tokens.numel() != M or not 0 <= column <= table.shape[1] - n:
        raise ValueError("tokens must be int64, one per row, and the slice inside the table")
    if norm_weight.shape != (W,) or (out_weight is not None and out_weight.shape != (W,)):
        raise ValueError("norm weights must have the stream's width")
    out = torch.empty(x.shape, dtype=x.dtype, device=x.device)
    tokens = tokens.contiguous()
    code = _capi.native().token_side(
        x2, x2.stride(0), tokens, gate_weight, proj_weight, table, table.shape[0],
        table.stride(0), int(column), norm_weight, residual, out_weight, out, M, W, n, float(eps),
        _dt(x.dtype))
    if code == _capi.ERR_IMPL:
        return None
    _capi.check(code, "based_token_side")
    return out


def _check_tied(q, cache, factor, B, H, G, d):
    if H % G or q.shape[2] != H * d or cache.shape[0] < B or cache.shape[2] != G * d or cache.dtype != q.dtype or cache.stride(2) != 1:
        raise ValueError("q must be [B, L, H d] and cache [>= B, max_len, G d] in its dtype, H a multiple of G")
    if factor.dtype != torch.float32 or factor.shape[0] < B or factor.shape[1] != G or factor.shape[2] < cache.shape[1] or factor.stride(2) != 1:
        raise ValueError("factor must be float32 [>= B, G, >= max_len]")


def tied_attention_state(batch: int, heads: int, kv_heads: int, dim: int, max_len: int, dtype, device) -> dict:
    """What :func:`tied_prepare_` and :func:`tied_attention` keep for ``batch`` sequences: the keys, their factors (rows padded to
    whole key tiles) and the zeroed counters of a decode step whose keys are split."""
    rows = max(_capi.TIED_DECODE_ROWS, heads // kv_heads)
    return {"keys": torch.zeros(batch, max_len, kv_heads * dim, dtype=dtype, device=device),
            "factor": torch.zeros(batch, kv_heads, (max_len + 127) // 128 * 128, dtype=torch.float32, device=device),
            "count": torch.zeros(batch * kv_heads * ((rows + 15) // 16), dtype=torch.int32, device=device)}


def tied_prepare_(q: torch.Tensor, k: torch.Tensor, q_weight: torch.Tensor, k_weight: torch.Tensor, cache: torch.Tensor,
                  factor: torch.Tensor, *, pos=0, eps: float = 1e-6, temp_coef: float = 0.0, temp_every: float = 1.0) -> torch.Tensor:
    """Queries ``q [B, L, H d]`` normed per head, times both norm weights and ``1 + temp_coef ln(floor((p + 1) / temp_every) +
    1)`` IN PLACE; keys ``k [B, L, G d]`` appended to ``cache [B, max_len, G d]`` as they are, their inverse root mean squares to
    ``factor [B, G, max_len]``."""
    _need_cuda(q, k, q_weight, k_weight, cache, factor)
    B, L, _ = q.shape
    d = q_weight.shape[0]
    H, G = q.shape[2] // d, k.shape[2] // d
    _same_dtype(q, q=q, k=k, q_weight=q_weight, k_weight=k_weight)
    _check_tied(q, cache, factor, B, H, G, d)
    if k.shape != (B, L, G * d) or k_weight.shape != (d,):
        raise ValueError("k must be [B, L, G d]")
    off, scalar = _position(pos, q)
    if q.numel() > 0:
        code = _capi.native().tied_prepare(
            q, k, q_weight, k_weight, cache, factor, B, L, H, G, d,
            cache.shape[1], _strides_bl(q), _strides_bl(k), _strides_bl(cache), _strides_bl(factor), off, scalar, float(eps),
            float(temp_coef), float(temp_every), _dt(q.dtype))
        _capi.check(code, "based_tied_prepare")
    return q


def tied_attention(q: torch.Tensor, cache: torch.Tensor, factor: torch.Tensor, count: torch.Tensor, heads: int, scale: float, *,
                   gate: Optional[torch.Tensor] = None, pos=0, sink: float = 0.0, out: torch.Tensor, impl: str = "auto") -> torch.Tensor:
    """Causal attention of prepared queries ``q [B, L, H d]`` at positions ``pos ..`` over ``cache [B, max_len, G d]``, whose rows
    are keys (scores times ``factor``) and values; ``sink`` scores of 0 without a value in each softmax sum; ``out [B, L, H d]``
    times ``sigmoid(gate [B, L, H d])``.  ``count``: int32 zeros, see :func:`tied_attention_state`."""
    _need_cuda(q, cache, factor, count, gate, out)
    if count.dtype != torch.int32 or not count.is_contiguous():
        raise TypeError("count must be a contiguous int32 tensor")
    B, L, W = q.shape
    d = W // heads
    G = cache.shape[2] // d
    _same_dtype(q, q=q, gate=gate, out=out)
    _check_tied(q, cache, factor, B, heads, G, d)
    if out.shape != q.shape or (gate is not None and gate.shape != q.shape):
        raise ValueError("gate and out must have q's shape")
    off, scalar = _position(pos, q)
    if out.numel() == 0:
        return out
    need = 0
    if q.dtype == torch.bfloat16 and (impl == "decode" or impl == "auto" and (off is not None or L * (heads // G) <= _capi.TIED_DECODE_ROWS)):
        need = _capi.lib().based_tied_attention_scratch_bytes(B, L, heads, G, d, cache.shape[1])
    scratch = torch.empty(need, dtype=torch.uint8, device=q.device) if need else None
    code = _capi.native().tied_attention(
        q, cache, factor, gate, out, B, L, heads, G, d, cache.shape[1],
        _strides_bl(q), _strides_bl(cache), _strides_bl(factor), _strides_bl(gate) if gate is not None else None, _strides_bl(out),
        off, scalar, float(scale), float(sink), _dt(q.dtype), _IMPLS[impl], scratch, need, count, count.numel())
    _capi.check(code, "based_tied_attention")
    return out


def _check_lightning(state, decay, B, H, d, dv):
    if state.shape[0] < B or state.shape[1:] != (H, d, dv) or state.dtype != torch.float32 or not state.is_contiguous():
        raise ValueError("state must be a contiguous float32 [>= B, H, d, dv] tensor")
    if decay.shape != (H,) or decay.dtype != torch.float32 or not decay.is_contiguous():
        raise ValueError("decay must be float32, one per head")


def lightning(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, decay: torch.Tensor, state: torch.Tensor, *, pos=0,
              out: Optional[torch.Tensor] = None, impl: str = "auto") -> torch.Tensor:
    """Linear attention with a constant decay per head: q, k ``[B, L, H d]``, v ``[B, L, H dv]`` before silu, ``state [B, H, d,
    dv]`` fp32 updated IN PLACE; the read-out ``[B, L, H dv]``."""
    _need_cuda(q, k, v, decay, state, out)
    B, L, _ = q.shape
    _, H, d, dv = state.shape
    _check_lightning(state, decay, B, H, d, dv)
    out = torch.empty(B, L, H * dv, dtype=q.dtype, device=q.device) if out is None else out
    _same_dtype(q, q=q, k=k, v=v, out=out)
    if q.shape[2] != H * d or k.shape != q.shape or v.shape != (B, L, H * dv) or out.shape != v.shape:
        raise ValueError("q, k must be [B, L, H d] and v, out [B, L, H dv]")
    off, scalar = _position(pos, q)
    if out.numel() == 0:
        return out
    lib = _capi.lib()
    need = lib.based_lightning_scratch_bytes(B, L, H, d, dv) if q.dtype == torch.bfloat16 and impl != "simt" else 0
    scratch = torch.empty(need, dtype=torch.uint8, device=q.device) if need else None
    code = _capi.native().lightning_split(q, k, v, decay, state, out, B, L,
                                     H, d, dv, _strides_bl(q), _strides_bl(k), _strides_bl(v), _strides_bl(out), off, scalar,
                                     _dt(q.dtype), _IMPLS[impl], scratch, need)
    _capi.check(code, "based_lightning")
    return out


def lightning_step(q, k, v, gate, decay, norm_weight, state, read, count, *, pos, eps: float, out: torch.Tensor) -> bool:
    """One token per row in one launch: q, k, v, gate are column slices ``[B, .]`` of one packed projection, ``state`` is updated
    IN PLACE, ``read [B, H dv]`` fp32 and ``count [B]`` int32 (zeros) are workspace; ``out [B, H dv]`` normed over all heads and
    gated.  Returns False, nothing launched, for sizes it does not take."""
    _need_cuda(q, k, v, gate, decay, norm_weight, state, read, count, out)
    B = q.shape[0]
    _, H, d, dv = state.shape
    _check_lightning(state, decay, B, H, d, dv)
    _same_dtype(q, q=q, k=k, v=v, gate=gate, norm_weight=norm_weight, out=out)
    if q.shape[1] != H * d or k.shape != q.shape or v.shape != (B, H * dv) or gate.shape != v.shape or out.shape != v.shape or norm_weight.shape != (H * dv,):
        raise ValueError("q, k must be [B, H d] and v, gate, out [B, H dv]")
    if len({t.stride(0) for t in (q, k, v, gate)}) > 1 and B > 1:
        raise ValueError("q, k, v and gate must be slices of one tensor")
    if read.dtype != torch.float32 or read.shape[0] < B or read.shape[1] != H * dv or not read.is_contiguous() or count.dtype != torch.int32 or count.numel() < B:
        raise ValueError("read must be contiguous float32 [>= B, H dv] and count int32 [>= B]")
    off, scalar = _position(pos, q)
    if B == 0:
        return True
    code = _capi.native().lightning_step(
        q, k, v, gate, q.stride(0), decay, norm_weight,
        state, read, count, out, out.stride(0), B, H, d, dv, off, scalar, float(eps),
        _dt(q.dtype))
    if code == _capi.ERR_IMPL:
        return False
    _capi.check(code, "based_lightning_step")
    return True


def lightning_step_rows(q, k, v, gate, decay, norm_weight, state, *, pos, eps: float) -> Optional[NormRows]:
    """:func:`lightning_step` with the norm's factor left to the product behind it: :class:`NormRows` ``[B, 1, H dv]`` for
    :func:`decode_linear`.  None, nothing launched, for dtypes and sizes it does not take."""
    _need_cuda(q, k, v, gate, decay, norm_weight, state)
    B = q.shape[0]
    _, H, d, dv = state.shape
    if q.dtype != torch.bfloat16 or not 0 < B <= STEP_MAX_ROWS:
        return None
    _check_lightning(state, decay, B, H, d, dv)
    _same_dtype(q, q=q, k=k, v=v, gate=gate, norm_weight=norm_weight)
    if q.shape[1] != H * d or k.shape != q.shape or v.shape != (B, H * dv) or gate.shape != v.shape or norm_weight.shape != (H * dv,):
        raise ValueError("q, k must be [B, H d] and v, gate [B, H dv]")
    if len({t.stride(0) for t in (q, k, v, gate)}) > 1 and B > 1:
        raise ValueError("q, k, v and gate must be slices of one tensor")
    off, scalar = _position(pos, q)
    pieces = _capi.lib().based_lightning_step_pieces(B, H, dv)
    out = torch.empty(B, 1, H * dv, dtype=q.dtype, device=q.device)
    ss = torch.empty(B, pieces, dtype=torch.float32, device=q.device)
    code = _capi.native().lightning_step_rows(q, k, v, gate, q.stride(0), decay, norm_weight, state, out, H * dv, ss, pieces, B, H, d, dv,
                                              off, scalar, _dt(q.dtype))
    if code == _capi.ERR_IMPL:
        return None
    _capi.check(code, "based_lightning_step_rows")
    return NormRows(out, ss, eps)
