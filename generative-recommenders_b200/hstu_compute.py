"""The LayerNorm + linear stages around the attention, with the reference's signatures
(generative_recommenders/ops/hstu_compute.py:54-335)."""

import weakref
from typing import Optional, Tuple

import torch

from . import _cabi
from .common import (HammerKernel, _require_cuda_backend, as_dtype, dtype_code, on_device, outside_autograd,
                     require_cuda, stream_ptr)
from . import hstu_attention as _attention
from .hstu_attention import _i32, _index, hstu_mha
from .layer_norm import layer_norm
from .mm import addmm

_ACT = {"none": 0, "sigmoid": 1, "silu": 2}


class _SiluColumnsFunction(torch.autograd.Function):
    """u = SiLU(x[:, :width]) written densely; x itself (the uvqk buffer) is left untouched."""

    @staticmethod
    def forward(ctx, x, width):
        rows = x.shape[0]
        u = torch.empty((rows, width), dtype=x.dtype, device=x.device)
        if rows > 0:
            with on_device(x.device):
                _cabi.check(
                    _cabi.lib().b200_hstu_silu_fwd(x.data_ptr(), x.stride(0), u.data_ptr(), u.stride(0), rows, width,
                                                   dtype_code(x), stream_ptr(x.device)),
                    "b200_hstu_silu_fwd")
        ctx.save_for_backward(x)
        ctx.width = width
        return u

    @staticmethod
    def backward(ctx, du):
        (x,) = ctx.saved_tensors
        rows, width = x.shape[0], ctx.width
        if du.stride(-1) != 1:
            du = du.contiguous()
        dx = torch.zeros_like(x) if x.shape[1] != width else torch.empty_like(x)
        if rows > 0:
            with on_device(x.device):
                _cabi.check(
                    _cabi.lib().b200_hstu_silu_bwd(du.data_ptr(), du.stride(0), x.data_ptr(), x.stride(0),
                                                   dx.data_ptr(), dx.stride(0), rows, width, dtype_code(x),
                                                   stream_ptr(x.device)),
                    "b200_hstu_silu_bwd")
        return dx, None


def _aligned16(t: torch.Tensor) -> torch.Tensor:
    """``t`` itself when its first element sits on a 16-byte boundary (what the tensor-core kernel's
    bulk loads need), else a fresh copy - a contiguous slice of a flat parameter buffer can start
    anywhere."""
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _fused_uqvk_supported(x, uvqk_weight, hv) -> bool:
    if x.dtype not in (torch.bfloat16, torch.float16) or x.dim() != 2 or x.shape[0] == 0:
        return False
    return _cabi.host().uvqk_supported(x, uvqk_weight, hv, dtype_code(x))


# Inference only: the workspace of the fused kernel holds what the preparation launches derive from
# the four parameter tensors (W' = diag(gamma) W and two column vectors).  While those tensors are
# alive and unmodified (same objects, same storage, same version counters) the workspace is kept
# and the preparation is skipped.  The version counter sees optimizer steps, load_state_dict and
# every other in-place operation on the parameter itself; it does NOT see a write through
# ``param.data`` (``param.data.copy_(new)``), which shares the storage but not the counter.  Code
# that refreshes weights that way calls ``clear_prepared_weights()`` afterwards, or switches the
# cache off with ``set_prepared_weights_cache(False)``.
_PREPARED = {}
_PREPARED_ON = True


def clear_prepared_weights() -> None:
    """Forget every cached preparation of the fused uvqk stage (see the comment above)."""
    global _PREPARED
    _PREPARED = {}   # (a call under way adds to the old one)


def set_prepared_weights_cache(on: bool) -> None:
    """Keep (default) or never keep the derived weights of the fused uvqk stage between
    inference calls."""
    global _PREPARED_ON
    _PREPARED_ON = bool(on)
    if not on:
        clear_prepared_weights()


def _prepared_state(w, nw, nb, b, stream):
    return (w.data_ptr(), w._version, nw.data_ptr(), nw._version, nb.data_ptr(), nb._version, b.data_ptr(),
            b._version, stream)


def _prepared_workspace(nw, nb, w, b, nbytes, device, keep):
    """``(workspace, prepared, remember)``: ``remember()``, if there is one, keeps the workspace for later
    calls.  It is called when the preparation is in the stream and not before: a call of another thread
    that found the workspace earlier could be queued ahead of it, and after a launch that returned an
    error there is nothing to find."""
    if not keep or not _PREPARED_ON or torch.cuda.is_current_stream_capturing():
        return torch.empty(nbytes, dtype=torch.uint8, device=device), False, None
    known, key = _PREPARED, id(w)
    # the workspace was prepared on this stream; a call on another stream is not ordered after that
    # preparation, so it prepares (and then owns) a new one
    stream = stream_ptr(device)
    hit = known.get(key)   # (an id can recur: the entry holds weak references to compare)
    if hit is not None:
        rw, rnw, rnb, rb, sig, ws = hit
        if (rw() is w and rnw() is nw and rnb() is nb and rb() is b and ws.numel() == nbytes
                and sig == _prepared_state(w, nw, nb, b, stream)):
            return ws, True, None
    ws = torch.empty(nbytes, dtype=torch.uint8, device=device)
    # Only module parameters are worth remembering, and only when all four tensors are the
    # parameters themselves: a cast copy made for one call never comes back.  Parameters made in
    # inference mode have no version.
    if not all(isinstance(t, torch.nn.Parameter) and not t.is_inference() for t in (w, nw, nb, b)):
        return ws, False, None
    sig = _prepared_state(w, nw, nb, b, stream)

    def remember():
        if len(known) > 256:
            known.clear()
        known[key] = (weakref.ref(w), weakref.ref(nw), weakref.ref(nb), weakref.ref(b), sig, ws)

    return ws, False, remember


def _fused_uqvk_launch(x, nw, nb, eps, w, b, hv, inference=False):
    """One launch of the fused kernel: returns (uvqk [M, N], u [M, hv], mean [M], rstd [M]).  For
    ``inference`` the derived weights may be kept, the pre-activation u columns of uvqk stay unwritten
    and mean and rstd are None."""
    M, D = x.shape
    N = w.shape[1]
    if w.shape[0] != D or nw.numel() < D or nb.numel() < D or b.numel() < N:   # (the kernel reads them by the width of x)
        raise RuntimeError("uvqk stage: parameters of another width than x")
    uvqk = torch.empty((M, N), dtype=x.dtype, device=x.device)
    u = torch.empty((M, hv), dtype=x.dtype, device=x.device)
    mean = torch.empty(M, dtype=torch.float32, device=x.device) if not inference else None
    rstd = torch.empty(M, dtype=torch.float32, device=x.device) if not inference else None
    nbytes = _cabi.lib().b200_hstu_ln_linear_workspace_bytes(D, N)
    ws, prepared, remember = _prepared_workspace(nw, nb, w, b, nbytes, x.device, inference)
    a = _cabi.LnLinearArgs()
    a.weights_prepared = 1 if prepared else 0
    a.skip_pre_activation = 1 if inference else 0   # only the backward reads it
    a.x, a.norm_weight, a.norm_bias, a.weight, a.bias = (x.data_ptr(), nw.data_ptr(), nb.data_ptr(),
                                                          w.data_ptr(), b.data_ptr())
    a.out, a.u = uvqk.data_ptr(), u.data_ptr()
    if not inference:
        a.mean, a.rstd = mean.data_ptr(), rstd.data_ptr()
    a.workspace, a.workspace_bytes = ws.data_ptr(), nbytes
    a.x_row_stride, a.out_row_stride, a.u_row_stride = x.stride(0), uvqk.stride(0), u.stride(0)
    a.M, a.D, a.N, a.silu_cols = M, D, N, hv
    a.eps, a.dtype = eps, dtype_code(x)
    with on_device(x.device):
        _cabi.check(_cabi.lib().b200_hstu_ln_linear_silu_fwd(a, stream_ptr(x.device)),
                    "b200_hstu_ln_linear_silu_fwd")
    if remember is not None:
        remember()
    return uvqk, u, mean, rstd


def _fused_uqvk_backward(x, nw, nb, w, uvqk, mean, rstd, eps, hv, du, d_uvqk):
    """Backward of the fused stage.  ``d_uvqk`` [M, N] already holds the gradients of the v, q, k
    columns; the u columns are filled here (``du * SiLU'``).  Recomputes ``LN(x)`` from the saved
    statistics (the reference's ``recompute_normed_x_in_backward``,
    generative_recommenders/ops/triton/triton_hstu_preprocess_and_attention.py:122-127, 185-203)
    and uses library GEMMs.  Returns (dx, d_norm_weight, d_norm_bias, d_weight, d_bias)."""
    return _cabi.host().uvqk_backward(x, nw, nb, w, uvqk, mean, rstd, eps, hv, du, d_uvqk, dtype_code(x))


def _stage_parameters(x, norm_weight, norm_bias, weight, bias):
    """The parameters as the fused kernel reads them (a parameter that is so already: itself)."""
    return (as_dtype(norm_weight, x.dtype).contiguous(), as_dtype(norm_bias, x.dtype).contiguous(),
            _aligned16(as_dtype(weight, x.dtype).contiguous()), as_dtype(bias, x.dtype).contiguous())


def _uqvk_views(uvqk, num_heads, attn_dim, hidden_dim):
    """(q, k, v) as ``[M, H, d]`` views of the uvqk buffer."""
    hv, ha = hidden_dim * num_heads, attn_dim * num_heads
    v, q, k = uvqk[:, hv:].split_with_sizes((hv, ha, ha), 1)
    return (q.unflatten(1, (num_heads, attn_dim)), k.unflatten(1, (num_heads, attn_dim)),
            v.unflatten(1, (num_heads, hidden_dim)))


def _fused_uqvk_inference(x, norm_weight, norm_bias, eps, weight, bias, num_heads, attn_dim, hidden_dim):
    """The fused stage where no gradient is wanted: ``(u, q, k, v)``."""
    nw, nb, w, b = _stage_parameters(x, norm_weight, norm_bias, weight, bias)
    uvqk, u, _, _ = _fused_uqvk_launch(x, nw, nb, eps, w, b, hidden_dim * num_heads, inference=True)
    return (u,) + _uqvk_views(uvqk, num_heads, attn_dim, hidden_dim)


class _FusedUqvkFunction(torch.autograd.Function):
    """``uvqk = LN(x) W + b`` and ``u = SiLU(uvqk[:, :hv])`` from one tensor-core kernel
    (csrc/ln_linear_sm100.cu)."""

    @staticmethod
    def forward(ctx, x, norm_weight, norm_bias, eps, weight, bias, num_heads, attn_dim, hidden_dim):
        hv, ha = hidden_dim * num_heads, attn_dim * num_heads
        nw, nb, w, b = _stage_parameters(x, norm_weight, norm_bias, weight, bias)
        uvqk, u, mean, rstd = _fused_uqvk_launch(x, nw, nb, eps, w, b, hv)
        ctx.set_materialize_grads(False)
        ctx.save_for_backward(x, nw, nb, w, uvqk, mean, rstd)
        ctx.cfg = (eps, hv, ha, norm_weight.dtype, norm_bias.dtype, weight.dtype, bias.dtype)
        # q, k, v are views of the uvqk buffer, handed out as separate results so that the backward
        # receives their gradients one by one instead of three zero-padded [M, N] sums
        return (u,) + _uqvk_views(uvqk, num_heads, attn_dim, hidden_dim)

    @staticmethod
    def backward(ctx, du, dq, dk, dv):
        x, nw, nb, w, uvqk, mean, rstd = ctx.saved_tensors
        eps, hv, ha, nw_dtype, nb_dtype, w_dtype, b_dtype = ctx.cfg
        M, N = uvqk.shape
        d_uvqk = torch.empty((M, N), dtype=x.dtype, device=x.device)
        for lo, width, g in ((hv, hv, dv), (2 * hv, ha, dq), (2 * hv + ha, ha, dk)):
            if g is None:
                d_uvqk[:, lo:lo + width].zero_()
            else:
                d_uvqk[:, lo:lo + width].copy_(g.reshape(M, width))
        dx, dnw, dnb, dw, db = _fused_uqvk_backward(x, nw, nb, w, uvqk, mean, rstd, eps, hv, du, d_uvqk)
        return (dx, as_dtype(dnw, nw_dtype), as_dtype(dnb, nb_dtype), None, as_dtype(dw, w_dtype),
                as_dtype(db, b_dtype), None, None, None)


def _attention_switches(x):
    return _attention._IMPL[_attention._forced_impl], dtype_code(x)


class _FusedPreprocessAttentionFunction(torch.autograd.Function):
    """The fused uvqk stage and the attention as one autograd node: the attention backward writes
    dq / dk / dv straight into the column blocks of ``d_uvqk``, which then feeds the stage's
    backward GEMMs - no gradient copies in between.  Returns (u, attn [M, H, dv], k, v)."""

    @staticmethod
    def forward(ctx, x, norm_weight, norm_bias, eps, weight, bias, num_heads, attn_dim, hidden_dim, seq_offsets,
                num_targets, bias_by_distance, max_seq_len, alpha, max_attn_len, contextual_seq_len,
                recompute_uvqk=False):
        nw, nb, w, b = _stage_parameters(x, norm_weight, norm_bias, weight, bias)
        plan = any(ctx.needs_input_grad[:6]) or ctx.needs_input_grad[11]
        ctx.set_materialize_grads(False)  # k / v usually get no gradient: do not add zeros for them
        u, out, k, v, uvqk, mean, rstd, ctx.planned_scratch = _cabi.host().uvqk_attention_forward(
            x, nw, nb, w, b, eps, num_heads, attn_dim, hidden_dim, seq_offsets, num_targets, bias_by_distance,
            max_seq_len, alpha, max_attn_len, contextual_seq_len, *_attention_switches(x), plan, _attention._CHECK_STATUS)
        if not plan:
            ctx.planned_scratch = None
        # recompute_uvqk: the [M, 4 H d] projection - the largest activation of the layer - is not kept;
        # the backward runs the fused kernel once more (the reference's recompute_uvqk_in_backward,
        # generative_recommenders/ops/triton/triton_hstu_preprocess_and_attention.py:122-127, 185-203).
        # k and v go out as views of that buffer either way: it lives on only while the caller keeps them
        # (the layer does so for its KV cache, otherwise it drops them at once).
        keep = None if recompute_uvqk else uvqk
        ctx.save_for_backward(x, nw, nb, w, b, keep, mean, rstd, seq_offsets, num_targets, bias_by_distance)
        ctx.cfg = (eps, num_heads, attn_dim, hidden_dim, max_seq_len, alpha, max_attn_len, contextual_seq_len,
                   norm_weight.dtype, norm_bias.dtype, weight.dtype, bias.dtype)
        return u, out, k, v

    @staticmethod
    def backward(ctx, du, dattn, dk_ext, dv_ext):
        x, nw, nb, w, b, uvqk, mean, rstd, seq_offsets, num_targets, bias_by_distance = ctx.saved_tensors
        (eps, H, A, V, max_seq_len, alpha, max_attn_len, contextual_seq_len,
         nw_dtype, nb_dtype, w_dtype, b_dtype) = ctx.cfg
        planned = None
        if dattn is not None:
            planned, ctx.planned_scratch = ctx.planned_scratch, None
        dx, dnw, dnb, dw, db, d_bias = _cabi.host().uvqk_attention_backward(
            x, nw, nb, w, b, uvqk, mean, rstd, eps, H, A, V, seq_offsets, num_targets, bias_by_distance, max_seq_len,
            alpha, max_attn_len, contextual_seq_len, *_attention_switches(x), du, dattn, dk_ext, dv_ext, planned,
            bias_by_distance is not None and ctx.needs_input_grad[11], _attention._CHECK_STATUS)
        return (dx, as_dtype(dnw, nw_dtype), as_dtype(dnb, nb_dtype), None, as_dtype(dw, w_dtype),
                as_dtype(db, b_dtype), None, None, None, None, None, d_bias, None, None, None, None, None)


_FUSED_UQVK = True


def set_fused_uqvk(on: bool) -> None:
    """Switch between the fused tensor-core uvqk stage (default, where the shapes allow it) and the
    three separate stages (LayerNorm kernel, library GEMM, SiLU kernel)."""
    global _FUSED_UQVK
    _FUSED_UQVK = bool(on)


def hstu_cached_attention(x, norm_weight, norm_bias, norm_eps, num_heads, attn_dim, hidden_dim, uvqk_weight, uvqk_bias,
                          k_cache, v_cache, cache_offsets, num_targets, max_seq_len, attn_alpha, max_attn_len,
                          contextual_seq_len):
    """The uvqk stage on the new rows of every sequence, their K and V behind the cached ones, and the attention
    of the new rows against both: ``(u, attn [M, H dv], k, v, seq_offsets)``, or None where the separate
    ops have to do it."""
    hv, ha, M = hidden_dim * num_heads, attn_dim * num_heads, x.shape[0]
    B = cache_offsets.numel() - 1
    if not (_FUSED_UQVK and x.is_cuda and B > 0 and M % B == 0
            and _cabi.host().cached_supported(x, uvqk_weight, hv, ha, k_cache, v_cache, cache_offsets)
            and outside_autograd(x, norm_weight, norm_bias, uvqk_weight, uvqk_bias, k_cache, v_cache)):
        return None
    require_cuda(norm_weight, norm_bias, uvqk_weight, uvqk_bias, k_cache, v_cache, cache_offsets, num_targets)
    nw, nb, w, b = _stage_parameters(x, norm_weight, norm_bias, uvqk_weight, uvqk_bias)
    nbytes = _cabi.lib().b200_hstu_ln_linear_workspace_bytes(*w.shape)
    ws, prepared, remember = _prepared_workspace(nw, nb, w, b, nbytes, x.device, True)
    result = _cabi.host().cached_attention(
        x, nw, nb, w, b, float(norm_eps), num_heads, attn_dim, hidden_dim, ws, prepared, k_cache, v_cache,
        cache_offsets, _index(num_targets), int(max_seq_len), float(attn_alpha), int(max_attn_len),
        int(contextual_seq_len), *_attention_switches(x), _attention._CHECK_STATUS)
    if remember is not None:
        remember()
    return result


def hstu_compute_uqvk(
    x: torch.Tensor,
    norm_weight: torch.Tensor,
    norm_bias: torch.Tensor,
    norm_eps: float,
    num_heads: int,
    attn_dim: int,
    hidden_dim: int,
    uvqk_weight: torch.Tensor,
    uvqk_bias: torch.Tensor,
    kernel: HammerKernel = HammerKernel.CUDA,
) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor]:
    """LN -> addmm -> split [u | v | q | k] -> SiLU(u); returns (u, q, k, v) with q, k, v as
    ``[L, H, d]`` views of the uvqk buffer (generative_recommenders/ops/hstu_compute.py:54-104)."""
    _require_cuda_backend(kernel)
    require_cuda(x, norm_weight, norm_bias, uvqk_weight, uvqk_bias)
    hv, ha = hidden_dim * num_heads, attn_dim * num_heads
    if _FUSED_UQVK and _fused_uqvk_supported(x, uvqk_weight, hv):
        if outside_autograd(x, norm_weight, norm_bias, uvqk_weight, uvqk_bias):
            return _fused_uqvk_inference(x, norm_weight, norm_bias, float(norm_eps), uvqk_weight, uvqk_bias,
                                         num_heads, attn_dim, hidden_dim)
        return _FusedUqvkFunction.apply(x, norm_weight, norm_bias, float(norm_eps), uvqk_weight, uvqk_bias,
                                        num_heads, attn_dim, hidden_dim)
    else:
        normed_x = layer_norm(x, weight=norm_weight, bias=norm_bias, eps=norm_eps, kernel=kernel)
        uvqk = addmm(uvqk_bias, normed_x, uvqk_weight, kernel)
        u = _SiluColumnsFunction.apply(uvqk[:, :hv], hv)
    v = uvqk[:, hv : 2 * hv].view(-1, num_heads, hidden_dim)
    q = uvqk[:, 2 * hv : 2 * hv + ha].view(-1, num_heads, attn_dim)
    k = uvqk[:, 2 * hv + ha :].view(-1, num_heads, attn_dim)
    return u, q, k, v


def _norm_mul_forward(attn, u, weight, bias, eps, num_heads, linear_dim, concat_u, concat_x, act, group_norm,
                      dropout_ratio, dropout_seed, want_mask=False, stats=True):
    """One launch of the norm-mul kernel; returns ``(out, mean, rstd)`` (inputs already contiguous in
    their last dimension, weight / bias already of the activation dtype); without ``stats`` the last two
    are None."""
    result = _cabi.host().norm_mul_forward(
        attn, u, weight, bias, eps, num_heads, linear_dim, concat_u, concat_x, act, group_norm, dropout_ratio, dropout_seed,
        dtype_code(attn), want_mask, stats)
    return result if want_mask else result[:3]


def _norm_mul_backward(dout, attn, u, weight, bias, mean, rstd, eps, num_heads, linear_dim, concat_u, concat_x, act,
                       group_norm, dropout_ratio, dropout_seed, dropout_mask=None):
    """Backward of the norm-mul kernel; returns ``(dattn, du, dweight, dbias)``.  ``dropout_mask``: the
    bits the forward stored; without them the kernel regenerates the mask from the seed."""
    return _cabi.host().norm_mul_backward(
        dout, attn, u, weight, bias, mean, rstd, eps, num_heads, linear_dim, concat_u, concat_x, act, group_norm,
        dropout_ratio, dropout_seed, dropout_mask, dtype_code(attn))


# By default the backward of the norm-mul stage regenerates the dropout mask from the seed and nothing
# is stored.  Switched on, the forward also writes the mask as bits (6 % of the output's bytes) and the
# backward reads them.  Measured on B200 at 1965 MHz, 200 k rows of bf16, [u | attn | y], ratio 0.3, forward +
# backward in us (repeats agree within 1 %): D = 256 156 + 207 regenerating, 169 + 225 stored;
# D = 512 270 + 330 and 314 + 305; D = 1024 592 + 840 and 803 + 3470 (the kernel for that width, with its
# accumulators in shared memory, only regenerates).  It pays at none of these, so it is off.  With recompute_y the
# mask is never stored.
_STORE_DROPOUT_MASK = False


def set_store_dropout_mask(on: bool) -> None:
    global _STORE_DROPOUT_MASK
    _STORE_DROPOUT_MASK = bool(on)


class _NormMulFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, attn, u, weight, bias, eps, num_heads, linear_dim, concat_u, concat_x, act, group_norm,
                dropout_ratio=0.0, dropout_seed=None):
        if attn.stride(-1) != 1:
            attn = attn.contiguous()
        if u.stride(-1) != 1:
            u = u.contiguous()
        weight = as_dtype(weight, attn.dtype).contiguous()
        bias = as_dtype(bias, attn.dtype).contiguous()
        keep_mask = _STORE_DROPOUT_MASK and any(ctx.needs_input_grad)   # (grad mode is off inside forward())
        out, mean, rstd, mask = _norm_mul_forward(attn, u, weight, bias, eps, num_heads, linear_dim, concat_u, concat_x,
                                                  act, group_norm, dropout_ratio, dropout_seed, want_mask=True) \
            if keep_mask else _norm_mul_forward(attn, u, weight, bias, eps, num_heads, linear_dim, concat_u, concat_x,
                                                act, group_norm, dropout_ratio, dropout_seed) + (None,)
        ctx.save_for_backward(attn, u, weight, bias, mean, rstd, dropout_seed, mask)
        ctx.cfg = (eps, num_heads, linear_dim, concat_u, concat_x, act, group_norm, dropout_ratio)
        return out

    @staticmethod
    def backward(ctx, dout):
        attn, u, weight, bias, mean, rstd, dropout_seed, mask = ctx.saved_tensors
        dattn, du, dw, db = _norm_mul_backward(dout, attn, u, weight, bias, mean, rstd, *ctx.cfg, dropout_seed, mask)
        return dattn, du, dw, db, None, None, None, None, None, None, None, None, None


class _OutputStageFunction(torch.autograd.Function):
    """The whole output stage, ``x + dropout(cat([u, attn, act(u) * Norm(attn)])) @ W``, as one autograd
    node that keeps its inputs and the row statistics only: the concatenated activation (three
    times as wide as ``attn``) is recomputed in the backward by one more launch of the norm-mul
    kernel - with the same dropout seed, hence the same mask - before the two backward GEMMs read it.
    This is the reference's ``recompute_y_in_backward``
    (generative_recommenders/ops/triton/triton_hstu_linear.py:1895-2040)."""

    @staticmethod
    def forward(ctx, attn, u, x, weight, bias, output_weight, eps, num_heads, linear_dim, concat_u, concat_x, act,
                group_norm, dropout_ratio, dropout_seed):
        if attn.stride(-1) != 1:
            attn = attn.contiguous()
        if u.stride(-1) != 1:
            u = u.contiguous()
        w = as_dtype(weight, attn.dtype).contiguous()
        b = as_dtype(bias, attn.dtype).contiguous()
        wo = as_dtype(output_weight, x.dtype)
        cfg = (eps, num_heads, linear_dim, concat_u, concat_x, act, group_norm, dropout_ratio)
        out, mean, rstd = _cabi.host().output_forward(attn, u, x, w, b, wo, *cfg, dropout_seed, dtype_code(attn), True,
                                                          False)
        ctx.save_for_backward(attn, u, w, b, wo, mean, rstd, dropout_seed)
        ctx.cfg = cfg
        ctx.dtypes = (weight.dtype, bias.dtype, output_weight.dtype)
        return out

    @staticmethod
    def backward(ctx, dout):
        attn, u, w, b, wo, mean, rstd, dropout_seed = ctx.saved_tensors
        if dout.stride(-1) != 1:
            dout = dout.contiguous()
        dattn, du, dw, db, d_wo = _cabi.host().output_backward(dout, attn, u, w, b, wo, mean, rstd, *ctx.cfg, dropout_seed,
                                                               dtype_code(attn))
        wdt, bdt, odt = ctx.dtypes
        return (dattn, du, dout, as_dtype(dw, wdt), as_dtype(db, bdt), as_dtype(d_wo, odt), None, None, None, None,
                None, None, None, None, None)


def _draw_dropout_seed(device) -> torch.Tensor:
    # from torch's CUDA generator: reproducible under torch.manual_seed, and a fresh value on every
    # replay when the step is captured in a CUDA graph
    return torch.randint(0, 2 ** 62, (1,), dtype=torch.int64, device=device)


def hstu_norm_mul_dropout(
    attn: torch.Tensor,
    u: torch.Tensor,
    norm_weight: torch.Tensor,
    norm_bias: torch.Tensor,
    norm_eps: float,
    dropout_ratio: float,
    training: bool,
    concat_u: bool = False,
    concat_x: bool = False,
    mul_u_activation_type: str = "none",
    group_norm: bool = False,
    num_heads: int = 1,
    linear_dim: int = -1,
    dropout_seed: Optional[torch.Tensor] = None,
) -> torch.Tensor:
    """``dropout(cat([u, attn, act(u) * Norm(attn)]))`` - the input of the output linear
    (generative_recommenders/ops/pytorch/pt_hstu_linear.py:23-82).

    In training the dropout mask is generated inside the kernel (counter-based Philox keyed by
    ``dropout_seed``, a one-element int64 tensor on the device; drawn from torch's CUDA generator when
    not given) and regenerated by the backward, like the reference's GPU path
    (ops/triton/triton_hstu_linear.py:365-492); the mask bits are this library's own.  The
    group-norm variant applies ``torch.nn.functional.dropout`` afterwards."""
    if mul_u_activation_type not in _ACT:
        raise ValueError("mul_u_activation_type must be one of none / sigmoid / silu")
    if group_norm and concat_u != concat_x:
        # the reference's group-norm branch only concatenates when both flags are set (:52-54)
        concat_u = concat_x = False
    act = 0 if group_norm else _ACT[mul_u_activation_type]
    if linear_dim <= 0:
        linear_dim = attn.shape[1] // num_heads
    drop = training and dropout_ratio > 0.0
    fused_drop = drop and not group_norm and dropout_ratio < 1.0
    if fused_drop and dropout_seed is None:
        dropout_seed = _draw_dropout_seed(attn.device)
    cfg = (float(norm_eps), int(num_heads), int(linear_dim), bool(concat_u), bool(concat_x), act, bool(group_norm),
           float(dropout_ratio) if fused_drop else 0.0, dropout_seed if fused_drop else None)
    if not group_norm and outside_autograd(attn, u, norm_weight, norm_bias):
        y, _, _ = _norm_mul_forward(
            attn if attn.stride(-1) == 1 else attn.contiguous(), u if u.stride(-1) == 1 else u.contiguous(),
            as_dtype(norm_weight, attn.dtype).contiguous(), as_dtype(norm_bias, attn.dtype).contiguous(), *cfg,
            stats=False)
    else:
        y = _NormMulFunction.apply(attn, u, norm_weight, norm_bias, *cfg)
    if drop and not fused_drop:
        y = torch.nn.functional.dropout(y, p=dropout_ratio, training=True)
    return y


def _output_inference(attn, u, x, norm_weight, norm_bias, norm_eps, output_weight, num_heads, linear_dim, concat_u,
                      concat_x, act, dropout_ratio, over_x=False):
    """The output stage (LayerNorm flavour) where no gradient is wanted; with ``over_x`` the result goes over
    x."""
    return _cabi.host().output_forward(
        attn if attn.stride(-1) == 1 else attn.contiguous(), u if u.stride(-1) == 1 else u.contiguous(), x,
        as_dtype(norm_weight, attn.dtype).contiguous(), as_dtype(norm_bias, attn.dtype).contiguous(),
        as_dtype(output_weight, x.dtype), float(norm_eps), int(num_heads),
        int(linear_dim) if linear_dim > 0 else attn.shape[1] // num_heads, bool(concat_u), bool(concat_x), act, False,
        float(dropout_ratio), _draw_dropout_seed(attn.device) if dropout_ratio > 0.0 else None, dtype_code(attn), False,
        over_x and x.is_contiguous() and not torch.is_autocast_enabled("cuda"))[0]


def _compute_output(attn, u, x, norm_weight, norm_bias, norm_eps, output_weight, num_heads, linear_dim, dropout_ratio,
                    training, concat_u, concat_x, mul_u_activation_type, group_norm, recompute_y_in_backward, kernel,
                    over_x=False):
    """``hstu_compute_output``; ``over_x``: the caller has no use for x any more, the result may go over it."""
    _require_cuda_backend(kernel)
    require_cuda(attn, u, x, norm_weight, norm_bias, output_weight)
    if recompute_y_in_backward and torch.is_grad_enabled() and mul_u_activation_type in _ACT and attn.shape[0] > 0:
        g_ = bool(group_norm)
        cu, cx = bool(concat_u), bool(concat_x)
        if g_ and cu != cx:
            cu = cx = False
        drop = training and dropout_ratio > 0.0
        if not (drop and g_):   # the group-norm variant draws its mask with torch's dropout: kept on the plain path
            seed = _draw_dropout_seed(attn.device) if (drop and dropout_ratio < 1.0) else None
            ld = linear_dim if linear_dim > 0 else attn.shape[1] // num_heads
            return _OutputStageFunction.apply(attn, u, x, norm_weight, norm_bias, output_weight, float(norm_eps),
                                              int(num_heads), int(ld), cu, cx, 0 if g_ else _ACT[mul_u_activation_type],
                                              g_, float(dropout_ratio) if seed is not None else 0.0, seed)
    drop = training and dropout_ratio > 0.0
    if (not group_norm and mul_u_activation_type in _ACT and not (drop and dropout_ratio >= 1.0)
            and outside_autograd(attn, u, x, norm_weight, norm_bias, output_weight)):
        return _output_inference(attn, u, x, norm_weight, norm_bias, norm_eps, output_weight, num_heads, linear_dim,
                                 concat_u, concat_x, _ACT[mul_u_activation_type], dropout_ratio if drop else 0.0,
                                 over_x=over_x)
    y = hstu_norm_mul_dropout(attn, u, norm_weight, norm_bias, norm_eps, dropout_ratio, training, concat_u, concat_x,
                              mul_u_activation_type, group_norm, num_heads, linear_dim)
    return addmm(x, y, as_dtype(output_weight, x.dtype), kernel)


def hstu_compute_output(
    attn: torch.Tensor,
    u: torch.Tensor,
    x: torch.Tensor,
    norm_weight: torch.Tensor,
    norm_bias: torch.Tensor,
    norm_eps: float,
    output_weight: torch.Tensor,
    num_heads: int,
    linear_dim: int,
    dropout_ratio: float,
    training: bool,
    concat_u: bool,
    concat_x: bool,
    mul_u_activation_type: str,
    group_norm: bool,
    recompute_y_in_backward: bool,
    kernel: HammerKernel = HammerKernel.CUDA,
) -> torch.Tensor:
    """``x + dropout(cat([u, attn, act(u) * Norm(attn)])) @ W_out``
    (generative_recommenders/ops/hstu_compute.py:107-214,
    generative_recommenders/ops/pytorch/pt_hstu_linear.py:85-120).
    With ``recompute_y_in_backward`` the stage is one autograd node that does not keep the
    concatenated activation (see ``_OutputStageFunction``)."""
    return _compute_output(attn, u, x, norm_weight, norm_bias, norm_eps, output_weight, num_heads, linear_dim,
                           dropout_ratio, training, concat_u, concat_x, mul_u_activation_type, group_norm,
                           recompute_y_in_backward, kernel)


def hstu_preprocess_and_attention(
    x: torch.Tensor,
    norm_weight: torch.Tensor,
    norm_bias: torch.Tensor,
    norm_eps: float,
    num_heads: int,
    attn_dim: int,
    hidden_dim: int,
    uvqk_weight: torch.Tensor,
    uvqk_bias: torch.Tensor,
    max_seq_len: int,
    seq_offsets: torch.Tensor,
    attn_alpha: float,
    causal: bool,
    num_targets: Optional[torch.Tensor],
    max_attn_len: int,
    contextual_seq_len: int,
    recompute_uvqk_in_backward: bool,
    recompute_normed_x_in_backward: bool,
    sort_by_length: bool,
    prefill: bool = False,
    kernel: HammerKernel = HammerKernel.CUDA,
    enable_tma: Optional[bool] = None,
    bias_by_distance: Optional[torch.Tensor] = None,
) -> Tuple[torch.Tensor, torch.Tensor, Optional[torch.Tensor], Optional[torch.Tensor]]:
    """uqvk stage followed by the attention; returns ``(u, attn_output [L, H*dv], k, v)``
    (generative_recommenders/ops/hstu_compute.py:217-335; like the reference's composite the
    attention runs with dropout off, :327-328)."""
    _require_cuda_backend(kernel)
    torch._assert(max_seq_len > 0, "max_seq_len must be larger than 0")
    torch._assert(x.dim() == 2, "x must be 2-D")
    torch._assert(x.shape[1] == uvqk_weight.shape[0], "x.shape[1] must equal uvqk_weight.shape[0]")
    torch._assert(
        uvqk_weight.shape[1] == 2 * num_heads * (hidden_dim + attn_dim),
        "uvqk_weight.shape[1] must equal 2 * num_heads * (hidden_dim + attn_dim)",
    )
    torch._assert(causal is True, "only causal attention is supported.")
    hv = hidden_dim * num_heads
    if (_FUSED_UQVK and x.is_cuda and _fused_uqvk_supported(x, uvqk_weight, hv)
            and attn_dim == hidden_dim and attn_dim in (64, 128)):
        # one autograd node for the stage and the attention (see _FusedPreprocessAttentionFunction)
        require_cuda(x, norm_weight, norm_bias, uvqk_weight, uvqk_bias, seq_offsets, num_targets, bias_by_distance)
        inference = outside_autograd(x, norm_weight, norm_bias, uvqk_weight, uvqk_bias, bias_by_distance)
        offs = _index(seq_offsets) if inference else _i32(seq_offsets)
        nt = _index(num_targets) if inference else _i32(num_targets)
        if nt is not None and nt.numel() != offs.numel() - 1:
            raise RuntimeError("num_targets must have one entry per sequence")
        rab = None if bias_by_distance is None else bias_by_distance.to(torch.float32).reshape(-1).contiguous()
        if inference:
            nw, nb, w, b = _stage_parameters(x, norm_weight, norm_bias, uvqk_weight, uvqk_bias)
            nbytes = _cabi.lib().b200_hstu_ln_linear_workspace_bytes(*w.shape)
            ws, prepared, remember = _prepared_workspace(nw, nb, w, b, nbytes, x.device, True)
            result = _cabi.host().uvqk_attention_inference(
                x, nw, nb, w, b, float(norm_eps), num_heads, attn_dim, hidden_dim, ws, prepared, offs, nt, rab,
                int(max_seq_len), float(attn_alpha), int(max_attn_len), int(contextual_seq_len),
                *_attention_switches(x), _attention._CHECK_STATUS)
            if remember is not None:
                remember()
            return result
        u, attn, k, v = _FusedPreprocessAttentionFunction.apply(
            x, norm_weight, norm_bias, float(norm_eps), uvqk_weight, uvqk_bias, num_heads, attn_dim, hidden_dim,
            offs, nt, rab, int(max_seq_len), float(attn_alpha), int(max_attn_len), int(contextual_seq_len),
            bool(recompute_uvqk_in_backward))
        return u, attn.view(-1, hidden_dim * num_heads), k, v
    if (x.is_cuda and x.shape[0] > 0 and x.stride(1) == 1 and not (_FUSED_UQVK and _fused_uqvk_supported(x, uvqk_weight, hv))
            and all(t.dtype is x.dtype for t in (norm_weight, norm_bias, uvqk_weight, uvqk_bias))
            and outside_autograd(x, norm_weight, norm_bias, uvqk_weight, uvqk_bias, bias_by_distance)
            and not torch.is_autocast_enabled("cuda")):   # (it changes the type between the stages)
        # the separate stages in one call
        require_cuda(norm_weight, norm_bias, uvqk_weight, uvqk_bias, seq_offsets, num_targets, bias_by_distance)
        offs, nt = _index(seq_offsets), _index(num_targets)
        if nt is not None and nt.numel() != offs.numel() - 1:
            raise RuntimeError("num_targets must have one entry per sequence")
        rab = None if bias_by_distance is None else bias_by_distance.to(torch.float32).reshape(-1).contiguous()
        return _cabi.host().separate_attention_inference(
            x, norm_weight.contiguous(), norm_bias.contiguous(), uvqk_weight, uvqk_bias, float(norm_eps), num_heads,
            attn_dim, hidden_dim, offs, nt, rab, int(max_seq_len), float(attn_alpha), int(max_attn_len),
            int(contextual_seq_len), *_attention_switches(x), _attention._CHECK_STATUS)
    u, q, k, v = hstu_compute_uqvk(
        x=x, norm_weight=norm_weight, norm_bias=norm_bias, norm_eps=norm_eps, num_heads=num_heads,
        attn_dim=attn_dim, hidden_dim=hidden_dim, uvqk_weight=uvqk_weight, uvqk_bias=uvqk_bias, kernel=kernel,
    )
    attn_output = hstu_mha(
        max_seq_len=max_seq_len, alpha=attn_alpha, q=q, k=k, v=v, seq_offsets=seq_offsets, causal=causal,
        dropout_pr=0.0, training=False, num_targets=num_targets, max_attn_len=max_attn_len,
        contextual_seq_len=contextual_seq_len, sort_by_length=sort_by_length, kernel=kernel,
        bias_by_distance=bias_by_distance,
    ).view(-1, hidden_dim * num_heads)
    return u, attn_output, k, v
