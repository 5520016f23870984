"""Chunked gated delta rule (GDN) - the `[B,T,H,D]` operator surface.

`chunk_gated_delta_rule` keeps the argument names and semantics of the reference's composed entry
`flash_gated_delta_rule` (examples/flash_gated_delta_rule.py:1126-1228): q,k `[B,T,HK,K]`,
v `[B,T,HV,V]`, g (log decay) and beta `[B,T,HV]`, `scale` defaulting to K^-0.5, `initial_state`
`[N,HV,K,V]`, `output_final_state`, optional in-kernel q/k L2 normalisation, packed variable-length
batches through `cu_seqlens`, and GVA (value head hv reads q/k head hv // (HV/HK)) without
materialising repeated q/k.
"""
from __future__ import annotations

import torch

from .. import host

CHUNK = 64


def _varlen_meta(cu_seqlens, device):
    """Host-side chunk bookkeeping for packed batches (the reference prepares the same
    (sequence, chunk) metadata on the host, examples/flash_gated_delta_rule.py:78-100)."""
    cu_host = [int(x) for x in (cu_seqlens.tolist() if isinstance(cu_seqlens, torch.Tensor) else cu_seqlens)]
    if len(cu_host) < 2 or cu_host[0] != 0 or any(b < a for a, b in zip(cu_host, cu_host[1:])):
        raise RuntimeError(f"cu_seqlens must start at 0 and be non-decreasing, got {cu_host}")
    lens = [b - a for a, b in zip(cu_host, cu_host[1:])]
    offs = [0]
    for L in lens:
        offs.append(offs[-1] + (L + CHUNK - 1) // CHUNK)
    cu = torch.tensor(cu_host, dtype=torch.int32, device=device)
    co = torch.tensor(offs, dtype=torch.int32, device=device)
    return cu, co, max(lens), offs[-1], len(lens), cu_host[-1]


def _as_rows(t):
    """The kernels address tokens by a flat row index: batch rows must sit back to back."""
    if t.stride(-1) != 1 or (t.shape[0] > 1 and t.stride(0) != t.shape[1] * t.stride(1)):
        return t.contiguous()
    return t


def _fold_batch(t):
    """A `[B,T,H,D]` view of head-first memory (`[B,H,T,D]` storage: batch stride = H x head stride) seen as one sequence of
    B*H heads, `[1,T,B*H,D]`, on the same storage.  Every (batch row, head) pair is an independent recurrence, so the kernels
    run head-first batches through this view without a copy.  None when the strides do not allow it."""
    return host().fold(t)


def _fold_plan(q, k, v, cu_seqlens):
    """Whether a fixed-length batch whose rows do not sit back to back (head-first storage) can run as one sequence of
    B*H heads instead of being copied: returns the folded (q, k, v) views or None."""
    return host().fold_plan(q, k, v, cu_seqlens)


def gdn_chunk_fwd(q, k, v, g, beta, scale, initial_state, output_final_state, cu_seqlens=None, save_for_backward=False,
                  output_dtype=None):
    """Launch the forward kernels.  Returns (o, final_state, saved) where saved holds gam, X and, when
    `save_for_backward`, the split per-chunk states and v_new that the backward kernels consume."""
    o, ht, gam, x_inv, s_img, vn_img, p_img, seg_m, geo = host().gdn_fwd(q, k, v, g, beta, scale, initial_state, output_final_state,
                                                                  cu_seqlens, save_for_backward, output_dtype)
    cu, co, n, max_len, total_chunks = geo
    return o, ht, dict(gam=gam, x_inv=x_inv, s_img=s_img, vn_img=vn_img, p_img=p_img, seg_m=seg_m, cu=cu, co=co, max_len=max_len,
                       total_chunks=total_chunks, N=n)


def gdn_chunk_bwd(q, k, v, beta, saved, do, dht, scale, want_dh0, grad_dtype=None):
    """Launch the backward kernels on the tensors the forward saved.
    Returns (dq, dk, dv, dg, dbeta, dh0 | None); gradients are bf16 unless `grad_dtype` says fp32."""
    s = saved
    return host().gdn_bwd(q, k, v, beta, s["gam"], s["x_inv"], s["s_img"], s["vn_img"], s["p_img"], s["seg_m"], s["cu"], s["co"], s["N"],
                          s["max_len"], s["total_chunks"], do, dht, scale, want_dh0, *(grad_dtype,) * 5)


class ChunkGatedDeltaRuleFunction:
    """The reference's autograd binding by name (examples/flash_gated_delta_rule.py:1026-1122): `apply` runs the native node,
    which saves q, k, v, beta, gam, X and the split per-chunk states / v_new instead of recomputing them."""

    @staticmethod
    def apply(q, k, v, g, beta, scale, initial_state, output_final_state, cu_seqlens, output_dtype, qk_l2norm):
        return host().gdn(q, k, v, g, beta, scale, initial_state, output_final_state, cu_seqlens, output_dtype, qk_l2norm)


def chunk_gated_delta_rule_fwd_bwd(q, k, v, g, beta, do, scale=None, initial_state=None, dht=None, cu_seqlens=None,
                                   output_dtype=None, grad_dtype=None):
    """Forward and backward in one call without the autograd graph (what a training step costs).
    Returns (o, final_state, (dq, dk, dv, dg, dbeta, dh0))."""
    scale = q.shape[-1] ** -0.5 if scale is None else float(scale)
    q, k, v, g, beta = (_as_rows(x) for x in (q, k, v, g, beta))
    o, ht, saved = gdn_chunk_fwd(q, k, v, g, beta, scale, initial_state, True, cu_seqlens, save_for_backward=True,
                                 output_dtype=output_dtype)
    grads = gdn_chunk_bwd(q, k, v, beta, saved, do, dht, scale, initial_state is not None, grad_dtype=grad_dtype)
    return o, ht, grads


chunk_gated_delta_rule_bwd = gdn_chunk_bwd


def chunk_gated_delta_rule(q, k, v, g, beta, scale=None, initial_state=None, output_final_state=False,
                           use_qk_l2norm_in_kernel=False, cu_seqlens=None, chunk_size=64, head_first=False,
                           output_dtype=None):
    """Returns ``(o [B,T,HV,V], final_state [N,HV,K,V] | None)``; differentiable w.r.t. q, k, v, g, beta, initial_state."""
    op = "chunk_gated_delta_rule"
    if head_first:   # [B,H,T,D] tokens and [B,H,T] gates: the same operator on transposed views, output back in [B,H,T,V]
        o, ht = chunk_gated_delta_rule(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), g.transpose(1, 2), beta.transpose(1, 2),
                                       scale=scale, initial_state=initial_state, output_final_state=output_final_state,
                                       use_qk_l2norm_in_kernel=use_qk_l2norm_in_kernel, cu_seqlens=cu_seqlens, chunk_size=chunk_size,
                                       output_dtype=output_dtype)
        return o.transpose(1, 2), ht
    # chunk_size is the reference's blocking parameter: o, the final state and every gradient are the same function of
    # the inputs for any blocking, so the fused kernels keep their own 64-token tiling for the sizes the reference tiles for
    if int(chunk_size) not in (16, 32, 64, 128):
        raise NotImplementedError(f"{op}: chunk_size must be one of 16, 32, 64, 128, got {chunk_size}")
    scale = q.shape[-1] ** -0.5 if scale is None else float(scale)
    return host().gdn(q, k, v, g, beta, scale, initial_state, output_final_state, cu_seqlens, output_dtype,
                      use_qk_l2norm_in_kernel)


def flash_gated_delta_rule(q, k, v, g, beta, scale=None, initial_state=None, output_final_state=False,
                           use_qk_l2norm_in_kernel=False, cu_seqlens=None, cu_seqlens_list=None, chunk_indices=None,
                           chunk_indices_list=None, chunk_size=64, head_first=False):
    """The reference's composed entry with its own layout and checks (examples/flash_gated_delta_rule.py:1126-1228):
    q, k `[B,H,T,K]`, v `[B,H,T,V]` (head-first), g, beta `[B,T,H]`; returns (o `[B,T,H,V]`, final_state `[N,H,K,V]` or None).
    The host-side chunk metadata arguments (`cu_seqlens_list`, `chunk_indices`, `chunk_indices_list`) are accepted and not
    needed: the chunk geometry follows from `cu_seqlens`.  GVA callers pass q, k with fewer heads than v."""
    del cu_seqlens_list, chunk_indices, chunk_indices_list
    if q.dtype != k.dtype or k.dtype != v.dtype:
        raise ValueError(f"q current type is {q.dtype}, k current type is {k.dtype}, v current type is {v.dtype}; they should be equal")
    if q.dtype == torch.float32:
        raise ValueError("ChunkGatedDeltaRuleFunction does not support float32. Please use float16/bfloat16.")
    if beta.ndim != 3 or g.ndim != 3:
        raise ValueError("g and beta must be rank-3 tensors with shape [B, T, H].")
    if q.ndim != 4 or k.ndim != 4 or v.ndim != 4:
        raise ValueError("q, k and v must be rank-4 tensors with shape [B, H, T, D].")
    if q.shape[:3] != k.shape[:3] or q.shape[0] != v.shape[0] or q.shape[2] != v.shape[2]:
        raise ValueError(f"q/k/v shape prefixes must match, got {q.shape}, {k.shape}, {v.shape}.")
    if g.shape != beta.shape:
        raise ValueError(f"g and beta shapes must match, got {g.shape} and {beta.shape}.")
    if g.shape[0] != v.shape[0] or g.shape[1] != v.shape[2] or g.shape[2] != v.shape[1]:
        raise ValueError(f"Expected q/k/v in [B, H, T, D] and g/beta in [B, T, H]; got q={tuple(q.shape)}, g={tuple(g.shape)}.")
    if head_first:
        import warnings
        warnings.warn("head_first is kept only for API compatibility. This entry always expects q/k/v as [B, H, T, D].", stacklevel=2)
    if chunk_size != 2 ** (int(chunk_size).bit_length() - 1):
        raise ValueError(f"chunk_size must be a power of 2, got {chunk_size}.")
    if cu_seqlens is not None and q.shape[0] != 1:
        raise ValueError(f"The batch size is expected to be 1 rather than {q.shape[0]} when using cu_seqlens. "
                         "Please flatten variable-length inputs before processing.")
    if cu_seqlens is not None and initial_state is not None and initial_state.shape[0] != len(cu_seqlens) - 1:
        raise ValueError("The number of initial states is expected to match the number of input sequences, "
                         f"got initial_state.shape[0]={initial_state.shape[0]} and sequences={len(cu_seqlens) - 1}.")
    return chunk_gated_delta_rule(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), g, beta, scale=scale,
                                  initial_state=initial_state, output_final_state=output_final_state,
                                  use_qk_l2norm_in_kernel=use_qk_l2norm_in_kernel, cu_seqlens=cu_seqlens, chunk_size=chunk_size)
