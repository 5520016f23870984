"""Fused-recurrent gated delta rule (decode).  Two entry points over one CUDA kernel:

* :func:`fused_recurrent_gated_delta_rule` - the `[B,T,H,D]` surface with `initial_state` /
  `final_state` of shape `[N,HV,K,V]` (upstream ``fla.ops`` naming, which the reference targets).
* :func:`recurrent_gated_delta_rule` - the reference's in-place state-pool operator
  (torch_custom/fla_npu/fla_npu/ops/ascendc/_aclnn_ctypes.py:654-846), same argument names.
"""
from __future__ import annotations

import torch

from .. import host

_GATE_TYPES = (torch.bfloat16, torch.float32, torch.float16)   # fp16 gates become fp32 in the library's conversion kernel


def _activation_ok(name, t):
    # fp16 activations are read exactly by the decode kernel (fp32 arithmetic on CUDA cores); q, k, v share one dtype
    if t.dtype not in (torch.bfloat16, torch.float16):
        raise TypeError(f"{name} dtype must be torch.bfloat16 or torch.float16, got {t.dtype}")


def fused_recurrent_gated_delta_rule(q, k, v, g=None, beta=None, scale=None, initial_state=None,
                                     output_final_state=False, use_qk_l2norm_in_kernel=False, cu_seqlens=None,
                                     transpose_state_layout=False, inplace_final_state=False, gk=None):
    """q,k `[B,T,HK,K]`, v `[B,T,HV,V]` bf16; g, beta `[B,T,HV]`; gk `[B,T,HV,K]` (per-key-channel log decay, optional);
    initial_state `[N,HV,K,V]` fp32|bf16 (`[N,HV,V,K]` with ``transpose_state_layout``).
    Returns ``(o [B,T,HV,V], final_state | None)``.

    With ``inplace_final_state`` the final state overwrites ``initial_state`` (serving pools) and that
    same tensor is returned.  With ``cu_seqlens`` (int32/int64 `[N+1]`) B must be 1.
    """
    scale = q.shape[-1] ** -0.5 if scale is None else scale
    return host().recurrent_fused(q, k, v, g, beta, scale, initial_state, output_final_state, use_qk_l2norm_in_kernel,
                                  cu_seqlens, transpose_state_layout, inplace_final_state, gk)


def recurrent_gated_delta_rule(query, key, value, state, *, beta, scale=1.0, actual_seq_lengths, ssm_state_indices,
                               num_accepted_tokens=None, g=None, gk=None):
    """Reference operator surface: run recurrent GDN and update ``state`` in place.

    query/key `[T,Nk,Dk]`, value `[T,Nv,Dv]`, beta `[T,Nv]` bf16; g `[T,Nv]` fp32; state
    `[blocks,Nv,Dv,Dk]` bf16|fp32 (V-first); ``actual_seq_lengths`` int32 `[B+1]` whose entry 0 is a
    skipped prefix length and entries 1.. are per-sequence token counts; ``ssm_state_indices`` int32 `[T]`.
    Returns the attention output `[T,Nv,Dv]` (bf16).
    """
    op = "recurrent_gated_delta_rule"
    if g is None and gk is None:
        raise RuntimeError(f"{op}: either g or gk must be provided.")
    if gk is not None:
        raise NotImplementedError(f"{op}: gk (per-channel decay) is not supported by this operator; "
                                  "the reference documents it as not supported yet as well")
    return host().recurrent_pool(query, key, value, state, beta, scale, actual_seq_lengths, ssm_state_indices,
                                 num_accepted_tokens, g)


def recurrent_kda(q, k, v, g, beta, initial_state=None, *, cu_seqlens=None, ssm_state_indices=None, A_log=None,
                  dt_bias=None, num_accepted_tokens=None, layout="BSND", scale=None, output_final_state=False,
                  inplace_final_state=True, use_qk_l2norm_in_kernel=False, use_gate_in_kernel=False,
                  use_beta_sigmoid_in_kernel=False, allow_neg_eigval=False, safe_gate=False, lower_bound=None,
                  state_v_first=False):
    """Recurrent KDA step over a state pool, with the reference operator's argument names
    (npu_recurrent_kda, torch_custom/fla_npu/fla_npu/ops/ascendc/_aclnn_ctypes.py:1298-1503).

    BSND: q,k `[B,T,H,K]`, v `[B,T,HV,V]`, g `[B,T,HV,K]`, beta `[B,T,HV]`; TND: the same without the batch dim.
    ``initial_state`` `[state_capacity,HV,K,V]` (`[..,V,K]` with ``state_v_first``) fp32|bf16, updated in place when
    ``inplace_final_state``.  ``ssm_state_indices``: packed `[T]` (state after token t goes to block indices[t]) or
    speculative `[seq_num,max_step]` (token s of sequence n goes to block indices[n,s]); a sequence starts from the
    block of its first token, or of token ``num_accepted_tokens[n] - 1``.  Returns ``(out, final_state | None)``.
    """
    op = "recurrent_kda"
    if layout not in ("BSND", "TND"):
        raise RuntimeError(f"{op}: layout must be BSND or TND.")
    tnd = layout == "TND"
    rank = 3 if tnd else 4
    if any(x.dim() != rank for x in (q, k, v, g)) or beta.dim() != rank - 1:
        raise RuntimeError(f"{op}: layout/rank mismatch. TND expects q/k [T,H,K], v [T,HV,V], g [T,HV,K], beta [T,HV]; "
                           "BSND expects q/k [B,T,H,K], v [B,T,HV,V], g [B,T,HV,K], beta [B,T,HV].")
    if q.shape != k.shape:
        raise RuntimeError(f"{op}: q and k must have identical shape.")
    for n, t in (("q", q), ("k", k), ("v", v)):
        _activation_ok(f"{op}: {n}", t)
    if not (q.dtype == k.dtype == v.dtype):
        raise TypeError(f"{op}: q, k, v must share one dtype, got {q.dtype}, {k.dtype}, {v.dtype}")
    if tnd:
        q, k, v, g, beta = (x.unsqueeze(0) for x in (q, k, v, g, beta))
    B, T, H, K = q.shape
    HV, V = v.shape[2], v.shape[3]
    if tuple(g.shape) != (B, T, HV, K) or tuple(beta.shape) != (B, T, HV) or tuple(v.shape[:2]) != (B, T):
        raise RuntimeError(f"{op}: v/g/beta shape mismatch.")
    if HV % H:
        raise RuntimeError(f"{op}: HV must be divisible by H.")
    if g.dtype not in _GATE_TYPES or beta.dtype not in _GATE_TYPES:
        raise RuntimeError(f"{op}: g and beta must use BF16 or FP32.")
    dev = q.device
    total = B * T
    if cu_seqlens is None:
        seq_num = B
        cu = None if not tnd else torch.tensor([0, T], dtype=torch.int32, device=dev)
    else:
        if not isinstance(cu_seqlens, torch.Tensor) or cu_seqlens.dim() != 1 or cu_seqlens.numel() < 2:
            raise RuntimeError(f"{op}: cu_seqlens must be a 1D INT32 or INT64 tensor.")
        cu = cu_seqlens.to(device=dev, dtype=torch.int32)
        seq_num = cu.numel() - 1
    tail = (HV, V, K) if state_v_first else (HV, K, V)
    if initial_state is None:
        if inplace_final_state:
            raise RuntimeError(f"{op}: inplace_final_state=True requires initial_state.")
        capacity = seq_num
    else:
        if initial_state.dtype not in (torch.float32, torch.bfloat16):
            raise RuntimeError(f"{op}: initial_state must use FP32 or BF16.")
        if initial_state.dim() != 4 or tuple(initial_state.shape[1:]) != tail:
            raise RuntimeError(f"{op}: initial_state must be [state_capacity,{','.join(map(str, tail))}].")
        if inplace_final_state and initial_state.requires_grad:
            raise RuntimeError(f"{op}: initial_state is updated in place and must not require grad")
        capacity = initial_state.shape[0]
    idx = None
    if ssm_state_indices is not None:
        if ssm_state_indices.dim() == 1 and ssm_state_indices.shape[0] >= total:
            idx = ssm_state_indices[:total].to(device=dev, dtype=torch.int32).contiguous()
        elif ssm_state_indices.dim() == 2 and ssm_state_indices.shape[0] == seq_num and ssm_state_indices.shape[1] > 0:
            # speculative [seq_num, max_step]: token s of sequence n -> indices[n, s]
            bounds = cu if cu is not None else torch.arange(0, total + 1, T, dtype=torch.int32, device=dev)
            tok = torch.arange(total, device=dev)
            seq_of = torch.bucketize(tok, bounds[1:].long(), right=True).clamp_(max=seq_num - 1)
            step = (tok - bounds[:-1].long()[seq_of]).clamp_(0, ssm_state_indices.shape[1] - 1)
            idx = ssm_state_indices.to(dev)[seq_of, step].to(torch.int32).contiguous()
        else:
            raise RuntimeError(f"{op}: ssm_state_indices must be INT32/INT64 packed [T] or speculative [seq_num,max_step].")
    elif capacity != seq_num:
        raise RuntimeError(f"{op}: without ssm_state_indices, state_capacity must equal seq_num.")
    if num_accepted_tokens is not None:
        if idx is None:
            raise RuntimeError(f"{op}: num_accepted_tokens requires ssm_state_indices.")
        if tuple(num_accepted_tokens.shape) != (seq_num,):
            raise RuntimeError(f"{op}: num_accepted_tokens must be INT32/INT64 [seq_num].")
        num_accepted_tokens = num_accepted_tokens.to(device=dev, dtype=torch.int32)
    gate_mode = 0
    lower = -5.0 if lower_bound is None else float(lower_bound)
    if use_gate_in_kernel:
        if A_log is None or A_log.dtype != torch.float32 or tuple(A_log.shape) != (HV,):
            raise RuntimeError(f"{op}: A_log must be FP32 [HV] when use_gate_in_kernel=True.")
        if safe_gate and not -5.0 <= lower < 0.0:
            raise RuntimeError(f"{op}: lower_bound must be in [-5,0) when safe_gate=True.")
        if dt_bias is not None:
            if dt_bias.dtype != torch.float32 or tuple(dt_bias.shape) not in ((HV * K,), (HV, K)):
                raise RuntimeError(f"{op}: dt_bias must be FP32 [HV*K] or [HV,K].")
            dt_bias = dt_bias.reshape(HV, K).contiguous()
        gate_mode = 2 if safe_gate else 1
    elif safe_gate or A_log is not None or dt_bias is not None:
        raise RuntimeError(f"{op}: A_log, dt_bias and safe_gate require use_gate_in_kernel=True.")
    scale = K ** -0.5 if scale is None else float(scale)
    beta_mode = (2 if allow_neg_eigval else 1) if use_beta_sigmoid_in_kernel else 0
    out, state_out = host().recurrent_kda(q, k, v, g, beta, initial_state, cu, idx, A_log, dt_bias, num_accepted_tokens, scale,
                                          inplace_final_state, use_qk_l2norm_in_kernel, gate_mode, beta_mode, lower, state_v_first,
                                          seq_num)
    if tnd:
        out = out.squeeze(0)
    return out, (state_out if output_final_state else None)
