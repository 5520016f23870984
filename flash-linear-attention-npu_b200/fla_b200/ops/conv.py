"""causal_conv1d forward / decode update.

`causal_conv1d` and `causal_conv1d_update` use the `[B,T,D]` surface the reference's composed entry
exposes (examples/flash_gated_delta_rule.py:422-443: x, weight `[D,W]`, bias, residual, initial_state,
activation, cu_seqlens, output_final_state).  States are `[N,D,W-1]` (the last W-1 inputs);
`npu_causal_conv1d` below keeps the reference low-level operator's signature and its
`[W,D]` weight / `[N,W-1,D]` state layouts (…/ops/ascendc/_aclnn_ctypes.py:951-985).
"""
from __future__ import annotations

import torch

from .. import host


def _act(activation) -> int:
    if activation in (None, 0, False):
        return 0
    if activation in ("silu", "swish", 1, True):
        return 1
    raise NotImplementedError(f"activation must be None, 'silu' or 'swish', got {activation!r}")


def causal_conv1d_bwd(x, weight, dy, bias=None, initial_state=None, dht=None, activation=None, cu_seqlens=None,
                      y_pre=None, need_dh0=None):
    """Gradients of :func:`causal_conv1d` (layouts as there).  Returns ``(dx, dw [D,W] f32, db [D] f32, dh0 | None)``.
    The pre-activation is recomputed from x (and bias) unless ``y_pre`` holds it."""
    want_dh0 = (initial_state is not None) if need_dh0 is None else need_dh0
    return host().conv_bwd(x, weight, dy, bias, initial_state, dht, _act(activation), cu_seqlens, y_pre, want_dh0)


def causal_conv1d(x, weight=None, bias=None, residual=None, initial_state=None, output_final_state=False,
                  activation=None, cu_seqlens=None):
    """x `[B,T,D]` bf16; weight `[D,W]`; initial_state / final_state `[N,D,W-1]`.
    Returns ``(y [B,T,D], final_state | None)``; differentiable in x, weight, bias, residual and initial_state (the reference
    wires its operator the same way, examples/flash_gated_delta_rule.py:323-419): the inputs are saved, the backward
    recomputes the pre-activation."""
    if weight is None:
        raise RuntimeError("causal_conv1d: weight is required")
    return host().conv(x, weight, bias, residual, initial_state, output_final_state, _act(activation), cu_seqlens)


def causal_conv1d_update(x, cache, residual=None, weight=None, bias=None, activation=None, cache_indices=None,
                         num_accepted_tokens=None, pad_slot_id=-1):
    """Decode step.  x `[N,D]` or `[N,T,D]`; cache `[slots,D,S]` (S >= W-1), updated in place.
    Returns y with the shape of x."""
    if weight is None:
        raise RuntimeError("causal_conv1d_update: weight is required")
    return host().conv_update(x, cache, residual, weight, bias, _act(activation), cache_indices, num_accepted_tokens, pad_slot_id)


def npu_causal_conv1d(x, weight, bias=None, conv_states=None, *, query_start_loc=None, cache_indices=None,
                      initial_state_mode=None, num_accepted_tokens=None, activation_mode=0, pad_slot_id=-1,
                      run_mode=0, head_num=0):
    """Reference low-level signature.  x `[B,T,D]` / `[T,D]` (varlen with query_start_loc) for run_mode 0,
    `[N,D]` / `[N,T,D]` for run_mode 1; weight `[W,D]`; conv_states `[slots,S,D]` updated in place.
    `head_num` > 0 (prefill only, …/_aclnn_ctypes.py:939-948): the output is `[B, head_num, T, D // head_num]`."""
    op = "npu_causal_conv1d"
    head_num = int(head_num)
    if head_num and int(run_mode) == 1:
        head_num = 0    # the reference re-lays the output only in prefill mode (_infer_causal_conv1d_y)
    w_dw = weight.transpose(0, 1)                                   # [D,W] view of the [W,D] tensor
    st = None if conv_states is None else conv_states.transpose(1, 2)  # [slots,D,S] view
    dev = x.device

    def as_i32(v):
        if v is None:
            return None
        return v.to(device=dev, dtype=torch.int32) if isinstance(v, torch.Tensor) else torch.tensor(
            list(v), dtype=torch.int32, device=dev)

    if int(run_mode) == 1:
        return causal_conv1d_update(x, st, weight=w_dw, bias=bias, activation=int(activation_mode),
                                    cache_indices=as_i32(cache_indices),
                                    num_accepted_tokens=as_i32(num_accepted_tokens), pad_slot_id=pad_slot_id)
    W = weight.shape[0]
    varlen = x.dim() == 2
    x3 = x.unsqueeze(0) if varlen else x
    cu = as_i32(query_start_loc) if varlen else None
    N = (cu.numel() - 1) if varlen else x3.shape[0]
    init = None
    idx = as_i32(cache_indices)
    if st is not None:
        if conv_states.requires_grad:
            raise RuntimeError(f"{op}: conv_states is updated in place and must not require grad")
        if st.shape[2] != W - 1:
            raise RuntimeError(f"{op}: prefill expects conv_states with state_len == W-1")
        if initial_state_mode is not None:
            sel = st if idx is None else st[idx.long()]
            mode = as_i32(initial_state_mode).bool()
            init = torch.where(mode[:, None, None], sel, torch.zeros_like(sel))
    if head_num:   # prefill output as [B, head_num, T, D / head_num] ([head_num, T, D / head_num] for packed input)
        y, final = host().conv_fwd(x3, w_dw, bias, None, init, st is not None, _act(int(activation_mode)), cu, head_num)
    else:
        y, final = causal_conv1d(x3, w_dw, bias, None, init, st is not None, int(activation_mode), cu)
    if st is not None:
        if idx is None:
            st[:N].copy_(final)
        else:
            keep = idx != pad_slot_id
            st[idx[keep].long()] = final[keep]
        torch.autograd.graph.increment_version(conv_states)
    return y.squeeze(0) if varlen else y   # packed input with head_num: [head_num, T, D / head_num]


def npu_causal_conv1d_bwd(x, y, weight, dy, initial_state=None, dht=None, *, query_start_loc=None, activation=0,
                          input_layout="BSND"):
    """Reference low-level signature (…/ops/ascendc/_aclnn_ctypes.py:988-1037): x, dy `[B,T,D]` (or `[T,D]` with
    ``query_start_loc``), y the forward's pre-activation, weight `[W,D]`, initial_state / dht `[B,W,D]` whose rows
    1..W-1 hold the W-1 stored inputs.  Returns ``(dx, dw [W,D], db [D], dh0 [B,W,D])`` in the dtype of x."""
    op = "npu_causal_conv1d_bwd"
    if input_layout not in ("BSND", "NTD", "TND"):
        raise NotImplementedError(f"{op}: input_layout {input_layout!r} is not provided")
    varlen = x.dim() == 2
    if varlen and query_start_loc is None:
        raise RuntimeError(f"{op}: query_start_loc is required for {input_layout} input.")
    W, D = weight.shape
    x3, dy3 = (t.unsqueeze(0) if varlen else t for t in (x, dy))
    y3 = None if y is None else (y.unsqueeze(0) if varlen else y)
    cu = None
    if varlen:
        cu = query_start_loc if isinstance(query_start_loc, torch.Tensor) else torch.tensor(list(query_start_loc))
        cu = cu.to(device=x.device, dtype=torch.int32)
    to_mine = lambda s: None if s is None else s[:, 1:, :].transpose(1, 2)   # noqa: E731  [B,W,D] -> [B,D,W-1] view
    dx, dw, db, dh0 = causal_conv1d_bwd(x3, weight.transpose(0, 1), dy3, None, to_mine(initial_state), to_mine(dht),
                                        int(activation), cu, y_pre=y3 if int(activation) else None, need_dh0=True)
    N = dh0.shape[0]
    dh0_ref = torch.zeros((N, W, D), dtype=x.dtype, device=x.device)
    if initial_state is not None:
        dh0_ref[:, 1:, :] = dh0.transpose(1, 2).to(x.dtype)
    return (dx.squeeze(0) if varlen else dx), dw.transpose(0, 1).to(x.dtype), db.to(x.dtype), dh0_ref
