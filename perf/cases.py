"""Performance cases of the linear-attention operators: what a model that runs on this library asks of it.

Every case goes through the public operators of `fla_b200.ops`, called the way the layers of a GDN model (Qwen3-Next: 16 q/k heads,
32 value heads, depthwise conv over the 8,192 projected channels) or of a KDA model (Kimi Linear: 32 heads, a gate per key channel)
call them; head counts below the full model's are tensor-parallel shards of it.  A pass is one layer's call:

  decode_gdn    one token per sequence: conv update over the cache, then the recurrent step on the fp32 state, both in place
  decode_pool   the reference operator's step over a V-first state pool with state indices and a few draft tokens per sequence
  decode_kda    the KDA step: gate and beta activations and the q/k normalisation in the kernel, state addressed by indices
  prefill_gdn   conv (final state kept) + chunked GDN forward (final state kept), q/k normalised in the kernel; fixed or packed
  prefill_kda   chunked KDA forward with the gate activation and the q/k normalisation in the kernel; fixed or packed
  train_gdn     chunked GDN forward and backward through autograd, alone or with the conv and the normalisation of the layer
  train_kda     chunked KDA forward and backward through autograd

Packed batches come with `cu_seqlens` as an int32 tensor on the device, the form in which the layers hand it on.
"""
import math
import os
import random
import sys

import torch
import torch.nn.functional as F

# the package lives in a folder of the working tree that is not itself importable by name
sys.path.insert(0, os.path.join(os.getcwd(), "flash-linear-attention-npu_b200"))

from fla_b200 import ops  # noqa: E402

D = 128           # head dim of q, k and v in every model served
W = 4             # conv width
CHUNK = 64        # tokens per chunk of the chunked form (the flop counts below)
MOST_TOKENS = 8 * 4096   # of a pass, at full head count


def listed():
    return [
        # a single user's chat turn: one sequence generating, nothing but launches and latency
        dict(name="decode_gdn_one", kind="decode_gdn", n=1, hk=16, hv=32),
        # a full serving batch (256 concurrent sequences, 0.5 GB of state)
        dict(name="decode_gdn_256", kind="decode_gdn", n=256, hk=16, hv=32),
        # speculative decoding on a 2-way shard: 1 to 4 draft tokens per sequence, every token's state kept in a bf16 pool
        dict(name="decode_pool_draft", kind="decode_pool", n=24, hk=8, hv=16, draft=4, state="bf16"),
        # a half-full KDA serving batch
        dict(name="decode_kda_45", kind="decode_kda", n=45, hk=32, hv=32),
        # the prompt of a short question, alone
        dict(name="prefill_gdn_short", kind="prefill_gdn", b=1, t=100, packed=0, hk=16, hv=32, conv=True, norm=True, h0=False, dtype="bf16"),
        # one long document: few independent chains, each 256 chunks long
        dict(name="prefill_gdn_long", kind="prefill_gdn", b=1, t=16384, packed=0, hk=16, hv=32, conv=True, norm=True, h0=False, dtype="bf16"),
        # continuous batching: 22 prompts of very different lengths packed together
        dict(name="prefill_gdn_packed", kind="prefill_gdn", b=1, t=11003, packed=22, hk=16, hv=32, conv=True, norm=True, h0=True, dtype="bf16"),
        # a large offline batch (inputs normalised by the caller, states carried in)
        dict(name="prefill_gdn_batch", kind="prefill_gdn", b=8, t=4096, packed=0, hk=16, hv=32, conv=True, norm=False, h0=True, dtype="bf16"),
        # the training step on a large fixed-length batch, the operator alone
        dict(name="train_gdn_batch", kind="train_gdn", b=8, t=4096, packed=0, hk=16, hv=32, conv=False, norm=False, h0=True),
        # the layer of a 4-way sharded model on packed documents: conv, normalisation, delta rule and all their gradients
        dict(name="train_gdn_layer_packed", kind="train_gdn", b=1, t=8191, packed=7, hk=4, hv=8, conv=True, norm=True, h0=False),
        # one long KDA prompt
        dict(name="prefill_kda_long", kind="prefill_kda", b=1, t=8192, packed=0, hk=32, hv=32, h0=False, dtype="bf16"),
        # the KDA training step on a large batch, intermediates kept for the backward
        dict(name="train_kda_batch", kind="train_kda", b=4, t=8192, packed=0, hk=32, hv=32, keep=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _tokens(rng, least, most=MOST_TOKENS):
    """(b, t, packed): a batch of equal lengths, one sequence, or a packed batch, of `least` to `most` tokens."""
    total = _log(rng, least, most)
    form = rng.choice(("one", "batch", "packed"))
    if form == "batch":
        b = min(_log(rng, 2, 16), max(1, total // 16))
        return b, max(1, total // b), 0
    if form == "packed":
        return 1, total, max(1, min(_log(rng, 2, 48), total // 8))
    return 1, min(total, 16384), 0


def draw(rng):
    kind = rng.choice(("decode_gdn", "decode_pool", "decode_kda", "prefill_gdn", "prefill_gdn", "prefill_kda", "train_gdn", "train_kda"))
    hk, hv = rng.choice(((2, 4), (4, 8), (8, 16), (16, 32)))
    if kind.endswith("kda"):
        hk = hv
    if kind == "decode_gdn":
        return dict(kind=kind, n=_log(rng, 1, 256), hk=hk, hv=hv)
    if kind == "decode_pool":
        return dict(kind=kind, n=_log(rng, 1, 96), hk=hk, hv=hv, draft=rng.randint(1, 4), state=rng.choice(("bf16", "f32")))
    if kind == "decode_kda":
        return dict(kind=kind, n=_log(rng, 1, 256), hk=hk, hv=hv)
    if kind == "prefill_gdn":
        b, t, packed = _tokens(rng, 16)
        dtype = rng.choice(("bf16", "bf16", "bf16", "f16"))     # the conv takes bf16 only: an fp16 caller runs its own
        return dict(kind=kind, b=b, t=t, packed=packed, hk=hk, hv=hv, conv=dtype == "bf16", norm=rng.random() < 0.75,
                    h0=rng.random() < 0.5, dtype=dtype)
    if kind == "prefill_kda":
        b, t, packed = _tokens(rng, 16)
        return dict(kind=kind, b=b, t=t, packed=packed, hk=hk, hv=hv, h0=rng.random() < 0.5, dtype=rng.choice(("bf16", "bf16", "f16")))
    if kind == "train_gdn":
        b, t, packed = _tokens(rng, 256)
        layer = rng.random() < 0.5
        return dict(kind=kind, b=b, t=t, packed=packed, hk=hk, hv=hv, conv=layer, norm=layer, h0=rng.random() < 0.5)
    b, t, packed = _tokens(rng, 256, MOST_TOKENS * 3 // 4)   # a pass that recomputes (keep=False) costs more than one that keeps
    return dict(kind=kind, b=b, t=t, packed=packed, hk=hk, hv=hv, keep=rng.random() < 0.5)


def _lengths(total, parts, rng):
    """`parts` ragged lengths that sum to `total`, spread like prompt lengths (a few long ones, many short ones)."""
    w = [math.exp(rng.gauss(0.0, 1.0)) for _ in range(parts)]
    s = sum(w)
    lens = [max(1, int(total * x / s)) for x in w]
    while sum(lens) > total:
        lens[lens.index(max(lens))] -= 1
    lens[0] += total - sum(lens)
    return lens


class _Maker:
    """Seeded device tensors."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def n(self, *shape, dtype=torch.bfloat16, scale=1.0):
        return (torch.randn(*shape, generator=self.g, device="cuda") * scale).to(dtype)

    def unit(self, *shape, dtype=torch.bfloat16):
        return F.normalize(torch.randn(*shape, generator=self.g, device="cuda"), dim=-1).to(dtype)

    def beta(self, *shape):
        return torch.sigmoid(torch.randn(*shape, generator=self.g, device="cuda")).to(torch.bfloat16)

    def decay(self, *shape):
        """Log decay of a GDN head: fp32, as the layer computes it from its projections."""
        return F.logsigmoid(torch.randn(*shape, generator=self.g, device="cuda"))

    def gate(self, *shape):
        """A KDA layer's raw gate and its A_log (1 to 16) and dt_bias (time steps of 0.001 to 0.1), as such layers initialise them."""
        hv, k = shape[-2:]
        a_log = torch.log(torch.rand(hv, generator=self.g, device="cuda") * 15.0 + 1.0)
        step = torch.exp(torch.rand(hv, k, generator=self.g, device="cuda") * math.log(100.0) + math.log(0.001))
        return dict(g=self.n(*shape, scale=0.5), a_log=a_log, dt_bias=step + torch.log(-torch.expm1(-step)))


def prepare(case, seed):
    c, m = dict(case), _Maker(seed)
    kind, hk, hv = c["kind"], c["hk"], c["hv"]
    host = random.Random(int(seed))
    dc = (2 * hk + hv) * D
    s = {"case": c}
    if kind == "decode_gdn":
        n = c["n"]
        s.update(x=m.n(n, dc), conv_state=m.n(n, dc, W - 1), weight=m.n(dc, W, scale=0.5), g=m.decay(n, 1, hv), beta=m.beta(n, 1, hv),
                 state=m.n(n, hv, D, D, dtype=torch.float32, scale=0.1))
        return s
    if kind == "decode_pool":
        lens = [1 + i % c["draft"] for i in range(c["n"])]
        host.shuffle(lens)
        t = sum(lens)
        slots = list(range(t + 8))
        host.shuffle(slots)
        dt = torch.bfloat16 if c["state"] == "bf16" else torch.float32
        s.update(q=m.unit(t, hk, D), k=m.unit(t, hk, D), v=m.n(t, hv, D), g=m.decay(t, hv), beta=m.beta(t, hv),
                 state=m.n(t + 8, hv, D, D, dtype=dt, scale=0.1),
                 lengths=torch.tensor([0] + lens, dtype=torch.int32, device="cuda"),
                 indices=torch.tensor(slots[:t], dtype=torch.int32, device="cuda"))
        return s
    if kind == "decode_kda":
        n = c["n"]
        slots = list(range(n + 3))
        host.shuffle(slots)
        s.update(q=m.n(n, 1, hk, D), k=m.n(n, 1, hk, D), v=m.n(n, 1, hv, D), beta=m.n(n, 1, hv),
                 state=m.n(n + 3, hv, D, D, dtype=torch.float32, scale=0.1), **m.gate(n, 1, hv, D),
                 indices=torch.tensor(slots[:n], dtype=torch.int32, device="cuda"))
        return s
    b, t = c["b"], c["t"]
    seqs = c["packed"] or b
    cu = None
    if c["packed"]:
        ends = [0]
        for x in _lengths(t, c["packed"], host):
            ends.append(ends[-1] + x)
        cu = torch.tensor(ends, dtype=torch.int32, device="cuda")
    s["cu"] = cu
    s["h0"] = m.n(seqs, hv, D, D, dtype=torch.float32, scale=0.1) if c.get("h0") else None
    dt = torch.float16 if c.get("dtype") == "f16" else torch.bfloat16
    if kind.endswith("kda"):
        if kind == "prefill_kda":       # q, k, the gate and beta as they leave the projections
            s.update(q=m.n(b, t, hk, D, dtype=dt), k=m.n(b, t, hk, D, dtype=dt), v=m.n(b, t, hv, D, dtype=dt),
                     beta=m.beta(b, t, hv), **m.gate(b, t, hv, D))
            return s
        s.update(q=m.unit(b, t, hk, D), k=m.unit(b, t, hk, D), v=m.n(b, t, hv, D),
                 g=(F.logsigmoid(m.n(b, t, hv, D, dtype=torch.float32)) / 16).to(torch.bfloat16), beta=m.beta(b, t, hv),
                 do=m.n(b, t, hv, D))
        s["wrt"] = [s[n].requires_grad_() for n in ("q", "k", "v", "g", "beta")]
        return s
    s.update(g=m.decay(b, t, hv), beta=m.beta(b, t, hv))
    if c["conv"]:
        s.update(x=m.n(b, t, dc), weight=m.n(dc, W, scale=0.5))
    if not c["conv"] or not c["norm"]:
        s.update(q=m.unit(b, t, hk, D, dtype=dt), k=m.unit(b, t, hk, D, dtype=dt))
    if not c["conv"]:
        s.update(v=m.n(b, t, hv, D, dtype=dt))
    if kind == "train_gdn":
        s.update(do=m.n(b, t, hv, D), dht=m.n(seqs, hv, D, D, dtype=torch.float32, scale=0.1))
        names = ("x", "weight") if c["conv"] else ("q", "k", "v")
        s["wrt"] = [s[n].requires_grad_() for n in names + ("g", "beta") + (("h0",) if c["h0"] else ())]
    return s


def _split(mixed, hk, hv):
    """q, k, v as views of the conv output."""
    q = mixed[..., : hk * D].unflatten(-1, (hk, D))
    k = mixed[..., hk * D: 2 * hk * D].unflatten(-1, (hk, D))
    v = mixed[..., 2 * hk * D:].unflatten(-1, (hv, D))
    return q, k, v


def run(s):
    c = s["case"]
    kind, hk, hv = c["kind"], c["hk"], c["hv"]
    if kind.startswith("train"):
        if kind == "train_kda":
            o, _ = ops.chunk_kda(s["q"], s["k"], s["v"], s["g"], s["beta"], cu_seqlens=s["cu"], disable_recompute=c["keep"])
            return [o.detach(), *torch.autograd.grad([o], s["wrt"], [s["do"]])]
        if c["conv"]:
            mixed, _ = ops.causal_conv1d(s["x"], s["weight"], activation="silu", cu_seqlens=s["cu"])
            q, k, v = _split(mixed, hk, hv)
        else:
            q, k, v = s["q"], s["k"], s["v"]
        o, ht = ops.chunk_gated_delta_rule(q, k, v, s["g"], s["beta"], initial_state=s["h0"], output_final_state=True,
                                           use_qk_l2norm_in_kernel=c["norm"], cu_seqlens=s["cu"])
        return [o.detach(), ht.detach(), *torch.autograd.grad([o, ht], s["wrt"], [s["do"], s["dht"]])]
    with torch.no_grad():
        if kind == "decode_gdn":
            mixed = ops.causal_conv1d_update(s["x"], s["conv_state"], weight=s["weight"], activation="silu")
            q, k, v = _split(mixed.unsqueeze(1), hk, hv)
            o, state = ops.fused_recurrent_gated_delta_rule(q, k, v, g=s["g"], beta=s["beta"], initial_state=s["state"],
                                                            use_qk_l2norm_in_kernel=True, inplace_final_state=True)
            return [o, state, s["conv_state"]]
        if kind == "decode_pool":
            o = ops.recurrent_gated_delta_rule(s["q"], s["k"], s["v"], s["state"], beta=s["beta"], scale=D ** -0.5,
                                               actual_seq_lengths=s["lengths"], ssm_state_indices=s["indices"], g=s["g"])
            return [o, s["state"]]
        if kind == "decode_kda":
            o, state = ops.recurrent_kda(s["q"], s["k"], s["v"], s["g"], s["beta"], s["state"], ssm_state_indices=s["indices"],
                                         A_log=s["a_log"], dt_bias=s["dt_bias"], output_final_state=True, use_qk_l2norm_in_kernel=True,
                                         use_gate_in_kernel=True, use_beta_sigmoid_in_kernel=True)
            return [o, state]
        if kind == "prefill_kda":
            o, ht = ops.chunk_kda(s["q"], s["k"], s["v"], s["g"], s["beta"], initial_state=s["h0"], output_final_state=True,
                                  use_qk_l2norm_in_kernel=True, use_gate_in_kernel=True, A_log=s["a_log"], dt_bias=s["dt_bias"],
                                  cu_seqlens=s["cu"])
            return [o, ht]
        out = []
        if c["conv"]:
            mixed, conv_state = ops.causal_conv1d(s["x"], s["weight"], activation="silu", output_final_state=True, cu_seqlens=s["cu"])
            out.append(conv_state)
            q, k, v = _split(mixed, hk, hv)
            if not c["norm"]:           # q, k normalised by the caller before the operator
                out.append(mixed[..., : 2 * hk * D])
                q, k = s["q"], s["k"]
        else:
            q, k, v = s["q"], s["k"], s["v"]
        o, ht = ops.chunk_gated_delta_rule(q, k, v, s["g"], s["beta"], initial_state=s["h0"], output_final_state=True,
                                           use_qk_l2norm_in_kernel=c["norm"], cu_seqlens=s["cu"])
        return [o, ht, *out]


def work(case):
    """Bytes: inputs once, outputs once.  Flops: the chunked form with triangular score blocks counted once (chunks of 64)."""
    c = case
    kind, hk, hv = c["kind"], c["hk"], c["hv"]
    dc = (2 * hk + hv) * D
    if kind.startswith("decode"):
        n = c["n"]
        tok = n if kind != "decode_pool" else sum(1 + i % c["draft"] for i in range(n))
        es = 2 if c.get("state") == "bf16" else 4
        # the state of each sequence read once and, for drafts, written once per token
        bts = (n + tok) * hv * D * D * es + tok * (2 * hk + 2 * hv) * D * 2
        bts += tok * hv * D * 2 + hv * D * 4 if kind == "decode_kda" else tok * hv * 6
        if kind == "decode_gdn":
            bts += n * dc * (W - 1) * 2 * 2 + n * dc * 2 + dc * W * 2
        return {"bytes": bts, "flops": tok * hv * D * D * 7 + (tok * dc * 2 * W if kind == "decode_gdn" else 0)}
    b, t = c["b"], c["t"]
    seqs, tok = c["packed"] or b, b * t
    th = tok * hv
    state = seqs * hv * D * D * 4
    qk, v = tok * hk * D * 2, th * D * 2
    fwd = th * (6 * D * D + 2 * CHUNK * D) + tok * hk * 2 * CHUNK * D + th * CHUNK * CHUNK // 3
    bwd = th * (12 * D * D + 5 * CHUNK * D) + tok * hk * 4 * CHUNK * D
    if kind == "prefill_kda":
        return {"bytes": 2 * qk + 2 * v + th * D * 2 + th * 2 + state * (2 if c["h0"] else 1), "flops": fwd}
    if kind == "train_kda":   # forward: q k v g beta in, o out; backward: dO in, the gradients out
        return {"bytes": 2 * (2 * qk + v + th * D * 2 + th * 2) + 2 * v, "flops": fwd + bwd}
    gates = th * 6
    conv = tok * dc * 2 if c["conv"] else 0
    if kind == "prefill_gdn":
        if c["conv"]:         # x in, o and the conv state out; q and k of the conv are only an output when the caller normalises
            bts = conv + v + gates + (0 if c["norm"] else 4 * qk) + seqs * dc * (W - 1) * 2
        else:
            bts = 2 * qk + 2 * v + gates
        return {"bytes": bts + state * (2 if c["h0"] else 1), "flops": fwd + (tok * dc * 2 * W if c["conv"] else 0)}
    io = conv if c["conv"] else 2 * qk + v
    bts = 2 * (io + gates) + 2 * v + state * (2 + (2 if c["h0"] else 0))
    return {"bytes": bts, "flops": fwd + bwd + (tok * dc * 6 * W if c["conv"] else 0)}


def tolerance(case):
    """fp32 states next to bf16 outputs in decoding (the rounding of the bf16 tensors decides); bf16 operands everywhere else."""
    if case["kind"] in ("decode_gdn", "decode_kda") or case.get("state") == "f32":
        return {"rel": 5e-3}
    return {"rel": 1e-2}
