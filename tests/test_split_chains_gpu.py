"""Chains split into segments over several SMs (few sequences and heads): equal, within the precision of the fp32 outputs, to the same
sequences inside a batch that is large enough not to be split."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(T, HK, HV, N, V=128, seed=0):
    g_ = torch.Generator(device="cuda").manual_seed(seed + T)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g_)   # noqa: E731
    unit = lambda *s: torch.nn.functional.normalize(rn(*s), dim=-1).bfloat16()   # noqa: E731
    return dict(q=unit(1, T, HK, 128), k=unit(1, T, HK, 128), v=rn(1, T, HV, V).bfloat16(),
                g=torch.nn.functional.logsigmoid(rn(1, T, HV) + 3), beta=torch.sigmoid(rn(1, T, HV)).bfloat16(),
                h0=0.1 * rn(N, HV, 128, V), do=rn(1, T, HV, V).bfloat16(), dht=0.1 * rn(N, HV, 128, V))


def _close(name, a, b, tol):
    a, b = a.double(), b.double()
    err = (a - b).abs().max() / b.pow(2).mean().sqrt()
    assert torch.isfinite(a).all() and err <= tol, f"{name}: {err:.2e}"


@pytest.mark.parametrize("T,HK,HV,V", [(1024, 1, 1, 128), (1111, 2, 4, 128), (4097, 2, 2, 128), (2300, 1, 2, 256)])
def test_gdn_split_forward_and_backward(T, HK, HV, V):
    from fla_b200.ops import chunk_gated_delta_rule_fwd_bwd
    d = _inputs(T, HK, HV, 1, V)

    def run(copies):
        x = {n: t.expand(copies, *t.shape[1:]).contiguous() for n, t in d.items()}
        o, ht, gr = chunk_gated_delta_rule_fwd_bwd(x["q"], x["k"], x["v"], x["g"], x["beta"], x["do"], initial_state=x["h0"], dht=x["dht"],
                                                   output_dtype=torch.float32, grad_dtype=torch.float32)
        return [t[:1] for t in (o, ht, *gr)]
    for n, a, b in zip(("o", "ht", "dq", "dk", "dv", "dg", "dbeta", "dh0"), run(1), run(-(-160 // HV))):
        _close(n, a, b, 2e-3)


@pytest.mark.parametrize("lens,HV", [([1500, 64, 0, 700, 5], 2), ([40, 2049], 4)])
def test_gdn_split_packed(lens, HV):
    from fla_b200.ops import chunk_gated_delta_rule, chunk_gated_delta_rule_fwd_bwd
    T = sum(lens)
    d = _inputs(T, HV, HV, len(lens))
    ends = [0]
    for x in lens:
        ends.append(ends[-1] + x)

    def run(copies):
        x = {n: t.repeat((1, copies) + (1,) * (t.dim() - 2)) if n not in ("h0", "dht") else t.repeat(copies, 1, 1, 1) for n, t in d.items()}
        cu = torch.tensor([0] + [c * T + e for c in range(copies) for e in ends[1:]], dtype=torch.int32, device="cuda")
        o, ht, gr = chunk_gated_delta_rule_fwd_bwd(x["q"], x["k"], x["v"], x["g"], x["beta"], x["do"], initial_state=x["h0"], dht=x["dht"],
                                                   cu_seqlens=cu, output_dtype=torch.float32, grad_dtype=torch.float32)
        o2, ht2 = chunk_gated_delta_rule(x["q"], x["k"], x["v"], x["g"], x["beta"], initial_state=x["h0"], output_final_state=True,
                                         cu_seqlens=cu, output_dtype=torch.float32)
        return [o[:, :T], ht[:len(lens)], *(t[:, :T] for t in gr[:5]), gr[5][:len(lens)], o2[:, :T], ht2[:len(lens)]]
    names = ("o", "ht", "dq", "dk", "dv", "dg", "dbeta", "dh0", "inference o", "inference ht")
    for n, a, b in zip(names, run(1), run(-(-160 // HV))):
        _close(n, a, b, 2e-3)


@pytest.mark.parametrize("keep", [False, True])
@pytest.mark.parametrize("T,HV,V", [(1024, 1, 128), (1111, 3, 128), (2300, 2, 256)])
def test_kda_split_forward_and_backward(T, HV, V, keep):
    from fla_b200.ops import chunk_kda, chunk_kda_fwd_bwd
    d = _inputs(T, HV, HV, 1, V)
    d["g"] = (-torch.rand(1, T, HV, 128, generator=torch.Generator(device="cuda").manual_seed(T), device="cuda") / 16).bfloat16()

    def run(copies):
        x = {n: t.expand(copies, *t.shape[1:]).contiguous() for n, t in d.items()}
        o, ht, gr = chunk_kda_fwd_bwd(x["q"], x["k"], x["v"], x["g"], x["beta"], x["do"], initial_state=x["h0"], dht=x["dht"],
                                      output_dtype=torch.float32, disable_recompute=keep)
        o2, ht2 = chunk_kda(x["q"], x["k"], x["v"], x["g"], x["beta"], initial_state=x["h0"], output_final_state=True, output_dtype=torch.float32)
        return [t[:1] for t in (o, ht, *gr, o2, ht2)]
    names = ("o", "ht", "dq", "dk", "dv", "dg", "dbeta", "dh0", "inference o", "inference ht")
    for n, a, b in zip(names, run(1), run(-(-160 // HV))):
        _close(n, a, b, 2e-3)
