"""Bookkeeping of packed batches on the device: chunk offsets made from the boundaries, and the state-pool step's offsets made
from its lengths, at batch sizes around the 32 sequences a warp handles at a time."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 70])
def test_chunk_offsets(n):
    from fla_b200 import host
    lens = [(i * 37) % 150 for i in range(n)]
    lens[0] = 65
    cu = [0]
    for x in lens:
        cu.append(cu[-1] + x)
    on = torch.empty(1, device="cuda")
    for form in (cu, torch.tensor(cu, device="cuda"), torch.tensor(cu, dtype=torch.int32, device="cuda")):
        cu_d, co, N, max_len, chunks = host().geometry(1, cu[-1], form, on)
        want = [0]
        for x in lens:
            want.append(want[-1] + (x + 63) // 64)
        assert cu_d.tolist() == cu and co.tolist() == want
        assert (N, max_len, chunks) == (n, max(lens), want[-1])


@pytest.mark.parametrize("n,prefix", [(1, 0), (32, 2), (33, 0), (70, 1)])
def test_pool_step_adds_up_its_lengths(n, prefix):
    from fla_b200.ops import fused_recurrent_gated_delta_rule, recurrent_gated_delta_rule
    lens = [1 + i % 3 for i in range(n)]
    T = prefix + sum(lens)
    g_ = torch.Generator(device="cuda").manual_seed(n)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g_)   # noqa: E731
    q, k = (torch.nn.functional.normalize(rn(T, 1, 128), dim=-1).bfloat16() for _ in range(2))
    v, g, beta = rn(T, 2, 128).bfloat16(), -rn(T, 2).abs(), torch.sigmoid(rn(T, 2)).bfloat16()
    first = [prefix]
    for x in lens:
        first.append(first[-1] + x)
    idx = torch.arange(T, dtype=torch.int32, device="cuda")
    pool = rn(T, 2, 128, 128)
    start = pool[first[:-1]].clone()
    o = recurrent_gated_delta_rule(q, k, v, pool, beta=beta, scale=0.5, g=g, ssm_state_indices=idx,
                                   actual_seq_lengths=torch.tensor([prefix] + lens, dtype=torch.int32, device="cuda"))
    live = slice(prefix, T)
    cu = torch.tensor([x - prefix for x in first], device="cuda")
    o2, s2 = fused_recurrent_gated_delta_rule(*(x[live].unsqueeze(0) for x in (q, k, v, g, beta)), scale=0.5, initial_state=start,
                                              output_final_state=True, cu_seqlens=cu, transpose_state_layout=True)
    assert torch.equal(o[live], o2[0])
    assert torch.equal(pool[[x - 1 for x in first[1:]]], s2)
