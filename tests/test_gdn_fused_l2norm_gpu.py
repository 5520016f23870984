"""chunk_gated_delta_rule(use_qk_l2norm_in_kernel=True) normalises inside its own kernels, forward and backward: equal to the l2norm
kernels run in front of and behind the operator, at lengths around the 64-token tile, with grouped heads and strided q, k."""
import pytest
import torch

from tests._util import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,HK,HV", [(1, 1, 2), (63, 2, 2), (65, 1, 4), (200, 2, 4)])
def test_fused_normalisation_matches_separate_passes(T, HK, HV):
    from fla_b200.ops import chunk_gated_delta_rule, l2norm_bwd, l2norm_fwd
    g_ = torch.Generator(device="cuda").manual_seed(T)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g_)   # noqa: E731
    mixed = rn(2, T, 2 * HK * 128).bfloat16()
    v, g, beta = rn(2, T, HV, 128).bfloat16(), -rn(2, T, HV).abs(), torch.sigmoid(rn(2, T, HV)).bfloat16()
    do = rn(2, T, HV, 128).bfloat16()

    def leaves(*ts):
        return [t.detach().clone().requires_grad_() for t in ts]
    m, v1, g1, b1 = leaves(mixed, v, g, beta)
    q1, k1 = (x.unflatten(-1, (HK, 128)) for x in m.chunk(2, dim=-1))
    o1, _ = chunk_gated_delta_rule(q1, k1, v1, g1, b1, use_qk_l2norm_in_kernel=True)
    got = torch.autograd.grad(o1, [m, v1, g1, b1], do)

    qn, qr = l2norm_fwd(q1.detach().contiguous())
    kn, kr = l2norm_fwd(k1.detach().contiguous())
    q2, k2, v2, g2, b2 = leaves(qn, kn, v, g, beta)
    o2, _ = chunk_gated_delta_rule(q2, k2, v2, g2, b2)
    dq, dk, dv, dg, db = torch.autograd.grad(o2, [q2, k2, v2, g2, b2], do)
    assert torch.equal(o1, o2) and torch.equal(got[1], dv)
    want = torch.cat([l2norm_bwd(n, r, d).flatten(-2) for n, r, d in ((qn, qr, dq), (kn, kr, dk))], dim=-1)
    # bf16 results, and the separate pass also rounds dq, dk to bf16 in between: some ulps at single elements, little over all
    assert_close("d(q, k)", got[0], want, 8e-2)
    assert (got[0].float() - want.float()).norm() <= 5e-3 * want.float().norm()
    assert_close("dg", got[2], dg, 1e-5)
    assert_close("dbeta", got[3].float(), db.float(), 1e-5)
