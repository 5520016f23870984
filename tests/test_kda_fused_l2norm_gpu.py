"""chunk_kda(use_qk_l2norm_in_kernel=True) normalises inside its prep kernel, and its backward goes through the normalisation in the
chunk-parallel kernel: equal to the l2norm kernels run in front of and behind the operator, at lengths around the 64-token tile."""
import pytest
import torch

from tests._util import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("keep", [False, True])
@pytest.mark.parametrize("T,HK,HV", [(1, 1, 1), (63, 2, 2), (65, 1, 2), (200, 2, 4)])
def test_fused_normalisation_matches_separate_passes(T, HK, HV, keep):
    from fla_b200.ops import chunk_kda, l2norm_bwd, l2norm_fwd
    g_ = torch.Generator(device="cuda").manual_seed(T)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g_)   # noqa: E731
    mixed = rn(2, T, 2 * HK * 128).bfloat16()
    v, g = rn(2, T, HV, 128).bfloat16(), (-rn(2, T, HV, 128).abs() / 16).bfloat16()
    beta, do = torch.sigmoid(rn(2, T, HV)).bfloat16(), rn(2, T, HV, 128).bfloat16()

    def leaves(*ts):
        return [t.detach().clone().requires_grad_() for t in ts]
    m, v1, g1, b1 = leaves(mixed, v, g, beta)
    q1, k1 = (x.unflatten(-1, (HK, 128)) for x in m.chunk(2, dim=-1))
    o1, _ = chunk_kda(q1, k1, v1, g1, b1, use_qk_l2norm_in_kernel=True, disable_recompute=keep)
    got = torch.autograd.grad(o1, [m, v1, g1, b1], do)

    qn, qr = l2norm_fwd(q1.detach().contiguous())
    kn, kr = l2norm_fwd(k1.detach().contiguous())
    q2, k2, v2, g2, b2 = leaves(qn, kn, v, g, beta)
    o2, _ = chunk_kda(q2, k2, v2, g2, b2, disable_recompute=keep)
    dq, dk, dv, dg, db = torch.autograd.grad(o2, [q2, k2, v2, g2, b2], do)
    assert torch.equal(o1, o2) and torch.equal(got[1], dv) and torch.equal(got[2], dg) and torch.equal(got[3], db)
    want = torch.cat([l2norm_bwd(n, r, d).flatten(-2) for n, r, d in ((qn, qr, dq), (kn, kr, dk))], dim=-1)
    # bf16 results, and the separate pass also rounds dq, dk to bf16 in between: some ulps at single elements, little over all
    assert_close("d(q, k)", got[0], want, 8e-2)
    assert (got[0].float() - want.float()).norm() <= 5e-3 * want.float().norm()
