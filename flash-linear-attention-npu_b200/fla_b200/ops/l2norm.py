"""Row-wise L2 normalisation kernels (reference: fla/ops/triton/triton_core/l2norm.py:131-234)."""
from __future__ import annotations

from .. import host


def l2norm_fwd(x, eps: float = 1e-6, output_dtype=None):
    """Returns ``(y, rstd)`` with ``y = x * rsqrt(sum(x^2, -1) + eps)`` and rstd of shape ``x.shape[:-1]`` (fp32)."""
    return host().l2norm_fwd(x, eps, output_dtype)


def l2norm_bwd(y, rstd, dy, eps: float = 1e-6):
    """Returns ``dx = dy * rstd - sum(dy * y, -1) * y * rstd`` in the dtype of ``y``."""
    return host().l2norm_bwd(y, rstd, dy, eps)
