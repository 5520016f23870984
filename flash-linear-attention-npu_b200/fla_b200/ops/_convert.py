"""fp16 tensors at the boundary of operators whose kernels multiply bf16 operands.

The reference's chunk and decode operators take fp16 as well as bf16 tensors and reject only fp32
(examples/flash_gated_delta_rule.py:1161-1162).  Here an fp16 tensor enters through the library's conversion kernel
(`fla_b200_convert`: rounded to bf16, 11 -> 8 significant bits) and results leave through it as fp16; gradients take the
same way back.  Nothing is cast through PyTorch."""
from __future__ import annotations

from .. import host


def convert(t, dtype, op: str = "convert"):
    """A dense copy of ``t`` (1 to 4 dims, innermost dim contiguous, any outer strides) in ``dtype``
    (float32 / bfloat16 / float16), made by the library's conversion kernel on the current stream."""
    del op
    return host().convert(t, dtype)


def to_dtype(t, dtype, op: str = "convert"):
    """``t`` in ``dtype`` (differentiable: the gradient is converted back); ``t`` itself when it already has that dtype or is None."""
    del op
    return host().to_dtype(t, dtype)
