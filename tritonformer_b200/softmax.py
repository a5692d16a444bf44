"""Softmax autograd Function over the last dimension (drop-in for tritonformer/softmax.py:6-21).

No autocast decoration, as in the reference; fp32, fp16 and bf16 inputs are accepted.  The
backward writes a new tensor instead of overwriting the incoming gradient.
"""
from torch.autograd import Function

from . import _host


class Softmax(Function):
    """softmax over the last dimension: apply(input)."""
    apply = staticmethod(_host.softmax)
