"""Softmax cross-entropy autograd Functions (drop-in for tritonformer/crossentropy.py:9-24).

`CrossEntropyLoss.apply(logits (N,V), labels (N,))` returns the per-row losses in the logits'
dtype, as the reference does.  `CrossEntropyLossFP32` is the same operator returning the
unrounded fp32 per-row losses; `lm_loss` is the model's shifted mean of them.
A label outside [0, V) marks a row to skip: zero loss, zero gradient.
"""
from torch.autograd import Function

from . import _host


class CrossEntropyLoss(Function):
    """Softmax Cross Entropy; per-row loss in the dtype of the logits."""

    @staticmethod
    def apply(input, labels):
        return _host.cross_entropy(input, labels, False)


class CrossEntropyLossFP32(Function):
    """Softmax Cross Entropy; per-row loss in fp32."""

    @staticmethod
    def apply(input, labels):
        return _host.cross_entropy(input, labels, True)


def lm_loss(logits, labels):
    """fp32 mean over the batch * (seq - 1) positions that have a next token of the loss of logits[b, t] (batch, seq,
    vocab) against labels[b, t + 1]: the shift, the per-row losses and their mean without a copy of either."""
    return _host.lm_loss(logits, labels)
