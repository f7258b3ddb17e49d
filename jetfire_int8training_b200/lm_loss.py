"""Cross-entropy of the language-model head on bf16 logits, without an fp32 copy of the logits.

`lm_cross_entropy(logits, targets)` equals `F.cross_entropy(logits.float().view(-1, V), targets.view(-1), ignore_index=-1)`
(the loss at the end of the reference's quantised GPT-2, INT8_GPT2/qmodel.py:433-439) up to fp32 rounding.  The forward pass
reads the logits once; the backward pass overwrites them IN PLACE with their gradient (the logits are an intermediate that
nothing else needs: the backward of the producing matmul uses its inputs, not its output), so no second [tokens, vocab] tensor
is ever allocated.  There is no CPU path.
"""
import torch

from ._lib import host

__all__ = ["lm_cross_entropy"]


class _LMLoss(torch.autograd.Function):
    @staticmethod
    def forward(ctx, logits, targets):
        loss, x, t, lse, count = host().lm_loss_forward(logits, targets)
        ctx.save_for_backward(x, t, lse, count)
        ctx.shape = logits.shape
        return loss

    @staticmethod
    def backward(ctx, grad_out):
        x, t, lse, count = ctx.saved_tensors
        host().lm_loss_backward(grad_out, x, t, lse, count)
        return x.view(ctx.shape), None


def lm_cross_entropy(logits, targets):
    """Mean softmax cross-entropy over the positions whose target lies in [0, vocab).  `logits` (bf16, [..., vocab]) is
    consumed: after backward() it holds its own gradient."""
    return _LMLoss.apply(logits, targets)
