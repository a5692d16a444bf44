"""GPU: values and layouts at the edge of what the operators accept: infinities and NaN, broadcast and overlapping rows,
saved-tensor hooks, transforms and tracing.  Where a kernel takes a call from another one, both have to agree on these too."""
import pytest
import torch

pytestmark = pytest.mark.gpu
HALF = [torch.float16, torch.bfloat16]


def _heads(h, t, hd, dtype, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(1, h, t, hd, device="cuda", generator=gen).to(dtype) for _ in range(4)]


@pytest.mark.parametrize("t,hd", [(64, 64), (192, 64), (192, 32), (192, 128), (320, 128), (256, 64)])
@pytest.mark.parametrize("where", ["v", "k"])
def test_attention_backward_keeps_slices_apart(t, hd, where):
    """An infinity in one head's last tile leaves the other heads' gradients exactly as they are without it."""
    from tritonformer_b200.attention import CausalAttention
    q, k, v, g = _heads(3, t, hd, torch.float16)
    grads = []
    for poisoned in (False, True):
        args = [x.clone() for x in (q, k, v)]
        if poisoned:
            args["qkv".index(where)][0, 0, t - 3, 1] = float("inf")
        args = [x.requires_grad_() for x in args]
        grads.append(torch.autograd.grad(CausalAttention.apply(*args), args, g))
    for clean, dirty in zip(*grads):
        # dQ of the clean heads is summed in any order: one 16-bit step
        assert (clean[0, 1:] - dirty[0, 1:]).abs().max().item() <= 2.0 ** -9 * clean.abs().max().item()


@pytest.mark.parametrize("t,hd", [(64, 64), (192, 64), (192, 32), (192, 128), (256, 64)])
def test_attention_backward_of_a_key_that_no_query_reaches(t, hd):
    """A key of -inf has probability zero for every query that sees it, so its dK and dV are zero and not NaN."""
    from tritonformer_b200.attention import CausalAttention
    q, k, v, g = _heads(2, t, hd, torch.float16)
    q = q.abs()
    k[0, 0, t - 3] = 0.0
    k[0, 0, t - 3, 0] = -float("inf")
    args = [x.requires_grad_() for x in (q, k, v)]
    dq, dk, dv = torch.autograd.grad(CausalAttention.apply(*args), args, g)
    assert torch.equal(dv[0, 0, t - 3], torch.zeros_like(dv[0, 0, t - 3]))
    assert torch.equal(dk[0, 0, t - 3], torch.zeros_like(dk[0, 0, t - 3]))
    assert dv.isfinite().all() and dk.isfinite().all()
