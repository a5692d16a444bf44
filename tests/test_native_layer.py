"""GPU: the native layer (one autograd node) against the same kernels driven one by one from Python, over the forms a layer
takes: biases, ALiBi as a table, head_dim 32 / 64 / 128, frozen parameters, separate and column-block projections, gradients
returned, added to .grad and written over it.  Both run the same products on the same values, so everything is equal to the
last bit but the q, k, v weight gradients, which one side may work out as one product of three times the width."""
import pytest
import torch

from test_edges import _fuse_projections, _layer

pytestmark = pytest.mark.gpu
EPS = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


PROJECTIONS = ("q_proj", "k_proj", "v_proj")


def _before(name, p, mode):
    """What lies in .grad before the step.  Projections whose gradients are no column blocks of one matrix are added to the
    buffer by the Python blocks in every mode, so theirs is cleared where it is to be written."""
    torch.manual_seed(p.numel())
    old = torch.randn_like(p, memory_format=torch.contiguous_format) * 0.1
    return old.zero_() if mode == "written" and any(w in name for w in PROJECTIONS) else old


def _projection_grads_agree(name, a, b, old):
    # each side rounds an fp32 sum over the rows once, or twice where it is rounded before it is added
    size = a.float().abs() + 2 * old.float().abs()
    bound = 3 * EPS[a.dtype] * size + 2.0 ** -20 * size.max()
    assert ((a.float() - b.float()).abs() <= bound).all(), name


def _run(layer, x, g, bias, python, mode, train_x=True):
    from tritonformer_b200 import linear
    for n, p in layer.named_parameters():
        p.grad = None
        if mode != "returned" and p.requires_grad:
            p.grad = _before(n, p, mode)
    xi = x.clone().requires_grad_(train_x)
    linear.PROFILE = [] if python else None  # recorded calls run the Python blocks
    try:
        if mode == "returned":
            y = layer(xi, bias)
            y.backward(g)
        else:
            with linear.accumulate_into_grad(overwrite=mode == "written", written=set()):
                y = layer(xi, bias)
                y.backward(g)
        if python:
            assert linear.PROFILE
    finally:
        linear.PROFILE = None
    torch.cuda.synchronize()
    return y.detach(), xi.grad, {n: p.grad for n, p in layer.named_parameters()}


FORMS = [dict(), dict(use_linear_bias=False), dict(num_attention_heads=4, head_dim=32), dict(num_attention_heads=1, head_dim=128),
         dict(ffn_dim=200), dict(hidden_size=256, num_attention_heads=4, ffn_dim=1024)]


@pytest.mark.parametrize("form", range(len(FORMS)))
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("mode", ["returned", "added", "written"])
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("alibi", [False, True])
def test_native_layer_is_the_python_layer(form, dtype, mode, fused, alibi):
    from tritonformer_b200.transformer import generate_alibi_mask
    layer = _layer(dtype, **FORMS[form])
    if fused:
        _fuse_projections(layer)
    d, heads = layer.input_layernorm.weight.numel(), layer.attention.num_attention_heads
    for t in (64, 256):  # one key tile and two: dQ has at most two shares, so its sum does not depend on their order
        gen = torch.Generator(device="cuda").manual_seed(t)
        x, g = (torch.randn(3, t, d, device="cuda", generator=gen).to(dtype) for _ in range(2))
        bias = generate_alibi_mask(256, heads)[0] if alibi else None
        (y0, dx0, p0), (y1, dx1, p1) = (_run(layer, x, g, bias, python, mode) for python in (True, False))
        assert torch.equal(y0, y1) and torch.equal(dx0, dx1)
        for n in p0:
            if any(w in n for w in PROJECTIONS):
                old = _before(n, p0[n], mode) if mode == "added" else torch.zeros_like(p0[n])
                _projection_grads_agree(n, p0[n], p1[n], old)
            else:
                assert torch.equal(p0[n], p1[n]), n


@pytest.mark.parametrize("frozen", ["q_proj", "attention", "mlp", "layernorm", "everything", "nothing"])
@pytest.mark.parametrize("train_x", [True, False])
def test_native_layer_with_frozen_parameters(frozen, train_x):
    layer = _layer()
    for n, p in layer.named_parameters():
        p.requires_grad_(not (frozen == "everything" or frozen in n))
    if frozen == "everything" and not train_x:
        pytest.skip("nothing to differentiate")
    x, g = (torch.randn(2, 128, 128, device="cuda").half() for _ in range(2))
    (y0, dx0, p0), (y1, dx1, p1) = (_run(layer, x, g, None, python, "returned", train_x) for python in (True, False))
    assert torch.equal(y0, y1)
    assert (dx1 is None) == (not train_x) and (dx0 is None or torch.equal(dx0, dx1))
    for n in p0:
        assert (p0[n] is None) == (p1[n] is None) == (frozen == "everything" or frozen in n), n
        if p0[n] is not None:
            _projection_grads_agree(n, p0[n], p1[n], torch.zeros_like(p0[n]))


def test_native_layer_launches():
    """Seven kernels forward; backward: eight products (the three projections' weight gradients one of them), the LayerNorms
    two each, attention three."""
    from tritonformer_b200 import _lib, linear
    layer = _fuse_projections(_layer(use_linear_bias=False))
    d = 128
    grads = torch.zeros(d, 3 * d, device="cuda").half()
    for i, p in enumerate((layer.attention.q_proj, layer.attention.k_proj, layer.attention.v_proj)):
        p.weight.grad = grads[:, i * d:(i + 1) * d]
    for p in layer.parameters():
        if p.grad is None:
            p.grad = torch.zeros_like(p)
    x = torch.randn(2, 128, d, device="cuda").half().requires_grad_()
    with linear.accumulate_into_grad():
        n0 = _lib.launch_count()
        y = layer(x)
        n1 = _lib.launch_count()
        y.backward(torch.randn_like(y))
        n2 = _lib.launch_count()
    assert (n1 - n0, n2 - n1) == (7, 8 + 4 + 3)


def test_captured_pattern_is_the_layers_own():
    import tritonformer_b200.fused as fused
    layer = _layer()
    x = torch.randn(2, 64, 128, device="cuda").half()
    patterns = []
    fused.CAPTURE_ACTIVATION_PATTERN = patterns
    try:
        with_capture = layer(x.requires_grad_())
        with torch.no_grad():
            layer(x)
    finally:
        fused.CAPTURE_ACTIVATION_PATTERN = None
    assert torch.equal(with_capture, layer(x)) and with_capture.grad_fn.name().find("Layer") >= 0
    assert len(patterns) == 2 and torch.equal(*patterns) and patterns[0].shape == (2, 64, 192)
    hidden = x + layer.attention(layer.input_layernorm(x), None)
    pre = layer.mlp.dense_h_to_4h(layer.post_attention_layernorm(hidden))
    assert ((pre > 0) != patterns[0]).float().mean().item() < 5e-3  # hidden is rounded once more there
