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


@pytest.mark.parametrize("t,hd", [(64, 64), (192, 64), (448, 64), (192, 128), (256, 32), (448, 32), (320, 128)])
@pytest.mark.parametrize("bias", [False, True])
def test_attention_with_keys_at_minus_infinity(t, hd, bias):
    """A key whose score is -inf for every query counts for nothing, wherever in a tile it lies: at its start the first query
    that sees it has no other key there.  Only queries with no other key at all have no result."""
    from tritonformer_b200.attention import BiasedCausalAttention, CausalAttention
    at = sorted({p for p in (1, 31, 32, 63, 64, 65, 127, 128, 129, 191, 192, 255, 256, 319, 320, t - 1) if p < t})
    sets = [[p] for p in at] + [[p, p + 1] for p in at if p + 1 < t] + [at, list(range(64, t)), [0], [0, 1, 2]]
    q, k, v, _ = _heads(len(sets), t, hd, torch.float16)
    q = q.abs() + 0.125
    for h, keys in enumerate(sets):
        k[0, h, keys, 0] = -float("inf")
    slopes = torch.tensor([2.0 ** -(1 + h % 6) for h in range(len(sets))], device="cuda")
    out = BiasedCausalAttention.apply(q, k, v, slopes) if bias else CausalAttention.apply(q, k, v)
    s = (q.double() @ k.double().transpose(-1, -2)) / hd ** 0.5
    if bias:
        i = torch.arange(t, device="cuda")
        s = s - slopes.double()[:, None, None] * (i[:, None] - i[None, :])
    s = s.masked_fill(~torch.ones(t, t, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    want = torch.softmax(s, -1) @ v.double()
    assert torch.equal(out.isnan(), want.isnan())
    # P and the result are rounded to 16 bits; values of about one
    assert (out.double() - want).nan_to_num(0.0).abs().max().item() <= 2.0 ** -11 * 8


@pytest.mark.parametrize("t,hd", [(64, 64), (192, 64), (192, 128), (128, 32), (192, 32)])
@pytest.mark.parametrize("dtype", HALF)
def test_attention_passes_nan_on(t, hd, dtype):
    """A NaN in any key reaches every query that sees it, at the sizes that are no whole tiles of the full width."""
    from tritonformer_b200.attention import CausalAttention
    q, k, v, _ = _heads(t - 1, t, hd, dtype)  # head i: NaN in key i
    for i in range(t - 1):
        k[0, i, i, 0] = float("nan")
    out = CausalAttention.apply(q, k, v)
    seen = torch.ones(t, t, dtype=torch.bool, device="cuda").tril()[:, : t - 1].t()  # (key, query)
    assert torch.equal(out[0].isnan().all(-1), seen)
    assert torch.equal(out[0].isnan().any(-1), seen)


@pytest.mark.parametrize("t,hd", [(192, 64), (704, 128), (320, 64), (512, 32), (192, 32)])
def test_attention_statistics_are_those_of_exact_exponentials(t, hd):
    """The log-sum-exp of the sizes that are no whole tiles of the full width: fp32 sums of exponentials that are good to a
    few units in the last place (2^-21 relative with 2^-22 for the sums), scores from fp32 products of 16-bit values."""
    from tritonformer_b200 import _lib as L
    h = 4
    q, k, v, _ = _heads(h, t, hd, torch.float16)
    out, lse = torch.empty_like(q), torch.empty(1, h, t, device="cuda")
    L.check(L.lib.tfb_attention_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(), 1, h, t, hd,
                                    *(L.strides3(x) for x in (q, k, v, out)), None, 0, None, 0, 0, 0, L.stream_ptr(q.device), None))
    s = (q.double() @ k.double().transpose(-1, -2)) / hd ** 0.5
    s = s.masked_fill(~torch.ones(t, t, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    want = torch.logsumexp(s, -1)
    # |score| <= about 8: 2^-22 of it for the product's sum and the scaling, as much for the result itself
    assert (lse.double() - want).abs().max().item() <= 2.0 ** -21 + 3 * 2.0 ** -22 * max(8.0, want.abs().max().item())


@pytest.mark.parametrize("cols", [1, 7, 9, 17, 257, 2047, 50257])
@pytest.mark.parametrize("dtype", HALF)
def test_cross_entropy_of_an_odd_vocabulary_passes_nan_on(cols, dtype):
    """A NaN logit in any column of a row makes its loss NaN; columns of -inf are left out of the sum."""
    from tritonformer_b200.crossentropy import CrossEntropyLossFP32
    at = sorted({c for c in (*range(9), cols // 2, cols - 9, cols - 2, cols - 1) if 0 <= c < cols})
    logits = torch.randn(len(at) * 8, cols, device="cuda").to(dtype)  # eight rows of each: every alignment of a row
    for i, c in enumerate(at):
        logits[i::len(at), c] = float("nan")
    labels = torch.zeros(logits.shape[0], dtype=torch.int64, device="cuda")
    assert CrossEntropyLossFP32.apply(logits, labels).isnan().all()
    masked = torch.randn(8, cols, device="cuda").to(dtype)
    masked[:, : cols - 1] = -float("inf")
    loss = CrossEntropyLossFP32.apply(masked, torch.full((8,), cols - 1, device="cuda"))
    assert loss.abs().max().item() <= 1e-6 * masked[:, -1].float().abs().max().item() + 1e-6


def _layer(dtype=torch.float16, seed=0, **kw):
    from tritonformer_b200.transformer import TransformerConfig, TransformerLayer
    cfg = dict(vocab_size=64, hidden_size=128, max_position_embeddings=128, num_attention_heads=2, head_dim=64, ffn_dim=192,
               num_hidden_layers=1, use_linear_bias=True, attn_bias=False)
    cfg.update(kw)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    layer = TransformerLayer(TransformerConfig(**cfg), device="cuda").to(dtype)
    with torch.no_grad():
        for n, p in layer.named_parameters():
            p.copy_(torch.randn(p.shape, device="cuda", generator=gen) * (0.05 if "layernorm" not in n else 0.2)
                    + (1.0 if n.endswith("layernorm.weight") else 0.0))
    return layer


def _fuse_projections(layer):
    """The q, k and v weights as column blocks of one matrix (Transformer.fuse_projection_weights)."""
    att = layer.attention
    parts = [att.q_proj, att.k_proj, att.v_proj]
    buf = torch.cat([p.weight.detach() for p in parts], 1)
    d = buf.shape[0]
    for i, p in enumerate(parts):
        p.weight = torch.nn.Parameter(buf[:, i * d:(i + 1) * d])
    return layer


class _ContiguousCopies(torch.autograd.graph.saved_tensors_hooks):
    """What saving on the host does to a saved tensor: a copy comes back, contiguous whatever the tensor was."""

    def __init__(self):
        super().__init__(lambda t: t.detach().clone(memory_format=torch.contiguous_format), lambda t: t.clone())


@pytest.mark.parametrize("hooks", [_ContiguousCopies, torch.autograd.graph.save_on_cpu])
@pytest.mark.parametrize("fused", [True, False])
def test_layer_backward_from_copies_of_the_saved_tensors(hooks, fused):
    import contextlib
    layer = _layer()
    if fused:
        _fuse_projections(layer)
    x = torch.randn(2, 128, 128, device="cuda").half()
    g = torch.randn_like(x)
    grads = []
    for context in (contextlib.nullcontext, hooks):
        xi = x.clone().requires_grad_()
        with context():
            y = layer(xi)
        grads.append(torch.autograd.grad(y, [xi] + list(layer.parameters()), g))
    for a, b in zip(*grads):
        assert torch.equal(a, b)


@pytest.mark.parametrize("hooks", [_ContiguousCopies, torch.autograd.graph.save_on_cpu])
@pytest.mark.parametrize("transposed", ["neither", "x", "w", "both"])
@pytest.mark.parametrize("m,k,n", [(5, 9, 13), (33, 33, 33), (40, 64, 24), (130, 257, 71)])
def test_linear_backward_from_copies_of_the_saved_tensors(hooks, transposed, m, k, n):
    import contextlib
    from tritonformer_b200.linear import LinearBias, LinearNoBiasReLU
    gen = torch.Generator(device="cuda").manual_seed(m)
    mk = lambda r, c, t: (torch.randn(c, r, device="cuda", generator=gen).half().t() if t
                          else torch.randn(r, c, device="cuda", generator=gen).half())
    x, w = mk(m, k, transposed in ("x", "both")), mk(k, n, transposed in ("w", "both"))
    b, g = mk(1, n, False)[0], mk(m, n, False)
    for fn, extra in ((LinearBias, (b,)), (LinearNoBiasReLU, ())):
        grads = []
        for context in (contextlib.nullcontext, hooks):
            args = [t.detach().requires_grad_() for t in (x, w, *extra)]
            with context():
                y = fn.apply(*args)
            grads.append(torch.autograd.grad(y, args, g))
        for a, c in zip(*grads):
            assert torch.equal(a, c)


def _calls(dtype=torch.float16):
    """(name, function of one floating tensor, that tensor) for every operator."""
    from tritonformer_b200.attention import BiasedCausalAttention, CausalAttention
    from tritonformer_b200.crossentropy import CrossEntropyLoss, CrossEntropyLossFP32, lm_loss
    from tritonformer_b200.embedding import Embedding
    from tritonformer_b200.layernorm import LayerNorm
    from tritonformer_b200.linear import LinearBias, LinearBiasReLU, LinearNoBias, LinearNoBiasReLU
    from tritonformer_b200.softmax import Softmax
    gen = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(*s, device="cuda", generator=gen).to(dtype)
    x, w, b, q = r(2, 64, 128), r(128, 64), r(64), r(2, 2, 64, 64)
    one, ids = r(128), torch.randint(0, 64, (2, 64), device="cuda", generator=gen)
    layer = _layer(dtype).requires_grad_(False)
    return [("linear", lambda t: LinearNoBias.apply(t, w), x), ("linear_weight", lambda t: LinearBias.apply(x, t, b), w),
            ("linear_relu", lambda t: LinearNoBiasReLU.apply(t, w), x),
            ("linear_bias_relu", lambda t: LinearBiasReLU.apply(x, w, t), b),
            ("layernorm", lambda t: LayerNorm.apply(t, one, one, 1e-5), x), ("softmax", lambda t: Softmax.apply(t), x),
            ("attention", lambda t: CausalAttention.apply(t, q, q), q),
            ("attention_slopes", lambda t: BiasedCausalAttention.apply(q, q, t, torch.tensor([0.5, 0.25], device="cuda")), q),
            ("cross_entropy", lambda t: CrossEntropyLoss.apply(t[0], ids[0]), x),
            ("cross_entropy_fp32", lambda t: CrossEntropyLossFP32.apply(t[0], ids[0]), x),
            ("lm_loss", lambda t: lm_loss(t, ids), x), ("embedding", lambda t: Embedding.apply(ids, t, None), w),
            ("layer", lambda t: layer(t), x)]


def test_forward_mode_and_transforms_are_refused():
    """Not implemented, and said so: a result without its tangent would pass for a constant."""
    import torch.autograd.forward_ad as fwd
    for name, fn, x in _calls():
        for grad in (False, True):
            with torch.set_grad_enabled(grad), fwd.dual_level():
                dual = fwd.make_dual(x.clone().requires_grad_(grad), torch.ones_like(x))
                with pytest.raises(NotImplementedError):
                    fn(dual)
                fn(x)
        with pytest.raises(RuntimeError):
            torch.func.grad(lambda t: fn(t).float().sum())(x)
        with torch.no_grad(), pytest.raises(RuntimeError):
            torch.func.vmap(fn)(torch.stack([x, x]))


def test_traced_operators_replay():
    """A traced call gives on new inputs what the operator gives, and differentiates."""
    for name, fn, x in _calls():
        example = x.clone()
        traced = torch.jit.trace(fn, example, check_trace=False)
        new = torch.randn_like(x).flip(0)
        with torch.no_grad():
            assert torch.equal(traced(new), fn(new)), name
        both = []
        for f in (fn, traced):
            t = new.clone().requires_grad_()
            y = f(t)
            both.append(torch.autograd.grad(y, t, torch.ones_like(y) * 0.5)[0])
        assert torch.equal(*both), name


@pytest.mark.parametrize("alibi", [False, True])
def test_traced_model_replays(alibi):
    from tritonformer_b200.transformer import Transformer, TransformerConfig
    torch.manual_seed(0)
    model = Transformer(TransformerConfig(vocab_size=96, hidden_size=128, max_position_embeddings=64, num_attention_heads=2,
                                          head_dim=64, ffn_dim=256, num_hidden_layers=2, use_linear_bias=True,
                                          attn_bias=alibi), device="cuda")
    with torch.no_grad():
        model.logits_out.weight.normal_(0.0, 0.02)
    ids = torch.randint(0, 96, (2, 2, 64), device="cuda")

    class Logits(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.model = model

        def forward(self, t):
            return self.model(t, None)

    traced = torch.jit.trace(Logits(), ids[0], check_trace=False)
    with torch.no_grad():
        assert torch.equal(traced(ids[1]), model(ids[1], None))


@pytest.mark.parametrize("form", ["LinearNoBias", "LinearBias", "LinearNoBiasReLU", "LinearBiasReLU"])
@pytest.mark.parametrize("k,n", [(128, 64), (77, 51)])
@pytest.mark.parametrize("dtype", HALF)
def test_linear_takes_broadcast_and_overlapping_rows(form, k, n, dtype):
    """Rows that repeat (stride 0) or overlap, as an input and as a gradient, give what their copies give."""
    import tritonformer_b200.linear as L
    fn, bias = getattr(L, form), "NoBias" not in form
    gen = torch.Generator(device="cuda").manual_seed(k)
    r = lambda *s: torch.randn(*s, device="cuda", generator=gen).to(dtype)
    w, b = r(k, n), r(n)
    inputs = [r(1, k).expand(9, k), r(k + 30).unfold(0, k, 3), r(2, 1, k).expand(2, 5, k), r(1, 1, k).expand(2, 5, k), r(6, k)]
    for x in inputs:
        rows = x.shape[:-1]
        for g in (r(n).expand(*rows, n), r(n + len(rows) * 16).unfold(0, n, 1)[: rows[-1]].expand(*rows, n), r(*rows, n)):
            sides = []
            for xi, gi in ((x, g), (x.contiguous(), g.contiguous())):
                args = [t.detach().requires_grad_() for t in ((xi, w, b) if bias else (xi, w))]
                y = fn.apply(*args)
                sides.append((y.detach(),) + torch.autograd.grad(y, args, gi))
            for one, two in zip(*sides):
                assert torch.equal(one, two)


@pytest.mark.parametrize("form", ["LinearNoBias", "LinearBias", "LinearNoBiasReLU", "LinearBiasReLU"])
def test_linear_gradient_of_a_sum_over_rows(form):
    import tritonformer_b200.linear as L
    x, w, b = (torch.randn(*s, device="cuda").half() for s in ((2, 7, 64), (64, 40), (40,)))
    args = [t.requires_grad_() for t in ((x, w, b) if "NoBias" not in form else (x, w))]
    y = getattr(L, form).apply(*args)
    got = torch.autograd.grad(y.sum((0, 1)), args, torch.ones(40, device="cuda").half())
    want = torch.autograd.grad(getattr(L, form).apply(*args), args, torch.ones_like(y))
    for a, c in zip(got, want):
        assert torch.equal(a, c)


@pytest.mark.parametrize("t,hd", [(64, 64), (192, 64), (192, 128), (128, 32), (192, 32)])
@pytest.mark.parametrize("which", ["q", "k", "v", "grad_heads", "grad_batch", "grad_rows"])
def test_attention_takes_broadcast_operands(t, hd, which):
    """One head's operand for all heads, or a gradient that repeats over heads, batch or positions."""
    from tritonformer_b200.attention import CausalAttention
    gen = torch.Generator(device="cuda").manual_seed(t + hd)
    q, k, v, g = (torch.randn(2, 3, t, hd, device="cuda", generator=gen).half() for _ in range(4))
    if which in "qkv":
        one = {"q": q, "k": k, "v": v}[which][:1, :1].expand(2, 3, t, hd)
        q, k, v = (one if n == which else x for n, x in (("q", q), ("k", k), ("v", v)))
    else:
        g = {"grad_heads": g[:, :1], "grad_batch": g[:1], "grad_rows": g[:, :, :1]}[which].expand(2, 3, t, hd)
    args = [x.detach().requires_grad_() for x in (q, k, v)]
    out = CausalAttention.apply(*args)
    got = (out.detach(),) + torch.autograd.grad(out, args, g)
    qd, kd, vd = (x.detach().double().requires_grad_() for x in (q, k, v))
    s = (qd @ kd.transpose(-1, -2)) / hd ** 0.5
    s = s.masked_fill(~torch.ones(t, t, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    ref = torch.softmax(s, -1) @ vd
    want = (ref.detach(),) + torch.autograd.grad(ref, (qd, kd, vd), g.double())
    for a, b in zip(got, want):  # P, dS, the output in delta and the result are each rounded to 16 bits
        assert ((a.double() - b).norm() / b.norm()).item() < 4 * 2.0 ** -11


@pytest.mark.parametrize("m,n,k", [(64, 64, 64), (256, 256, 256), (300, 248, 640), (640, 1000, 512)])
def test_one_wave_product_with_an_epilogue_operand_after_an_expired_wait(m, n, k):
    """While the status word is set a product writes nothing and leaves no load of its addend or mask on the way; the
    products behind it are right again once the word is cleared."""
    from tritonformer_b200 import _lib as L, linear as LIN
    assert L.device_status() == 0
    gen = torch.Generator(device="cuda").manual_seed(n)
    a, b, add, mask = (torch.randn(*s, device="cuda", generator=gen).half() for s in ((m, k), (k, n), (m, n), (m, n)))
    b *= k ** -0.5
    L.check(L.lib.tfb_debug_wait_probe(1_000_000, None, L.stream_ptr(a.device)))
    out = torch.full((m, n), 777.0, device="cuda", dtype=torch.float16)
    for _ in range(20):
        LIN.gemm(a, k, 1, b, n, 1, m, n, k, addend=add, out=out)
        LIN.gemm(a, k, 1, b, n, 1, m, n, k, mask=mask, out=out)
    assert bool((out == 777.0).all())
    assert L.device_status(reset=True) == 0x7E00
    want = a.double() @ b.double()
    for _ in range(5):
        got = LIN.gemm(a, k, 1, b, n, 1, m, n, k, addend=add)
        assert (got.double() - (want + add.double())).abs().max().item() <= 2.0 ** -10 * (want.abs().max().item() + 8)
    assert L.device_status() == 0


def test_what_a_backward_refuses_is_an_assertion_error():
    from tritonformer_b200.attention import CausalAttention
    args = [torch.randn(1, 2, 128, 64, device="cuda").half().requires_grad_() for _ in range(3)]
    out = CausalAttention.apply(*args)
    unaligned = torch.randn(out.numel() + 1, device="cuda").half()[1:].view_as(out)
    with pytest.raises(AssertionError, match="grad_out needs a 16-byte aligned base"):
        out.backward(unaligned)
    with pytest.raises(AssertionError, match="multiple of 64"):
        CausalAttention.apply(*(a[:, :, :100] for a in args))


def test_a_layer_refuses_an_empty_batch_where_it_comes_in():
    layer = _layer()
    for shape in ((0, 64, 128), (2, 0, 128)):
        for grad in (False, True):
            with torch.set_grad_enabled(grad), pytest.raises(AssertionError, match="attention: bad shape"):
                layer(torch.empty(shape, device="cuda", dtype=torch.float16))


@pytest.mark.parametrize("reentrant", [False, True])
def test_layer_under_checkpointing(reentrant):
    from torch.utils.checkpoint import checkpoint
    layer = _fuse_projections(_layer())
    x = torch.randn(2, 128, 128, device="cuda").half()
    g = torch.randn_like(x)
    grads = []
    for run in (layer, lambda t: checkpoint(layer, t, use_reentrant=reentrant)):
        layer.zero_grad(set_to_none=True)
        xi = x.clone().requires_grad_()
        run(xi).backward(g)
        grads.append([xi.grad] + [p.grad for p in layer.parameters()])
    for a, b in zip(*grads):
        assert torch.equal(a, b)
