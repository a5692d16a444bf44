"""CPU: the Python side of the native host path."""
import torch


def test_a_traced_call_replays_and_differentiates():
    from tritonformer_b200._trace import record
    scale = lambda x, w, k: (x @ w) * k

    class Model(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.w = torch.nn.Parameter(torch.randn(3, 4))
            self.frozen = torch.nn.Parameter(torch.randn(3, 4), requires_grad=False)

        def forward(self, x):
            return record(scale, x, self.w, 2.0) + record(scale, x, self.frozen, 3.0).relu()

    torch.manual_seed(0)
    model = Model()
    traced = torch.jit.trace(model, torch.randn(2, 3), check_trace=False)
    x = torch.randn(5, 3)
    grads = []
    for f in (lambda t: scale(t, model.w, 2.0) + scale(t, model.frozen, 3.0).relu(), traced):
        xi = x.clone().requires_grad_()
        y = f(xi)
        grads.append((y.detach(),) + torch.autograd.grad(y.square().sum(), (xi, model.w)))
    for a, b in zip(*grads):
        assert torch.allclose(a, b, rtol=1e-6, atol=1e-6)
    with torch.no_grad():
        assert torch.allclose(traced(x), model(x))


def test_overlap_switches_act_when_they_are_set(monkeypatch):
    from tritonformer_b200 import linear
    told = []
    real = linear._host

    class Host:
        def __getattr__(self, name):
            return getattr(real, name)

        def set_grad_mode(self, *mode):
            told.append(mode)
            real.set_grad_mode(*mode)

    monkeypatch.setattr(linear, "_host", Host())
    before = linear.FORK_WEIGHT_GRAD
    try:
        linear.FORK_WEIGHT_GRAD = False
        assert told[-1] == (False, False, False, False)
        linear.FORK_WEIGHT_GRAD = True
        assert told[-1] == (False, False, False, True)
        with linear.accumulate_into_grad(overwrite=True):
            assert told[-1] == (True, True, False, True)
            linear.FORK_WEIGHT_GRAD = False
            assert told[-1] == (True, True, False, False)
        assert told[-1] == (False, False, False, False)
    finally:
        linear.FORK_WEIGHT_GRAD = before
    assert told[-1][3] == before


def test_a_table_that_was_used_can_be_saved(tmp_path):
    from tritonformer_b200.attention import _resolve_bias
    from tritonformer_b200.transformer import generate_alibi_mask
    table = generate_alibi_mask(64, 4, device="cpu")[0]
    found = _resolve_bias(table, 4, 64, torch.float16)
    assert found.table is None and found.rounded == 1
    torch.save(table, tmp_path / "table.pt")
    again = torch.load(tmp_path / "table.pt")  # weights only
    assert torch.equal(again, table)
    assert torch.equal(_resolve_bias(again, 4, 64, torch.float16).slopes, found.slopes)


def test_tensors_without_data_are_refused_before_anything_is_launched():
    import pytest
    from torch._subclasses.fake_tensor import FakeTensorMode
    from tritonformer_b200.attention import CausalAttention
    from tritonformer_b200.layernorm import LayerNorm
    from tritonformer_b200.linear import LinearNoBias
    from tritonformer_b200.softmax import Softmax
    with FakeTensorMode():
        x, w, q = (torch.empty(s, device="cuda", dtype=torch.float16) for s in ((4, 64), (64, 64), (1, 2, 64, 64)))
        for call in (lambda: Softmax.apply(x), lambda: LinearNoBias.apply(x, w), lambda: CausalAttention.apply(q, q, q),
                     lambda: LayerNorm.apply(x, w[0], w[0], 1e-5), lambda: LinearNoBias.apply(x, w.requires_grad_())):
            with pytest.raises(NotImplementedError):
                call()
