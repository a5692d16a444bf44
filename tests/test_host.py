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
