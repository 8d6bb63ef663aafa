"""Calls that are refused on the host. A training step that is refused leaves the
model as it was: the step after it is the step of a model that never saw the
refused call, bit for bit. Outputs that the device cannot store to (host memory
that is not pinned) are an error of the call, and the model goes on working."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("refused_after", [0, 1, 3])
def test_a_refused_step_does_not_count(refused_after):
    import torch
    from optimisation_solver_b200.mlp import Mlp

    inputs, hidden, outputs, batch = 64, 64, 64, 8
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)

    def randn(*shape):
        return torch.randn(shape, generator=gen, device="cuda")

    steps = [(randn(batch, inputs).to(torch.bfloat16), randn(batch, outputs)) for _ in range(4)]
    weight = torch.rand(outputs, generator=gen, device="cuda")
    # One element past a 16-byte boundary: TMA cannot read it.
    shifted = torch.zeros(batch * inputs + 8, device="cuda", dtype=torch.bfloat16)[1:1 + batch * inputs]
    shapes = dict(W1=(hidden, inputs), b1=(hidden,), W2=(hidden, hidden), b2=(hidden,), W3=(outputs, hidden),
                  b3=(outputs,))

    def train(refuse):
        net = Mlp(inputs, hidden, outputs, batch, seed=3)
        losses = []
        for k, (x, t) in enumerate(steps):
            if refuse and k == refused_after:
                with pytest.raises(RuntimeError, match="16-byte"):
                    net.train_step(shifted.view(batch, inputs), t, weight, 1e-3)
            losses.append(net.train_step(x, t, weight, 1e-3))
        got = {k: torch.empty(s, device="cuda") for k, s in shapes.items()}
        net.get_params(got)
        return losses, got

    want_losses, want = train(False)
    losses, got = train(True)
    assert losses == want_losses
    for k in shapes:
        assert torch.equal(got[k], want[k]), k


@pytest.mark.parametrize("where", ["host", "pinned"])
def test_outputs_in_host_memory(where):
    import torch
    from optimisation_solver_b200.mlp import Mlp

    inputs, hidden, outputs, batch = 64, 64, 128, 8
    gen = torch.Generator(device="cuda")
    gen.manual_seed(9)
    x = torch.randn((batch, inputs), generator=gen, device="cuda").to(torch.bfloat16)
    target = torch.randn((batch, outputs), generator=gen, device="cuda")
    weight = torch.rand(outputs, generator=gen, device="cuda")
    net = Mlp(inputs, hidden, outputs, batch, seed=1)
    want, want_grad = torch.empty((batch, outputs), device="cuda"), torch.empty((hidden, inputs), device="cuda")
    net.forward(x, want)
    net.gradients(x, target, weight, {"W1": want_grad})
    out, grad = torch.zeros((batch, outputs)), torch.zeros((hidden, inputs))
    if where == "host":
        with pytest.raises(RuntimeError, match="device memory"):
            net.forward(x, out)
        with pytest.raises(RuntimeError, match="device memory"):
            net.gradients(x, target, weight, {"W1": grad})
        assert not out.any() and not grad.any()
        again = torch.empty_like(want)
        net.forward(x, again)
        assert torch.equal(again, want)
    else:
        out, grad = out.pin_memory(), grad.pin_memory()
        net.forward(x, out)
        net.gradients(x, target, weight, {"W1": grad})
        assert torch.equal(out, want.cpu()) and torch.equal(grad, want_grad.cpu())
