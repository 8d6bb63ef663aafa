"""A training step's fused kernels at the edges of their tiles: batches below,
at and above the 128 rows of a tile and not a power of two (the gradient's
division by the batch), inputs that end inside a tile, one and two K splits of
the last layer, the products that read operands as they are stored.

`gradients` is checked against the oracle (tolerance of test_gpu_mlp.py).
A first Adam step is then a function of the gradients alone, with every
operation rounded once in FP32, so it is compared bit for bit with numpy:
m = (1 - b1) g, v = ((1 - b2) g) g, p -= lr (m / c1) / (sqrt(v / c2) + eps).
"""
import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu

SIZES = [(8, 64, 64, 8), (264, 64, 128, 120), (136, 128, 192, 128), (1000, 192, 448, 136), (520, 512, 4032, 256),
         (2000, 512, 22016, 264)]


@pytest.mark.parametrize("inputs,hidden,outputs,batch", SIZES)
def test_step_is_adam_on_the_gradients(inputs, hidden, outputs, batch):
    import torch
    from optimisation_solver_b200.mlp import Mlp

    f = np.float32
    rng = np.random.default_rng(inputs + batch)
    shapes = dict(W1=(hidden, inputs), b1=(hidden,), W2=(hidden, hidden), b2=(hidden,), W3=(outputs, hidden),
                  b3=(outputs,))
    p = {k: (rng.standard_normal(s) / np.sqrt(s[-1])).astype(f) for k, s in shapes.items()}
    x = mo.bf16(rng.standard_normal((batch, inputs)))
    target = rng.standard_normal((batch, outputs)).astype(f)
    weight = (rng.random(outputs) / outputs).astype(f)

    def put(a):
        return torch.as_tensor(a, device="cuda")

    xb, tt, wt = put(x.astype(f)).to(torch.bfloat16), put(target), put(weight)
    net = Mlp(inputs, hidden, outputs, batch)
    net.set_params({k: put(v) for k, v in p.items()})
    grads = {k: torch.full(s, float("nan"), device="cuda") for k, s in shapes.items()}
    loss = net.gradients(xb, tt, wt, grads)
    want_loss, want = mo.gradients(x, target, weight, *(p[k].astype(np.float64) for k in shapes))
    assert abs(loss - want_loss) <= 2e-3 * abs(want_loss)
    g = {k: v.cpu().numpy() for k, v in grads.items()}
    for k in shapes:
        assert np.linalg.norm(g[k] - want[k]) <= 2e-2 * max(np.linalg.norm(want[k]), 1e-12), k

    lr = f(1e-3)
    assert net.train_step(xb, tt, wt, float(lr)) == loss
    got = {k: torch.empty(s, device="cuda") for k, s in shapes.items()}
    net.get_params(got)
    b1, b2, eps, one = f(0.9), f(0.999), f(1e-8), f(1)
    for k in shapes:
        m, v = (one - b1) * g[k], ((one - b2) * g[k]) * g[k]
        step = lr * (m / (one - b1)) / (np.sqrt(v / (one - b2)) + eps)
        assert np.array_equal(got[k].cpu().numpy(), p[k] - step), k


@pytest.mark.parametrize("first,second,batch,pad", [(1, 1, 1, 6), (2000, 20000, 3, 0), (1023, 1, 5, 0),
                                                    (700, 325, 70, 7)])
def test_feature_pair_is_the_concatenation(first, second, batch, pad):
    """Bit for bit the features of the concatenated array, at rows that end
    before, at and after a thread block's 1024 elements."""
    import ctypes as C

    import torch
    from optimisation_solver_b200 import native

    gen = torch.Generator(device="cuda")
    gen.manual_seed(first + batch)
    a, b = (torch.randn((batch, k), generator=gen, device="cuda", dtype=torch.float64) for k in (first, second))
    count = first + second
    mean, inv = (torch.rand(count, generator=gen, device="cuda") for _ in range(2))
    one, two = (torch.full((batch, count + pad), float("nan"), device="cuda").to(torch.bfloat16) for _ in range(2))
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    L = native.lib()
    both = torch.cat([a, b], dim=1)
    assert L.pdlpgpu_encode_features(p(both), batch, count, count + pad, p(mean), p(inv), p(one)) == 0
    assert L.pdlpgpu_encode_feature_pair(p(a), first, p(b), second, batch, count + pad, p(mean), p(inv), p(two)) == 0
    torch.cuda.synchronize()
    want = torch.zeros((batch, count + pad), device="cuda", dtype=torch.bfloat16)
    want[:, :count] = ((both.float() - mean) * inv).to(torch.bfloat16)
    assert torch.equal(one.view(torch.int16), two.view(torch.int16))
    assert torch.equal(one.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("M,N,K,splits", [(1, 1, 8, 1), (129, 257, 72, 1), (129, 130, 1032, 40), (64, 200, 4104, 8),
                                           (1000, 1544, 2568, 4), (300, 129, 520, 3), (1600, 2561, 136, 1),
                                           (1664, 2570, 712, 5), (2300, 1801, 64, 2)])
def test_products_of_every_kernel(M, N, K, splits):
    """The product at the edges of the three kernels plain products go to
    (one tile and less, one row or column more than a tile, odd widths, more
    splits than accumulators). Tolerance of test_gpu_mlp.py; and the splits'
    sum in order is what one run after another gives, so a second call
    matches the first bit for bit."""
    import torch
    from optimisation_solver_b200.mlp import gemm_bf16

    rng = np.random.default_rng(M + N + K + splits)
    a, b = mo.bf16(rng.standard_normal((M, K))), mo.bf16(rng.standard_normal((N, K)))
    ta, tb = (torch.as_tensor(v.astype(np.float32), device="cuda").to(torch.bfloat16) for v in (a, b))
    c, again = (torch.full((M, N), float("nan"), device="cuda") for _ in range(2))
    gemm_bf16(ta, tb, c, splits)
    gemm_bf16(ta, tb, again, splits)
    got = c.cpu().numpy().astype(np.float64)
    assert np.abs(got - a @ b.T).max() <= 1e-5 * (np.abs(a) @ np.abs(b).T).max()
    assert torch.equal(c, again)
