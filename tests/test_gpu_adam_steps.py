"""Adam's arithmetic after the first step and at the ends of FP32's range.

Ten steps with changing batches: bias corrections of every step, moments of
several gradients. The outputs' loss weights run over forty decades, so the
gradients of the last layer do too: second moments that vanish beside a first
moment, that are subnormal, that lie on both sides of the bounds between which
the kernel divides without branches, and up to 1e30. The last step's targets
hold a NaN. Every operation is rounded once in FP32 (the two moment updates'
sums by one fused multiply-add), so parameters are compared bit for bit with
numpy on the gradients that the model reports before each step.
"""
import ctypes
import ctypes.util

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

f = np.float32


def _fma(a, b, c):
    """float32 fma: the exact product and sum in float64, rounded to odd there,
    then once to float32."""
    p = np.asarray(a, np.float64) * np.asarray(b, np.float64)   # exact
    c = np.asarray(c, np.float64)
    s = p + c
    t = s - p
    err = (p - (s - t)) + (c - t)
    even = (s.view(np.int64) & 1) == 0
    odd = np.where((err != 0) & even & np.isfinite(s), np.nextafter(s, np.where(err > 0, np.inf, -np.inf)), s)
    return odd.astype(f)


def _powf(x, y):
    libm = ctypes.CDLL(ctypes.util.find_library("m"))
    libm.powf.restype = ctypes.c_float
    libm.powf.argtypes = [ctypes.c_float, ctypes.c_float]
    return f(libm.powf(float(x), float(y)))


@pytest.mark.parametrize("lr", [1e-3, 0.5, 1e-20, 0.0])
def test_ten_steps_of_every_magnitude(lr):
    import torch
    from optimisation_solver_b200.mlp import Mlp

    inputs, hidden, outputs, batch = 72, 64, 512, 40
    rng = np.random.default_rng(7)
    shapes = dict(W1=(hidden, inputs), b1=(hidden,), W2=(hidden, hidden), b2=(hidden,), W3=(outputs, hidden),
                  b3=(outputs,))
    p = {k: (rng.standard_normal(s) / np.sqrt(s[-1])).astype(f) for k, s in shapes.items()}

    def put(a):
        return torch.as_tensor(a, device="cuda")

    net = Mlp(inputs, hidden, outputs, batch)
    net.set_params({k: put(v) for k, v in p.items()})
    weight = put((10.0 ** rng.uniform(-27.0, 14.0, outputs)).astype(f))
    m = {k: np.zeros(s, f) for k, s in shapes.items()}
    v = {k: np.zeros(s, f) for k, s in shapes.items()}
    b1, b2, eps, one, rate = f(0.9), f(0.999), f(1e-8), f(1), f(lr)
    grads = {k: torch.empty(s, device="cuda") for k, s in shapes.items()}
    got = {k: torch.empty(s, device="cuda") for k, s in shapes.items()}
    seen = set()
    for step in range(1, 12):
        x = put(rng.standard_normal((batch, inputs)).astype(f)).to(torch.bfloat16)
        target = rng.standard_normal((batch, outputs)).astype(f)
        if step == 11:
            target[3, 200] = np.nan
        target = put(target)
        net.gradients(x, target, weight, grads)
        net.train_step(x, target, weight, lr)
        net.get_params(got)
        c1, c2 = one - _powf(b1, step), one - _powf(b2, step)
        with np.errstate(all="ignore"):
            for k in shapes:
                g = grads[k].cpu().numpy()
                m[k] = _fma(one - b1, g, b1 * m[k])
                v[k] = _fma((one - b2) * g, g, b2 * v[k])
                p[k] = p[k] - rate * (m[k] / c1) / (np.sqrt(v[k] / c2) + eps)
                assert np.array_equal(got[k].cpu().numpy(), p[k], equal_nan=True), (step, k)
            third = np.abs(v["W3"])
            seen |= {name for name, hit in dict(
                vanished=(third == 0) & (m["W3"] != 0), subnormal=(third > 0) & (third < 1.17e-38),
                low=(third >= 1.17e-38) & (third < 1e-25), middle=(third > 1e-25) & (third < 1e25),
                high=third > 1e25, nan=np.isnan(third)).items() if hit.any()}
    assert seen == {"vanished", "subnormal", "low", "middle", "high", "nan"}
