"""Forward passes of batches of many rows and few columns, whose last layer's
row tiles are dealt over several CTAs: one row tile a CTA and several, a last
one that is not full, one accumulator set and two, one K split and many. Each
128 rows of the batch repeat the same inputs, so their outputs repeat bit for
bit whichever CTA computed them; the first rows are compared with the oracle
(tolerance of test_gpu_mlp.py).
"""
import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inputs,hidden,outputs,batch", [
    (64, 64, 64, 136), (64, 64, 64, 8192), (72, 256, 128, 1000), (64, 512, 320, 5000), (128, 1024, 2048, 1928),
    (64, 4096, 64, 1160), (256, 512, 4800, 512), (64, 128, 22016, 264)])
def test_rows_do_not_depend_on_their_tile(inputs, hidden, outputs, batch):
    import torch
    from optimisation_solver_b200.mlp import Mlp

    rng = np.random.default_rng(inputs + outputs + batch)
    shapes = dict(W1=(hidden, inputs), b1=(hidden,), W2=(hidden, hidden), b2=(hidden,), W3=(outputs, hidden),
                  b3=(outputs,))
    p = {k: (rng.standard_normal(s) / np.sqrt(s[-1])).astype(np.float32) for k, s in shapes.items()}
    base = mo.bf16(rng.standard_normal((128, inputs)))
    x = torch.as_tensor(base.astype(np.float32), device="cuda").to(torch.bfloat16)
    net = Mlp(inputs, hidden, outputs, batch)
    net.set_params({k: torch.as_tensor(v, device="cuda") for k, v in p.items()})
    out = torch.full((batch, outputs), float("nan"), device="cuda")
    net.forward(x.repeat(-(-batch // 128), 1)[:batch].contiguous(), out)
    for first in range(128, batch, 128):
        rows = min(128, batch - first)
        assert torch.equal(out[first:first + rows], out[:rows]), first
    rows = min(128, batch)
    want, _, _ = mo.forward(base[:rows], *(p[k].astype(np.float64) for k in shapes))
    got = out[:rows].cpu().numpy()
    assert np.linalg.norm(got - want) <= 1e-2 * np.linalg.norm(want)
