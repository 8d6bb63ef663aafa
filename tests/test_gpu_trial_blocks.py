"""pdlpgpu_trial_noalloc at the edges of its blocks of lines: one line, a line
more and less than the 32 and 256 lines of a block, lines of 32 and 33 entries
(a thread's or a warp's sum), lines that straddle the 3072 products a block
holds at a time, empty lines, and more lines than one pass of the grid.

Reference: the trial's formulas in numpy FP64 (pdhg_kernel.cpp:47-187). A sum
of L products in any order is within L * 2^-53 * sum |product| of the exact
one; with values and vectors of magnitude about 1 and lines of at most 10^4
entries, 1e-10 of the largest entry bounds every output.
"""
import ctypes as C

import numpy as np
import pytest

from optimisation_solver_b200 import native

pytestmark = pytest.mark.gpu

TOL = 1e-10


def _csr(lengths, width, rng):
    start = np.zeros(lengths.size + 1, dtype=np.int64)
    np.cumsum(lengths, out=start[1:])
    index = rng.integers(0, width, int(start[-1])).astype(np.int32)
    return start, index, rng.standard_normal(int(start[-1]))


def _product(start, index, values, v):
    line = np.repeat(np.arange(start.size - 1), np.diff(start))
    return np.bincount(line, weights=values * v[index], minlength=start.size - 1)


def _lengths(kind, count, rng):
    if kind == "short":
        return rng.integers(0, 9, count)
    if kind == "around_32":
        return rng.integers(30, 36, count)
    out = rng.integers(0, 4, count)          # "long": a few lines of thousands among short ones
    out[rng.integers(0, count, 3)] = (3072, 3071, 9001)
    return out


@pytest.mark.parametrize("kind", ["short", "around_32", "long"])
@pytest.mark.parametrize("rows,cols", [(1, 1), (31, 33), (255, 257), (256, 9500), (3000, 10001),
                                       (90_000, 700_001)])
def test_trial_blocks(rows, cols, kind):
    import torch

    rng = np.random.default_rng(rows + len(kind))
    a = _csr(_lengths(kind, rows, rng), cols, rng)
    at = _csr(_lengths(kind, cols, rng), rows, rng)   # each half is checked on its own matrix
    c, x = rng.standard_normal(cols), rng.random(cols)
    xl, xu = np.zeros(cols), np.where(rng.random(cols) < 0.5, np.inf, 1.0)
    rl, ru = np.where(rng.random(rows) < 0.5, -np.inf, -0.1), np.full(rows, 0.1)
    tau, sigma = 0.5 + rng.random(cols), 0.5 + rng.random(rows)
    y, ax = rng.standard_normal(rows), rng.standard_normal(rows)
    step, weight = 0.7, 1.3

    def put(v):
        return torch.as_tensor(v, device="cuda")

    args = [put(v) for v in (*a, *at, c, xl, xu, tau, 1.0 / tau, rl, ru, sigma, 1.0 / sigma, x, y, ax)]
    ox, oy, oax = (torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
                   for n in (cols, rows, rows))
    red = torch.full((3,), float("nan"), dtype=torch.float64, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    rc = native.lib().pdlpgpu_trial_noalloc(rows, cols, *[p(t) for t in args], step, weight, p(ox),
                                            p(oy), p(oax), p(red),
                                            C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, native.last_error()
    torch.cuda.synchronize()

    want_x = np.maximum(xl, np.minimum(x - step / weight * tau * (c + _product(*at, y)), xu))
    want_ax = _product(*a, want_x)
    s = step * weight * sigma
    v = y + s * (2.0 * want_ax - ax)
    want_y = np.maximum(v - s * ru, 0.0) + np.minimum(v - s * rl, 0.0)
    dx, dy = want_x - x, want_y - y
    for got, want in ((ox, want_x), (oax, want_ax), (oy, want_y)):
        assert np.abs(got.cpu().numpy() - want).max() <= TOL * max(1.0, np.abs(want).max())
    terms = (dx * dx / tau, dy * dy / sigma, dy * (want_ax - ax))
    for got, term in zip(red.cpu().numpy(), terms):
        assert abs(got - term.sum()) <= TOL * max(1.0, np.abs(term).sum())
