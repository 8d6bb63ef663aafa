"""The trials of small LPs on each side of the lines at which their kernel or
its layout changes: clusters of eight and sixteen CTAs, short and long lines,
one slice a worker and several, nothing staged; one instance, a few of a
moderate size, and more than the device holds at once. Every route adds in the
two-kernel path's order, so all results are equal bit for bit.
"""
import numpy as np
import pytest

from optimisation_solver_b200 import generators as g
from optimisation_solver_b200.lp import PdlpOptions
from optimisation_solver_b200.pdlp import PdlpSolver

pytestmark = pytest.mark.gpu

SHAPES = [
    (2040, 4080, 5, 1), (2060, 4120, 5, 1),      # the last cluster of eight, the first of sixteen
    (3500, 7000, 7, 1), (3500, 7000, 8, 1),      # copies from five entries a line on (FP32)
    (900, 1800, 17, 1), (900, 1800, 19, 1),      # and from twelve (FP64)
    (4090, 8180, 5, 1), (4110, 8220, 5, 1),      # a second slice a worker
    (6500, 13000, 5, 1), (16300, 32700, 5, 1), (17000, 34000, 5, 1),   # nothing staged; more slices than four a worker
    (8000, 16000, 5, 2), (8000, 16000, 5, 3), (10000, 20000, 5, 3), (10000, 20000, 5, 4), (8000, 16000, 5, 9),
    (30000, 60000, 3, 1), (300, 5000, 40, 1), (1200, 1500, 60, 1), (6500, 13000, 30, 1), (7000, 14000, 30, 1),
]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("rows,cols,degree,count", SHAPES)
def test_routes_match_two_kernels(rows, cols, degree, count, precision):
    lps = [g.planted_lp(rows + 3 * k, cols + k, degree=degree, seed=k).lp for k in range(count)]
    options = PdlpOptions(iteration_limit=230).with_tolerance(1e-9)

    def solve(**ext):
        solver = PdlpSolver(precision, **ext)
        return solver.solve_batch(lps, options) if count > 1 else [solver.solve(lps[0], options)]

    for a, b in zip(solve(), solve(two_kernel_trials=1)):
        assert (a.status, a.iterations, a.step_trials, a.restart_count) == \
            (b.status, b.iterations, b.step_trials, b.restart_count)
        for k in ("primal", "row_dual", "dual_ray", "primal_ray"):
            assert np.array_equal(getattr(a, k), getattr(b, k)), k
        assert a.primal_objective == b.primal_objective
