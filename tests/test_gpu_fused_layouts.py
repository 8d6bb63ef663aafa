"""The fused trials' layouts (vectors copied to every CTA, half of them, none,
nothing staged) at the sizes where they change: one line, the edges of a slice
and of a worker's share, lines longer than an unrolled group, clusters of 1 to
16 CTAs, several slices a worker, every lane load width; and the decisions
that rank 0 takes for all (a clock, an iteration limit inside an interval). The
fused trials add in the two-kernel path's order, so all results are equal bit
for bit: no tolerance.
"""
import numpy as np
import pytest

from optimisation_solver_b200 import generators as g
from optimisation_solver_b200.lp import PdlpOptions
from optimisation_solver_b200.pdlp import PdlpSolver
from tests import cases

pytestmark = pytest.mark.gpu


def _flow(nodes):
    graph = g.flow_graph(nodes, seed=3)
    supply, cost = g.flow_parameters(graph, 1, 5)
    return g.flow_lp(graph, supply[0], cost[0])


LPS = {
    "one_line": cases.upper_bound_row,
    "31x33": lambda: g.planted_lp(31, 33, degree=3, seed=1).lp,
    "33x64_dense": lambda: g.planted_lp(33, 64, degree=30, seed=2).lp,
    "257x513": lambda: g.planted_lp(257, 513, seed=3).lp,
    "513x1025": lambda: g.planted_lp(513, 1025, seed=4).lp,
    "2048x4096": lambda: g.planted_lp(2048, 4096, seed=5).lp,
    "2049x8193": lambda: g.planted_lp(2049, 8193, seed=6).lp,
    "6000x3000": lambda: g.planted_lp(6000, 3000, degree=12, seed=7).lp,
    "16000x33000": lambda: g.planted_lp(16000, 33000, seed=8).lp,
    "flow_150": lambda: _flow(150),
    "flow_2000": lambda: _flow(2000),
}


def _compare(lp, precision, options, **ext):
    a = PdlpSolver(precision, **ext).solve(lp, options)
    b = PdlpSolver(precision, two_kernel_trials=1, **ext).solve(lp, options)
    assert (a.status, a.iterations, a.step_trials, a.restart_count) == \
        (b.status, b.iterations, b.step_trials, b.restart_count)
    for k in ("primal", "row_dual", "dual_ray", "primal_ray"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k
    assert a.primal_objective == b.primal_objective


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", list(LPS))
def test_layouts_match_two_kernels(name, precision):
    # 470 iterations: the limit falls inside an interval of 100 trials.
    _compare(LPS[name](), precision, PdlpOptions(iteration_limit=470).with_tolerance(1e-9))


@pytest.mark.parametrize("width", [1, 2, 4])
@pytest.mark.parametrize("name", ["257x513", "6000x3000", "16000x33000"])
def test_load_widths_match_two_kernels(name, width):
    _compare(LPS[name](), "mixed", PdlpOptions(iteration_limit=330).with_tolerance(1e-9),
             vector_width=width)


@pytest.mark.parametrize("name", ["31x33", "2048x4096", "16000x33000"])
def test_a_clock_that_does_not_run_out_changes_nothing(name):
    _compare(LPS[name](), "fp64", PdlpOptions(
        iteration_limit=330, time_limit_seconds=600.0).with_tolerance(1e-9))
