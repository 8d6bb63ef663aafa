"""Fused trials under a time limit and with a fixed step, whose decisions are
taken in every CTA like the others. A clock that does not run out and a fixed
step change nothing against the two-kernel path, bit for bit: main loop,
averaging and polishing (whose step and controller differ when the step is
fixed), clusters of one and of sixteen CTAs. A clock that runs out ends the
solve with the status and message of the two-kernel path and a point of an
interrupted run: fewer iterations than the limit, finite residuals.
"""
import numpy as np
import pytest

from optimisation_solver_b200 import generators as g
from optimisation_solver_b200.lp import PdlpOptions, PdlpStatus
from optimisation_solver_b200.pdlp import PdlpSolver
from tests import cases

pytestmark = pytest.mark.gpu

LPS = {
    "31x33": lambda: g.planted_lp(31, 33, degree=3, seed=1).lp,
    "1000x2000": lambda: g.planted_lp(1000, 2000, seed=11).lp,
    "6000x12000": lambda: g.planted_lp(6000, 12000, seed=8).lp,
    "polished": lambda: cases.random_feasible(300, 420, 21),
}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("averaging", [True, False])
@pytest.mark.parametrize("limit,adaptive", [(0.0, False), (600.0, True), (600.0, False)])
@pytest.mark.parametrize("name", list(LPS))
def test_limits_and_fixed_steps_match_two_kernels(name, limit, adaptive, averaging, precision):
    lp = LPS[name]()
    options = PdlpOptions(iteration_limit=470, time_limit_seconds=limit, use_adaptive_linesearch=adaptive,
                          use_averaging=averaging, polishing_iterations=330).with_tolerance(1e-11)
    a = PdlpSolver(precision).solve(lp, options)
    b = PdlpSolver(precision, two_kernel_trials=1).solve(lp, options)
    assert (a.status, a.iterations, a.step_trials, a.restart_count) == \
        (b.status, b.iterations, b.step_trials, b.restart_count)
    assert (a.final_step_size, a.final_primal_weight) == (b.final_step_size, b.final_primal_weight)
    for k in ("primal", "row_dual", "dual_ray", "primal_ray"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k
    assert a.primal_objective == b.primal_objective


@pytest.mark.parametrize("frequency", [100, 5000])
@pytest.mark.parametrize("name", ["31x33", "1000x2000", "6000x12000"])
def test_a_clock_that_runs_out_ends_the_solve(name, frequency):
    lp = LPS[name]()
    PdlpSolver("fp64").solve(lp, PdlpOptions(iteration_limit=10))   # loads the kernels
    base = dict(iteration_limit=2_000_000, use_feasibility_polishing=False, detect_infeasibility=False,
                termination_check_frequency=frequency)
    for seconds in (1e-6, 0.25):   # run out before the first trial, and in the middle
        options = PdlpOptions(time_limit_seconds=seconds, **base).with_tolerance(1e-300)
        a = PdlpSolver("fp64").solve(lp, options)
        b = PdlpSolver("fp64", two_kernel_trials=1).solve(lp, options)
        assert a.status == b.status == PdlpStatus.TIME_LIMIT
        assert a.status_message == b.status_message
        assert a.iterations < options.iteration_limit and a.step_trials >= a.iterations
        assert np.isfinite(a.primal_residual) and np.isfinite(a.dual_residual)
        assert (a.iterations > 0) == (b.iterations > 0) == (seconds > 0.1)
