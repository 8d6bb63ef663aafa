"""Fused trials over check intervals longer than the step factors a CTA keeps
in shared memory (160 iterations): every trial takes the factors of its own
iteration whatever part of the interval it is in, so all results equal the
two-kernel path's bit for bit and there is no tolerance. Intervals: one
iteration past the factors kept, a few times them, the most trials of a launch
and more; the main loop and feasibility polishing, whose iterations count from
zero again.
"""
import numpy as np
import pytest

from optimisation_solver_b200 import generators as g
from optimisation_solver_b200.lp import PdlpOptions
from optimisation_solver_b200.pdlp import PdlpSolver
from tests import cases

pytestmark = pytest.mark.gpu

LPS = {
    "31x33": lambda: g.planted_lp(31, 33, degree=3, seed=1).lp,
    "1000x2000": lambda: g.planted_lp(1000, 2000, seed=11).lp,
    "16000x33000": lambda: g.planted_lp(16000, 33000, seed=8).lp,
    "polished": lambda: cases.random_feasible(300, 420, 21),
}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("polishing", [False, True])
@pytest.mark.parametrize("frequency", [161, 400, 1020, 3000])
@pytest.mark.parametrize("name", list(LPS))
def test_long_check_intervals_match_two_kernels(name, frequency, polishing, precision):
    lp = LPS[name]()
    options = PdlpOptions(iteration_limit=1250, termination_check_frequency=frequency,
                          use_feasibility_polishing=polishing, polishing_iterations=700).with_tolerance(1e-10)
    a = PdlpSolver(precision).solve(lp, options)
    b = PdlpSolver(precision, two_kernel_trials=1).solve(lp, options)
    assert (a.status, a.iterations, a.step_trials, a.restart_count) == \
        (b.status, b.iterations, b.step_trials, b.restart_count)
    assert (a.final_step_size, a.final_primal_weight) == (b.final_step_size, b.final_primal_weight)
    for k in ("primal", "row_dual", "dual_ray", "primal_ray"):
        assert np.array_equal(getattr(a, k), getattr(b, k)), k
    assert a.primal_objective == b.primal_objective
