"""Solves of LPs of different sizes on several host threads at once. Their
fused trials are launches of the same kernels with different amounts of shared
memory; each solve must come out as it does alone, bit for bit, whatever the
other threads launch between its set-up and its launches.
"""
import threading

import numpy as np
import pytest

from optimisation_solver_b200 import generators as g
from optimisation_solver_b200.lp import PdlpOptions
from optimisation_solver_b200.pdlp import PdlpSolver

pytestmark = pytest.mark.gpu

SIZES = [(31, 33), (200, 400), (1000, 2000), (2000, 4000), (500, 900), (120, 300)]


@pytest.mark.parametrize("graphs", [True, False])
def test_solves_on_threads_match_solves_alone(graphs):
    options = PdlpOptions(iteration_limit=330).with_tolerance(1e-10)
    solver = PdlpSolver("fp64", disable_graphs=0 if graphs else 1)
    lps = [g.planted_lp(m, n, degree=4, seed=m).lp for m, n in SIZES]
    alone = [solver.solve(lp, options) for lp in lps]
    wrong = []
    start = threading.Barrier(len(lps))

    def work(k):
        start.wait(timeout=60)
        for _ in range(40):
            r = solver.solve(lps[k], options)
            if (r.status, r.status_message, r.iterations) != \
                    (alone[k].status, alone[k].status_message, alone[k].iterations) or \
                    not np.array_equal(r.primal, alone[k].primal) or \
                    not np.array_equal(r.row_dual, alone[k].row_dual):
                wrong.append((SIZES[k], str(r.status), r.status_message, r.iterations))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(lps))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:5]
