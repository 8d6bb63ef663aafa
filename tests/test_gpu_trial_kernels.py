"""The trial kernels over every shape of the CTA map: entries of one slice and of
many, more entries than one tile of a CTA holds, lines longer than a group of
entries in flight, every lane load width.

With a fixed step the iterates do not depend on how the map is cut: a line's sum
has one order, so all cuts agree bit for bit. With the adaptive step they depend
on the movement sums, whose order follows the cut: N terms of one sign differ by
at most N eps relative (1e-10 here), five steps by less than 1e-8 of the point.
"""
import numpy as np
import pytest

from optimisation_solver_b200 import generators as g
from optimisation_solver_b200.lp import PdlpOptions
from optimisation_solver_b200.pdlp import PdlpSolver

pytestmark = pytest.mark.gpu


def _degrees(n, seed):
    d = np.random.default_rng(seed).integers(1, 5, size=n)
    d[:3] = (700, 300, 37)      # lines over several groups and whole warps
    return d


LPS = {
    "1x2": lambda: g.planted_lp(1, 2, degree=1, seed=1).lp,
    "65x257": lambda: g.planted_lp(65, 257, seed=2).lp,
    "900x5000_long": lambda: g.planted_lp(900, 5000, seed=3, degrees=_degrees(5000, 3)).lp,
    "6000x3000": lambda: g.planted_lp(6000, 3000, degree=12, seed=4).lp,
    "40000x460000": lambda: g.planted_lp(40000, 460000, degree=2, seed=5).lp,
}


@pytest.fixture(scope="module")
def lps():
    cache = {}
    return lambda name: cache.setdefault(name, LPS[name]())


def _solve(lp, precision, limit, adaptive, **ext):
    o = PdlpOptions(iteration_limit=limit, use_adaptive_linesearch=adaptive,
                    use_feasibility_polishing=False).with_tolerance(1e-12)
    r = PdlpSolver(precision, two_kernel_trials=1, **ext).solve(lp, o)
    return r.iterations, np.array(r.primal), np.array(r.row_dual)


@pytest.mark.parametrize("slots", [1, 700, 100_000])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", list(LPS))
def test_every_cut_gives_the_same_iterates(name, precision, slots, lps):
    lp = lps(name)
    base = _solve(lp, precision, 12, False)
    cut = _solve(lp, precision, 12, False, cta_slots=slots)
    assert base[0] == cut[0]
    assert np.array_equal(base[1], cut[1]) and np.array_equal(base[2], cut[2])
    base = _solve(lp, "fp64", 5, True)
    cut = _solve(lp, "fp64", 5, True, cta_slots=slots)
    for a, b in zip(base[1:], cut[1:]):
        assert np.max(np.abs(a - b)) <= 1e-8 * max(1.0, np.max(np.abs(a)))


@pytest.mark.parametrize("width", [1, 2, 4])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_every_cut_at_each_load_width(precision, width, lps):
    for name in ("900x5000_long", "6000x3000"):
        base = _solve(lps(name), precision, 12, False, vector_width=width)
        for slots in (1, 100_000):
            cut = _solve(lps(name), precision, 12, False, vector_width=width, cta_slots=slots)
            assert np.array_equal(base[1], cut[1]) and np.array_equal(base[2], cut[2])
