"""Phase times: refused before the first iteration, then parts that add up to
the whole, in every form of the solver and the batch."""

from __future__ import annotations

import time

import pytest

from cuminlp_gb300 import _abi as A
from cuminlp_gb300 import generators as G
from cuminlp_gb300._lib import CmnError
from cuminlp_gb300.problem import Problem, sqr
from cuminlp_gb300.solver import Batch, DeviceProblem, Solver

pytestmark = pytest.mark.gpu

SHARED = dict(bisection_budget=3, batch_parents=64, frontier_cap=1024)


@pytest.fixture(scope="module", autouse=True)
def _built():
    from cuminlp_gb300 import build
    build.build_library()


def check_phases(of, step):
    with pytest.raises(CmnError):
        of.phase_ms()
    t0 = time.perf_counter()
    step()
    wall = (time.perf_counter() - t0) * 1e3
    ms = of.phase_ms()
    assert len(ms) == 5 and all(x > 0 for x in ms)
    assert sum(ms[:4]) == pytest.approx(ms[4], abs=1e-6) and ms[4] < wall


@pytest.mark.parametrize("precision", ["fp64", "fp32", "lazy"])
@pytest.mark.parametrize("iterations", [1, 4])
def test_phase_times(precision, iterations):
    dp = DeviceProblem(G.miqcqp_n32())
    s = Solver(dp, precision=precision, iter_limit=1 << 30, **SHARED)
    check_phases(s, lambda: s.step(iterations))
    if precision == "lazy":
        assert all(0 < x <= s.phase_ms()[4] for x in s.lazy_ms())
    b = Batch(2, dp.n_vars, precision=s.options.precision, **SHARED)
    b.add(dp, iter_limit=1 << 30)
    check_phases(b, lambda: b.step(iterations))


@pytest.mark.parametrize("bits", [1, 4])
def test_lazy_times_after_the_stop(bits):
    # a program with shared slots takes the interpreter; the iterations queued
    # behind the last one that expanded boxes leave its times as they are
    p = Problem()
    x = [p.var(-2.0, 3.0) for _ in range(5)]
    s = sqr(x[0]) + 1.0
    p.set_objective(sqr(x[1] - x[2]) / s + 0.5 * s + x[3] * x[4])
    p.add_constraint(s * x[3], A.CMP_LE, 4.0)
    solver = Solver(DeviceProblem(p), precision="lazy", iter_limit=1 << 30, batch_iter_limit=5, bisection_budget=bits,
                    batch_parents=64, frontier_cap=1024)
    solver.step(0)
    whole = solver.phase_ms()[4]
    assert all(0 < t <= whole for t in solver.lazy_ms())
