"""The pool's rebuild over several blocks of tiles (4,096 entries each) against
the oracle: the cap at and beside a tile's edge, evictions, and many equal lower
bounds split by position across tiles."""

from __future__ import annotations

import pytest

from cuminlp_gb300 import generators as G
from cuminlp_gb300.problem import Problem
from tests.test_gpu_solver import compare

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from cuminlp_gb300 import build
    build.build_library()


def tied_problem() -> Problem:
    """Lower bounds that change along two of the five variables only, and stay
    below the best value (the terms cancel, their bounds do not)."""
    p = Problem()
    x = [p.var(-2.0, 2.0) for _ in range(5)]
    p.set_objective(x[0] * x[1] - x[0] * x[1] + x[0] - x[0])
    return p


@pytest.mark.parametrize("cap,parents", [(4095, 1500), (4096, 4096), (4097, 700), (9000, 2100)])
def test_pool_of_several_tiles(cap, parents):
    for p in (tied_problem(), G.miqcqp_n32(1)):
        g = compare(p, 8, bisection_budget=3, batch_parents=parents, frontier_cap=cap)
        assert g["frontier_size"] == cap and g["counters"]["dropped_viable"] > 0
