"""Programs with shared slots over few boxes (independent runs of the program
on different warps, level by level) give the oracle's enclosures bit for bit:
partial tiles, both sides of the box count where one lane per box takes over,
every operator, and the regions of a role's box."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from cuminlp_gb300 import _abi as A
from cuminlp_gb300.problem import Expr, Problem, pow, sqr, sqrt
from cuminlp_gb300.solver import Bounder, DeviceProblem, eval_boxes
from tests.conftest import bits_equal
from tests.gpu_common import random_boxes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from cuminlp_gb300 import build
    build.build_library()


def wide_problem(n: int) -> Problem:
    """n loosely coupled groups: shared intermediates, sum chains read by
    nodes, constants, and checks of both kinds inside the groups."""
    p = Problem()
    x = [p.var(-2.0, 3.0) if i % 3 else p.int_var(-1.0, 4.0) for i in range(n)]
    g = p.graph
    total = None
    for i in range(n):
        a, b, c = x[i], x[(i + 1) % n], x[(i + 2) % n]
        s = sqr(a) + 1.0
        chain = 2.0 * (a * b) - 0.5 * sqr(c) + b
        low = Expr(g, g.emit(A.OP_MIN, (s.id, chain.id)))
        t = sqr(b - c) / s + sqrt(s) * low - pow(chain, 3) / (s + sqr(low))
        t = t + Expr(g, g.emit(A.OP_ABS, (chain.id,))) + p.fixed(2.0) * p.fixed(-1.5)
        total = t if total is None else total + t
        if i % 4 == 0:
            p.add_constraint(s * chain - t, A.CMP_LE, 4.0 + i)
        if i % 5 == 2:
            p.add_constraint(low + a, A.CMP_EQ, 0.5)
    p.set_objective(total)
    return p


@pytest.mark.parametrize("precision", [A.PRECISION_FP64, A.PRECISION_FP32_SCREEN])
@pytest.mark.parametrize("n,boxes", [(5, 1), (9, 31), (17, 33), (17, 3001), (40, 257), (6, 19456), (6, 19457)])
def test_boxes(n, boxes, precision):
    p = wide_problem(n)
    lo, hi = random_boxes(p, boxes, np.random.default_rng(boxes), 0.3)
    g = eval_boxes(DeviceProblem(p), lo, hi, precision)
    o = O.OracleProblem(p).eval_boxes(lo, hi, precision)
    assert np.array_equal(g[2], o[2])
    assert bits_equal(g[0], o[0]) and bits_equal(g[1], o[1])


@pytest.mark.parametrize("bits", [1, 5, 8])
def test_role_regions(bits):
    p = wide_problem(11)
    kinds, vids, widths, _ = O.bisection_choose(p.root_box(), p.var_kinds, bits)
    n = int(np.prod(widths))
    fe, lb = Bounder(DeviceProblem(p), kinds, n).bound(p.root_box(), vids, widths)
    ofe, olb = O.OracleProblem(p).bound(p.root_box(), kinds, vids, widths, n)
    assert np.array_equal(fe, ofe) and bits_equal(lb, olb)
