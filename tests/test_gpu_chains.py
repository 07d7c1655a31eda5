"""The evaluator of sum-chain programs (a tile of boxes per block, constraints
decided in FP32 where its error bound allows) gives the oracle's verdicts bit
for bit where it could go wrong: partial tiles, comparisons closer than the
FP32 error, equality and shared-root readers, subtracted and constant chain
terms, and bounds outside the FP32 filter's range."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from cuminlp_gb300 import _abi as A
from cuminlp_gb300 import generators as G
from cuminlp_gb300._lib import check as status, lib
from cuminlp_gb300.problem import Expr, Problem
from cuminlp_gb300.solver import Bounder, DeviceProblem, Sampler, eval_boxes
from tests.conftest import bits_equal
from tests.gpu_common import random_boxes
from tests.test_gpu_solver import compare

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from cuminlp_gb300 import build
    build.build_library()


def mixed_problem() -> Problem:
    """Chains of every reader and term form: <= and == checks, a constant and
    a variable start, subtracted terms, terms without a coefficient, one root
    read by the objective and a check, a product of a variable by itself."""
    p = Problem()
    x = [p.var(-3.0, 2.0), p.var(0.5, 4.0), p.var(-1.0, 1.0), p.int_var(0.0, 5.0), p.bin_var()]
    obj = 2.0 * (x[0] * x[1]) - 3.0 * (x[2] * x[3]) + x[4] * x[0] - (x[1] * x[2])
    p.set_objective(obj)
    p.add_constraint(obj, A.CMP_LE, 4.0)
    p.add_constraint(p.fixed(1.5) + x[0] * x[2] - 0.25 * x[3], A.CMP_LE, 1.0)
    p.add_constraint(x[0] + 2.0 * x[1] - x[2], A.CMP_EQ, 1.0)
    same = Expr(p.graph, p.graph.emit(A.OP_MUL, (x[2].id, x[2].id)))
    p.add_constraint(-1.0 * same + 0.5 * (x[1] * x[1]) - 2.0 * x[4], A.CMP_LE, 2.0)
    return p


def near_problem(rhs_shift: float) -> Problem:
    """One <= chain whose lower bound sits `rhs_shift` from the right side on
    a whole lattice of boxes: 0 and one FP64 ulp are inside the FP32 error."""
    p = Problem()
    x = [p.var(-4.0, 4.0) for _ in range(6)]
    acc = 1.25 * (x[0] * x[1])
    for i in range(1, 5):
        acc = acc + (0.5 + i) * (x[i] * x[i + 1])
    p.set_objective(acc + 3.0 * x[0])
    p.add_constraint(acc + 0.5 * (x[0] * x[0]), A.CMP_LE, -6.0 + rhs_shift)
    return p


def check(p: Problem, lo, hi):
    g = eval_boxes(DeviceProblem(p), lo, hi)
    o = O.OracleProblem(p).eval_boxes(lo, hi, A.PRECISION_FP64)
    assert np.array_equal(g[2], o[2])
    assert bits_equal(g[0], o[0]) and bits_equal(g[1], o[1])


@pytest.mark.parametrize("count", [1, 31, 32, 33, 257, 4099])
def test_partial_tiles(count):
    rng = np.random.default_rng(count)
    for p in (mixed_problem(), G.miqcqp_n32(1)):
        check(p, *random_boxes(p, count, rng, 0.3))


@pytest.mark.parametrize("shift", [0.0, 2.0 ** -50, -(2.0 ** -50), 2.0 ** -22, -(2.0 ** -22), 1.0])
def test_comparisons_inside_the_fp32_error(shift):
    # boxes on a quarter lattice: the chain's bound is exact, and -6 is one of
    # its values
    rng = np.random.default_rng(5)
    lo = rng.integers(-8, 8, (6, 3000)) / 4.0
    hi = lo + rng.integers(0, 3, lo.shape) / 4.0
    p = near_problem(shift)
    o = O.OracleProblem(p).eval_boxes(lo, hi, A.PRECISION_FP64)
    assert 0 < np.sum(o[2]) < lo.shape[1]
    check(p, lo, hi)


@pytest.mark.parametrize("value", [0.0, -0.0, 1e-300, 1e-20, 5e-324, 1e13, 1e200, np.inf, -np.inf])
def test_bounds_outside_the_filter_range(value):
    rng = np.random.default_rng(3)
    for p in (mixed_problem(), near_problem(0.25)):
        lo, hi = random_boxes(p, 200, rng, 0.3)
        at = rng.integers(0, lo.shape[0], 40), rng.integers(0, 200, 40)
        lo[at] = np.minimum(value, hi[at])
        both = rng.random(40) < 0.5
        hi[at[0][both], at[1][both]] = np.maximum(value, lo[at[0][both], at[1][both]])
        check(p, lo, hi)


@pytest.mark.parametrize("bits", [1, 3, 6, 9])
def test_role_regions(bits):
    p = G.miqcqp_n32(2)
    kinds, vids, widths, _ = O.bisection_choose(p.root_box(), p.var_kinds, bits)
    n = int(np.prod(widths))
    fe, lb = Bounder(DeviceProblem(p), kinds, n).bound(p.root_box(), vids, widths)
    ofe, olb = O.OracleProblem(p).bound(p.root_box(), kinds, vids, widths, n)
    assert np.array_equal(fe, ofe) and bits_equal(lb, olb)


@pytest.mark.parametrize("precision", ["fp64", "fp32", "lazy"])
@pytest.mark.parametrize("bits,parents", [(1, 3), (3, 33), (5, 20)])
def test_solver_iterations(precision, bits, parents):
    for p in (mixed_problem(), G.qcqp(G.QCQPSpec(n=9, m=3, n_int=2, int_lb=0, int_ub=6, rhs=(1.0, 3.0)), 77)):
        compare(p, 9, bisection_budget=bits, batch_parents=parents, frontier_cap=500, precision=precision)


def flat_problem() -> Problem:
    """An objective with few values: most points tie, so the FP32 bounds leave
    many of a tile's points to FP64."""
    p = Problem()
    x = [p.int_var(0.0, 3.0), p.var(-2.0, 2.0), p.var(-1.0, 1.0)]
    p.set_objective(x[0] + 2.0 * (x[0] * x[0]))
    p.add_constraint(x[1] * x[1] + x[2] * x[2] + 0.5 * (x[1] * x[2]), A.CMP_LE, 3.0)
    return p


def equality_problem() -> Problem:
    """An == chain that integer points meet exactly, beside a <= chain."""
    p = Problem()
    x = [p.int_var(-3.0, 4.0) for _ in range(4)] + [p.var(-2.0, 2.0)]
    p.set_objective(x[0] * x[1] - 2.0 * (x[2] * x[4]) + x[3] * x[3])
    p.add_constraint(2.0 * (x[0] * x[2]) + 1.0 * x[1], A.CMP_EQ, 3.0)
    p.add_constraint(x[4] * x[4] + 0.5 * (x[0] * x[4]), A.CMP_LE, 2.0)
    return p


@pytest.mark.parametrize("bits,points", [(1, 1), (4, 3), (6, 1), (9, 2), (12, 1)])
def test_sampled_candidates(bits, points):
    for p in (G.miqcqp_n32(3), G.qcqp_n4(2), mixed_problem(), flat_problem(), equality_problem(),
              G.qcqp(G.QCQPSpec(n=7, m=0), 5)):
        kinds, vids, widths, _ = O.bisection_choose(p.root_box(), p.var_kinds, bits)
        n = int(np.prod(widths))
        c = Sampler(DeviceProblem(p), kinds, n, sample_points=points).sample(p.root_box(), vids, widths, 11)
        found, value, point, index = O.OracleProblem(p).sample(p.root_box(), kinds, vids, widths, n, points, 11)
        assert c.found == found and (not found or (c.value == value and bits_equal(c.point, point) and c.index == index))


@pytest.mark.parametrize("bits,points", [(2, 1), (3, 2), (5, 1)])
def test_solver_samples(bits, points):
    # fathomed integer boxes (exact points, admissibility) among sampled ones
    for p in (flat_problem(), equality_problem()):
        compare(p, 8, bisection_budget=bits, batch_parents=40, frontier_cap=600, sample_points=points)


@pytest.mark.parametrize("bits,parents", [(2, 400), (3, 64), (3, 65), (4, 32), (4, 33), (5, 17), (4, 1300)])
def test_few_and_many_siblings(bits, parents):
    # both sides of the child counts where the objective's values are shared
    compare(G.miqcqp_n32(4), 7, bisection_budget=bits, batch_parents=parents, frontier_cap=6000)


@pytest.mark.parametrize("bits", [8, 10, 13, 14, 15])
def test_few_and_many_regions(bits):
    test_role_regions(bits)


def long_problem(n: int = 12, readers: bool = False) -> Problem:
    """An objective of more than 64 terms and <= chains of its length; with
    `readers` an == chain and a root shared by the objective and a check."""
    rng = np.random.default_rng(n)
    p = Problem()
    x = [p.int_var(-3.0, 6.0) if i % 5 == 4 else p.var(-4.0, 4.0) for i in range(n)]

    def chain():
        acc = float(rng.normal()) * x[0]
        for i in range(n):
            for j in range(i, n):
                t = x[i] * x[j]
                acc = acc - t if (i + j) % 7 == 3 else acc + float(rng.normal()) * t
        return acc

    obj = chain()
    p.set_objective(obj)
    p.add_constraint(chain(), A.CMP_LE, 20.0)
    p.add_constraint(chain(), A.CMP_LE, 35.0)
    if readers:
        p.add_constraint(obj, A.CMP_LE, 300.0)
        p.add_constraint(x[4] + 2.0 * x[9] - x[0] * x[1], A.CMP_EQ, 1.0)
    return p


OUTSIDE = [0.0, -0.0, 1e-300, 1e-20, 5e-324, 1e13, 1e30, 1e200, np.inf, -np.inf]


def outside_boxes(p: Problem, value: float):
    rng = np.random.default_rng(7)
    lo, hi = random_boxes(p, 200, rng, 0.3)
    at = rng.integers(0, lo.shape[0], 40), rng.integers(0, 200, 40)
    lo[at] = np.minimum(value, hi[at])
    both = rng.random(40) < 0.5
    hi[at[0][both], at[1][both]] = np.maximum(value, lo[at[0][both], at[1][both]])
    return lo, hi


@pytest.mark.parametrize("value", OUTSIDE)
def test_bounds_outside_the_filter_range_by_lane_groups(value):
    # programs long enough for lane groups on both objective bounds
    for p in (long_problem(), long_problem(readers=True)):
        check(p, *outside_boxes(p, value))


@pytest.mark.parametrize("value", OUTSIDE)
def test_fp32_bounds_outside_the_fast_range(value):
    for p in (mixed_problem(), near_problem(0.25), long_problem()):
        lo, hi = outside_boxes(p, value)
        g = eval_boxes(DeviceProblem(p), lo, hi, A.PRECISION_FP32_SCREEN)
        o = O.OracleProblem(p).eval_boxes(lo, hi, A.PRECISION_FP32_SCREEN)
        assert np.array_equal(g[2], o[2])
        assert bits_equal(g[0], o[0]) and bits_equal(g[1], o[1])


def outside_problem(n: int = 10) -> Problem:
    """Variables whose bounds leave the fast ranges at either end beside
    ordinary ones, so that parents inside and outside share a tile."""
    p = Problem()
    x = [p.var(-3e12, 3e12), p.var(-1e-14, 2e-14), p.int_var(0.0, 5.0)] + [p.var(-2.0, 3.0) for _ in range(n - 3)]
    obj = 1e-12 * (x[0] * x[3]) + 3.0 * (x[1] * x[4]) - x[2] * x[5]
    for i in range(3, n - 1):
        obj = obj + 0.5 * (x[i] * x[i + 1])
    p.set_objective(obj)
    p.add_constraint(1e-12 * x[0] + x[3] * x[4] - 2.0 * x[2], A.CMP_LE, 4.0)
    p.add_constraint(x[5] * x[5] + 1e11 * (x[1] * x[6]), A.CMP_LE, 6.0)
    return p


@pytest.mark.parametrize("precision", ["fp64", "fp32", "lazy"])
@pytest.mark.parametrize("bits,parents", [(2, 31), (4, 70)])
def test_solver_outside_the_fast_range(precision, bits, parents):
    compare(outside_problem(), 9, bisection_budget=bits, batch_parents=parents, frontier_cap=900, precision=precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32", "lazy"])
@pytest.mark.parametrize("bits,parents", [(1, 40), (3, 65), (5, 33)])
def test_solver_other_readers(precision, bits, parents):
    compare(long_problem(readers=True), 8, bisection_budget=bits, batch_parents=parents, frontier_cap=2000,
            precision=precision)


def chain_problem(n: int, terms: int, constraints: int, equalities: int = 0, shared: bool = False) -> Problem:
    """Chains of about `terms` products each."""
    rng = np.random.default_rng(100 * n + terms)
    p = Problem()
    x = [p.var(-4.0, 4.0) for _ in range(n)]

    def chain():
        acc = float(rng.normal()) * x[0]
        for _ in range(terms):
            i, j = rng.integers(0, n, 2)
            acc = acc + float(rng.normal()) * (x[i] * x[j])
        return acc

    obj = chain()
    p.set_objective(obj)
    for k in range(constraints):
        p.add_constraint(chain(), A.CMP_EQ if k < equalities else A.CMP_LE, 3.0 + k)
    if shared:
        p.add_constraint(obj, A.CMP_LE, 5.0)
    return p


# shapes that change the path with the number of boxes: no constraint, short
# and long ones, equalities, a root with two readers
PATHS = [(2, 2, 0), (3, 12, 0), (6, 70, 0), (2, 2, 1), (4, 12, 1), (6, 25, 3), (9, 60, 2), (4, 10, 2, 1),
         (6, 30, 6, 5), (5, 60, 3, 1), (6, 25, 4, 0, True), (40, 20, 1), (40, 70, 0)]


@pytest.mark.parametrize("boxes", [511, 2049, 8191, 10240, 16385, 40000, 98304, 131072])
def test_either_path(boxes):
    for shape in PATHS:
        p = chain_problem(*shape)
        if boxes > 20000 and p.n_vars > 6:
            continue
        rng = np.random.default_rng(boxes)
        lo, hi = random_boxes(p, boxes, rng, 0.3)
        dp, op = DeviceProblem(p), O.OracleProblem(p)
        for precision in (A.PRECISION_FP64, A.PRECISION_FP32_SCREEN):
            g, o = eval_boxes(dp, lo, hi, precision), op.eval_boxes(lo, hi, precision)
            assert np.array_equal(g[2], o[2])
            assert bits_equal(g[0], o[0]) and bits_equal(g[1], o[1])
            # the lower bound alone
            lb, fe = np.empty(boxes), np.empty(boxes, dtype=np.uint8)
            status(lib().cmn_eval_boxes(dp.handle, precision, A.ptr(lo), A.ptr(hi), boxes, boxes, A.ptr(lb), None,
                                        A.ptr(fe), 0, None))
            assert np.array_equal(fe, o[2]) and bits_equal(lb, o[0])


@pytest.mark.parametrize("bits", [6, 13, 14, 16])
def test_either_path_of_regions(bits):
    for shape in PATHS:
        p = chain_problem(*shape)
        kinds, vids, widths, _ = O.bisection_choose(p.root_box(), p.var_kinds, bits)
        n = int(np.prod(widths))
        b, op = Bounder(DeviceProblem(p), kinds, n), O.OracleProblem(p)
        fe, lb = b.bound(p.root_box(), vids, widths)
        ofe, olb = op.bound(p.root_box(), kinds, vids, widths, n)
        assert np.array_equal(fe, ofe) and bits_equal(lb, olb)
        clb, cub, cfe = b.bound_children(p.root_box(), vids, widths, 4)
        olb, oub, ofe = op.aggregate_bound(p.root_box(), kinds, vids, widths, n, 4)
        assert np.array_equal(cfe, ofe) and bits_equal(clb, olb) and bits_equal(cub, oub)


@pytest.mark.parametrize("n,constraints", [(150, 1), (150, 4), (400, 0), (400, 2)])
def test_tiles_of_many_variables(n, constraints):
    # few tiles fit an SM: boxes of one wave and of several, on either path
    rng = np.random.default_rng(n)
    p = Problem()
    x = [p.var(-4.0, 4.0) for _ in range(n)]

    def chain(products):
        acc = float(rng.normal()) * x[0]
        for i in range(n):
            t = x[i] * x[int(rng.integers(0, n))] if products else x[i]
            acc = acc + float(rng.normal()) * t
        return acc

    p.set_objective(chain(True))
    for k in range(constraints):
        p.add_constraint(chain(k % 2 == 1), A.CMP_LE, 4.0)
    dp, op = DeviceProblem(p), O.OracleProblem(p)
    for boxes in (700, 24000):
        lo, hi = random_boxes(p, boxes, rng, 0.2)
        for precision in (A.PRECISION_FP64, A.PRECISION_FP32_SCREEN):
            g, o = eval_boxes(dp, lo, hi, precision), op.eval_boxes(lo, hi, precision)
            assert np.array_equal(g[2], o[2])
            assert bits_equal(g[0], o[0]) and bits_equal(g[1], o[1])
