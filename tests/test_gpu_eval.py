"""Fused evaluator (a) on the GPU against the CPU oracle: bit-exact node
enclosures (signs of zero aside) in FP64 and in the FP32 screen, over
random, degenerate and zero-straddling boxes."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from cuminlp_gb300 import _abi as A
from cuminlp_gb300 import generators as G
from cuminlp_gb300._lib import check, lib
from cuminlp_gb300.problem import Problem
from cuminlp_gb300.solver import DeviceProblem, eval_boxes
from tests.conftest import bits_equal
from tests.gpu_common import ops_problem, random_boxes, with_objective

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from cuminlp_gb300 import build
    build.build_library()


def check_eval(problem, n_boxes, seed, precision, scale=0.2):
    rng = np.random.default_rng(seed)
    lo, hi = random_boxes(problem, n_boxes, rng, scale)
    dp = DeviceProblem(problem)
    glb, gub, gfe = eval_boxes(dp, lo, hi, precision)
    olb, oub, ofe = O.OracleProblem(problem).eval_boxes(lo, hi, precision)
    assert bits_equal(glb, olb), np.flatnonzero(glb != olb)[:10]
    assert bits_equal(gub, oub)
    assert np.array_equal(gfe, ofe)
    return glb, gub, gfe


@pytest.mark.parametrize("precision", [A.PRECISION_FP64, A.PRECISION_FP32_SCREEN])
@pytest.mark.parametrize("n_vars,boxes,seed", [(4, 20000, 101), (32, 3000, 102), (64, 600, 103)])
def test_eval_boxes_match_oracle(n_vars, boxes, seed, precision):
    p = G.BY_N[n_vars]()
    lb, ub, fe = check_eval(p, boxes, seed, precision)
    assert np.all(lb <= ub)
    if n_vars == 4:
        assert 0 < fe.sum() < len(fe)  # both verdicts occur


@pytest.mark.parametrize("precision", [A.PRECISION_FP64, A.PRECISION_FP32_SCREEN])
def test_every_operator_matches_oracle(precision):
    check_eval(ops_problem(), 20000, 7, precision, scale=0.5)


@pytest.mark.parametrize("precision", [A.PRECISION_FP64, A.PRECISION_FP32_SCREEN])
def test_node_enclosures_match_oracle(precision):
    # each sampled node of the n=32 MIQCQP as the objective: its enclosure on every
    # box must equal the oracle's node-by-node evaluation
    p = G.miqcqp_n32()
    rng = np.random.default_rng(5)
    cands = [n.id for n in p.graph.nodes if n.op not in (A.OP_CONST,)]
    picks = sorted(set(rng.choice(cands, 60, replace=False).tolist()) | {p.objective_root})
    lo, hi = random_boxes(p, 512, rng, 0.3)
    op = O.OracleProblem(p)
    box0 = np.stack([lo[:, 3], hi[:, 3]], 1).reshape(-1)
    nlo, nhi = op.eval_nodes(box0, fp32=precision == A.PRECISION_FP32_SCREEN)
    for nid in picks:
        q = with_objective(p, nid)
        glb, gub, _ = eval_boxes(DeviceProblem(q), lo, hi, precision)
        olb, oub, _ = O.OracleProblem(q).eval_boxes(lo, hi, precision)
        assert bits_equal(glb, olb) and bits_equal(gub, oub), nid
        # and the whole-DAG oracle agrees on box 3
        assert bits_equal(np.float64(nlo[nid]), glb[3]) and bits_equal(np.float64(nhi[nid]), gub[3])


def test_fp32_screen_contains_fp64():
    p = G.miqcqp_n64()
    rng = np.random.default_rng(11)
    lo, hi = random_boxes(p, 2000, rng, 0.05)
    dp = DeviceProblem(p)
    lb64, ub64, fe64 = eval_boxes(dp, lo, hi, A.PRECISION_FP64)
    lb32, ub32, fe32 = eval_boxes(dp, lo, hi, A.PRECISION_FP32_SCREEN)
    assert np.all(lb32 <= lb64) and np.all(ub32 >= ub64)
    assert np.all(fe32 >= fe64)  # the screen never excludes what FP64 keeps


def test_enclosure_contains_sampled_points():
    p = G.miqcqp_n32()
    rng = np.random.default_rng(3)
    lo, hi = random_boxes(p, 256, rng, 0.1)
    dp = DeviceProblem(p)
    lb, ub, _ = eval_boxes(dp, lo, hi)
    op = O.OracleProblem(p)
    for b in range(0, 256, 8):
        for _ in range(20):
            x = rng.uniform(lo[:, b], hi[:, b])
            obj, _ = op.eval_point(x)
            assert lb[b] <= obj <= ub[b]


@pytest.mark.parametrize("precision", [A.PRECISION_FP64, A.PRECISION_FP32_SCREEN])
def test_quotients_of_signed_zeros(precision):
    # every order of zeros, denormals and finite ends in the dividend, over
    # positive and negative divisors: the bounds' zeros keep the oracle's sign
    p = Problem()
    x, y = p.var(-2.0, 2.0), p.var(0.5, 4.0)
    p.set_objective(x / y)
    ends = np.array([-2.0, -5e-324, -0.0, 0.0, 5e-324, 1e-300, 3.0])
    divisors = np.array([-4.0, -0.5, -5e-324, 5e-324, 0.5, 4.0])
    lo, hi = [], []
    for a in ends:
        for b in ends:
            for c in divisors:
                for d in divisors:
                    if a <= b and c <= d and c * d > 0:
                        lo.append((a, c))
                        hi.append((b, d))
    lo, hi = np.array(lo).T.copy(), np.array(hi).T.copy()
    g = eval_boxes(DeviceProblem(p), lo, hi, precision)
    o = O.OracleProblem(p).eval_boxes(lo, hi, precision)
    for a, b in zip(g[:2], o[:2]):
        nan = np.isnan(a) & np.isnan(b)
        assert np.all(nan | (a.view(np.uint64) == b.view(np.uint64)))


@pytest.mark.parametrize("stride", [5, 6, (1 << 28) - 1, 1 << 28])
def test_host_planes_of_any_stride(stride):
    # a few boxes of planes up to 2 GiB apart (untouched memory between them)
    p = Problem()
    x, y = p.var(-2.0, 2.0), p.var(-3.0, 4.0)
    p.set_objective(x * y + 2.0 * x)
    p.add_constraint(x + y, A.CMP_LE, 1.0)
    lo, hi = random_boxes(p, 5, np.random.default_rng(1), 0.3)
    far = [np.empty(stride + 5), np.empty(stride + 5)]
    for f, b in zip(far, (lo, hi)):
        f[:5], f[stride:stride + 5] = b[0], b[1]
    lb, ub, fe = np.empty(5), np.empty(5), np.empty(5, dtype=np.uint8)
    dp = DeviceProblem(p)
    check(lib().cmn_eval_boxes(dp.handle, A.PRECISION_FP64, A.ptr(far[0]), A.ptr(far[1]), 5, stride, A.ptr(lb),
                               A.ptr(ub), A.ptr(fe), 0, None))
    o = O.OracleProblem(p).eval_boxes(lo, hi, A.PRECISION_FP64)
    assert bits_equal(lb, o[0]) and bits_equal(ub, o[1]) and np.array_equal(fe, o[2])
