"""Stages whose Cases are no boxes -- conditions on data, on remainders, on
two variables, alternatives -- and boxed ones read at a data-dependent
index: they run in blocks like any other stage, every part evaluated and
the last one that holds taken.  Kernels run on the CPU against the
definitions."""

import numpy as np
import pytest

from polymage_b200.compiler import buildPipeline
from polymage_b200.constructs import (Case, Cast, Condition, Float, Function,
                                      Image, Int, Interval, Parameter,
                                      Variable)
from tests import emulate
from tests.dsl_eval import Evaluator

R, C = Parameter(Int, "R"), Parameter(Int, "C")
x, y, z = (Variable(Int, n) for n in "xyz")


def _cond(v, op, k):
    return Condition(v, op, k)


CASES = {
    "data": lambda a: [Case(_cond(a(x, y), ">", 0.5), a(x, y - 1) + 1),
                       Case(_cond(a(x, y), "<=", 0.3), a(x + 1, y))],
    "parity": lambda a: [
        Case(_cond(x % 2, "==", 0) & _cond(y % 2, "==", 0), a(x, y + 1)),
        Case(_cond(x % 2, "==", 1) & _cond(y % 2, "==", 0), a(x - 1, y)),
        Case(_cond(y % 2, "==", 1) & _cond(x, ">=", 9), a(x + 1, y - 1))],
    "or": lambda a: [Case(_cond(x, ">=", 9) | _cond(y, ">=", 30),
                          a(x - 1, y) + 2),
                     Case(_cond(x, "<", 5), a(x, y + 1))],
    "diagonal": lambda a: [Case(_cond(x, ">=", y), a(x, y - 1)),
                           Case(_cond(x, "<", y - 3), a(x, y + 1) * 3)],
    "plain last": lambda a: [a(x, y) + a(x, y + 1)],
}


def _build(case, opts):
    img = Image(Float, "img", [R, C])
    a = Function(([x, y], [Interval(Int, 0, R - 2), Interval(
        Int, 0, C - 1)]), Float, "a")
    a.defn = [(img(x, y) + img(x + 1, y)) * 0.5]
    b = Function(([x, y], [Interval(Int, 1, R - 3), Interval(
        Int, 1, C - 2)]), Float, "b")
    b.defn = CASES[case](a)
    g = Function(([x, y], [Interval(Int, 2, R - 4), Interval(
        Int, 2, C - 3)]), Float, "g")
    g.defn = [b(x, y - 1) + b(x + 1, y) + b(x - 1, y)]
    return buildPipeline([g, b], param_estimates=[(R, 500), (C, 500)],
                         tile_sizes=[8, 32], pipe_name="forms_" +
                         case.replace(' ', '_'), options=list(opts))


@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("opts", [(), ('inline_budget=0',)])
def test_parts_that_are_no_boxes(case, opts, tmp_path):
    p = _build(case, opts)
    src = p.generate_code().source
    body = src[src.index("_body("):src.index("extern \"C\" __global__")]
    assert body.count("const bool pm_fbox") == sum(
        len(g.plan.steps) for g in p.groups) > 1
    prm = {'R': 31, 'C': 74}
    inputs = {'img': np.random.default_rng(6).random((31, 74)).astype(
        np.float32)}
    got = emulate.run(p, prm, inputs, tmp_path, fill=0)
    ev = Evaluator(prm, inputs)
    for out in p.ordered_params()[2]:
        # float32 sums of three values below 4
        assert np.abs(got[out.name] - ev.array(out)).max() <= \
            8 * 16 * 2.0 ** -24


def test_boxed_case_at_a_data_dependent_index(tmp_path):
    """A stage in registers, defined on some bins and read at any: no tile
    can drop its Case, and none goes point by point for it."""
    img, idx = Image(Float, "grid", [R, C, 8]), Image(Int, "idx", [R, C])
    dom = [Interval(Int, 0, R - 1), Interval(Int, 0, C - 1)]
    f = Function(([x, y, z], dom + [Interval(Int, 0, 7)]), Float, "f")
    f.defn = [Case(_cond(z, ">=", 2) & _cond(z, "<=", 5),
                   img(x, y, z) + 1)]
    g = Function(([x, y], dom), Float, "g")
    g.defn = [f(x, y, Cast(Int, idx(x, y)))]
    p = buildPipeline([g], param_estimates=[(R, 500), (C, 500)],
                      tile_sizes=[8, 32], pipe_name="forms_bins")
    src = p.generate_code().source
    assert [n.role for n in p.groups[-1].plan.nodes if n.name == "f"] == \
        ['inline']
    inside = src[src.index("const bool pm_inside = "):]
    assert "r_f_lo2" not in inside[:inside.index(";")]
    rng = np.random.default_rng(7)
    inputs = {'grid': rng.random((13, 70, 8)).astype(np.float32),
              'idx': rng.integers(0, 8, (13, 70)).astype(np.int32)}
    prm = {'R': 13, 'C': 70}
    got = emulate.run(p, prm, inputs, tmp_path)["g"]
    # one float32 sum below 2
    assert np.abs(got - Evaluator(prm, inputs).array(g)).max() <= 2.0 ** -23
