"""Quotients of parameters that a launch carries precomputed: computed in
their own precision, and none whose evaluation on the host could trap."""

import numpy as np

from polymage_b200.compiler import buildPipeline
from polymage_b200.constructs import (Case, Condition, Double, Float,
                                      Function, Image, Int, Interval,
                                      Parameter, Variable)
from polymage_b200.expr_ast import Value
from tests import emulate

R, C, N, M = (Parameter(Int, n) for n in "RCNM")
h = Parameter(Float, "h")
x, y = Variable(Int, "x"), Variable(Int, "y")
DOM = [Interval(Int, 0, R - 1), Interval(Int, 0, C - 1)]


def _build(typ, defn, name, *prms):
    img = Image(typ, "img", [R, C])
    g = Function(([x, y], DOM), typ, "g")
    g.defn = defn(img)
    return buildPipeline([g], param_estimates=[(R, 50), (C, 50)] +
                         list(prms), tile_sizes=[8, 32], pipe_name=name)


def test_equal_texts_of_different_precision(tmp_path):
    """1.0 / h in float and in double print alike."""
    p = _build(Double, lambda img: [
        img(x, y) * (Value(1.0, Float) / h) +
        img(x, y) * (Value(1.0, Double) / h) * 3], "quot_types", (h, 3))
    img = np.random.default_rng(1).random((9, 40))
    got = emulate.run(p, {'R': 9, 'C': 40, 'h': 3.0}, {'img': img},
                      tmp_path)["g"]
    one, third = np.float64(np.float32(1) / np.float32(3)), 1 / 3.0
    # float64 rounding of four operations
    assert np.abs(got - (img * one + img * third * 3)).max() <= 4 * 2.0 ** -52


def test_integer_quotients_stay_in_their_case(tmp_path):
    """1.0 / (N / M) with M = 0 under a Case that does not hold."""
    p = _build(Float, lambda img: [
        Case(Condition(M, ">", 0), img(x, y) * (1.0 / (N / M))),
        Case(Condition(M, "<=", 0), img(x, y) + 2)], "quot_int",
        (N, 6), (M, 2))
    src = p.generate_code().source
    assert "h_0" not in src
    img = np.random.default_rng(2).random((9, 40)).astype(np.float32)
    for m, want in ((2, img / 3), (0, img + 2)):
        got = emulate.run(p, {'R': 9, 'C': 40, 'N': 6, 'M': m},
                          {'img': img}, tmp_path)["g"]
        assert np.abs(got - want).max() <= 2 * 2.0 ** -23


def test_the_solvers_quotients_are_still_precomputed():
    from polymage_b200.apps import catalog
    src = dict(catalog.default_builds())["jacobi2d"]().generate_code().source
    assert "D.h_0 = (double)" in src
