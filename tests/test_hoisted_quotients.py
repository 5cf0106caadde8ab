"""Quotients of parameters that a launch carries precomputed: computed in
their own precision."""

import numpy as np

from polymage_b200.compiler import buildPipeline
from polymage_b200.constructs import (Double, Float, Function, Image,
                                      Int, Interval, Parameter, Variable)
from polymage_b200.expr_ast import Value
from tests import emulate

R, C = Parameter(Int, "R"), Parameter(Int, "C")
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


def test_the_solvers_quotients_are_still_precomputed():
    from polymage_b200.apps import catalog
    src = dict(catalog.default_builds())["jacobi2d"]().generate_code().source
    assert "D.h_0 = (double)" in src
