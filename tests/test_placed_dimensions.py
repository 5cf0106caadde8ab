"""Dimensions of constant extent that lie at a place given by parameters
(``[R, R + 5]``): tiles, regions and buffers follow the parameters of the
call.  Kernels run on the CPU against the definitions."""

import numpy as np
import pytest

from polymage_b200.compiler import buildPipeline
from polymage_b200.constructs import (Case, Condition, Float, Function,
                                      Image, Int, Interval, Max, Parameter,
                                      Variable)
from tests import emulate
from tests.dsl_eval import Evaluator

R, C = Parameter(Int, "R"), Parameter(Int, "C")
x, y = Variable(Int, "x"), Variable(Int, "y")
PLACED, COLS = Interval(Int, R, R + 5), Interval(Int, 0, C - 1)


def _outer(img):
    f = Function(([x, y], [PLACED, COLS]), Float, "f")
    f.defn = [img(x - R, y) + 1]
    g = Function(([x, y], [PLACED, COLS]), Float, "g")
    g.defn = [Case(Condition(x, "<=", R + 4), f(x, y) + f(x + 1, Max(
        y - 1, 0)) + f(x, Max(y - 2, 0)))]
    return g


def _inner(img):
    f = Function(([y, x], [COLS, PLACED]), Float, "f")
    f.defn = [img(x - R, y) + 1]
    g = Function(([y, x], [COLS, PLACED]), Float, "g")
    g.defn = [f(y, x) + f(Max(y - 1, 0), R + 1) + f(Max(y - 2, 0), R)]
    return g


@pytest.mark.parametrize("defn", [_outer, _inner])
@pytest.mark.parametrize("opts", [('inline_budget=0',),
                                  ('inline_budget=100000',),
                                  ('inline_budget=0', ('materialize',
                                                       ['f']))])
@pytest.mark.parametrize("rows", [0, 21])
def test_values_at_their_place(defn, opts, rows, tmp_path):
    g = defn(Image(Float, "img", [6, C]))
    p = buildPipeline([g], param_estimates=[(R, 500), (C, 500)],
                      tile_sizes=[4, 16], pipe_name="placed" +
                      defn.__name__, options=list(opts))
    img = np.random.default_rng(rows).random((6, 45)).astype(np.float32)
    prm = {'R': rows, 'C': 45}
    got = emulate.run(p, prm, {'img': img}, tmp_path, fill=0)["g"]
    ref = Evaluator(prm, {'img': img}).array(g)
    # float32 sums of three values below 2
    assert np.abs(got - ref).max() <= 4 * 8 * 2.0 ** -24


@pytest.mark.parametrize("opts", [('fuse_all',), ()])
def test_live_out_across_a_dimension_of_bins(opts, tmp_path):
    """A plane and a volume of bins: the plane's columns lie along the bins
    of the volume's tiles, which are fewer."""
    img = Image(Float, "img", [R, C])
    z = Variable(Int, "z")
    rows = Interval(Int, 1, R - 2)
    f = Function(([x, y], [Interval(Int, 0, R - 1), COLS]), Float, "f")
    f.defn = [img(x, y) + 1]
    f2 = Function(([x, y], [rows, COLS]), Float, "f2")
    f2.defn = [f(x - 1, y) + f(x + 1, y)]
    g2 = Function(([x, y], [rows, Interval(Int, 1, C - 2)]), Float, "g2")
    g2.defn = [f2(x, y - 1) + f2(x, y + 1)]
    g3 = Function(([x, y, z], [rows, COLS, Interval(Int, 0, 4)]), Float,
                  "g3")
    g3.defn = [img(x - 1, y) * z + img(x + 1, y)]
    p = buildPipeline([g2, g3], param_estimates=[(R, 500), (C, 500)],
                      tile_sizes=[2, 8, 32], pipe_name="plane_volume",
                      options=list(opts) + ['inline_budget=0'])
    prm = {'R': 13, 'C': 45}
    inputs = {'img': np.random.default_rng(4).random((13, 45)).astype(
        np.float32)}
    got = emulate.run(p, prm, inputs, tmp_path, fill=0)
    ev = Evaluator(prm, inputs)
    for g in (g2, g3):
        # float32 sums of products below 10
        assert np.abs(got[g.name] - ev.array(g)).max() <= 4 * 16 * 2.0 ** -24


@pytest.mark.parametrize("rows", [9, 40, 43])
@pytest.mark.parametrize("rblock", [2, 4])
def test_rows_that_start_at_a_parameter(rows, rblock, tmp_path):
    """Tiles start at R / 4 + 5: the row that a block starts at has no
    known remainder, so the halves of its index do not fold."""
    img = Image(Float, "img", [R + 8, C + 8])
    cols = Interval(Int, 4, 2 * C - 4)
    f = Function(([x, y], [Interval(Int, 2, 2 * R), cols]), Float, "f")
    f.defn = [img(x / 2 - 1, y / 2) + img(x / 2, y / 2)]
    g = Function(([x, y], [Interval(Int, R / 4 + 5, 3 * R),
                           Interval(Int, 8, 3 * C)]), Float, "g")
    g.defn = [f(x / 2, y / 2) + f(x / 2 + 1, y / 2 + 1) +
              f(x / 2, y / 2 + 1)]
    p = buildPipeline([g], param_estimates=[(R, 500), (C, 500)],
                      tile_sizes=[16, 32], pipe_name="start_rows",
                      options=['inline_budget=0', 'rblock=%d' % rblock])
    prm = {'R': rows, 'C': 25}
    inputs = {'img': np.random.default_rng(rows).random(
        (rows + 8, 33)).astype(np.float32)}
    got = emulate.run(p, prm, inputs, tmp_path)["g"]
    # float32 sums of six values below 1
    assert np.abs(got - Evaluator(prm, inputs).array(g)).max() <= \
        8 * 8 * 2.0 ** -24
