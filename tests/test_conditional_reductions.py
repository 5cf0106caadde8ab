"""Sums whose parts read under a condition: the pixel that gives a value or
a bin may lie outside the image where the condition does not hold.  Every
form of the sum runs on the CPU, which refuses reads outside a buffer."""

import numpy as np
import pytest

from polymage_b200.compiler import buildPipeline
from polymage_b200.constructs import (Case, Cast, Condition, Double, Float,
                                      Function, Image, Int, Interval, Max,
                                      Min, Op, Parameter, Reduce, Reduction,
                                      Variable)
from tests import emulate
from tests.dsl_eval import Evaluator

R, C = Parameter(Int, "R"), Parameter(Int, "C")
x, y, i, j, b = (Variable(Int, n) for n in "xyijb")
BINS = 6


@pytest.mark.parametrize("form,k,opts", [
    ("cells", 8, ()), ("privatized", 8, ('no_cells',)),
    ("atomics", 8, ('no_cells', 'no_privatize')), ("other cells", 5, ())])
@pytest.mark.parametrize("bins", ["all", "low"])
def test_reads_stay_under_their_condition(form, k, opts, bins, tmp_path):
    img, idx = Image(Float, "img", [R, C]), Image(Int, "idx", [R, C])
    dom = [Interval(Int, 0, R / k + 1), Interval(Int, 0, C / 8 + 1),
           Interval(Int, 0, BINS - 1)]
    h = Reduction(([i, j, b], dom), ([x, y], [
        Interval(Int, 0, R - 1), Interval(Int, 0, C - 1)]), Float, "h")
    cond = Condition(x, "<=", R - 2) & Condition(y, ">=", 1)
    if bins == "low":
        cond = cond & Condition(b, "<=", 2)
    h.defn = [Case(cond, Reduce(h(x / k, y / 8, Cast(Int, idx(x + 1, y - 1))),
                                img(x + 1, y - 1), Op.Sum))]
    h.default = 0
    g = Function(([i, j, b], dom), Float, "g")
    g.defn = [h(i, j, b) + 1]
    p = buildPipeline([g], param_estimates=[(R, 500), (C, 500)],
                      tile_sizes=[16, 64], pipe_name="cond_red",
                      options=list(opts))
    rows, cols = 21, 45
    rng = np.random.default_rng(k)
    inputs = {'img': rng.random((rows, cols)).astype(np.float32),
              'idx': rng.integers(-1, BINS + 1, (rows, cols)).astype(
                  np.int32)}
    got = emulate.run(p, {'R': rows, 'C': cols}, inputs, tmp_path)["g"]
    ref = np.ones(got.shape)
    X, Y = np.mgrid[0:rows - 1, 1:cols]
    z = inputs['idx'][1:, :-1]
    ok = (z >= 0) & (z < (3 if bins == "low" else BINS))
    np.add.at(ref, (X[ok] // k, Y[ok] // 8, z[ok]),
              inputs['img'][1:, :-1][ok].astype(np.float64))
    # float32 sums of at most 64 values below 1
    assert np.abs(got - ref).max() <= 64 * 64 * 2.0 ** -24


TARGETS = {
    "row bin": lambda v, w: (v / 8, w / 8, Min(v / 8, 3)),
    "low rows": lambda v, w: (Min(v / 8, 1), w / 8, 2),
    "last row": lambda v, w: (Min(v / 5, R / 8), w / 8, 2),
    "first rows": lambda v, w: (Max(v / 8 - 1, 0), w / 8, 2),
}


@pytest.mark.parametrize("target", sorted(TARGETS))
@pytest.mark.parametrize("opts", [(), ('no_privatize',)])
def test_clamped_targets(target, opts, tmp_path):
    """Targets with a clamped index: a tile near the clamp adds into more
    cells than one far from it."""
    img = Image(Float, "img", [R, C])
    dom = [Interval(Int, 0, R / 8 + 1), Interval(Int, 0, C / 8 + 1),
           Interval(Int, 0, BINS - 1)]
    h = Reduction(([i, j, b], dom), ([x, y], [
        Interval(Int, 0, R - 1), Interval(Int, 0, C - 1)]), Float, "h")
    h.defn = [Reduce(h(*TARGETS[target](x, y)), img(x, y), Op.Sum)]
    h.default = 0
    g = Function(([i, j, b], dom), Float, "g")
    g.defn = [h(i, j, b) + 1]
    p = buildPipeline([g], param_estimates=[(R, 30), (C, 500)],
                      tile_sizes=[16, 64], pipe_name="clamp_red",
                      options=list(opts))
    prm = {'R': 30, 'C': 45}
    inputs = {'img': np.random.default_rng(7).random((30, 45)).astype(
        np.float32)}
    got = emulate.run(p, prm, inputs, tmp_path)["g"]
    ref = Evaluator(prm, inputs).array(g)
    # float32 sums of at most 240 values below 1
    assert np.abs(got - ref).max() <= 240 * 240 * 2.0 ** -24


@pytest.mark.parametrize("typ,bins,threads,taken", [
    (Float, 60, 1024, False), (Double, 64, 512, False),
    (Double, 64, 256, False), (Double, 64, 128, True),
    (Float, 64, 256, True), (Float, 28, 1024, True)])
def test_cells_fit_an_sm(typ, bins, threads, taken):
    """Per-thread bins that an SM cannot hold, or only for few threads,
    leave the sum to the atomic form."""
    img, idx = Image(typ, "img", [R, C]), Image(Int, "idx", [R, C])
    h = Reduction(([i, j, b], [Interval(Int, 0, R / 8), Interval(
        Int, 0, C / 8), Interval(Int, 0, bins - 1)]), ([x, y], [
            Interval(Int, 0, R - 1), Interval(Int, 0, C - 1)]), typ, "h")
    h.defn = [Case(Condition(b, ">=", 0), Reduce(
        h(x / 8, y / 8, Cast(Int, idx(x, y))), img(x, y), Op.Sum))]
    h.default = 0
    p = buildPipeline([h], param_estimates=[(R, 500), (C, 500)],
                      tile_sizes=[16, 256], pipe_name="cell_fit",
                      options=['threads=%d' % threads])
    plan = p.groups[0].plan
    assert (plan.cells is not None) == taken
    assert plan.smem_bytes <= 227 * 1024 and plan.smem_bytes > 0
