"""Stages defined on the inner bins of a dimension of constant extent and
read at any of them: the loops leave out the bins that the Case does not
cover, which hold 0, and every covered bin has to be computed -- also those
that the unconditional form does not reach, because a clamp binds there or
a stage evaluated in registers has another Case.  Kernels run on the CPU
against the point-by-point evaluation of the definitions."""

import numpy as np
import pytest

from polymage_b200.compiler import buildPipeline
from polymage_b200.constructs import (Case, Cast, Condition, Float, Function,
                                      Image, Int, Interval, Min, Parameter,
                                      Variable)
from tests import emulate
from tests.dsl_eval import Evaluator

BINS = 16
R, C = Parameter(Int, "R"), Parameter(Int, "C")
x, y, z = (Variable(Int, n) for n in "xyz")


def _case(lo, hi, expr):
    return [Case(Condition(z, ">=", lo) & Condition(z, "<=", hi), expr)]


def _bound_clamp(grid, dom):
    """A clamp that binds inside the covered bins."""
    return _case(2, 13, grid(x, y, Min(z + 1, 10)) + grid(x, y, z) + 5)


def _narrower_inline(grid, dom):
    """A stage in registers whose Case covers fewer bins."""
    a = Function(([x, y, z], dom), Float, "a")
    a.defn = _case(4, 9, grid(x, y, z) * 2)
    return _case(2, 13, a(x, y, z) + 5)


def _inline_before(grid, dom):
    a = Function(([x, y, z], dom), Float, "a")
    a.defn = _case(1, 12, grid(x, y, z) * 2)
    return _case(2, 13, a(x, y, z - 2) + a(x, y, z + 1))


@pytest.mark.parametrize("defn", [_bound_clamp, _narrower_inline,
                                  _inline_before])
@pytest.mark.parametrize("rows,cols", [(9, 21)])
def test_every_covered_bin_is_computed(defn, rows, cols, tmp_path):
    grid = Image(Float, "grid", [R, C, BINS])
    idx = Image(Int, "idx", [R, C])
    dom = [Interval(Int, 0, R - 1), Interval(Int, 0, C - 1),
           Interval(Int, 0, BINS - 1)]
    f = Function(([x, y, z], dom), Float, "f")
    f.defn = defn(grid, dom)
    g = Function(([x, y], dom[:2]), Float, "g")
    g.defn = [f(x, y, Cast(Int, idx(x, y))) + f(x, y, 3)]
    p = buildPipeline([g], param_estimates=[(R, 500), (C, 500)],
                      tile_sizes=[8, 16], pipe_name="cov" + defn.__name__,
                      options=[('materialize', ['f'])])
    n, = [n for q in p.groups for n in q.plan.nodes if n.name == "f"]
    assert n.role == 'smem'
    rng = np.random.default_rng(rows)
    inputs = {'grid': rng.random((rows, cols, BINS)).astype(np.float32),
              'idx': rng.integers(0, BINS, (rows, cols)).astype(np.int32)}
    prm = {'R': rows, 'C': cols}
    got = emulate.run(p, prm, inputs, tmp_path)["g"]
    ref = Evaluator(prm, inputs).array(g)
    # float32 sums of at most six values below 8
    assert np.abs(got - ref).max() <= 6 * 16 * 2.0 ** -24
