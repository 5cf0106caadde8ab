"""Live-outs that their readers need up to a point short of their domain's
end: computed that far, on every path.  Kernels run on the CPU against the
definitions."""

import numpy as np
import pytest

from polymage_b200.compiler import buildPipeline
from polymage_b200.constructs import (Case, Condition, Float, Function,
                                      Image, Int, Interval, Parameter,
                                      Variable)
from tests import emulate
from tests.dsl_eval import Evaluator

R, C = Parameter(Int, "R"), Parameter(Int, "C")
x, y = Variable(Int, "x"), Variable(Int, "y")


@pytest.mark.parametrize("cond", ["box", "data", "either"])
@pytest.mark.parametrize("opts", [(), ('guarded',), ('no_inside',)])
def test_coarse_half_of_a_fine_grid(cond, opts, tmp_path):
    img = Image(Float, "img", [2 * R + 2, 2 * C + 2])
    fine = [Interval(Int, 0, 2 * R), Interval(Int, 0, 2 * C)]
    f = Function(([x, y], fine), Float, "f")
    inner = Condition(x, "<=", R) & Condition(y, "<=", C)
    f.defn = [Case({"box": inner, "data": Condition(img(x, y), ">", 0.5),
                    "either": inner | Condition(x, "<=", 3)}[cond],
                   img(x, y) + img(x + 1, y + 1))]
    g = Function(([x, y], [Interval(Int, 1, R), Interval(Int, 1, C)]),
                 Float, "g")
    g.defn = [f(x, y) + f(x - 1, y) + f(x, y - 1)]
    p = buildPipeline([g], param_estimates=[(R, 100), (C, 100)],
                      tile_sizes=[8, 16], group_size=1,
                      pipe_name="need_" + cond, options=list(opts))
    rows, cols = 13, 35
    inputs = {'img': np.random.default_rng(3).random(
        (2 * rows + 2, 2 * cols + 2)).astype(np.float32)}
    prm = {'R': rows, 'C': cols}
    got = emulate.run(p, prm, inputs, tmp_path)["g"]
    ref = Evaluator(prm, inputs).array(g)
    # float32 sums of six values below 1
    assert np.abs(got - ref).max() <= 6 * 6 * 2.0 ** -24
