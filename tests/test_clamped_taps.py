"""Taps whose index is clamped, and indices that divide: the region that a
tile keeps of a producer has to hold what its points read, also where the
bounds of a clamp are not the edges of the producer's domain.  Kernels run
on the CPU (tests/emulate.py) against the point-by-point evaluation of the
definitions; shared memory that no loop or copy wrote reads as NaN."""

import numpy as np
import pytest

from polymage_b200.compiler import buildPipeline
from polymage_b200.constructs import (Case, Condition, Float, Function,
                                      Image, Int, Interval, Max, Min,
                                      Parameter, Variable)
from tests import emulate
from tests.dsl_eval import Evaluator

BINS = 12
R, C, M = (Parameter(Int, n) for n in "RCM")
x, y, z = (Variable(Int, n) for n in "xyz")


def _run(out, inputs, prm, tmp_path, tile, name, options=(), est=500):
    """One device call against the definition; the plan's nodes."""
    p = buildPipeline([out], param_estimates=[
        (q, prm[q.name] if q is M else est) for q in (R, C, M)
        if q.name in prm], tile_sizes=list(tile), pipe_name=name,
        options=list(options))
    got = emulate.run(p, prm, inputs, tmp_path)[out.name]
    ref = Evaluator(prm, inputs).array(out)
    # float32 sums of at most eight values below 2
    assert np.abs(got - ref).max() <= 8 * 16 * 2.0 ** -24
    return dict((n.name, n) for g in p.groups for n in g.plan.nodes)


def _grid(f_of):
    """A stage of BINS bins in shared memory, read at ``f_of(f)``."""
    img = Image(Float, "img", [R, C, BINS])
    dom = [Interval(Int, 0, R - 1), Interval(Int, 0, C - 1),
           Interval(Int, 0, BINS - 1)]
    f = Function(([x, y, z], dom), Float, "f")
    f.defn = [img(x, y, z) + 1]
    g = Function(([x, y, z], dom), Float, "g")
    g.defn = [f_of(f)]
    return g


BIN_TAPS = {
    "max": lambda f: f(x, y, Max(z - 1, 4)) + f(x, y, Max(z - 2, 4)),
    "min": lambda f: f(x, y, Min(z + 1, 6)) + f(x, y, Min(z, 5)),
    "both": lambda f: f(x, y, Min(Max(z - 2, 3), 7)) + f(x, y, Max(z, 2)),
    "row": lambda f: f(x, y, Min(x, 3)) + f(x, y, Min(x + 1, 3)),
    "column": lambda f: f(x, y, Min(y / 8, 4)) + f(x, y, Min(y / 4, 5)),
    "scales": lambda f: f(x, y, Min(z, 5)) + f(x, y, Min(2 * z, 9)),
    "parameter": lambda f: f(x, y, Min(z, M)) + f(x, y, Max(z, M)),
}


@pytest.mark.parametrize("taps", sorted(BIN_TAPS))
@pytest.mark.parametrize("role", ["smem", "stage"])
@pytest.mark.parametrize("tile", [(8, 16, BINS), (8, 16, 5)])
def test_clamps_in_a_dimension_of_constant_extent(taps, role, tile,
                                                  tmp_path):
    g = _grid(BIN_TAPS[taps])
    prm = {'R': 11, 'C': 45}
    if taps == "parameter":
        prm['M'] = 7
    rng = np.random.default_rng(1)
    _run(g, {'img': rng.random((11, 45, BINS)).astype(np.float32)}, prm,
         tmp_path, tile, "bin_" + taps,
         [('materialize', ['f'])] if role == 'smem' else
         ['inline_budget=100000', 'stage_pointwise'])
