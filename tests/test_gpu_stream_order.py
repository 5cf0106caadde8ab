"""Calls in a row on one stream, each of which reads what the last one wrote
and overwrites its input: a launch may start while the previous kernel still
runs, and must read nothing before that kernel has ended.  Inputs are read
straight from HBM in one build and staged in the other, on sizes from a few
CTAs (every launch of the row fits on the GPU at once) to many."""

import numpy as np
import pytest

from polymage_b200.compiler import buildPipeline
from polymage_b200.constructs import (Float, Function, Image, Int, Interval,
                                      Max, Min, Parameter, Variable)

R, C = Parameter(Int, "R"), Parameter(Int, "C")
x, y = Variable(Int, "x"), Variable(Int, "y")


def _build(option):
    """out = the average of the 4 neighbours, clamped at the edges."""
    img = Image(Float, "img", [R, C])
    dom = [Interval(Int, 0, R - 1), Interval(Int, 0, C - 1)]
    f = Function(([x, y], dom), Float, "f")
    s = img(Max(x - 1, 0), y) + img(Min(x + 1, R - 1), y) + \
        img(x, Max(y - 1, 0)) + img(x, Min(y + 1, C - 1))
    f.defn = [s * 0.25]
    return buildPipeline([f], param_estimates=[(R, 500), (C, 500)],
                         tile_sizes=[16, 64], pipe_name="order_" + option,
                         options=[option])


@pytest.mark.parametrize("option", ["no_stage", "stage_pointwise"])
def test_kernels_wait_before_they_name_their_arrays(option):
    src = _build(option).generate_code().source
    body = src[src.index("_g0_body("):]
    assert body.index("pm_grid_dep_wait();") < body.index("__restrict__")


@pytest.mark.gpu
@pytest.mark.parametrize("option", ["no_stage", "stage_pointwise"])
@pytest.mark.parametrize("rows,cols", [(16, 64), (61, 203), (256, 1024),
                                       (1500, 2049)])
def test_ping_pong(option, rows, cols, cuda):
    import torch
    cp = _build(option).build()
    prm = {'R': rows, 'C': cols}
    img = np.random.default_rng(rows).random((rows, cols)).astype(
        np.float32)
    a, b = torch.from_numpy(img).to(cuda), torch.zeros(
        rows, cols, device=cuda)
    steps = 40
    for _ in range(steps):
        cp.run_dev(prm, {'img': a}, {'f': b})
        a, b = b, a
    torch.cuda.synchronize()
    cp.check()
    ref = img.astype(np.float64)
    for _ in range(steps):
        p = np.pad(ref, 1, mode='edge')
        ref = (p[:-2, 1:-1] + p[2:, 1:-1] + p[1:-1, :-2] + p[1:-1, 2:]) / 4
    # each step rounds three float32 sums of values below 4, and averages
    assert np.abs(a.cpu().numpy() - ref).max() <= steps * 2 ** -23
