"""Sums over an image into grid cells with data-dependent bins, computed in
the grid-cell form (per-thread bins, one warp per cell): cell shapes other
than the bilateral grid's, images that end inside a cell, a warp and a
tile, values outside the bins, integer sums (exact) and float ones (each
cell at most 512 values below 1: |error| <= 512 * 2^-24 * 512)."""

import numpy as np
import pytest

from polymage_b200.compiler import buildPipeline
from polymage_b200.constructs import (Case, Cast, Condition, Float, Image,
                                      Int, Interval, Op, Parameter, Reduce,
                                      Reduction, Variable)

BINS = 6


def _build(k0, k1, typ, opts=()):
    R, C = Parameter(Int, "R"), Parameter(Int, "C")
    x, y = Variable(Int, "x"), Variable(Int, "y")
    c, i, j, b = (Variable(Int, n) for n in "cijb")
    img = Image(Float, "img", [R, C])
    name = "cells_%d_%d_%s" % (k0, k1, "f" if typ is Float else "i")
    h = Reduction(([c, i, j, b],
                   [Interval(Int, 0, 1), Interval(Int, 0, R / k0 + 1),
                    Interval(Int, 0, C / k1), Interval(Int, 0, BINS - 1)]),
                  ([x, y], [Interval(Int, 0, R - 1), Interval(Int, 0, C - 1)]),
                  typ, name)
    z = Cast(Int, img(x, y) * BINS)
    h.defn = [Case(Condition(c, "==", 0),
                   Reduce(h(0, x / k0 + 1, y / k1, z),
                          img(x, y) if typ is Float else 3, Op.Sum)),
              Case(Condition(c, "==", 1),
                   Reduce(h(1, x / k0 + 1, y / k1, z), 1, Op.Sum))]
    h.default = 0
    return buildPipeline([h], param_estimates=[(R, 100), (C, 300)],
                         tile_sizes=[16, 256], pipe_name=name,
                         options=list(opts))


@pytest.mark.parametrize("k0,k1", [(8, 8), (2, 32), (32, 2), (5, 16)])
@pytest.mark.parametrize("typ", [Float, Int])
def test_plans_take_the_cell_form(k0, k1, typ):
    plan = [g.plan for g in _build(k0, k1, typ).groups][0]
    assert plan.cells[0] == (k0, k1) and plan.tile[0] % k0 == 0
    plan = [g.plan for g in _build(k0, k1, typ, ["no_cells"]).groups][0]
    assert plan.cells is None


@pytest.mark.gpu
@pytest.mark.parametrize("k0,k1,typ", [(8, 8, Int), (2, 32, Int),
                                       (32, 2, Float), (5, 16, Float)])
def test_sums_match(k0, k1, typ, cuda):
    import torch
    cp = _build(k0, k1, typ).build()
    dt = np.float32 if typ is Float else np.int32
    for R, C in [(1, 1), (k0, k1), (k0 + 1, 33), (31, 257), (70, 255),
                 (64, 600)]:
        rng = np.random.default_rng(R * C)
        img = (rng.random((R, C)) * 1.2).astype(np.float32)
        out = torch.full((2, R // k0 + 2, C // k1 + 1, BINS), 7,
                         dtype=torch.from_numpy(np.zeros(0, dt)).dtype,
                         device=cuda)
        cp.run_dev({'R': R, 'C': C}, {'img': torch.from_numpy(img).to(cuda)},
                   {cp.outputs[0].name: out})
        torch.cuda.synchronize()
        cp.check()
        ref = np.zeros(out.shape)
        z = (img * np.float32(BINS)).astype(np.int64)
        X, Y = np.mgrid[0:R, 0:C]
        ok = z < BINS
        cell = (X[ok] // k0 + 1, Y[ok] // k1, z[ok])
        np.add.at(ref[0], cell, img[ok].astype(np.float64)
                  if typ is Float else 3)
        np.add.at(ref[1], cell, 1)
        err = np.abs(out.cpu().numpy() - ref).max()
        assert err <= (0 if typ is Int else 512 * 512 * 2.0 ** -24)
