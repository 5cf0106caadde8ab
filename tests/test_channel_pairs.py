"""Two-channel stages whose channels are interleaved in shared memory,
read by the forms that know the layout and by those that do not: the
kernels of small pipelines run on the CPU (tests/emulate.py, which refuses
misaligned and out-of-bounds accesses) against the point-by-point
evaluation of their definitions."""

import numpy as np
import pytest

from polymage_b200.apps import catalog
from polymage_b200.compiler import buildPipeline
from polymage_b200.constructs import (Cast, Float, Function, Image, Int,
                                      Interval, Parameter, UInt, Variable)
from tests import emulate
from tests.dsl_eval import Evaluator

R, C = Parameter(Int, "R"), Parameter(Int, "C")
x, y, c = (Variable(Int, n) for n in "xyc")
ROWS, COLS = Interval(Int, 1, R), Interval(Int, 1, C)
CH = Interval(Int, 0, 1)


def _filtered(typ):
    """A two-channel stage that is kept in shared memory."""
    img = Image(typ, "img", [2, R + 4, C + 4])
    f = Function(([c, x, y], [CH, Interval(Int, 0, R + 2),
                              Interval(Int, 0, C + 2)]), typ, "f")
    f.defn = [img(c, x, y) + 2 * img(c, x + 1, y + 1)]
    return img, f


def _build(out, name, tile, *options):
    p = buildPipeline([out], param_estimates=[(R, 500), (C, 500)],
                      tile_sizes=list(tile), pipe_name=name,
                      options=['inline_budget=0'] + list(options))
    f, = [n for g in p.groups for n in g.plan.nodes if n.name == "f"]
    assert f.role == 'smem'
    return p, f


def _check(p, inputs, sizes, tmp_path):
    prm = {'R': sizes[0], 'C': sizes[1]}
    got = emulate.run(p, prm, inputs, tmp_path)
    ev = Evaluator(prm, inputs)
    for out in p.ordered_params()[2]:
        ref = ev.array(out)
        # float32 sums of at most six products of values below 3
        assert np.abs(got[out.name] - ref).max() <= 32 * 2.0 ** -23


def test_data_dependent_channel(tmp_path):
    img, f = _filtered(Float)
    m = Image(Int, "m", [R + 4, C + 4])
    g = Function(([x, y], [ROWS, COLS]), Float, "g")
    ch = Cast(Int, m(x, y))
    g.defn = [f(ch, x - 1, y) + f(ch, x + 1, y)]
    p, _ = _build(g, "pairs_dd", (16, 64), 'stage_pointwise')
    rng = np.random.default_rng(1)
    _check(p, {'img': rng.random((2, 41, 94)).astype(np.float32),
               'm': rng.integers(0, 2, (41, 94)).astype(np.int32)},
           (37, 90), tmp_path)


def _binned(typ, bins=6):
    img = Image(typ, "img", [2, R + 4, C + 4, bins])
    z = Variable(Int, "z")
    f = Function(([c, x, y, z], [CH, Interval(Int, 0, R + 2), Interval(
        Int, 0, C + 2), Interval(Int, 0, bins - 1)]), typ, "f")
    f.defn = [img(c, x, y, z) + img(c, x + 1, y + 1, z)]
    m = Image(Int, "m", [R + 4, C + 4])
    return f, Cast(Int, m(x, y))


def _binned_inputs(sizes, scale, dt, bins=6):
    rng = np.random.default_rng(3)
    shape = (sizes[0] + 4, sizes[1] + 4)
    return {'img': (rng.random((2,) + shape + (bins,)) * scale).astype(dt),
            'm': rng.integers(0, bins, shape).astype(np.int32)}


def test_tiles_of_one_channel(tmp_path):
    """Tiles of channel 1 read only that channel of the stage: its region
    does not start at the domain's first one."""
    f, k = _binned(Float)
    g = Function(([c, x, y], [CH, ROWS, COLS]), Float, "g")
    g.defn = [f(c, x - 1, y, k) + f(c, x + 1, y, k) +
              f(1, x, y - 1, k) * f(1, x, y + 1, k)]
    p, n = _build(g, "pairs_tile", (1, 8, 32))
    assert n.ext[0] == 2 and not n.pairs
    _check(p, _binned_inputs((17, 50), .25, np.float32), (17, 50), tmp_path)


@pytest.mark.parametrize("typ", [Float, Int, UInt])
def test_types(typ, tmp_path):
    """Interleaved channels of every 4-byte type: both channels of a
    data-dependent bin."""
    f, k = _binned(typ)
    g = Function(([x, y], [ROWS, COLS]), typ, "g")
    g.defn = [f(0, x, y, k) + 3 * f(1, x, y, k) + f(0, x - 1, y, k)]
    p, n = _build(g, "pairs_" + typ.c_type_name(), (8, 32))
    assert n.pairs == (typ is not UInt)
    flt = typ is Float
    _check(p, _binned_inputs((17, 50), .25 if flt else 50, np.float32 if flt
                             else np.int64), (17, 50), tmp_path)


def test_only_gathered_stages_are_interleaved():
    """A row filter of two channels reads 16-byte vectors of each channel;
    the bilateral grid's slicing gathers pairs, and its blurs pass them
    on."""
    img, f = _filtered(Float)
    g = Function(([c, x, y], [CH, ROWS, COLS]), Float, "g")
    g.defn = [f(c, x, y - 1) + 2 * f(c, x, y) + f(c, x, y + 1)]
    p, n = _build(g, "pairs_rows", (16, 64), 'channel_tile_all')
    assert n.ext[0] == 2 and not n.pairs
    src = p.generate_code().source
    assert "const float4*>(&sm_f" in src and "float2" not in src
    p = dict(catalog.default_builds())["bilateral"]()
    assert [n.name for q in p.groups for n in getattr(q.plan, 'nodes', [])
            if n.in_smem and n.pairs] == ["blury", "blurx", "blurz"]
