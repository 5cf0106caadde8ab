"""Taps whose index is clamped, and indices that divide: the region that a
tile keeps of a producer has to hold what its points read, also where the
bounds of a clamp are not the edges of the producer's domain.  Kernels run
on the CPU (tests/emulate.py) against the point-by-point evaluation of the
definitions; shared memory that no loop or copy wrote reads as NaN."""

import ctypes
import subprocess

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
def test_clamps_in_a_dimension_of_constant_extent(taps, role, tmp_path):
    g = _grid(BIN_TAPS[taps])
    tile = (8, 16, 5 if role == 'smem' else BINS)
    prm = {'R': 11, 'C': 45}
    if taps == "parameter":
        prm['M'] = 7
    rng = np.random.default_rng(1)
    _run(g, {'img': rng.random((11, 45, BINS)).astype(np.float32)}, prm,
         tmp_path, tile, "bin_" + taps,
         [('materialize', ['f'])] if role == 'smem' else
         ['inline_budget=100000', 'stage_pointwise'])


def _rows(taps, cond=None, lo=0, hi=R - 1):
    """A filter of two images' rows, the second through shared memory."""
    img = Image(Float, "img", [R, C])
    dom = [Interval(Int, lo, hi), Interval(Int, 0, C - 1)]
    f = Function(([x, y], [Interval(Int, 0, R - 1), dom[1]]), Float, "f")
    f.defn = [img(x, y) + 1]
    g = Function(([x, y], dom), Float, "g")
    e = taps(f)
    g.defn = [e] if cond is None else [Case(cond, e)]
    return g


def _img(rows, cols):
    return {'img': np.random.default_rng(rows).random(
        (rows, cols)).astype(np.float32)}


# bounds off the producer's edges by a literal, by a parameter, and taps
# whose bounds differ; x / 2 and x * 2 with them; indices that run down
ROW_TAPS = {
    "literal": (lambda f: f(Min(x + 1, 20), y) + f(Min(x + 2, 20), y), {}),
    "literals": (lambda f: f(Max(x - 1, 9), y) + f(Min(x + 1, 20), y), {}),
    "crop": (lambda f: f(Min(Max(x - 1, M), R - 1 - M), y) +
             f(Min(Max(x + 1, M), R - 1 - M), y), {'M': 8}),
    "crop_far": (lambda f: f(Min(Max(x - 1, M), R - 1 - M), y) +
                 f(Min(Max(x + 1, M), R - 1 - M), y), {'M': 30}),
    "one_sided": (lambda f: f(Max(x - 1, M), y) +
                  f(Min(x + 1, R - 1 - M), y), {'M': 8}),
    "one_sided_8": (lambda f: f(Max(x - 1, 8), y) + f(Min(x + 1, R - 9), y),
                    {}),
    "one_sided_2": (lambda f: f(Max(x - 1, 2), y) + f(Min(x + 1, R - 3), y),
                    {}),
    "edges": (lambda f: f(Max(x - 1, 0), y) + f(Min(x + 1, R - 1), y), {}),
    "one_tap": (lambda f: f(Max(x - 9, 0), y) + f(Max(x - 8, 0), y), {}),
    "columns": (lambda f: f(x, Max(y - 3, M)) + f(x, Min(y, C - M)),
                {'M': 2}),
    "half": (lambda f: f(Min(Max(x / 2 - 1, M), R - 1), y) +
             f(Min(x / 2 + 1, R - 1), y), {'M': 3}),
    "twice": (lambda f: f(Min(2 * x, R - 1 - M), y) +
              f(Min(2 * x + 1, R - 1 - M), y), {'M': 1}),
    "down": (lambda f: f(Max(R - 1 - M - x, 0), y) +
             f(Max(R - 2 - M - x, 0), y), {'M': 3}),
    "quotient": (lambda f: f(Max((x - 3) / 2, 0), y) +
                 f(Max((x - 1) / 2, 0), y), {}),
}


@pytest.mark.parametrize("taps", sorted(ROW_TAPS))
@pytest.mark.parametrize("role", ["smem", "stage"])
def test_clamps_inside_the_domain(taps, role, tmp_path):
    e, prm = ROW_TAPS[taps]
    rows, cols = (97, 21) if role == 'smem' else (97, 70)
    _run(_rows(e), _img(rows, cols), dict(prm, R=rows, C=cols), tmp_path,
         (16, 32), "row_" + taps,
         [('materialize', ['f'])] if role == 'smem' else
         ['inline_budget=100000', 'stage_pointwise'])


@pytest.mark.parametrize("taps", ["quotient", "half", "one_sided_2",
                                  "edges", "crop", "twice"])
@pytest.mark.parametrize("tile", [(1, 32), (3, 48)])
def test_thin_tiles(taps, tile, tmp_path):
    """Tiles of a few rows: a tap rounded towards zero or clamped easily
    lies outside what the tile's other taps read."""
    e, prm = ROW_TAPS[taps]
    _run(_rows(e), _img(37, 50), dict(prm, R=37, C=50), tmp_path, tile,
         "thin_" + taps, ['inline_budget=0', 'stage_pointwise'])


def test_negative_numerators_without_a_clamp(tmp_path):
    """(x - 3) / 2 at x = 2 is 0, which rounding down would miss."""
    g = _rows(lambda f: f((x - 3) / 2, y) + f((x - 3) / 2, Max(y - 1, 0)),
              lo=2)
    for tile in ((1, 32), (4, 16)):
        _run(g, _img(21, 40), {'R': 21, 'C': 40}, tmp_path, tile,
             "negative%d" % tile[0], ['inline_budget=0', 'stage_pointwise'])


def test_negative_domains(tmp_path):
    """Tiles whose numerators are all negative."""
    img = Image(Float, "img", [R, C])
    cols = Interval(Int, 0, C - 1)
    f = Function(([x, y], [Interval(Int, -20, R - 21), cols]), Float, "f")
    f.defn = [img(x + 20, y) + 1]
    g = Function(([x, y], [Interval(Int, 0, 2 * R - 50), cols]), Float, "g")
    g.defn = [f((x - 35) / 2, y) + f((x - 35) / 2, Max(y - 1, 0))]
    for tile in ((4, 32), (3, 16)):
        _run(g, _img(33, 40), {'R': 33, 'C': 40}, tmp_path, tile,
             "negdom%d" % tile[0], ['inline_budget=0', 'stage_pointwise'])


@pytest.mark.parametrize("opts", [(), ('no_fold_clamps',),
                                  ('shared_regions',)])
def test_crops_of_several_stages(opts, tmp_path):
    """A chain of cropped stages, one of them an output too, and a second
    consumer with the same crop."""
    def crop(v, hi):
        return Min(Max(v, M), hi - 1 - M)
    img = Image(Float, "img", [R, C])
    dom = [Interval(Int, 0, R - 1), Interval(Int, 0, C - 1)]
    fs = []
    for n in "fgh":
        fs.append(Function(([x, y], dom), Float, n))
    f, g, h = fs
    f.defn = [img(crop(x - 1, R), y) + img(crop(x + 1, R), crop(y, C))]
    g.defn = [Case(Condition(x, ">=", 3), f(crop(x + 2, R), y) +
                   f(crop(x - 2, R), y))]
    h.defn = [g(x, crop(y - 1, C)) + g(x, crop(y + 1, C)) +
              f(crop(x, R), y)]
    prm = {'R': 45, 'C': 71, 'M': 6}
    inputs = _img(45, 71)
    for outs in ([h], [h, g]):
        p = buildPipeline(outs, param_estimates=[(R, 500), (C, 500), (M, 6)],
                          tile_sizes=[8, 16], pipe_name="crops%d" % len(outs),
                          options=['inline_budget=0'] + list(opts))
        got = emulate.run(p, prm, inputs, tmp_path, fill=0)
        ev = Evaluator(prm, inputs)
        for o in outs:
            # float32 sums of at most ten values below 1
            assert np.abs(got[o.name] - ev.array(o)).max() <= \
                10 * 16 * 2.0 ** -24


def test_edge_clamps_keep_their_stages():
    """Clamps at the producer's edges, or at most a tap's offset inside
    them, move no region; a crop moves it; taps that may lie anywhere apart
    keep a stage out of the tile."""
    for taps, moved in (("edges", False), ("literal", True),
                        ("crop", True), ("one_sided_8", True),
                        ("one_sided", None), ("literals", None)):
        e, prm = ROW_TAPS[taps]
        p = buildPipeline(
            [_rows(e)], param_estimates=[(R, 500), (C, 500)] +
            ([(M, 8)] if prm else []), tile_sizes=[16, 32],
            pipe_name="keep_" + taps, options=['inline_budget=0'])
        n = [n for q in p.groups for n in q.plan.nodes if n.name == "f" and
             n.role != 'out']
        assert [bool(q.moved) if q.in_smem else None for q in n] == [moved]


@pytest.mark.parametrize("opts", [('no_stage',), ('stage_pointwise',)])
@pytest.mark.parametrize("crop", [5, 60])
def test_bands_copy_what_their_tiles_read(opts, crop, tmp_path):
    """The host entry copies a prefix of each input before a band of tiles
    runs: the footprint function has to cover the clamped rows, also those
    far from the band."""
    img = Image(Float, "img", [R, C])
    g = Function(([x, y], [Interval(Int, 0, R - 1), Interval(
        Int, 0, C - 1)]), Float, "g")

    def at(v):
        return img(Min(Max(v, M), R - 1 - M), y)
    g.defn = [at(x - 1) + at(x + 1)]
    p = buildPipeline([g], param_estimates=[(R, 500), (C, 500), (M, 5)],
                      tile_sizes=[16, 32], pipe_name="bands%d" % crop,
                      options=list(opts))
    src = p.generate_code().source
    k = "pm_bands%d_g0" % crop
    body = src[src.index("static void %s_footprint(" % k):]
    body = body[body.index("{") + 1:body.index("\n}\n")]
    rows, cols = 150, 40
    (tmp_path / "fp.cpp").write_text("""
static int pm_imin(int a, int b) { return a < b ? a : b; }
static int pm_imax(int a, int b) { return a > b ? a : b; }
static int pm_floordiv(int a, int b) { int q = a / b; return (q * b != a &&
  ((a < 0) != (b < 0))) ? q - 1 : q; }
struct D_t { int p_R, p_C, p_M, glo[2], ghi[2], gn[2], tile_base; };
extern "C" void fp(const D_t* Dp, int tile, long long* in_end, int* a_lo,
                   int* a_hi) { const D_t& D = *Dp;
""" + body + "}\n")
    so = str(tmp_path / "fp.so")
    subprocess.run(["g++", "-O1", "-w", "-shared", "-fPIC",
                    str(tmp_path / "fp.cpp"), "-o", so], check=True)
    D = (ctypes.c_int * 10)(rows, cols, crop, 0, 0, rows - 1, cols - 1,
                            -(-rows // 16), -(-cols // 32), 0)
    end = (ctypes.c_longlong * 1)()
    lo, hi = (ctypes.c_int * 2)(), (ctypes.c_int * 2)()
    lib = ctypes.CDLL(so)
    for tile in range(D[7] * D[8]):
        lib.fp(D, tile, end, lo, hi)
        last = min(lo[0] + 15, rows - 1)
        need = max(min(max(v, crop), rows - 1 - crop)
                   for q in (lo[0], last) for v in (q - 1, q + 1))
        assert end[0] >= need * cols + hi[1] + 1, (tile, lo[0], end[0])
