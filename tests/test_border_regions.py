"""Regions of border tiles, from the generated code itself: the region
inference that each kernel's host twin (``<kernel>_footprint``) carries is
compiled for the CPU and run for every tile of small, odd-sized images.

A kernel's buffers have static extents, and its interior form relies on the
origins of regions having fixed residues modulo 4 (16-byte vector reads).
Regions are not clamped to the image along parametric dimensions, so both
have to hold on every tile: a region larger than its buffer would read or
write out of it, another residue would misalign a vector read."""

import ctypes
import re
import subprocess

import pytest

from polymage_b200.apps import catalog
from polymage_b200.codegen import StencilGen
from polymage_b200.evaluate import eval_int

CASES = [("harris", (61, 83)), ("unsharp", (37, 131)),
         ("campipe", (131, 197)), ("bilateral", (77, 93)),
         ("pyramid", (157, 211)), ("pyramid8", (37, 53)),
         ("pyramid8", (130, 257)), ("laplacian", (156, 188)),
         ("interpolate", (211, 157)), ("jacobi2d", (45, 0)),
         ("jacobi3d", (37, 0)), ("vcycle", (13, 0)), ("vcycle3d", (6, 0)),
         ("mg3p", (34, 0)), ("nlmeans", (37, 41))]


@pytest.mark.parametrize("name,sizes", CASES)
def test_regions_fit_their_buffers_on_every_tile(name, sizes, tmp_path,
                                                 monkeypatch):
    gens = []
    init = StencilGen.__init__

    def record(self, *args):
        init(self, *args)
        gens.append(self)
    monkeypatch.setattr(StencilGen, "__init__", record)
    p = dict(catalog.default_builds())[name]()
    src = p.generate_code().source
    env = p.int_env()
    for k in list(env):
        env[k] = sizes[1] if k.name in ('C', 'cols') else \
            sizes[0] if k.name in ('R', 'rows', 'N', 'n') else env[k]
    helpers = ("static int pm_imin(int a, int b) { return a < b ? a : b; }\n"
               "static int pm_imax(int a, int b) { return a > b ? a : b; }\n"
               "static int pm_floordiv(int a, int b) { int q = a / b; return "
               "(q * b != a && ((a < 0) != (b < 0))) ? q - 1 : q; }\n")
    text = [helpers]
    jobs = []
    for g in gens:
        plan = g.plan
        body = src[src.index("static void %s_footprint(" % g.k):]
        body = body[body.index("{") + 1:body.index("(void)t0;")]
        bufs = [n for n in plan.nodes if n.in_smem]
        if not bufs:
            continue
        prms = sorted(set(re.findall(r"= D\.(p_\w+);", body)))
        out = "".join("out[%d] = r_%s_lo%d; out[%d] = r_%s_hi%d;\n" % (
            2 * i, nm, d, 2 * i + 1, nm, d) for i, (nm, d) in enumerate(
                (g.node_name(n), d) for n in bufs for d in range(n.ndims)))
        text.append("struct D_%s { float %s; int glo[8], ghi[8], gn[8], "
                    "tile_base; };\n" % (g.k, ", ".join(prms + ["pad_"])))
        text.append('extern "C" void %s(const float* prm, const int* glo, '
                    "const int* ghi, const int* gn, int tile, int* out) {\n"
                    "D_%s D; D.tile_base = 0;\n" % (g.k, g.k))
        text += ["D.%s = prm[%d];\n" % (q, i) for i, q in enumerate(prms)]
        text.append("for (int d = 0; d < 8; ++d) { D.glo[d] = glo[d]; "
                    "D.ghi[d] = ghi[d]; D.gn[d] = gn[d]; }\n")
        text.append(body + "(void)t0;\n" + out + "}\n")
        jobs.append((g, bufs, prms))
    cpp = tmp_path / "regions.cpp"
    cpp.write_text("".join(text))
    so = str(tmp_path / "regions.so")
    subprocess.run(["g++", "-O1", "-w", "-shared", "-fPIC", str(cpp), "-o",
                    so], check=True)
    lib = ctypes.CDLL(so)
    values = dict(("p_" + k.name, v) for k, v in env.items())
    ints = ctypes.c_int * 8
    checked = 0
    for g, bufs, prms in jobs:
        plan = g.plan
        na = plan.anchor.ndims
        glo, ghi = [None] * na, [None] * na
        for n in plan.nodes:
            if n.role != 'out':
                continue
            for d, dom in enumerate(n.func.domain):
                k = d if n.func is plan.anchor else n.owned_map[d]
                a = eval_int(dom.lowerBound, env)
                b = eval_int(dom.upperBound, env)
                glo[k] = a if glo[k] is None else min(glo[k], a)
                ghi[k] = b if ghi[k] is None else max(ghi[k], b)
        gn = [(h - l + t) // t for l, h, t in zip(glo, ghi, plan.tile)]
        if min(gn) < 1:
            continue
        total = 1
        for v in gn:
            total *= v
        prm = (ctypes.c_float * (len(prms) + 1))(
            *[values.get(q, 1.0) for q in prms])
        g.inner_residues()
        nout = 2 * sum(n.ndims for n in bufs)
        out = (ctypes.c_int * nout)()
        for tile in range(total):
            getattr(lib, g.k)(prm, ints(*glo), ints(*ghi), ints(*gn), tile,
                              out)
            i = 0
            for n in bufs:
                for d in range(n.ndims):
                    lo, hi = out[i], out[i + 1]
                    i += 2
                    assert hi - lo + 1 <= n.ext[d], (g.k, n.name, d, lo, hi)
                r = g._loop_res.get(n.func)
                if r is not None:
                    assert lo % 4 == r, (g.k, n.name, lo, r)
            checked += 1
    assert checked > 0
