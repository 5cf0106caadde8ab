"""Kernel parameters of launches that stand for several groups: the
estimate that bounds them covers what a launch carries, and only groups
without a dependence share one."""

import subprocess

import pytest

from polymage_b200 import codegen
from polymage_b200.apps import catalog
from polymage_b200.compiler import buildPipeline
from polymage_b200.constructs import (Double, Float, Function, Image, Int,
                                      Interval, Parameter, Variable)
from polymage_b200.expr_ast import Value
from polymage_b200.pipe import body_refs
from tests import emulate

R, C = Parameter(Int, "R"), Parameter(Int, "C")
x, y = Variable(Int, "x"), Variable(Int, "y")
DOM = [Interval(Int, 0, R - 1), Interval(Int, 0, C - 1)]


def _quotients(n):
    """A stage that multiplies by ``n`` different quotients of h."""
    h = Parameter(Float, "h")
    img = Image(Double, "img", [R, C])
    f = Function(([x, y], DOM), Double, "f")
    e = img(x, y)
    for i in range(n):
        e = e * (Value(float(i + 1), Double) / h)
    f.defn = [e]
    return buildPipeline([f], param_estimates=[(R, 50), (C, 50), (h, 1)],
                         tile_sizes=[8, 32], pipe_name="quotients")


@pytest.mark.parametrize("build", [
    lambda: _quotients(40), dict(catalog.default_builds())["jacobi2d"],
    dict(catalog.default_builds())["harris"]])
def test_the_estimate_covers_a_launch(build, tmp_path, monkeypatch):
    gens = []
    init = codegen.StencilGen.__init__

    def record(self, *args):
        init(self, *args)
        gens.append(self)
    monkeypatch.setattr(codegen.StencilGen, "__init__", record)
    src = emulate._device_source(build().generate_code().source)
    src += "int main() { return %s ? 0 : 1; }\n" % " && ".join(
        "sizeof(%s_launch) <= %d" % (g.k, codegen._launch_param_bytes(g))
        for g in gens)
    (tmp_path / "a.cpp").write_text(src)
    exe = str(tmp_path / "a.exe")
    subprocess.run(["g++", "-O0", "-w", "-std=c++17", "-I", emulate.CUDA_INC,
                    str(tmp_path / "a.cpp"), "-o", exe,
                    "-Wl,--unresolved-symbols=ignore-all"], check=True)
    assert subprocess.run([exe]).returncode == 0


def _chain(n):
    """n stages, each of which reads the one before."""
    prev = Image(Float, "img", [R, C])
    for i in range(n):
        f = Function(([x, y], DOM), Float, "f%d" % i)
        f.defn = [prev(x, y) + 1]
        prev = f
    return buildPipeline([prev], param_estimates=[(R, 500), (C, 500)],
                         tile_sizes=[8, 32], group_size=1,
                         pipe_name="chain_of_groups",
                         options=['merge_launches'])


def test_a_chain_of_groups_keeps_its_launches():
    p = _chain(4)
    mod = p.generate_code()
    assert not mod.meta.get('merges')
    assert mod.meta['launches'] == len(p.groups) == 4


def test_no_merged_group_reads_another_of_its_launch():
    """Dependences from the definitions themselves."""
    from polymage_b200.apps.harris import build_harris
    p = build_harris(tile_sizes=(32, 64), group_size=3,
                     options=('merge_launches',))
    mod = p.generate_code()
    assert mod.meta['merges']
    made = dict(("pm_harris_g%d" % g.level_time,
                 [c.func for c in g.comps]) for g in p.groups)
    for run in mod.meta['merges']:
        for k in run:
            reads = [r.objectRef for f in made[k] for r in body_refs(f)]
            for other in run:
                assert other == k or not any(
                    r is f for r in reads for f in made[other])
