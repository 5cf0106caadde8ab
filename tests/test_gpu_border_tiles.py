"""Border tiles on the GPU: sizes one below, at and one above the tile
sizes of the shipped builds, down to images smaller than a tile, with row
pitches that TMA can stage (multiples of 16 bytes) and that it cannot, and
an input whose base is 4 bytes past a 16-byte boundary.  A tile there runs
the unconditional code on the blocks inside its valid box and point by
point around it, over buffers whose layout does not depend on the border.

Oracles: the float64 restatements, with each pipeline's tolerance
(float32: rounding of tens of operations on values below 1; float64:
1e-10 relative)."""

import numpy as np
import pytest

import oracle.bilateral as OB
import oracle.harris as OH
import oracle.interpolate as OI
import oracle.jacobi as OJ
import oracle.multigrid as OM
import oracle.pyramid as OP
import oracle.unsharp as OU
from polymage_b200.apps import catalog

pytestmark = pytest.mark.gpu


def _run(name, params, inputs, cuda, shift=0):
    """Outputs of a device call; inputs ``shift`` elements past an aligned
    base."""
    import torch
    cp = catalog.build(name)
    ins = {}
    for k, a in inputs.items():
        t = torch.zeros(a.size + 8, dtype=torch.from_numpy(a[:0]).dtype,
                        device=cuda)
        v = t[shift:shift + a.size].view(a.shape)
        v.copy_(torch.from_numpy(a))
        ins[k] = v
    outs = dict((f.name, torch.zeros(
        cp.shape_of(f, params), dtype=torch.float64 if f.typ.size() == 8
        else torch.float32, device=cuda)) for f in cp.outputs)
    cp.run_dev(params, ins, outs)
    torch.cuda.synchronize()
    cp.check()
    return [outs[f.name].cpu().numpy() for f in cp.outputs]


@pytest.mark.parametrize("rows,cols,shift", [
    (4, 4, 0), (5, 7, 0), (35, 67, 0), (36, 68, 0), (36, 68, 1),
    (37, 69, 0), (67, 132, 0), (100, 64, 0)])
def test_harris(rows, cols, shift, cuda):
    img = OH.make_input(rows, cols, seed=rows + cols)
    out, = _run("harris", {'R': rows - 2, 'C': cols - 2}, {'img': img},
                cuda, shift)
    ref = OH.harris(img)
    assert np.abs(out - ref).max() <= 1e-5 * max(np.abs(ref).max(), 1e-30)


@pytest.mark.parametrize("rows,cols,shift", [
    (1, 1, 0), (3, 5, 0), (63, 127, 0), (64, 128, 0), (64, 128, 1),
    (65, 129, 0), (66, 132, 0), (67, 260, 0), (129, 254, 0)])
def test_unsharp(rows, cols, shift, cuda):
    img = OU.make_input(rows, cols, seed=rows + cols)
    thr = float(np.float32(0.001))
    out, = _run("unsharp", {'R': rows, 'C': cols, 'threshold': thr,
                            'weight': 3.0}, {'img': img}, cuda, shift)
    ref = OU.unsharp(img, thr, 3.0)
    # points within rounding of the threshold may take either arm
    near = OU.margin(img, thr) <= 1e-6
    assert np.abs(np.where(near, 0, out - ref)).max() <= 1e-5


@pytest.mark.parametrize("rows,cols,shift", [
    (31, 127, 0), (32, 128, 0), (32, 128, 1), (33, 129, 0), (40, 260, 0)])
def test_bilateral(rows, cols, shift, cuda):
    img = OB.make_input(rows, cols, seed=rows + cols)
    out, = _run("bilateral", {'rows': rows, 'cols': cols}, {'input': img},
                cuda, shift)
    assert np.abs(out - OB.bilateral(img)).max() <= 1e-5


@pytest.mark.parametrize("R,C,shift", [
    (8, 8, 0), (31, 63, 0), (32, 64, 0), (32, 64, 1), (33, 65, 0),
    (129, 191, 0)])
def test_pyramid8(R, C, shift, cuda):
    a, b, m = OP.make_inputs(R, C, seed=R + C)
    out, = _run("pyramid8", {'R': R, 'C': C},
                {'img1': a, 'img2': b, 'mask': m}, cuda, shift)
    assert np.abs(out - OP.pyramid_blend_clamped(a, b, m, L=8)).max() <= 2e-5


@pytest.mark.parametrize("R,C,shift", [
    (513, 512, 0), (512, 514, 1), (527, 577, 0)])
def test_interpolate(R, C, shift, cuda):
    img = OI.make_input(R, C, seed=R + C)
    out, = _run("interpolate", {'R': R, 'C': C}, {'img': img}, cuda, shift)
    assert np.abs(out - OI.interpolate(img)).max() <= 1e-5


def _close64(out, ref):
    assert np.abs(out - ref).max() <= 1e-10 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("N,shift", [(1, 0), (5, 0), (31, 0), (62, 0),
                                     (62, 1), (63, 0), (66, 0)])
def test_jacobi2d(N, shift, cuda):
    V, F = OJ.make_input(N, seed=N)
    out, = _run("jacobi2d", {'N': N}, {'V_': V, 'F_': F}, cuda, shift)
    _close64(out, OJ.jacobi2d(V, F, T=catalog.JACOBI2D['T']))


@pytest.mark.parametrize("N,shift", [(1, 0), (7, 0), (14, 0), (30, 1),
                                     (31, 0), (33, 0), (66, 0)])
def test_jacobi3d(N, shift, cuda):
    rng = np.random.default_rng(N)
    V, F = rng.random((N + 2,) * 3), rng.random((N + 2,) * 3)
    out, = _run("jacobi3d", {'N': N}, {'V_': V, 'F_': F}, cuda, shift)
    _close64(out, OJ.jacobi3d(V, F, T=catalog.JACOBI3D['T']))


@pytest.mark.parametrize("n,shift", [(1, 0), (3, 1), (7, 0), (9, 0)])
def test_vcycle3d(n, shift, cuda):
    kw = catalog.VCYCLE3D
    V, F = OM.make_input3d(n, L=kw['L'], seed=n)
    out, = _run("vcycle3d", {'n': n}, {'V_': V, 'F_': F}, cuda, shift)
    _close64(out, OM.v_cycle3d(V, F, n, L=kw['L'], nu1=kw['nu1'],
                               nu2=kw['nu2'], nuc=kw['nuc']))
