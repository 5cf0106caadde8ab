"""Timed workloads of the shipped pipelines.

Each case is one call of a shipped pipeline (``polymage_b200.apps.catalog``)
on device buffers, through ``CompiledPipeline.run_dev`` for one image and
``CompiledPipeline.run_batch`` for a batch of uneven images, as a program
that keeps its images on the GPU calls them:

* ``harris``, ``unsharp``, ``campipe``, ``bilateral``, ``pyramid8``,
  ``interpolate``: image processing, float32 (the camera pipe int16 raw to
  uint8 RGB, every byte computed in integers);
* ``jacobi2d``, ``jacobi3d``, ``vcycle3d``: time-iterated and multigrid
  solvers, float64.

A built library takes any size, so sizes range over what these programs
meet: thumbnails to 4096 x 4096, even and odd sides.  ``listed`` holds the
benchmark sizes of each pipeline, a small call and ragged ones; ``draw``
gives further sizes of the same pipelines.  ``exact`` restates each float
pipeline in plain torch, in float64.
"""

import math

import numpy as np
import torch

from polymage_b200.apps import catalog
from polymage_b200.apps.campipe import MATRIX_3200, MATRIX_7000

THRESHOLD = 0.001
WEIGHT = 3.0


def listed():
    return [
        # a thumbnail or a crop: the call's latency counts
        {"name": "harris_256", "app": "harris", "rows": 256, "cols": 256},
        # corner detection on one 4-megapixel frame
        {"name": "harris_2048", "app": "harris", "rows": 2048, "cols": 2048},
        # sharpening a full-HD frame after a crop: odd sides, rows that do
        # not start on 16 bytes
        {"name": "unsharp_1079x1917", "app": "unsharp", "rows": 1079,
         "cols": 1917},
        # sharpening a large photograph
        {"name": "unsharp_4096", "app": "unsharp", "rows": 4096,
         "cols": 4096},
        # one raw frame of a 5-megapixel sensor
        {"name": "campipe_1968x2592", "app": "campipe", "rows": 1968,
         "cols": 2592},
        # edge-preserving smoothing of one 4-megapixel frame
        {"name": "bilateral_1536x2560", "app": "bilateral", "rows": 1536,
         "cols": 2560},
        # an album: uneven images in one call
        {"name": "bilateral_batch24", "app": "bilateral_batch", "count": 24,
         "low": 512, "high": 2048, "sides_seed": 1},
        # blending two 4-megapixel photographs through 8 levels
        {"name": "pyramid8_2048", "app": "pyramid8", "rows": 2048,
         "cols": 2048},
        # filling the low-alpha pixels of an RGBA image, 10 levels
        {"name": "interpolate_2048", "app": "interpolate", "rows": 2048,
         "cols": 2048},
        # ten smoothing steps of a 2-D Poisson problem
        {"name": "jacobi2d_2048", "app": "jacobi2d", "n": 2048},
        # ten smoothing steps of a 3-D Poisson problem
        {"name": "jacobi3d_128", "app": "jacobi3d", "n": 128},
        # one multigrid V-cycle, finest grid 255^3
        {"name": "vcycle3d_255", "app": "vcycle3d", "n": 31},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


# sides of a drawn case, per pipeline
_RANGES = {
    "harris": (128, 4096),
    "unsharp": (128, 4096),
    "campipe": (160, 2592),
    "bilateral": (128, 2560),
    "pyramid8": (160, 2048),
    "interpolate": (160, 2048),
    "jacobi2d": (160, 2048),
    "jacobi3d": (32, 128),
    "vcycle3d": (8, 31),
}


def draw(rng):
    app = rng.choice(sorted(_RANGES) + ["bilateral_batch"])
    if app == "bilateral_batch":
        return {"app": app, "count": rng.randint(4, 24), "low": 256,
                "high": 2048, "sides_seed": rng.randint(0, 1 << 20)}
    low, high = _RANGES[app]
    if app in ("jacobi2d", "jacobi3d", "vcycle3d"):
        return {"app": app, "n": _log_int(rng, low, high)}
    rows = _log_int(rng, low, high)
    cols = min(high, max(low, int(round(rows * rng.uniform(0.6, 1.7)))))
    return {"app": app, "rows": rows, "cols": cols}


# ---- inputs -----------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(seed)
    return g


def _uniform(g, shape, dtype=torch.float32):
    return torch.rand(shape, generator=g, device=_device(), dtype=dtype)


def _photo(g, channels, rows, cols):
    """Smooth shading, object edges and sensor noise, in [0, 1)."""
    coarse = _uniform(g, (1, channels, rows // 64 + 2, cols // 64 + 2))
    shade = torch.nn.functional.interpolate(
        coarse, (rows, cols), mode="bilinear", align_corners=True)[0]
    blocks = _uniform(g, (1, channels, rows // 24 + 2, cols // 24 + 2))
    edges = torch.nn.functional.interpolate(blocks, (rows, cols))[0]
    noise = _uniform(g, (channels, rows, cols))
    return (0.55 * shade + 0.35 * edges + 0.0999 * noise).contiguous()


def _batch_sides(case):
    rng = np.random.default_rng(case["sides_seed"])
    sides = rng.integers(case["low"], case["high"] + 1, (case["count"], 2))
    return [(int(r), int(c)) for r, c in sides]


def _finest(n):
    """Points per side of the V-cycle's finest grid (3 levels above ``n``)."""
    return ((n + 1) << catalog.VCYCLE3D["L"]) - 1


def _inputs(case, seed):
    """(parameters, input tensors) of a single-image case."""
    g = _generator(seed)
    app = case["app"]
    if app == "harris":
        r, c = case["rows"], case["cols"]
        return {"R": r - 2, "C": c - 2}, {"img": _photo(g, 1, r, c)[0]}
    if app == "unsharp":
        r, c = case["rows"], case["cols"]
        img = torch.zeros((3, r + 4, c + 4), device=_device())
        img[:, 2:r + 2, 2:c + 2] = _photo(g, 3, r, c)
        return ({"R": r, "C": c, "threshold": THRESHOLD, "weight": WEIGHT},
                {"img": img})
    if app == "campipe":
        r, c = case["rows"], case["cols"]
        raw = (_photo(g, 1, r, c)[0] * 1024).to(torch.int16)
        # the colour matrices feed only a table, which the host computes
        return ({"R": r, "C": c, "colour_temp": 3700.0, "contrast": 50.0,
                 "gamma": 2.0},
                {"img": raw,
                 "matrix_3200": torch.tensor(MATRIX_3200,
                                             dtype=torch.float32),
                 "matrix_7000": torch.tensor(MATRIX_7000,
                                             dtype=torch.float32)})
    if app == "bilateral":
        r, c = case["rows"], case["cols"]
        return {"rows": r, "cols": c}, {"input": _photo(g, 1, r, c)[0]}
    if app == "pyramid8":
        r, c = case["rows"], case["cols"]
        return ({"R": r, "C": c},
                {"img1": _photo(g, 3, r, c), "img2": _photo(g, 3, r, c),
                 "mask": _photo(g, 1, r, c)[0]})
    if app == "interpolate":
        r, c = case["rows"], case["cols"]
        img = torch.zeros((4, r + 2, c + 2), device=_device())
        img[0:3, 1:r + 1, 1:c + 1] = _photo(g, 3, r, c)
        img[3, 1:r + 1, 1:c + 1] = 0.25 + 0.75 * _photo(g, 1, r, c)[0]
        return {"R": r, "C": c}, {"img": img}
    if app in ("jacobi2d", "jacobi3d"):
        n = case["n"]
        shape = (n + 2,) * (2 if app == "jacobi2d" else 3)
        return {"N": n}, {"V_": _uniform(g, shape, torch.float64),
                          "F_": _uniform(g, shape, torch.float64)}
    if app == "vcycle3d":
        shape = (_finest(case["n"]) + 2,) * 3
        return {"n": case["n"]}, {"V_": _uniform(g, shape, torch.float64),
                                  "F_": _uniform(g, shape, torch.float64)}
    raise ValueError(app)


def _batch_inputs(case, seed):
    g = _generator(seed)
    return [_photo(g, 1, r, c)[0] for r, c in _batch_sides(case)]


_DTYPES = {4: torch.float32, 8: torch.float64, 1: torch.uint8}


def _outputs(cp, params):
    return dict((f.name, torch.zeros(cp.shape_of(f, params),
                                     dtype=_DTYPES[f.typ.size()],
                                     device=_device()))
                for f in cp.outputs)


# ---- the measured calls -----------------------------------------------------
def prepare(case, seed):
    if case["app"] == "bilateral_batch":
        cp = catalog.build("bilateral")
        images = _batch_inputs(case, seed)
        params = [{"rows": im.shape[0], "cols": im.shape[1]}
                  for im in images]
        return {"pipeline": cp, "batch": True, "params": params,
                "inputs": [{"input": im} for im in images],
                "outputs": [_outputs(cp, p) for p in params]}
    cp = catalog.build(case["app"])
    params, inputs = _inputs(case, seed)
    return {"pipeline": cp, "batch": False, "params": params,
            "inputs": inputs, "outputs": _outputs(cp, params)}


def run(state):
    cp = state["pipeline"]
    if state["batch"]:
        cp.run_batch(state["params"], state["inputs"], state["outputs"])
    else:
        cp.run_dev(state["params"], state["inputs"], state["outputs"])
    return state["outputs"]


# floating-point operations per output point (multiplies, adds, compares),
# each stage evaluated once per point of its domain
_FLOPS = {"harris": 53, "unsharp": 72, "campipe": 0, "bilateral": 40,
          "pyramid8": 230, "interpolate": 70}


def work(case):
    app = case["app"]
    if app == "bilateral_batch":
        px = sum(r * c for r, c in _batch_sides(case))
        return {"bytes": 8 * px, "flops": 40 * px}
    if app in ("jacobi2d", "jacobi3d"):
        dims = 2 if app == "jacobi2d" else 3
        n = case["n"]
        steps = (catalog.JACOBI2D if dims == 2 else catalog.JACOBI3D)["T"]
        return {"bytes": 24 * (n + 2) ** dims,
                "flops": steps * (2 * dims + 5) * n ** dims}
    if app == "vcycle3d":
        n = _finest(case["n"])
        # smoothing steps and the defect on each level, a factor 8 apart
        per_point = 11 * (catalog.VCYCLE3D["nu1"] + 1) + 30
        return {"bytes": 24 * (n + 2) ** 3,
                "flops": int(per_point * n ** 3 * 8 / 7)}
    r, c = case["rows"], case["cols"]
    nbytes = {
        "harris": 8 * r * c,
        "unsharp": 12 * (r + 4) * (c + 4) + 12 * r * c,
        "campipe": 2 * r * c + 3 * (r - 48) * (c - 64) + 96,
        "bilateral": 8 * r * c,
        "pyramid8": 28 * r * c + 12 * r * c,
        "interpolate": 16 * (r + 2) * (c + 2) + 12 * r * c,
    }[app]
    return {"bytes": nbytes, "flops": _FLOPS[app] * r * c}


# ---- the same in plain torch, float64 ----------------------------------------
def exact(case, seed):
    app = case["app"]
    if app == "campipe":
        return None                      # bytes, computed in integers
    if app == "bilateral_batch":
        return [{"filtered": _exact_bilateral(im)}
                for im in _batch_inputs(case, seed)]
    _, ins = _inputs(case, seed)
    if app == "harris":
        return {"harris": _exact_harris(ins["img"].double())}
    if app == "unsharp":
        return {"mask": _exact_unsharp(ins["img"].double())}
    if app == "bilateral":
        return {"filtered": _exact_bilateral(ins["input"])}
    if app == "pyramid8":
        return {"blend": _exact_pyramid(ins["img1"].double(),
                                        ins["img2"].double(),
                                        ins["mask"].double(),
                                        catalog.PYRAMID8["L"])}
    if app == "interpolate":
        return {"interpolate": _exact_interpolate(ins["img"].double(), 10)}
    if app in ("jacobi2d", "jacobi3d"):
        dims = 2 if app == "jacobi2d" else 3
        kw = catalog.JACOBI2D if dims == 2 else catalog.JACOBI3D
        u = ins["V_"]
        for _ in range(kw["T"]):
            w = torch.zeros_like(u)
            _relax(w, u, ins["F_"])
            u = w
        return {"jacobi": u}
    if app == "vcycle3d":
        kw = catalog.VCYCLE3D
        return {kw["name"]: _exact_vcycle(ins["V_"], ins["F_"], kw["L"],
                                          kw["nu1"], True)}
    raise ValueError(app)


def _exact_harris(img):
    h, w = img.shape

    def at(a, dx, dy):
        return a[1 + dx:a.shape[0] - 1 + dx, 1 + dy:a.shape[1] - 1 + dy]

    def sobel(a):                        # derivative along the last axis
        return ((at(a, -1, 1) - at(a, -1, -1)) +
                2 * (at(a, 0, 1) - at(a, 0, -1)) +
                (at(a, 1, 1) - at(a, 1, -1))) / 12

    def box(a):
        return sum(at(a, dx, dy) for dx in (-1, 0, 1) for dy in (-1, 0, 1))

    iy = sobel(img)
    ix = sobel(img.t()).t()
    sxx, syy, sxy = box(ix * ix), box(iy * iy), box(ix * iy)
    trace = sxx + syy
    out = torch.zeros_like(img)
    out[2:h - 2, 2:w - 2] = sxx * syy - sxy * sxy - 0.04 * trace * trace
    return out


def _exact_unsharp(img):
    rows, cols = img.shape[1] - 4, img.shape[2] - 4
    taps = (1, 4, 6, 4, 1)
    # the column blur is defined on columns 1 .. cols, and reads 0 outside
    blurx = torch.zeros_like(img[:, 2:rows + 1])
    blurx[:, :, 1:cols + 1] = sum(
        t * img[:, k:rows - 1 + k, 1:cols + 1]
        for k, t in enumerate(taps)) / 16
    blur = sum(t * blurx[:, :, k:cols - 1 + k]
               for k, t in enumerate(taps)) / 16
    src = img[:, 2:rows + 1, 2:cols + 1]
    sharp = src * (1 + WEIGHT) - blur * WEIGHT
    out = torch.zeros((3, rows, cols), dtype=img.dtype, device=img.device)
    out[:, :rows - 1, :cols - 1] = torch.where(
        (src - blur).abs() < float(np.float32(THRESHOLD)), src, sharp)
    return out


def _exact_bilateral(img):
    rows, cols = img.shape
    dev = img.device
    gx, gy, gz = rows // 8 + 4, cols // 8 + 4, 14
    x = torch.arange(rows, device=dev)[:, None]
    y = torch.arange(cols, device=dev)[None, :]
    z = (img * 10).long()                # the intensity bin, in float32
    cell = (((2 + x // 8) * gy + 2 + y // 8) * gz + 2 + z).reshape(-1)
    v = img.double()
    grid = torch.zeros((2, gx * gy * gz), dtype=torch.float64, device=dev)
    grid[0].index_add_(0, cell, v.reshape(-1))
    grid[1].index_add_(0, cell, torch.ones_like(v).reshape(-1))
    grid = grid.reshape(2, gx, gy, gz)
    inner = torch.zeros(grid.shape[1:], dtype=torch.float64, device=dev)
    inner[2:rows // 8 + 2, 2:cols // 8 + 2, 2:12] = 1
    for axis in (3, 1, 2):
        grid = inner * sum(t * torch.roll(grid, 2 - k, axis)
                           for k, t in enumerate((1, 4, 6, 4, 1)))

    def at(dx, dy, dz):
        i = ((2 + x // 8 + dx) * gy + 2 + y // 8 + dy) * gz + 2 + z + dz
        return grid.reshape(2, -1)[:, i]

    xf, yf = (x % 8).double() / 8, (y % 8).double() / 8

    def plane(dz):
        return torch.lerp(
            torch.lerp(at(0, 0, dz), at(1, 0, dz), xf.expand(rows, cols)),
            torch.lerp(at(0, 1, dz), at(1, 1, dz), xf.expand(rows, cols)),
            yf.expand(rows, cols))

    value, weight = torch.lerp(plane(0), plane(1), v * 10 - z)
    return torch.where(weight > 0, value / weight, v)[None]


def _take(a, index, axis):
    return a.index_select(axis, index.clamp(0, a.shape[axis] - 1))


def _half(a, axis):
    x = torch.arange((a.shape[axis] + 1) // 2, device=a.device)
    return sum(t * _take(a, 2 * x + k - 2, axis)
               for k, t in enumerate((1, 4, 6, 4, 1))) / 16


def _double(a, n, axis):
    x = torch.arange(n, device=a.device)
    h = x // 2
    here, after = _take(a, h, axis), _take(a, h + 1, axis)
    even = (_take(a, h - 1, axis) + 6 * here + after) / 8
    shape = [1] * a.dim()
    shape[axis] = n
    return torch.where((x % 2 == 0).reshape(shape), even, (here + after) / 2)


def _exact_pyramid(img1, img2, mask, levels):
    def down(a):
        return _half(_half(a, -2), -1)

    def up(a, like):
        return _double(_double(a, like.shape[-2], -2), like.shape[-1], -1)

    pyr = [[img1, img2, mask]]
    for _ in range(levels - 1):
        pyr.append([down(a) for a in pyr[-1]])
    out = None
    for l in range(levels - 1, -1, -1):
        a, b, m = pyr[l]
        if l < levels - 1:
            a = a - up(pyr[l + 1][0], a)
            b = b - up(pyr[l + 1][1], b)
        blend = a * m + b * (1 - m)
        out = blend if out is None else blend + up(out, blend)
    return out


def _exact_interpolate(img, levels):
    rows, cols = img.shape[1] - 2, img.shape[2] - 2
    dev = img.device

    def index(n):
        return torch.arange(1, n + 1, device=dev)

    def down(a, l, axis):
        i = 2 * index((rows if axis == 1 else cols) >> l)
        return (a.index_select(axis, i - 2) + 2 * a.index_select(axis, i - 1)
                + a.index_select(axis, i)) / 4

    def pad(core):
        return torch.nn.functional.pad(core, (1, 1, 1, 1))

    pyr = [img * img[3:4]]
    for l in range(1, levels):
        # the row filter is zero outside the interior columns
        dx = torch.nn.functional.pad(
            down(pyr[-1], l, 1)[:, :, 1:(cols >> (l - 1)) + 1], (1, 1))
        pyr.append(pad(down(dx, l, 2)))
    out = pyr[-1]
    for l in range(levels - 2, -1, -1):
        i, j = index(rows >> l), index(cols >> l)
        ux = (out.index_select(1, (i + 1) // 2) +
              out.index_select(1, (i + 2) // 2)) / 2
        ux = torch.nn.functional.pad(
            ux[:, :, 1:(cols >> (l + 1)) + 1], (1, 1))
        upy = (ux.index_select(2, (j + 1) // 2) +
               ux.index_select(2, (j + 2) // 2)) / 2
        d = pyr[l][:, 1:(rows >> l) + 1, 1:(cols >> l) + 1]
        out = pad(d + (1 - d[3:4]) * upy)
    core = out[:, 1:rows + 1, 1:cols + 1]
    return core[0:3] / core[3:4]


def _interior(u):
    return u[(slice(1, -1),) * u.dim()]


def _laplacian(u):
    n = u.shape[0] - 2
    acc = 2 * u.dim() * _interior(u)
    for axis in range(u.dim()):
        for start in (0, 2):
            s = [slice(1, -1)] * u.dim()
            s[axis] = slice(start, start + n)
            acc = acc - u[tuple(s)]
    return acc


def _relax(w, u, f):
    """One weighted Jacobi step into the interior of ``w``; ``u`` None is
    the zero iterate."""
    dims = f.dim()
    h = 1.0 / (f.shape[0] - 1)
    omega = {2: 4.0 / 5.0, 3: 8.0 / 9.0}[dims]
    c = omega * h * h / (2 * dims)
    if u is None:
        _interior(w).copy_(c * _interior(f))
    else:
        _interior(w).copy_(_interior(u) -
                           c * (_laplacian(u) / (h * h) - _interior(f)))


def _exact_vcycle(u, f, level, nu1, finest):
    """Pre-smoothing, coarse-grid correction of the defect, no
    post-smoothing; nothing is solved on the coarsest grid.  The boundary
    keeps the input's values on the finest grid and is 0 below it."""
    if level == 0:
        return u
    for _ in range(nu1):
        w = u.clone() if finest else torch.zeros_like(f)
        _relax(w, u, f)
        u = w
    h = 1.0 / (f.shape[0] - 1)
    r = torch.zeros_like(f)
    _interior(r).copy_(_interior(f) - _laplacian(u) / (h * h))
    for axis in range(3):                # full weighting, [1 2 1]/4 an axis
        i = torch.arange(1, r.shape[axis] // 2, device=r.device) * 2
        r = (r.index_select(axis, i - 1) + 2 * r.index_select(axis, i) +
             r.index_select(axis, i + 1)) / 4
    e = _exact_vcycle(None, torch.nn.functional.pad(r, (1,) * 6), level - 1,
                      nu1, False)
    if e is None:
        return u
    for axis in range(3):
        i = torch.arange(1, f.shape[axis] - 1, device=f.device)
        e = (e.index_select(axis, i // 2) +
             e.index_select(axis, (i + 1) // 2)) / 2
    out = u.clone()
    _interior(out).add_(e)
    return out
