"""The work a user of this framework has it do, as timed cases.

Every case is one call (or the short sequence of calls one user action makes)
through the public entry points, on the deterministic atlases the tests, the
bench and the serving stream use (torus: 4 long charts, icosphere: 16 compact
charts, genus-2: 32 thin charts with much boundary).  What a program keeps from
call to call, the hierarchy, the assembled and updated system and its handles,
is kept here too (`_model`); what is new with every call, textures, right-hand
sides, sources, masks, weights and the buffers they live in, is made from the
seed by `prepare`.

Paths (a case's "path"):
  filter     screened-Poisson texture filtering, device buffers, FP32 V-cycles
             inside FP64 refinement to 1e-6 (gdtp_solve_device)
  filter64   the same problem with the plain FP64 V-cycle (gdtp_solve_fp64_device)
  lic        line-integral convolution: anisotropic metric, flexible CG
             (gdtp_solve_device with the krylov knob)
  stream     a sequence of textures from pinned host memory (solve_stream)
  reweight   the filtering app's weight slider: update, then the solve
  geodesic   heat-method distances from k sources, host in and out
  vcycle     one V-cycle on host vectors, what the drop-in headers call
  brush      the sharpening brush: masked cell stiffness (device buffers)
"""
import ctypes as C
import math
from collections import OrderedDict

import numpy as np
import torch

from gradientdomaintextureprocessing_b200 import _lib, meshgen
from gradientdomaintextureprocessing_b200.geodesics import Geodesics
from gradientdomaintextureprocessing_b200.hierarchy import InitializeHierarchy
from gradientdomaintextureprocessing_b200.metric import InitializeAnisotropicMetric, across_for_ratio
from gradientdomaintextureprocessing_b200.system import Brush, System, texel_signal, texture_filtering_rhs

TOL = 1e-6
STIFFNESS, SHARPNESS = 1e-3, 2.0     # the filtering app's screened Poisson weights
LIC_STIFFNESS, LIC_RATIO = 1e-4, 1e3
STREAM_PROBLEMS = 4
# active texels of an atlas as a share of its image, at about 512^2
_COVER = {"torus": 0.89, "icosphere": 0.30, "genus2": 0.065}
_EXACT_MAX = 55_000                  # unknowns of the largest dense 64-bit solve


def listed():
    def case(name, path, mesh, width, height, k):
        return {"name": name, "path": path, "mesh": mesh, "width": width, "height": height, "k": k}

    return [
        # the smallest interactive solve: one small RGB texture, launches and latency
        case("filter_torus_256_rgb", "filter", "torus", 256, 256, 3),
        # an ordinary odd-sized grey-scale texture on an atlas of thin charts
        case("filter_genus2_1013x1187_grey", "filter", "genus2", 1013, 1187, 1),
        # the headline: a 2048^2 RGB texture of a 16-chart atlas
        case("filter_icosphere_2048_rgb", "filter", "icosphere", 2048, 2048, 3),
        # a server's batch: five RGB requests of one model solved together
        case("filter_icosphere_725x611_batch15", "filter", "icosphere", 725, 611, 15),
        # the double-precision option
        case("filter64_icosphere_1024_rgb", "filter64", "icosphere", 1024, 1024, 3),
        # line-integral convolution of one noise texture along a tangent field
        case("lic_genus2_1024", "lic", "genus2", 1024, 1024, 1),
        # end to end from and to host memory, as a batch tool filters a set of textures
        case("stream_icosphere_1024_rgb", "stream", "icosphere", 1024, 1024, 3),
        # the slider: new weights, then the new solution
        case("reweight_icosphere_1024_rgb", "reweight", "icosphere", 1024, 1024, 3),
        # one click in the geodesics app
        case("geodesic_icosphere_512_1", "geodesic", "icosphere", 512, 512, 1),
        # the largest: all distances from 64 sources
        case("geodesic_icosphere_1024_64", "geodesic", "icosphere", 1024, 1024, 64),
        # one frame of the unchanged app behind the drop-in headers
        case("vcycle_torus_640x480_rgb", "vcycle", "torus", 640, 480, 3),
        # one stroke of the brush
        case("brush_icosphere_1024_rgb", "brush", "icosphere", 1024, 1024, 3),
    ]


def _size(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    path = rng.choice(["filter", "filter", "filter", "filter", "filter64", "lic", "stream", "reweight", "geodesic", "vcycle", "brush"])
    mesh = "icosphere" if path in ("geodesic", "stream") else "genus2" if path == "lic" else rng.choice(["torus", "icosphere", "genus2"])
    k = {"lic": 1, "brush": 3, "vcycle": 3, "stream": 3}.get(path) or rng.choice([1, 1, 3, 3, 3, 4, 6, 9, 15])
    if path == "geodesic":
        k = _size(rng, 1, 64)
    low = 256 if mesh == "genus2" else 128
    high = {"filter": 2048, "filter64": 1400}.get(path, 1024)
    if k > 4 and path != "geodesic":
        high = min(high, 1024)
    width = _size(rng, low, high)
    height = min(high, max(low, int(width * rng.uniform(0.75, 1.33))))
    return {"path": path, "mesh": mesh, "width": width, "height": height, "k": k}


# ----------------------------------------------------------------------------
# what a program keeps
# ----------------------------------------------------------------------------
_kept = OrderedDict()


def _mesh(case):
    w, h, small = case["width"], case["height"], min(case["width"], case["height"])
    if case["mesh"] == "torus":
        return meshgen.torus_atlas(w, h, texture="value_noise")
    if case["mesh"] == "icosphere":
        return meshgen.icosphere_atlas(w, h, subdiv=6 if small >= 1024 else 5)
    return meshgen.genus2_atlas(w, h, nu=352 if small >= 2048 else 176, nv=144 if small >= 2048 else 72)


def _model(case):
    """The case's hierarchy and its system (or geodesics pair); the two last used are kept."""
    key = (case["mesh"], case["width"], case["height"], case["path"])
    if key in _kept:
        _kept.move_to_end(key)
        return _kept[key]
    while len(_kept) >= 2:
        _kept.popitem(last=False)
    mesh = _mesh(case)
    h = InitializeHierarchy(mesh, case["width"], case["height"], levels=4)
    if case["path"] == "geodesic":
        model = Geodesics(h)
    elif case["path"] == "lic":
        field = meshgen.gaussian_bump_field(mesh, bumps=8, seed=0)
        metric = InitializeAnisotropicMetric(mesh, field, across=across_for_ratio(LIC_RATIO))
        model = System(h, parameter_metric=metric)
        model.update(LIC_STIFFNESS, 1.0)
        model.set("krylov", 1)
    else:
        model = System(h)
        model.update(STIFFNESS, 1.0)
    _kept[key] = (h, model)
    return _kept[key]


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------
def _texture(case, generator):
    """Smooth value noise with fine noise on top, in [0, 1.1], height x width x k."""
    k, w, h = case["k"], case["width"], case["height"]
    lattice = torch.rand((1, k, 33, 33), generator=generator)
    smooth = torch.nn.functional.interpolate(lattice, size=(h, w), mode="bilinear", align_corners=False)
    image = smooth + 0.1 * torch.rand((1, k, h, w), generator=generator)
    return np.ascontiguousarray(image[0].permute(1, 2, 0).numpy())


def _signal(case, h, generator):
    return texel_signal(h, _texture(case, generator)).reshape(-1, case["k"])


def _filter_rhs(case, h, system, generator):
    return texture_filtering_rhs(system, _signal(case, h, generator), STIFFNESS, SHARPNESS)


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def prepare(case, seed):
    g = torch.Generator().manual_seed(seed)
    path, k = case["path"], case["k"]
    h, model = _model(case)
    state = {"path": path, "k": k, "model": model, "report": _lib.Report()}
    if path in ("filter", "filter64", "reweight"):
        b = _filter_rhs(case, h, model, g)
        state["weight"] = STIFFNESS * (1.0 + 0.5 * float(torch.rand((), generator=g)))
        state["b"] = torch.from_numpy(b).cuda()
        state["x"] = torch.zeros_like(state["b"])
    elif path == "lic":
        noise = torch.rand((model.n, 1), generator=g, dtype=torch.float64).numpy()
        state["b"] = torch.from_numpy(model.apply(noise, which=1)).cuda()
        state["x"] = torch.zeros_like(state["b"])
    elif path == "stream":
        state["b"] = [_pinned(_filter_rhs(case, h, model, g)) for _ in range(STREAM_PROBLEMS)]
        state["x"] = [_pinned(np.zeros_like(b)) for b in state["b"]]
    elif path == "geodesic":
        deep = h.array("deepGlobal").reshape(-1)
        state["sources"] = deep[torch.randperm(len(deep), generator=g)[:k].numpy()].astype(np.int32)
    elif path == "vcycle":
        f = _signal(case, h, g)
        state["b"] = texture_filtering_rhs(model, f, STIFFNESS, SHARPNESS).astype(np.float32)
        state["x"] = f.astype(np.float32)
    else:
        cells = h.counts(0)["numCells"]
        mask = torch.rand(cells, generator=g, dtype=torch.float64)
        mask[mask < 0.7] = 0.0       # a stroke leaves most cells alone
        state["brush"] = Brush(model, _signal(case, h, g))
        state["mask"] = mask.cuda()
        state["x"] = torch.empty((model.n, k), dtype=torch.float64, device="cuda")
    return state


# ----------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------
def _pointer(t):
    return C.c_void_p(t.data_ptr())


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _solve(state, entry, iterations):
    state["x"].zero_()
    _lib.check(entry(state["model"].handle, _pointer(state["b"]), _pointer(state["x"]), state["k"], TOL, iterations, _stream(),
                     C.byref(state["report"])))
    return state["x"]


def run(state):
    path, model = state["path"], state["model"]
    if path == "filter":
        return _solve(state, _lib.lib().gdtp_solve_device, 60)
    if path == "filter64":
        return _solve(state, _lib.lib().gdtp_solve_fp64_device, 60)
    if path == "lic":
        return _solve(state, _lib.lib().gdtp_solve_device, 1000)
    if path == "reweight":
        model.update(state["weight"], 1.0)
        return _solve(state, _lib.lib().gdtp_solve_device, 60)
    if path == "stream":
        return model.solve_stream(state["b"], state["x"], tol=TOL)[0]
    if path == "geodesic":
        return model.distance(state["sources"], tol=TOL)[0]
    if path == "vcycle":
        return model.vcycle(state["x"], state["b"])
    _lib.check(_lib.lib().gdtp_brush_apply_device(state["brush"]._b, _pointer(state["mask"]), _pointer(state["x"]), _stream()))
    return state["x"]


def work(case):
    """Right-hand sides (or signal, mask) read once, results written once, and the
    finest operator (9 double coefficients a texel) read and applied once."""
    texels = _COVER[case["mesh"]] * case["width"] * case["height"]
    values = texels * case["k"]
    vector = 4.0 if case["path"] == "vcycle" else 8.0
    count = STREAM_PROBLEMS if case["path"] == "stream" else 1
    read = {"geodesic": 0.0, "vcycle": 2.0}.get(case["path"], 1.0)
    solves = 2 if case["path"] == "geodesic" else count
    return {"bytes": count * (1.0 + read) * vector * values + 72.0 * texels, "flops": 18.0 * values * solves}


# ----------------------------------------------------------------------------
# 64-bit values
# ----------------------------------------------------------------------------
def _dense(case, h, system):
    """The finest operator as a dense matrix on the GPU, scattered from the system's coefficients."""
    n = system.n
    a = torch.zeros(n * n, dtype=torch.float64, device="cuda")

    def add(rows, cols, values):
        at = torch.as_tensor(rows.astype(np.int64) * n + cols.astype(np.int64)).cuda()
        a.index_add_(0, at, torch.from_numpy(np.ascontiguousarray(values, dtype=np.float64)).cuda())

    coefficients = system.array("coef.deep", 0)
    for start, end, previous, following, first in h.array("rasterLines"):
        i = np.arange(end - start + 1)
        for c in range(9):
            row = (previous, start, following)[c // 3]
            add(start + i, row + i + c % 3 - 1, coefficients[first + i, c])
    boundary = h.array("boundaryGlobal").reshape(-1)
    for block in ("bb", "bd"):
        ptr, col, val = (system.array(f"coef.{block}.{p}", 0) for p in ("ptr", "col", "val"))
        rows = boundary[np.repeat(np.arange(len(ptr) - 1), np.diff(ptr))]
        add(rows, boundary[col] if block == "bb" else col, val)
    return a.view(n, n)


def exact(case, seed):
    """Solutions by a dense Cholesky factorisation in 64 bits, where the texels are
    few enough for one; the matrix entries are the problem's data (the assembled
    system).  The V-cycle, the brush and the distances have no closed form in
    terms of that matrix, and larger systems do not fit a dense factorisation."""
    if case["path"] not in ("filter", "filter64", "lic", "reweight") or _COVER[case["mesh"]] * case["width"] * case["height"] > 1.3 * _EXACT_MAX:
        return None
    state = prepare(case, seed)
    h, system = _model(case)
    if system.n > _EXACT_MAX:
        return None
    if case["path"] == "reweight":
        system.update(state["weight"], 1.0)
    a = _dense(case, h, system)
    scale = a.diagonal().rsqrt().clone()
    a *= scale[:, None]
    a *= scale[None, :]
    factor = torch.linalg.cholesky(a)
    x = torch.cholesky_solve(state["b"] * scale[:, None], factor) * scale[:, None]
    if case["path"] == "reweight":
        system.update(STIFFNESS, 1.0)
    return x
