"""The work a program has this library do, as cases to time and to check: the elliptic solves of
one surface timestep (flexure, hillslope diffusion on the raster and on the cube grid), the
flexure step's grid helpers, and a training step of the learned first guess.

Every case goes through the entry points a user calls: the C ABI's `_dev` calls on device arrays
through a handle made once per raster (dt_flex_solve_dev, dt_diff_solve_dev, dt_cube_diff_solve_dev),
the deeptime_gpu.grid functions and the deeptime_gpu.unet model. Inputs follow the library's own
workloads (seeded rigidity 10^(21 + 3u), |k|^-2 and |k|^-2.5 topographies, log-uniform
diffusivities), drawn on the GPU.

`exact` restates each system in plain torch in 64 bits and solves it tightly, without this
library's code.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "deep-time_b200"))

from deeptime_gpu import _lib as L  # noqa: E402
from deeptime_gpu import cube as C  # noqa: E402
from deeptime_gpu import diffusion as Dm  # noqa: E402
from deeptime_gpu import flexure as F  # noqa: E402
from deeptime_gpu import grid as Gr  # noqa: E402
from deeptime_gpu import unet as U  # noqa: E402

WEIGHTS = os.path.join(ROOT, "deep-time_b200", "weights", "unet_flexure.bin")
G = 9.81
RHO_MANTLE, RHO_WATER = 3300.0, 1030.0
GIRTH_M = 40.0e6  # the planet's girth: the production rasters' dx is this over their width


# ---- the cases ---------------------------------------------------------------------------------

def listed():
    return [
        # The timestep's own flexure call: the solve raster the step coarsens to (39 km cells), the
        # reference's bank preconditioner and max|z| < 2 m rule, a land-sea restoring density.
        # Once per timestep; a handful of iterations, so set-up and launches count.
        dict(name="flexure_step_1024x328", kind="flexure_step", w=1024, h=328),
        # The same call where the coarsened raster is no power of two either way: 1500 x 750.
        dict(name="flexure_step_1500x750", kind="flexure_step", w=1500, h=750),
        # The plain FP64 method at its benchmark size and tolerance (mean-D preconditioner, 1e-10):
        # small rasters, many cheap iterations.
        dict(name="flexure_plain_512x256", kind="flexure_plain", w=512, h=256),
        # The headline solve: FP32 PCG with FP64 reliable updates, the bank, the U-Net's first
        # guess, to 1e-8 at 2.5 km.
        dict(name="flexure_mixed_4096x2048", kind="flexure_mixed", w=4096, h=2048),
        # The timestep loop's cell (1.25 km) over half its raster each way: the largest.
        dict(name="flexure_mixed_8192x4096", kind="flexure_mixed", w=8192, h=4096),
        # The FP32 solve on the sphere's row metric (latitudes +-58 degrees), from x = 0.
        dict(name="flexure_sphere_2048x1024", kind="flexure_sphere", w=2048, h=1024),
        # The timestep's own diffusion call at the first-level raster: FP64 CG, the FP32
        # damped-Jacobi cycle, the LOD first guess, RMS residual 1e-5 m, a land-sea diffusivity.
        dict(name="diffusion_step_2048x656", kind="diffusion_step", w=2048, h=656),
        # The multigrid benchmark: FP32 CG on red-black Gauss-Seidel cycles with FP64 reliable
        # updates to 1e-10, kappa dt / dx^2 log-uniform over [0.1, 100].
        dict(name="diffusion_mixed_2048x1024", kind="diffusion_mixed", w=2048, h=1024),
        # The timestep loop's diffusion at a raster far beyond the L2.
        dict(name="diffusion_mixed_8192x4096", kind="diffusion_mixed", w=8192, h=4096),
        # The cube grid's implicit diffusion, 6 x 256^2 cells, RMS 1e-6 m.
        dict(name="cube_256", kind="cube", n=256, dt=7.0),
        # The flexure step's grid work around its solve: Te blur, coarsening, prolongation,
        # binomial filter, on the first-level raster.
        dict(name="step_grid_2048x656", kind="step_grid", w=2048, h=656, f=2),
        # One training batch of the first guess: loss and gradients, forward and backward.
        dict(name="unet_gradients_16x512x256", kind="unet", batch=16, w=512, h=256),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["flexure_step", "flexure_step", "flexure_plain", "flexure_mixed", "flexure_sphere", "diffusion_step",
                       "diffusion_step", "diffusion_mixed", "diffusion_mixed", "cube", "step_grid", "unet"])
    if kind == "flexure_step":  # any width and height the step's coarsening leaves
        w = _size(rng, 200, 2048)
        if rng.random() < 0.4:
            w = 1 << int(round(math.log2(w)))
        return dict(kind=kind, w=w, h=max(64, int(w * rng.uniform(0.3, 0.5))))
    if kind == "flexure_plain":
        w = 1 << rng.randint(7, 11)
        return dict(kind=kind, w=w, h=w // rng.choice([1, 2, 4]) if rng.random() < 0.6 else _size(rng, 64, w // 2))
    if kind == "flexure_mixed":  # the first guess works on 10 km cells, 1024 across and a multiple of 8 down
        s = rng.choice([1, 2, 4, 8])
        return dict(kind=kind, w=1024 * s, h=s * 8 * rng.randint(8, 64))
    if kind == "flexure_sphere":
        w = 1 << rng.randint(8, 11)
        return dict(kind=kind, w=w, h=_size(rng, 100, w // 2))
    if kind == "diffusion_step":
        w = _size(rng, 128, 6000)
        return dict(kind=kind, w=w, h=max(48, int(w * rng.uniform(0.2, 0.6))))
    if kind == "diffusion_mixed":
        w = _size(rng, 128, 6000)
        if rng.random() < 0.5:
            w = 1 << int(round(math.log2(w)))
        return dict(kind=kind, w=w, h=max(32, int(w * rng.uniform(0.25, 0.55))))
    if kind == "cube":
        return dict(kind=kind, n=_size(rng, 24, 320), dt=round(rng.uniform(1.0, 60.0), 2))
    if kind == "step_grid":
        f = rng.choice([1, 2, 3, 4])
        ws = _size(rng, 100, 2048)
        return dict(kind=kind, w=f * ws, h=f * max(16, int(ws * rng.uniform(0.25, 0.6))), f=f)
    return dict(kind=kind, batch=rng.randint(1, 16), w=512 * rng.choice([1, 1, 2]), h=8 * rng.randint(4, 32))


# ---- inputs ------------------------------------------------------------------------------------

def _gen(seed, k):
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * int(seed) + k)
    return g


def _randn(shape, g):
    return torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)


def _freq(h, w):
    fy = torch.fft.fftfreq(h, device="cuda", dtype=torch.float64)[:, None]
    fx = torch.fft.rfftfreq(w, device="cuda", dtype=torch.float64)[None, :]
    return fy, fx


def _smooth01(w, h, sigma, g):
    """White noise smoothed over `sigma` cells (x periodic, y mirrored), rescaled to [0, 1]."""
    v = _randn((h, w), g)
    ext = torch.cat([v, v.flip(0)])
    fy, fx = _freq(2 * h, w)
    gain = torch.exp(-2.0 * (math.pi * sigma) ** 2 * (fx * fx + fy * fy))
    u = torch.fft.irfft2(torch.fft.rfft2(ext) * gain, s=ext.shape)[:h]
    return ((u - u.min()) / (u.max() - u.min())).contiguous()


def _topography(w, h, beta, std, g):
    """A zero-mean Gaussian random field of spectrum |k|^-beta and the given standard deviation."""
    fy, fx = _freq(h, w)
    k2 = fx * fx + fy * fy
    k2[0, 0] = 1.0
    amp = k2 ** (-beta / 4.0)
    amp[0, 0] = 0.0
    f = torch.fft.irfft2(torch.fft.rfft2(_randn((h, w), g)) * amp, s=(h, w))
    return (f * (std / f.std(unbiased=False))).contiguous()


def _benchmark_inputs(w, h, dx, seed):
    """(d, c, b, dx) of the benchmark's recipe: the rigidity smoothed over 80 km."""
    d = 10.0 ** (21.0 + 3.0 * _smooth01(w, h, 80.0e3 / dx, _gen(seed, 1))) / G
    b = 2700.0 * _topography(w, h, 2.0, 1500.0, _gen(seed, 2))
    return d, torch.full_like(d, RHO_MANTLE), b, dx


def _step_inputs(w, h, seed):
    """The timestep's call: a rigidity over provinces, and water over the low ground."""
    d = 10.0 ** (21.0 + 3.0 * _smooth01(w, h, 8.0, _gen(seed, 1))) / G
    topo = _topography(w, h, 2.0, 1500.0, _gen(seed, 2))
    c = torch.where(topo < -500.0, RHO_MANTLE - RHO_WATER, RHO_MANTLE).to(torch.float64).contiguous()
    return d, c, 2700.0 * topo, GIRTH_M / w


def _sphere_metric(h):
    """Rows of equal area between sines of latitude +-0.85: (a, b) of the row metric."""
    s = np.clip((0.5 * h - np.arange(h + 1)) * (0.85 / (0.5 * h)), -1.0, 1.0)
    m = 0.5 * (s[:-1] + s[1:])
    a = 1.0 / np.maximum(1.0 - m * m, 1e-12)
    b = 1.0 - s * s
    b[0] = b[-1] = 0.0
    return a, b


def _flexure_inputs(case, seed):
    w, h = case["w"], case["h"]
    if case["kind"] == "flexure_step":
        return _step_inputs(w, h, seed)
    # 10 km cells at 512 for the plain method, 2.5 km at 4096 for the others
    return _benchmark_inputs(w, h, (5.12e6 if case["kind"] == "flexure_plain" else 10.24e6) / w, seed)


def _diffusion_inputs(case, seed):
    """(h, kd, dt, dx)."""
    w, h = case["w"], case["h"]
    topo = _topography(w, h, 2.5, 800.0, _gen(seed, 1))
    if case["kind"] == "diffusion_step":
        # slow soil creep on land, a fast shelf under water: a sharp edge at the shore
        dx, dt = GIRTH_M / w, 1.0e5
        s = torch.where(topo > 0.0, 0.02, 4.0) * 10.0 ** (_smooth01(w, h, 6.0, _gen(seed, 2)) - 0.5)
    else:
        dx, dt = 2500.0, 1.0
        s = 10.0 ** (-1.0 + 3.0 * _smooth01(w, h, max(1.0, w / 256.0), _gen(seed, 2)))
    return topo, (s * dx * dx / dt).contiguous(), dt, dx


_GEOMETRY = {}  # the cube's neighbour table by n: a program builds it once


def _cube_inputs(case, seed):
    """(slots, lap, areas, kd, h): a symmetric coupling Laplacian on the cube's topology."""
    n = case["n"]
    if n not in _GEOMETRY:
        slots = C.topology(n)
        m = np.where(slots != C.NO_CELL, slots, 0).astype(np.int64)
        back = np.argmax(slots[m] == np.arange(len(slots))[:, None, None], axis=2)
        _GEOMETRY.clear()
        _GEOMETRY[n] = slots, m, back
    slots, m, back = _GEOMETRY[n]
    rng = np.random.default_rng(seed)
    cells = 6 * n * n
    areas = 1.0 + 0.2 * rng.random(cells)
    raw = rng.random((cells, 8))
    raw[:, 0::2] = 0.8 + 0.4 * raw[:, 0::2]
    raw[:, 1::2] = 0.05 + 0.15 * raw[:, 1::2]
    lap = np.where(m > np.arange(cells)[:, None], raw, raw[m, back])
    lap = np.where(slots != C.NO_CELL, lap, 0.0)
    kd = np.where(rng.random(cells) < 0.3, 0.02, 1.0) * (0.5 + rng.random(cells))
    return slots, lap, areas, kd, 1000.0 * rng.standard_normal(cells)


_LEVELS, _BASE, _PAD = 4, 32, 32


def _unet_layers():
    """(cin, cout) of the 3 x 3 convolutions in parameter order."""
    out = []
    for k in range(_LEVELS):
        c = _BASE << k
        out += [(_PAD if k == 0 else c // 2, c), (c, c)]
    for k in range(_LEVELS - 2, -1, -1):
        c = _BASE << k
        out += [(3 * c, c), (c, c)]
    return out


def _unet_inputs(case, seed):
    """(parameters, x, target) of a half-trained network: He-scaled weights, small biases."""
    g = _gen(seed, 1)
    parts = []
    for cin, cout in _unet_layers():
        fan = 9 * (2 if cin == _PAD and not parts else cin)
        parts += [torch.randn(9 * cin * cout, device="cuda", generator=g) * math.sqrt(2.0 / fan),
                  torch.randn(cout, device="cuda", generator=g) * 0.05]
    parts += [torch.randn(_BASE, device="cuda", generator=g) / math.sqrt(_BASE), torch.zeros(1, device="cuda")]
    shape = (case["batch"], case["h"], case["w"])
    x = torch.randn(shape + (2,), device="cuda", generator=g)
    return torch.cat(parts), x, torch.randn(shape, device="cuda", generator=g) * 0.3


def _handle_stream():
    return torch.cuda.Stream()


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def prepare(case, seed):
    kind, lib = case["kind"], L.lib()
    st = {"kind": kind}
    if kind.startswith("flexure"):
        w, h = case["w"], case["h"]
        st["d"], st["c"], st["b"], dx = _flexure_inputs(case, seed)
        st["x"] = torch.zeros_like(st["b"])
        st["solver"] = F.Solver(w, h, dx, _sphere_metric(h) if kind == "flexure_sphere" else None)
        st["stream"] = _handle_stream()
        L.check(lib.dt_flex_set_stream(st["solver"]._h, ctypes.c_void_p(st["stream"].cuda_stream)))
        if kind == "flexure_step":
            st["params"] = F.params(tol=2.0, max_iterations=60)
        elif kind == "flexure_plain":
            st["params"] = F.params(precond=L.PRECOND_MEAN_D, stop=L.STOP_REL_RESIDUAL, tol=1e-10, max_iterations=20000)
        else:
            mixed = kind == "flexure_mixed"
            st["params"] = F.params(stop=L.STOP_REL_RESIDUAL, precision=L.PREC_MIXED_RELIABLE, tol=1e-8,
                                    max_iterations=20000, warm_start=L.WARM_UNET if mixed else L.WARM_NONE)
            if mixed:
                st["model"] = U.UNet(seed=1)
                st["model"].load(WEIGHTS)
                L.check(lib.dt_flex_set_unet(st["solver"]._h, st["model"]._h, ctypes.c_double(10_000.0)))
    elif kind.startswith("diffusion"):
        st["h"], st["kd"], st["dt"], dx = _diffusion_inputs(case, seed)
        st["x"] = torch.empty_like(st["h"])
        st["ws"] = Dm.Workspace(Dm.Dims(case["w"], case["h"], dx, True))
        st["stream"] = _handle_stream()
        L.check(lib.dt_diff_set_stream(st["ws"]._h, ctypes.c_void_p(st["stream"].cuda_stream)))
        st["params"] = Dm.params() if kind == "diffusion_step" else Dm.params(
            cycle=L.CYCLE_RBGS, precision=L.DIFF_MIXED_RELIABLE, stop=L.STOP_REL_RESIDUAL, tol=1e-10, max_iterations=2000)
    elif kind == "cube":
        slots, lap, areas, kd, h = _cube_inputs(case, seed)
        st["cube"] = C.CubeDiffusion(case["n"], slots, lap, areas)
        st["kd"], st["h"] = torch.from_numpy(kd).cuda(), torch.from_numpy(h).cuda()
        st["x"], st["dt"] = torch.empty_like(st["h"]), case["dt"]
        st["stream"] = _handle_stream()
        L.check(lib.dt_cube_set_stream(st["cube"]._h, ctypes.c_void_p(st["stream"].cuda_stream)))
    elif kind == "step_grid":
        w, h, f = case["w"], case["h"], case["f"]
        st["te"] = 8.0 + 52.0 * _smooth01(w, h, 4.0, _gen(seed, 1))
        st["load"] = 2700.0 * _topography(w, h, 2.0, 1500.0, _gen(seed, 2))
        st["deflection"] = _topography(w // f, h // f, 3.0, 900.0, _gen(seed, 3))
        st["f"] = f
    else:
        p, st["input"], st["target"] = _unet_inputs(case, seed)
        st["model"] = U.UNet(seed=1)
        st["model"].set_params(p.cpu().numpy())
        st["shape"] = (case["batch"], case["h"], case["w"])
    torch.cuda.synchronize()  # the handles' streams are not the one the inputs were made on
    return st


# ---- one pass ----------------------------------------------------------------------------------

def run(st):
    kind, lib, rep = st["kind"], L.lib(), L.Report()
    if kind.startswith("flexure"):
        L.check(lib.dt_flex_solve_dev(st["solver"]._h, _ptr(st["d"]), _ptr(st["c"]), _ptr(st["b"]), _ptr(st["x"]),
                                      ctypes.byref(st["params"]), ctypes.byref(rep)))
        return st["x"]
    if kind.startswith("diffusion") or kind == "cube":
        with torch.cuda.stream(st["stream"]):  # the solve replaces the field in place
            st["x"].copy_(st["h"])
        dt = ctypes.c_double(st["dt"])
        if kind == "cube":
            L.check(lib.dt_cube_diff_solve_dev(st["cube"]._h, _ptr(st["x"]), _ptr(st["kd"]), dt, ctypes.c_double(1e-6),
                                               ctypes.byref(rep)))
        else:
            L.check(lib.dt_diff_solve_dev(st["ws"]._h, _ptr(st["x"]), _ptr(st["kd"]), dt, ctypes.byref(st["params"]),
                                          ctypes.byref(rep)))
        return st["x"]
    if kind == "step_grid":
        f = st["f"]
        te = Gr.box_blur(st["te"].clone(), 2, 2)
        load = Gr.restrict(st["load"], f)
        w = Gr.binomial(Gr.prolong_linear(st["deflection"], f), 1)
        return {"te": te, "load": load, "deflection": w}
    loss = st["model"].loss_and_grad_dev(st["input"].data_ptr(), st["target"].data_ptr(), *st["shape"])
    return {"loss": loss, "gradients": st["model"].gradients()}


def work(case):
    """Inputs read once and outputs written once; for the solves, nothing of the iterations that the
    answer's accuracy asks for. The network's arithmetic: three products per weight and pixel."""
    kind = case["kind"]
    if kind == "unet":
        px = case["batch"] * case["w"] * case["h"]
        flops, depth = 0.0, [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0]
        for (cin, cout), k in zip(_unet_layers(), depth):
            flops += 3 * 2 * 9 * cin * cout * (px >> (2 * k))
        params = sum(9 * a * b + b for a, b in _unet_layers()) + _BASE + 1
        return {"bytes": 12 * px + 8 * params, "flops": flops}
    if kind == "cube":
        cells = 6 * case["n"] ** 2
        return {"bytes": cells * 8 * 3, "flops": cells * 20}
    cells = case["w"] * case["h"]
    if kind == "step_grid":
        part = cells // case["f"] ** 2
        return {"bytes": 8 * (4 * cells + 2 * part), "flops": cells * 20}
    fields = 4 if kind.startswith("flexure") else 3
    return {"bytes": cells * 8 * fields, "flops": cells * (25 if fields == 4 else 9)}


# ---- the same in 64 bits -----------------------------------------------------------------------

def _shift(v, n):
    """v's neighbour above (n = -1) or below (n = 1), the edge rows repeated."""
    return torch.cat([v[:1], v[:-1]]) if n < 0 else torch.cat([v[1:], v[-1:]])


def _lap(v, dx, metric):
    we, ea = torch.roll(v, 1, 1), torch.roll(v, -1, 1)
    no, so = _shift(v, -1), _shift(v, 1)
    if metric is None:
        return (we + ea + no + so - 4.0 * v) / (dx * dx)
    a, bn, bs = metric
    return (a * (we + ea - 2.0 * v) + bn * (no - v) + bs * (so - v)) / (dx * dx)


def _cg(apply, precondition, b, tol, cap):
    x = torch.zeros_like(b)
    r = b.clone()
    z = precondition(r)
    p, rz, stop = z.clone(), torch.dot(r.ravel(), z.ravel()), tol * tol * torch.dot(b.ravel(), b.ravel())
    for it in range(cap):
        ap = apply(p)
        alpha = rz / torch.dot(p.ravel(), ap.ravel())
        x.add_(alpha * p)
        r.sub_(alpha * ap)
        if it % 10 == 9 and bool(torch.dot(r.ravel(), r.ravel()) <= stop):
            break
        z = precondition(r)
        rz, old = torch.dot(r.ravel(), z.ravel()), rz
        p = z + (rz / old) * p
    return x


def _exact_flexure(case, seed):
    if case["w"] * case["h"] > 1 << 23:
        return None  # minutes of plain torch
    d, c, b, dx = _flexure_inputs(case, seed)
    h, w = b.shape
    metric, ax, by = None, 1.0, 1.0
    if case["kind"] == "flexure_sphere":
        a, bb = (torch.from_numpy(v).cuda() for v in _sphere_metric(h))
        metric = a[:, None], bb[:-1, None], bb[1:, None]
        ax, by = float(a.mean()), float(bb.mean())
    ky = torch.arange(2 * h, device="cuda", dtype=torch.float64)[:, None] * (math.pi / h)
    kx = torch.arange(w // 2 + 1, device="cuda", dtype=torch.float64)[None, :] * (2.0 * math.pi / w)
    lam = (ax * (2.0 * torch.cos(kx) - 2.0) + by * (2.0 * torch.cos(ky) - 2.0)) / (dx * dx)
    symbol = 1.0 / (d.mean() * lam * lam + c.mean())

    def precondition(r):
        ext = torch.cat([r, r.flip(0)])
        return torch.fft.irfft2(torch.fft.rfft2(ext) * symbol, s=ext.shape)[:h].contiguous()

    return _cg(lambda v: _lap(d * _lap(v, dx, metric), dx, metric) + c * v, precondition, b, 1e-13, 3000)


def _exact_diffusion(case, seed):
    h0, kd, dt, dx = _diffusion_inputs(case, seed)
    east = 0.5 * (kd + torch.roll(kd, -1, 1)) * (dt / (dx * dx))
    west = torch.roll(east, 1, 1)
    south = torch.cat([0.5 * (kd[:-1] + kd[1:]), torch.zeros_like(kd[:1])]) * (dt / (dx * dx))
    north = torch.cat([torch.zeros_like(kd[:1]), south[:-1]])
    diag = 1.0 + east + west + south + north

    def apply(v):
        return (diag * v - east * torch.roll(v, -1, 1) - west * torch.roll(v, 1, 1) - south * _shift(v, 1)
                - north * _shift(v, -1))

    return _cg(apply, lambda r: r / diag, h0, 1e-14, 2000)


def _exact_cube(case, seed):
    slots, lap, areas, kd, h = _cube_inputs(case, seed)
    some = slots != C.NO_CELL
    m = np.where(some, slots, 0).astype(np.int64)
    here = np.arange(len(kd))[:, None]

    def mean(a, b):
        return 0.5 * (kd[a] + kd[b])

    dif = np.empty(lap.shape)
    for k in range(8):
        if k % 2 == 0:
            dif[:, k] = mean(here[:, 0], m[:, k])
        else:  # a diagonal takes the least of the quad's four sides
            a, b, far = m[:, k - 1], m[:, (k + 1) % 8], m[:, k]
            dif[:, k] = np.minimum(np.minimum(mean(here[:, 0], a), mean(a, far)), np.minimum(mean(far, b), mean(b, here[:, 0])))
    k = np.where(some, case["dt"] / areas.mean() * dif * lap, 0.0)
    k, m = torch.from_numpy(k).cuda(), torch.from_numpy(m).cuda()
    mu = torch.from_numpy(areas / areas.mean()).cuda()
    diag = mu + k.sum(1)
    return _cg(lambda v: diag * v - (k * v[m]).sum(1), lambda r: r / diag, mu * torch.from_numpy(h).cuda(), 1e-14, 2000)


def _exact_grid(case, seed):
    w, h, f = case["w"], case["h"], case["f"]
    te = 8.0 + 52.0 * _smooth01(w, h, 4.0, _gen(seed, 1))
    for _ in range(2):  # radius 2: five cells, x wrapping, y mirrored at its edges
        te = sum(torch.roll(te, k, 1) for k in range(-2, 3)) / 5.0
        ext = torch.cat([te[:2].flip(0), te, te[-2:].flip(0)])
        te = sum(ext[k:k + h] for k in range(5)) / 5.0
    load = 2700.0 * _topography(w, h, 2.0, 1500.0, _gen(seed, 2))
    load = load.reshape(h // f, f, w // f, f).mean((1, 3))
    v = _topography(w // f, h // f, 3.0, 900.0, _gen(seed, 3))
    x = (torch.arange(w, device="cuda", dtype=torch.float64) + 0.5) / f - 0.5
    y = ((torch.arange(h, device="cuda", dtype=torch.float64) + 0.5) / f - 0.5).clamp(0, h // f - 1)
    i, j = x.floor().long(), y.floor().long()
    tx, ty = x - i, (y - j)[:, None]
    rows = v[:, i % (w // f)] * (1.0 - tx) + v[:, (i + 1) % (w // f)] * tx
    v = rows[j] * (1.0 - ty) + rows[(j + 1).clamp(max=h // f - 1)] * ty
    v = 0.25 * torch.roll(v, 1, 1) + 0.5 * v + 0.25 * torch.roll(v, -1, 1)
    return {"te": te, "load": load, "deflection": 0.25 * _shift(v, -1) + 0.5 * v + 0.25 * _shift(v, 1)}


def _exact_unet(case, seed):
    p, x, target = _unet_inputs(case, seed)
    p = p.double().requires_grad_()
    fn, at, layers = torch.nn.functional, 0, []
    for cin, cout in _unet_layers():
        wt = p[at:at + 9 * cin * cout].reshape(3, 3, cin, cout).permute(3, 2, 0, 1)
        layers.append((wt, p[at + 9 * cin * cout:at + (9 * cin + 1) * cout]))
        at += (9 * cin + 1) * cout

    def conv(v, k):
        wt, bias = layers[k]
        return torch.relu(fn.conv2d(fn.pad(v, (1, 1, 0, 0), mode="circular"), wt[:, :v.shape[1]], bias, padding=(1, 0)))

    loss = 0.0
    for one, want in zip(x.double(), target.double()):  # an image at a time: the activations in 64 bits are large
        cur, skips = one.permute(2, 0, 1)[None], []
        for k in range(_LEVELS):
            cur = conv(conv(cur, 2 * k), 2 * k + 1)
            if k + 1 < _LEVELS:
                skips.append(cur)
                cur = fn.avg_pool2d(cur, 2)
        for k in range(_LEVELS - 2, -1, -1):
            up = torch.cat([fn.interpolate(cur, scale_factor=2, mode="nearest"), skips[k]], dim=1)
            at_k = 2 * _LEVELS + 2 * (_LEVELS - 2 - k)
            cur = conv(conv(up, at_k), at_k + 1)
        out = torch.einsum("nchw,c->nhw", cur, p[at:at + _BASE]) + p[at + _BASE]
        part = torch.mean((out[0] - want) ** 2) / len(x)
        part.backward(retain_graph=True)
        loss += float(part.detach())
    return {"loss": loss, "gradients": p.grad.detach()}


def exact(case, seed):
    kind = case["kind"]
    if kind.startswith("flexure"):
        return _exact_flexure(case, seed)
    if kind.startswith("diffusion"):
        return _exact_diffusion(case, seed)
    return {"cube": _exact_cube, "step_grid": _exact_grid, "unet": _exact_unet}[kind](case, seed)
