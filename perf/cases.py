"""Performance cases of the solver library, through its Python binding.

Each case is one kind of call that a flow or potential solver makes over and
over on a kept context (octree, plans and tables built once): a single block
convolution, Poisson solves on uniform and refined octrees of several block
sizes, batches of small problems, the integrating factor, IF-HERK time steps
with and without an immersed boundary, and the Fourier-in-z block operators.

Inputs are made on the GPU from the seed; the octree of a case depends on the
case alone. All contexts work on one stream, as in a program whose solves follow
one another, and their outputs are ready on it.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "iblgf-amr_b200"))

import iblgf_b200 as B  # noqa: E402

EXTENTS = (4, 6, 8, 10, 14, 16)


# ------------------------------------------------------------------- cases
def listed():
    poisson = {"kind": "poisson", "layout": 20261203}
    return [
        # the block convolution on its own (a host code that drives the blocks
        # itself): the smallest call
        {"name": "conv_block_fp64", "kind": "conv", "extent": 16, "precision": "fp64", "scale": 0.25},
        # a small uniform box, as in unit-sized set-ups: launches and latency
        dict(poisson, name="poisson_uniform_6_fp64", extent=6, bx=4, by=4, bz=4, levels=0, gaussians=0,
             precision="fp64"),
        # 64^3 cells, one level: an ordinary uniform solve
        dict(poisson, name="poisson_uniform_64_fp32", extent=16, bx=4, by=4, bz=4, levels=0, gaussians=0,
             precision="fp32"),
        # an uneven box with another block size and one refinement level
        dict(poisson, name="poisson_ragged_10_fp32", extent=10, bx=5, by=3, bz=4, levels=1, gaussians=6,
             precision="fp32"),
        # three mesh levels, 21.8 million leaf cells: the benchmark's solve
        dict(poisson, name="poisson_amr_3level_fp32", extent=16, bx=8, by=8, bz=8, levels=2, gaussians=16,
             precision="fp32"),
        # two mesh levels in plain double precision
        dict(poisson, name="poisson_amr_2level_fp64", extent=16, bx=8, by=8, bz=8, levels=1, gaussians=16,
             precision="fp64"),
        # many independent problems of 1 to 64 blocks solved together
        {"name": "batch_256_fp32", "kind": "batch", "problems": 256, "most": 64, "extent": 16, "layout": 20261203,
         "precision": "fp32"},
        # the viscous term's integrating factor at a low Reynolds number
        {"name": "integrating_factor_fp64", "kind": "factor", "extent": 16, "bx": 6, "by": 4, "bz": 4, "levels": 0,
         "gaussians": 4, "layout": 7, "alpha": 0.25, "precision": "fp64"},
        # time steps of a vortex ring: small blocks, and the three-level ring
        {"name": "ns_ring_small_fp64", "kind": "ring", "extent": 6, "per_radius": 4, "levels": 1, "Re": 1000.0,
         "precision": "fp64"},
        {"name": "ns_ring_3level_fp32", "kind": "ring", "extent": 16, "per_radius": 8, "levels": 2, "Re": 1000.0,
         "precision": "fp32"},
        # time steps past a sphere with its force solve on every stage
        {"name": "ns_sphere_fp64", "kind": "sphere", "size": "large", "spacing": 1.7, "Re": 300.0,
         "precision": "fp64"},
        # the operators of one Fourier-in-z stage on 2-D blocks
        {"name": "fourier_z_operators", "kind": "fourier", "blocks": 1024, "nb": 18, "modes": 16, "planes": 48},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _logint(rng, lo, hi):
    return max(lo, min(hi, int(_log(rng, lo, hi + 1))))


def draw(rng):
    kind = rng.choice(("conv", "poisson", "poisson", "poisson", "batch", "factor", "ring", "ring", "sphere", "fourier"))
    extent, precision = rng.choice(EXTENTS), rng.choice(("fp32", "fp64"))
    layout = rng.randrange(1, 1 << 30)
    if kind == "conv":
        return {"kind": kind, "extent": extent, "precision": precision, "scale": rng.uniform(0.1, 1.0)}
    if kind in ("poisson", "factor"):
        levels = rng.choice((0, 1, 2)) if kind == "poisson" else rng.choice((0, 0, 1))
        most = (512, 192, 48)[levels]
        while True:
            b = [_logint(rng, 1, 10) for _ in range(3)]
            if b[0] * b[1] * b[2] <= most:
                break
        c = {"kind": kind, "extent": extent, "bx": b[0], "by": b[1], "bz": b[2], "levels": levels,
             "gaussians": _logint(rng, 2, 20), "layout": layout, "precision": precision}
        if kind == "factor":
            c["alpha"] = _log(rng, 1e-4, 0.5)
        return c
    if kind == "batch":
        return {"kind": kind, "problems": _logint(rng, 3, 256), "most": _logint(rng, 8, 64), "extent": extent,
                "layout": layout, "precision": precision}
    if kind == "ring":
        return {"kind": kind, "extent": extent, "per_radius": rng.choice((3, 4, 5, 6)), "levels": rng.choice((0, 1)),
                "Re": _log(rng, 50.0, 3000.0), "precision": precision}
    if kind == "sphere":
        return {"kind": kind, "size": "small", "spacing": rng.uniform(1.5, 2.0), "Re": _log(rng, 100.0, 500.0),
                "precision": "fp64"}
    modes = _logint(rng, 1, 24)
    return {"kind": kind, "blocks": _logint(rng, 8, 900), "nb": rng.choice(EXTENTS) + 2, "modes": modes,
            "planes": rng.choice((2, 3)) * modes}


# ----------------------------------------------------------------- octrees
def _box(case):
    """Lower corner and block counts of the block region (cells, blocks) and the bounding box around it."""
    e, n = case["extent"], (case["bx"], case["by"], case["bz"])
    start = tuple(-((k + 1) // 2) * e for k in n)
    m = 1
    while m < max(n):
        m *= 2
    half = max(m * e // 2, e)
    return start, n, (-2 * half,) * 3, (4 * half,) * 3


def _gaussians(case):
    """Amplitude, width and centre (cells) of the source's Gaussians: a pair of opposite sign and seeded others."""
    start, n, _, _ = _box(case)
    e = case["extent"]
    size = [k * e for k in n]
    mid = [s + d / 2.0 for s, d in zip(start, size)]
    off = min(0.75 * e, 0.25 * size[0])
    g = [(s, 0.25 * e, (mid[0] + s * off, mid[1], mid[2])) for s in (1.0, -1.0)]
    rng = np.random.Generator(np.random.PCG64(case["layout"]))
    for _ in range(case["gaussians"]):
        width, amp = rng.uniform(2.0, 6.0) * e / 16.0, rng.uniform(-1.0, 1.0)
        at = rng.uniform(-0.25, 0.25, size=3)
        g.append((amp, width, tuple(mid[d] + at[d] * size[d] for d in range(3))))
    return g


def _factors(g, axis, x):
    return np.stack([np.exp(-((x - c[axis]) ** 2) / (2.0 * s * s)) for _, s, c in g])


def _largest(g, lo, n, dx):
    """max |f| over the cell centres of a box of n[d] cells from cell lo[d] on, spacing dx."""
    fx, fy, fz = (_factors(g, d, (lo[d] + np.arange(n[d]) + 0.5) * dx) for d in range(3))
    fx = fx * np.array([a for a, _, _ in g])[:, None]
    yz = (fy[:, :, None] * fz[:, None, :]).reshape(len(g), -1)
    return float(np.abs(fx.T @ yz).max())


def _refiner(case):
    """Refine where the source exceeds 1e-3 (base level) or 1e-2 of its largest value, on the block grown by 2 cells."""
    start, n, _, _ = _box(case)
    e, g = case["extent"], _gaussians(case)
    top = _largest(g, start, [k * e for k in n], 1.0)

    def refine(base, extent, rl, diff):
        if rl >= case["levels"]:
            return False
        return _largest(g, [b - 2 for b in base], (extent[0] + 4,) * 3, 0.5 ** rl) > top * (1e-3 if rl == 0 else 1e-2)
    return refine


def _octree(case, stream):
    start, n, lo, size = _box(case)
    e = case["extent"]
    return B.Solver(lo, size, e, 1.0, [(start, tuple(k * e for k in n))], n_levels=case["levels"],
                    predicate=_refiner(case) if case["levels"] else None, precision=_precision(case),
                    stream=stream.cuda_stream)


def _precision(case):
    return B.FP32 if case["precision"] == "fp32" else B.FP64


def _rng(seed):
    return np.random.Generator(np.random.PCG64(int(seed)))


class _Device:
    """A field's device memory as torch sees it; keeps its context alive."""

    def __init__(self, solver, field):
        self.solver = solver
        self.__cuda_array_interface__ = {"shape": (solver.n, solver.Nb, solver.Nb, solver.Nb), "typestr": "<f8",
                                         "data": (solver.device_ptr(field), False), "version": 3}


def _view(solver, field):
    return torch.as_tensor(_Device(solver, field), device="cuda")


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def _sum_of_gaussians(g, amp, base, dx, e):
    """Values at the cell centres of the blocks with lower corners base (level cells) and spacings dx: (blocks, z, y, x)."""
    i = torch.arange(e, device="cuda", dtype=torch.float64) + 0.5
    out = torch.zeros((len(dx), e, e, e), dtype=torch.float64, device="cuda")
    b, h = _t(np.asarray(base, np.float64)), _t(np.asarray(dx, np.float64))
    for (_, s, c), a in zip(g, amp):
        f = [torch.exp(-(((b[:, d, None] + i) * h[:, None] - c[d]) ** 2) / (2.0 * s * s)) for d in range(3)]
        out.addcmul_((f[2] * float(a))[:, :, None, None], f[1][:, None, :, None] * f[0][:, None, None, :])
    return out


def _amplitudes(case, seed):
    r = _rng(seed)
    return [a * r.uniform(0.5, 1.5) for a, _, _ in _gaussians(case)]


def _fill_source(case, solver, field, seed):
    leaf = np.nonzero(solver.leaf)[0]
    dx = 0.5 ** (solver.levels[leaf] - solver.base_level)
    v = _view(solver, field)
    v.zero_()
    v[_t(leaf), 1:-1, 1:-1, 1:-1] = _sum_of_gaussians(_gaussians(case), _amplitudes(case, seed), solver.bbase[leaf],
                                                     dx, case["extent"])


# ----------------------------------------------------------------- prepare
class State:
    pass


@functools.lru_cache(maxsize=None)
def _stream():
    return torch.cuda.Stream()


def prepare(case, seed):
    s = State()
    s.kind, s.stream = case["kind"], _stream()
    globals()["_prepare_" + s.kind](case, int(seed), s)
    torch.cuda.synchronize()
    return s


def _prepare_conv(case, seed, s):
    e = case["extent"]
    nb, p = e + 2, 2 * (e + 2) - 1
    s.g = B.Solver((-e, -e, -e), (2 * e,) * 3, e, 1.0, [((-e, -e, -e), (e, e, e))], precision=_precision(case),
                   stream=s.stream.cuda_stream)
    s.src, s.kernel, s.out = _conv_inputs(nb, p, seed)
    s.scale = case["scale"]


def _conv_inputs(nb, p, seed):
    """A block, a kernel that decays like the Green's function, and a block to add to."""
    r = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *n: torch.randn(n, generator=r, device="cuda", dtype=torch.float64)  # noqa: E731
    i = torch.arange(p, device="cuda", dtype=torch.float64) - (nb - 1)
    d = (i[:, None, None] ** 2 + i[None, :, None] ** 2 + i[None, None, :] ** 2 + 0.06).sqrt()
    return rnd(nb, nb, nb), -(1.0 + 0.01 * rnd(p, p, p)) / (4 * math.pi * d), rnd(nb, nb, nb)


def _prepare_poisson(case, seed, s):
    s.g = _octree(case, s.stream)
    s.src, s.tgt = s.g.field(), s.g.field()
    torch.cuda.synchronize()
    _fill_source(case, s.g, s.src, seed)
    torch.cuda.synchronize()
    s.g.apply_lgf(s.src, s.tgt)  # the plans of a running program
    s.out = _view(s.g, s.tgt)


def _prepare_factor(case, seed, s):
    s.g = _octree(case, s.stream)
    s.src, s.tgt, s.alpha = s.g.field(), s.g.field(), case["alpha"]
    torch.cuda.synchronize()
    _fill_source(case, s.g, s.src, seed)
    torch.cuda.synchronize()
    s.g.apply_if(s.src, s.tgt, s.alpha)
    s.out = _view(s.g, s.tgt)


def _batch_problems(case):
    """Block counts log-uniform from 1 to `most`, the blocks filling a near-cube; 4 Gaussians per problem."""
    rng = np.random.Generator(np.random.PCG64(case["layout"]))
    e, out = case["extent"], []
    counts = [int(min(max(math.floor(math.exp(rng.uniform(0.0, math.log(case["most"])))), 1), case["most"]))
              for _ in range(case["problems"])]
    for n in counts:
        a = math.ceil(round(n ** (1.0 / 3.0), 9))
        b = math.ceil(math.sqrt(n / a))
        dims = (a, b, math.ceil(n / (a * b)))
        start = [-((d + 1) // 2) * e for d in dims]
        at = [tuple(start[k] + q * e for k, q in enumerate((i % a, (i // a) % b, i // (a * b)))) for i in range(n)]
        m = 1
        while m < max(dims):
            m *= 2
        half = max(m * e // 2, e)
        g = [(rng.uniform(-1.0, 1.0), rng.uniform(2.0, 6.0) * e / 16.0,
              tuple(rng.uniform(start[k], start[k] + dims[k] * e) for k in range(3))) for _ in range(4)]
        out.append({"bd_base": (-2 * half,) * 3, "bd_extent": (4 * half,) * 3, "blocks": [(c, (e, e, e)) for c in at],
                    "gaussians": g})
    return out


def _batch_sources(case, seed):
    """The sources on all blocks of all problems, (blocks, z, y, x), and the blocks' lower corners."""
    r, e, parts, at = _rng(seed), case["extent"], [], []
    for p in _batch_problems(case):
        base = np.array([b[0] for b in p["blocks"]])
        amp = [a * r.uniform(0.5, 1.5) for a, _, _ in p["gaussians"]]
        parts.append(_sum_of_gaussians(p["gaussians"], amp, base, np.ones(len(base)), e))
        at.append(base)
    return parts, at


def _prepare_batch(case, seed, s):
    problems = _batch_problems(case)
    s.g = B.BatchSolver(case["extent"], 1.0, problems, precision=_precision(case), stream=s.stream.cuda_stream)
    s.src, s.tgt = s.g.field(), s.g.field()
    torch.cuda.synchronize()
    field = _view(s.g, s.src)
    where, pick, first = [], [], 0
    parts, corners = _batch_sources(case, seed)
    for i, at in enumerate(corners):
        view = s.g.problem(i)
        index = {tuple(c): first + k for k, c in enumerate(at.tolist())}
        for o in np.nonzero(view.leaf)[0]:
            where.append(view.offset + int(o))
            pick.append(index[tuple(view.bbase[o].tolist())])
        first += len(at)
    field[_t(np.array(where)), 1:-1, 1:-1, 1:-1] = torch.cat(parts)[_t(np.array(pick))]
    torch.cuda.synchronize()
    s.g.apply_lgf(s.src, s.tgt)
    s.out = _view(s.g, s.tgt)


def _smooth_noise(r, X):
    """A smooth field of order one: products of sines and cosines with seeded wave numbers."""
    k = r.uniform(0.5, 2.0, size=3)
    return torch.sin(k[0] * X[0]) * torch.cos(k[1] * X[1]) * torch.cos(k[2] * X[2])


def _faces(solver, dx_base, comp):
    """Coordinates of the faces normal to `comp` of every node of every block (broadcastable)."""
    i = torch.arange(solver.Nb, device="cuda", dtype=torch.float64) - 1.0
    dx = _t(dx_base * 0.5 ** (solver.levels - solver.base_level).astype(np.float64))
    b = _t(solver.bbase.astype(np.float64))
    x = [(b[:, d, None] + i + (0.0 if d == comp else 0.5)) * dx[:, None] for d in range(3)]
    return x[0][:, None, None, :], x[1][:, None, :, None], x[2][:, :, None, None]


def _start_flow(s, case, seed, value):
    """Velocity fields from value(X, comp) plus 1 % smooth seeded noise; two steps build the plans and the step's
    graph, then the start values are put back."""
    r = _rng(seed)
    noise = [_rng(r.integers(1 << 30)) for _ in range(3)]
    s.u, s.p, s.T = [s.g.field() for _ in range(3)], s.g.field(), 0.0
    torch.cuda.synchronize()
    s.out = [_view(s.g, f) for f in s.u + [s.p]]
    start = []
    for k in range(3):
        X = _faces(s.g, s.dx, k)
        start.append(value(X, k) + s.noise * _smooth_noise(noise[k], X))
    for v, f in zip(start, s.out):
        f.copy_(v)
    torch.cuda.synchronize()
    s.g.ns_step(s.u, s.p, s.dt, s.Re, 0.0, 2)
    s.g.synchronize()
    for v, f in zip(start, s.out):
        f.copy_(v)
    s.out[3].zero_()


def _ring_mesh(case):
    e, dx, levels = case["extent"], 1.0 / case["per_radius"], case["levels"]
    half = -(-3 * case["per_radius"] // e) * e
    thresh = ((), (1e-2,), (2e-3, 2e-2))[levels]

    def refine(base, extent, rl, diff):
        if rl >= levels:
            return False
        x, y, z = ((base[d] + np.arange(extent[0] + 4) - 1.5) * dx / 2 ** rl for d in range(3))
        rho = np.sqrt(x[:, None] ** 2 + y[None, :] ** 2)
        near = np.exp(-((rho - 1.0) ** 2) / 0.04).max() * np.exp(-(z ** 2) / 0.04).max()
        return bool(near > thresh[rl])
    return e, dx, half, levels, refine


def _prepare_ring(case, seed, s):
    e, s.dx, half, levels, refine = _ring_mesh(case)
    s.Re, s.noise = case["Re"], 0.005
    s.dt = 0.35 * s.dx / 2 ** levels / 0.5
    s.g = B.Solver((-2 * half,) * 3, (4 * half,) * 3, e, s.dx, [((-half,) * 3, (2 * half,) * 3)], n_levels=levels,
                   predicate=refine if levels else None, precision=_precision(case), stream=s.stream.cuda_stream)
    w2 = 0.3 ** 2  # curl of a0 exp(-d^2 / w^2) (-y, x, 0), d the distance to the core circle, speed about 0.5

    def value(X, k):
        x, y, z = X
        rho = torch.sqrt(x * x + y * y).clamp_min(1e-12)
        q = 0.5 / 2.0 * torch.exp(-((rho - 1.0) ** 2 + z * z) / w2)
        if k < 2:
            return q * 2.0 * z / w2 * (x if k == 0 else y)
        return q * (2.0 - 2.0 * rho * (rho - 1.0) / w2)
    _start_flow(s, case, seed, value)


# box, spacing and refinement radii around the sphere (a wake behind the large one)
SPHERES = {"small": (6, 1.0 / 8, (-12, -12, -12), (12, 12, 12), (1.1,)),
           "large": (16, 1.0 / 10, (-32, -32, -32), (64, 32, 32), (1.6, 1.0))}


def _sphere_mesh(case):
    e, dx, lo, hi, radii = SPHERES[case["size"]]

    def refine(base, extent, rl, diff):
        if rl >= len(radii):
            return False
        h, r = dx / 2 ** rl, radii[rl]
        a = [(base[d] - 2) * h for d in range(3)]
        b = [(base[d] + extent[d] + 2) * h for d in range(3)]
        q = [min(max(0.0, a[d]), b[d]) for d in range(3)]
        if case["size"] == "large" and rl == 0 and b[0] > -r and a[0] < 4.0 and q[1] ** 2 + q[2] ** 2 < r * r:
            return True
        return q[0] ** 2 + q[1] ** 2 + q[2] ** 2 < r * r
    return e, dx, lo, hi, len(radii), refine


def _sphere_points(h):
    n = int(math.floor(math.pi / (h * h * math.sqrt(3.0) / 2.0))) + 1
    x = np.arange(n) + 0.5
    phi, theta = np.arccos(1.0 - 2.0 * x / n), 4.0 * math.pi * x / (1.0 + math.sqrt(5.0))
    return 0.5 * np.stack([np.cos(theta) * np.sin(phi), np.sin(theta) * np.sin(phi), np.cos(phi)], 1)


def _prepare_sphere(case, seed, s):
    e, s.dx, lo, hi, levels, refine = _sphere_mesh(case)
    s.Re, s.noise = case["Re"], 0.1
    s.dt = 0.35 * s.dx / 2 ** levels
    m = 1
    while m * e < max(max(abs(v) for v in lo), max(abs(v) for v in hi)):
        m *= 2
    s.g = B.Solver((-2 * m * e,) * 3, (4 * m * e,) * 3, e, s.dx, [(lo, tuple(h - l for l, h in zip(lo, hi)))],
                   n_levels=levels, predicate=refine, precision=_precision(case), stream=s.stream.cuda_stream)
    s.g.ib_set_points(_sphere_points(case["spacing"] * s.dx / 2 ** levels), s.Re)
    s.g.ns_options((-1.0, 0.0, 0.0))  # the body at rest in a stream of speed one
    _start_flow(s, case, seed, lambda X, k: torch.zeros((), dtype=torch.float64, device="cuda"))


def _fourier_inputs(case, seed):
    r = torch.Generator(device="cuda").manual_seed(seed)
    n, nb, sep, pl = case["blocks"], case["nb"], 2 * case["modes"], case["planes"]
    rnd = lambda c: torch.randn((n, c, nb, nb), generator=r, device="cuda", dtype=torch.float64)  # noqa: E731
    return {"cell": rnd(sep), "face": rnd(3 * sep), "edge": rnd(3 * sep), "u": rnd(3 * pl), "w": rnd(3 * pl)}


def _prepare_fourier(case, seed, s):
    s.g = B.Solver((-32, -32, -32), (64, 64, 64), 16, 1.0, [((-16, -16, -16), (32, 32, 32))],
                   stream=s.stream.cuda_stream)
    s.modes, s.planes, s.inp = case["modes"], case["planes"], _fourier_inputs(case, seed)
    new = lambda c: torch.zeros((case["blocks"], c, case["nb"], case["nb"]), dtype=torch.float64, device="cuda")  # noqa: E731
    sep = 2 * s.modes
    s.out = {"laplace": new(sep), "gradient": new(3 * sep), "divergence": new(sep), "curl": new(3 * sep),
             "curl_transpose": new(3 * sep), "nonlinear": new(3 * s.planes)}


# --------------------------------------------------------------------- run
def run(s):
    if s.kind in ("poisson", "batch"):
        s.g.apply_lgf(s.src, s.tgt)
    elif s.kind == "factor":
        s.g.apply_if(s.src, s.tgt, s.alpha)
    elif s.kind in ("ring", "sphere"):
        s.T = s.g.ns_step(s.u, s.p, s.dt, s.Re, s.T, 1)
    elif s.kind == "conv":
        s.g.conv_block(s.src.data_ptr(), s.kernel.data_ptr(), s.out.data_ptr(), s.scale)
    else:
        g, i, o, m = s.g, s.inp, s.out, s.modes
        g.helm2d_op("curl", i["face"], o["curl"], m, 0.1, 2.0)
        g.helm2d_nonlinear(i["u"], i["w"], o["nonlinear"], s.planes)
        g.helm2d_op("divergence", i["face"], o["divergence"], m, 0.1, 2.0)
        g.helm2d_op("gradient", i["cell"], o["gradient"], m, 0.1, 2.0)
        g.helm2d_op("laplace", i["cell"], o["laplace"], m, 0.1, 2.0)
        g.helm2d_op("curl_transpose", i["edge"], o["curl_transpose"], m, 0.1, 2.0, -1.0)
    return s.out


# -------------------------------------------------------------------- work
def _refined(base_blocks, levels, refine, e):
    """Leaf blocks per level of the octree that the rule asks for."""
    out, at = [], [tuple(b) for b in base_blocks]
    for rl in range(levels + 1):
        up = [b for b in at if rl < levels and refine(b, (e, e, e), rl, levels - rl)]
        out.append(len(at) - len(up))
        at = [tuple(2 * b[d] + ((k >> d) & 1) * e for d in range(3)) for b in up for k in range(8)]
    return out


def _blocks_of(start, n, e):
    return [(start[0] + i * e, start[1] + j * e, start[2] + k * e)
            for k in range(n[2]) for j in range(n[1]) for i in range(n[0])]


@functools.lru_cache(maxsize=None)
def _leaf_blocks(items):
    case = dict(items)
    kind = case["kind"]
    if kind in ("poisson", "factor"):
        start, n, _, _ = _box(case)
        refine = _refiner(case) if case["levels"] else None
        return sum(_refined(_blocks_of(start, n, case["extent"]), case["levels"], refine, case["extent"]))
    if kind == "batch":
        return sum(len(p["blocks"]) for p in _batch_problems(case))
    if kind == "ring":
        e, _, half, levels, refine = _ring_mesh(case)
        return sum(_refined(_blocks_of((-half,) * 3, (2 * half // e,) * 3, e), levels, refine, e))
    e, _, lo, hi, levels, refine = _sphere_mesh(case)
    return sum(_refined(_blocks_of(lo, [(h - l) // e for l, h in zip(lo, hi)], e), levels, refine, e))


def _transforms(e):
    """Operations of the forward and the inverse transform of a block (padded to 2 (e + 2) - 1 points per axis)."""
    p = 2 * (e + 2) - 1
    return 2 * 2.5 * p ** 3 * math.log2(p ** 3)


def work(case):
    """Each input value read and each output value written once; per leaf block and solve its two transforms."""
    kind = case["kind"]
    if kind == "conv":
        nb = case["extent"] + 2
        return {"bytes": 8.0 * (3 * nb ** 3 + (2 * nb - 1) ** 3), "flops": 1.5 * _transforms(case["extent"])}
    if kind == "fourier":
        n = case["blocks"] * case["nb"] ** 2 * 8.0
        sep = 2 * case["modes"]
        return {"bytes": n * (4 * sep + 9 * case["planes"] + 4 * sep + 4 * sep + 2 * sep + 6 * sep), "flops":
                n / 8.0 * (6 * 3 * sep + 30 * case["planes"])}
    e = SPHERES[case["size"]][0] if kind == "sphere" else case["extent"]
    blocks = _leaf_blocks(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
    if kind in ("ring", "sphere"):  # velocity in, velocity and pressure out; three solves and integrating factors
        return {"bytes": 8.0 * 7 * blocks * e ** 3, "flops": 3.0 * blocks * _transforms(e)}
    return {"bytes": 16.0 * blocks * e ** 3, "flops": float(blocks * _transforms(e))}


# --------------------------------------------------------------- tolerance
def tolerance(case):
    """About four times what other transforms or sums show: FP32 against FP64 solves 3e-7 (largest 1.5e-5), FP64 solves
    and time steps in another order of sums 1e-14 to 2e-13 (the velocity past the sphere largest 6e-12, through the
    force solve), FP32 time steps with other transforms for the integrating factor 1.5e-5 (largest 1.5e-4, both of the
    pressure, a potential divided by the step size)."""
    kind = case["kind"]
    if kind == "fourier":
        return {"rel": 1e-15, "max": 1e-13}
    if kind == "sphere":
        return {"rel": 1e-11, "max": 1e-9}
    if kind == "ring":
        return {"rel": 6e-5, "max": 6e-4} if case["precision"] == "fp32" else {"rel": 1e-12, "max": 1e-11}
    return {"rel": 2e-6, "max": 1e-4} if case["precision"] == "fp32" else {"rel": 4e-13, "max": 4e-12}


# ------------------------------------------------------------------- exact
def exact(case, seed):
    """The results in 64 bits by plain sums or FFTs: block convolution and block operators, and the free-space solves
    and integrating factors on one mesh level (a refined mesh has no plain counterpart: None)."""
    kind = case["kind"]
    if kind == "conv":
        nb = case["extent"] + 2
        p = 2 * nb - 1
        src, kernel, out = _conv_inputs(nb, p, int(seed))
        n = (p + nb - 1,) * 3
        full = torch.fft.irfftn(torch.fft.rfftn(src, s=n) * torch.fft.rfftn(kernel, s=n), s=n)
        w = slice(nb - 1, 2 * nb - 1)
        return out + case["scale"] * full[w, w, w]
    if kind == "fourier":
        return _exact_fourier(case, int(seed))
    if kind == "batch":
        parts, corners = _batch_sources(case, seed)
        out = []
        for p, v, at in zip(_batch_problems(case), parts, corners):
            out.append(_on_octree(p["bd_base"], p["bd_extent"], case["extent"], v, at, _free_space))
        return torch.cat(out)
    if kind in ("poisson", "factor") and case["levels"] == 0:
        start, n, lo, size = _box(case)
        e = case["extent"]
        at = np.array(_blocks_of(start, n, e))
        v = _sum_of_gaussians(_gaussians(case), _amplitudes(case, seed), at, np.ones(len(at)), e)
        if kind == "poisson":
            return _on_octree(lo, size, e, v, at, _free_space)
        f = _bessel(np.array([case["alpha"]]), 64)[0]
        if f[e] > 1e-17:  # the library sums over adjacent blocks only
            return None
        return _on_octree(lo, size, e, v, at, lambda s: _smooth(s, f))
    return None


def _bessel(t, n):
    """e^{-2t} I_k(2t), k < n: the Fourier coefficients of exp(-2t (1 - cos theta))."""
    m = 8192
    th = 2.0 * np.pi * np.arange(m) / m
    t = torch.as_tensor(t, dtype=torch.float64, device="cuda")
    c = torch.as_tensor(1.0 - np.cos(th), device="cuda")
    return (torch.fft.rfft(torch.exp(-2.0 * t[:, None] * c[None, :]), dim=1).real[:, :n] / m).cpu().numpy()


@functools.lru_cache(maxsize=4)
def _green(n):
    """The lattice Green's function of the seven-point Laplacian for offsets 0 .. n-1 per axis: minus the integral over
    t of prod e^{-2t} I_k(2t), Gauss-Legendre on dyadic intervals up to 2^18 and the expansion of the tail."""
    x, w = np.polynomial.legendre.leggauss(28)
    edges = [0.0] + [2.0 ** k for k in range(-2, 19)]
    t = np.concatenate([0.5 * (b - a) * (x + 1) + a for a, b in zip(edges, edges[1:])])
    w = np.concatenate([0.5 * (b - a) * w for a, b in zip(edges, edges[1:])])
    f = torch.as_tensor(_bessel(t, n), device="cuda")
    yz = (f[:, :, None] * f[:, None, :]).reshape(len(t), -1)
    g = ((f * torch.as_tensor(w, device="cuda")[:, None]).T @ yz).reshape(n, n, n)
    T, i = 2.0 ** 18, torch.arange(n, device="cuda", dtype=torch.float64) ** 2
    q = (i[:, None, None] + i[None, :, None] + i[None, None, :]) / 4.0
    tail = 2 * T ** -0.5 - (q - 3.0 / 16) * (2.0 / 3) * T ** -1.5 + q * q / 2 * (2.0 / 5) * T ** -2.5 - q ** 3 / 6 * (2.0 / 7) * T ** -3.5
    return -(g + tail / (4 * math.pi) ** 1.5)


def _free_space(src):
    """The solution of the seven-point equation on the box of src (z, y, x) grown by one cell."""
    m = [d + 2 for d in src.shape]
    g = _green(max(m))[:m[0], :m[1], :m[2]]
    n = [2 * k for k in m]
    full = torch.zeros(n, dtype=torch.float64, device="cuda")
    for a in (0, 1):
        for b in (0, 1):
            for c in (0, 1):
                part = g
                at = []
                for axis, back in enumerate((a, b, c)):
                    if back:
                        part = part.narrow(axis, 1, m[axis] - 1).flip(axis)
                        at.append(slice(n[axis] - m[axis] + 1, n[axis]))
                    else:
                        at.append(slice(0, m[axis]))
                full[tuple(at)] = part
    pad = torch.zeros(n, dtype=torch.float64, device="cuda")
    pad[1:m[0] - 1, 1:m[1] - 1, 1:m[2] - 1] = src
    return torch.fft.irfftn(torch.fft.rfftn(pad) * torch.fft.rfftn(full), s=n)[:m[0], :m[1], :m[2]]


def _smooth(src, f):
    """src convolved with f[|x|] f[|y|] f[|z|], on its box grown by one cell."""
    pad = torch.nn.functional.pad(src, (1,) * 6)
    for axis in range(3):
        n = pad.shape[axis]
        i = torch.arange(n)
        d = (i[:, None] - i[None, :]).abs()
        k = torch.as_tensor(f, device="cuda")[d.clamp_max(len(f) - 1).cuda()] * (d < len(f)).cuda()
        pad = torch.movedim(torch.tensordot(k, pad, dims=([1], [axis])), 0, axis)
    return pad


def _on_octree(lo, size, e, values, corners, solve):
    """solve() of the blocks' values, on the blocks with their one-cell margins in the octree's order: all ancestors'
    blocks (zero) by level from the root, then the base blocks, each level by its interleaved coordinates."""
    c = (np.asarray(corners) - np.asarray(lo)) // e
    low = np.asarray(corners).min(0)
    n = (np.asarray(corners).max(0) - low) // e + 1
    box = torch.zeros(tuple(int(k) * e for k in n[::-1]), dtype=torch.float64, device="cuda")
    for v, at in zip(values, np.asarray(corners) - low):
        box[at[2]:at[2] + e, at[1]:at[1] + e, at[0]:at[0] + e] = v
    u = solve(box)

    def order(x):
        key = [sum(((int(q[d]) >> b) & 1) << (3 * b + d) for b in range(20) for d in range(3)) for q in x]
        return np.argsort(np.array(key, dtype=np.int64), kind="stable")
    level = int(max(size) // e).bit_length()
    above = sum(len(np.unique(c >> k, axis=0)) for k in range(1, level + 1))
    nb = e + 2
    out = torch.zeros((above + len(c), nb, nb, nb), dtype=torch.float64, device="cuda")
    for i, o in enumerate(order(c)):
        a = (np.asarray(corners)[o] - low).tolist()
        out[above + i] = u[a[2]:a[2] + nb, a[1]:a[1] + nb, a[0]:a[0] + nb]
    return out


def _exact_fourier(case, seed):
    i = _fourier_inputs(case, seed)
    dx, lz, m, pl = 0.1, 2.0, case["modes"], case["planes"]
    om = (2.0 * math.pi * torch.arange(m, device="cuda", dtype=torch.float64) / lz)[None, :, None, None]

    def at(f, x=0, y=0):
        return torch.roll(f, (-y, -x), (2, 3))

    def inner(f):
        out = torch.zeros_like(f)
        out[:, :, 1:-1, 1:-1] = f[:, :, 1:-1, 1:-1]
        return out

    def group(f, k, n):
        return f[:, k * n:(k + 1) * n]

    def dz(f):  # i omega f, real and imaginary parts interleaved
        out = torch.empty_like(f)
        out[:, 0::2], out[:, 1::2] = -f[:, 1::2] * om, f[:, 0::2] * om
        return out
    s = 2 * m
    c, F, E = i["cell"], [group(i["face"], k, s) for k in range(3)], [group(i["edge"], k, s) for k in range(3)]
    back = lambda f, **o: (f - at(f, **o)) / dx  # noqa: E731
    fwd = lambda f, **o: (at(f, **o) - f) / dx  # noqa: E731
    out = {
        "laplace": (at(c, x=1) + at(c, x=-1) + at(c, y=1) + at(c, y=-1) - 4 * c) / dx ** 2 + dz(dz(c)),
        "gradient": torch.cat([back(c, x=-1), back(c, y=-1), dz(c)], 1),
        "divergence": fwd(F[0], x=1) + fwd(F[1], y=1) + dz(F[2]),
        "curl": torch.cat([back(F[2], y=-1) - dz(F[1]), dz(F[0]) - back(F[2], x=-1),
                           back(F[1], x=-1) - back(F[0], y=-1)], 1),
        "curl_transpose": -torch.cat([fwd(E[2], y=1) - dz(E[1]), dz(E[0]) - fwd(E[2], x=1),
                                      fwd(E[1], x=1) - fwd(E[0], y=1)], 1),
    }
    U, W = [group(i["u"], k, pl) for k in range(3)], [group(i["w"], k, pl) for k in range(3)]
    zy, zx = W[2] * (U[1] + at(U[1], x=-1)), W[2] * (U[0] + at(U[0], y=-1))
    xy, yx = W[0] * U[1], W[1] * U[0]
    out["nonlinear"] = torch.cat([
        0.5 * W[1] * (U[2] + at(U[2], x=-1)) - 0.25 * (zy + at(zy, y=1)),
        0.25 * (zx + at(zx, x=1)) - 0.5 * W[0] * (U[2] + at(U[2], y=-1)),
        0.5 * (xy + at(xy, y=1) - yx - at(yx, x=1))], 1)
    return {k: inner(v) for k, v in out.items()}
