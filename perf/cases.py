"""Performance cases of the channel solver: the calls that a two-phase channel-flow program makes in each time step.

A program holds its fields on the GPU, makes the solver handles once and calls, per Runge-Kutta substep, the surface
tension, the material properties, the momentum predictor and the pressure projection (FAST_MODE, direct solver), or
the MG_MODE projection; an ensemble projects many small channels in one call.  Sizes are those of the benchmark's
configurations, of the tests and of the grids in between: nx/2 and nz are 2^a or 3*2^a, ny is anything.

``prepare`` builds what such a program has in hand (seeded fields with bubbles, the handles), ``run`` makes one pass,
``exact`` computes the same outputs in plain torch, in 64 bits.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from tbfsolver_b200.fields import Field, VField, field_shape
from tbfsolver_b200.grid import Grid
from tbfsolver_b200.solver import (PCG, VOF, Ensemble, FlowControl, MomentumEqn, PoissonEqn, FastPoissonSolver,
                                   compute_surface_tension)

DT, ALPHA = 1e-4, 1.0
GAMMA, XI = 1.5, -0.5          # Adams-Bashforth 2
RHOL, RHOG, MUL, MUG = 1.0, 0.02, 5e-3, 1e-4
SIGMA, GCH, RET = 0.05, 0.3, 180.0
LX, LY, LZ = 2.0 * math.pi, 2.0, math.pi
CELL = ("cl", "sx", "sy", "sz")
# the multigrid solver stops at ||r||/||q|| <= 1e-10, the mixed one at 1e-10 on residual and divergence
TOL_ITER = 1e-10


def _case(kind, nx, ny, nz, **kw):
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "stretched": True, "by": max(1, nx // 96), "wait": True}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest channel of the tests: launches and host latency
        dict(_case("projection", 32, 24, 16), name="projection 32x24x16"),
        # a coarse production run, no power of two anywhere, driven asynchronously
        dict(_case("projection", 96, 100, 48, stretched=False, wait=False), name="projection 96x100x48"),
        # a middle-sized channel; the program reads max|div u| after every projection
        dict(_case("projection", 256, 256, 128), name="projection 256x256x128"),
        # the headline channel
        dict(_case("projection", 512, 384, 256), name="projection 512x384x256"),
        # the largest channel that the direct solver's transforms take in x and z
        dict(_case("projection", 1024, 512, 512, by=8), name="projection 1024x512x512"),
        # the mixed-precision refined projection of the headline channel
        dict(_case("mixed", 512, 384, 256), name="mixed 512x384x256"),
        # MG_MODE: variable-coefficient PCG with multigrid, six levels
        dict(_case("mg", 256, 256, 128, levels=6), name="mg 256x256x128"),
        # the momentum predictor alone, with a TVD limiter
        dict(_case("momentum", 256, 200, 128, scheme=3), name="momentum vanleer 256x200x128"),
        # the surface tension of the headline channel
        dict(_case("surface", 512, 384, 256), name="surface 512x384x256"),
        # one substep of a bubbly flow with surface tension
        dict(_case("substep", 256, 256, 128, scheme=2, tension=True), name="substep tension 256x256x128"),
        # one substep of the headline channel without surface tension
        dict(_case("substep", 512, 384, 256, scheme=2, tension=False), name="substep 512x384x256"),
        # sixteen channels of the reference's minimal box projected in one call
        dict(_case("ensemble", 128, 192, 64, by=1, members=16), name="ensemble 16"),
    ]


def _member_size(case, m):
    """Grid of ensemble member m: the case's sizes and the next smaller ones."""
    half = lambda n, q: (n, n * 3 // 4, n // 2)[q]  # noqa: E731
    return half(case["nx"], m % 3), half(case["ny"], (m // 3) % 3), half(case["nz"], (m // 2) % 3)


def draw(rng):
    kind = rng.choice(("projection",) * 4 + ("solve", "mixed", "mg", "momentum", "surface", "substep", "substep",
                                            "ensemble"))
    lens = [8, 12, 16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512]
    top = {"projection": 6e7, "solve": 6e7, "mixed": 5e7, "mg": 4e6, "momentum": 5e7, "surface": 5e7, "substep": 5e7,
           "ensemble": 2e6}[kind]
    bot = {"mg": 3e4, "mixed": 1e5}.get(kind, 1e4)
    while True:
        cells = math.exp(rng.uniform(math.log(bot), math.log(top)))
        nx = 2 * rng.choice(lens)
        nz = rng.choice(lens)
        ny = int(cells / (nx * nz))
        if kind == "mg":  # every extent divisible by 2^(levels-1), at least two cells on the coarsest level
            levels = rng.choice((3, 4, 5))
            f = 2 ** (levels - 1)
            ny -= ny % f
            n_c = (nx // f) * (ny // f) * (nz // f)
            if nx % f or nz % f or min(nx, ny, nz) < 2 * f or n_c > 600:
                continue
            h = (LX / nx, LY / ny, LZ / nz)  # point smoothing wants cells that are not too flat
            if max(h) > 3.2 * min(h):
                continue
        if kind == "ensemble" and (nx % 16 or nz % 8 or ny < 32 or nx > 256 or nz > 128 or ny > 256):
            continue
        if 8 <= ny <= 512 and nz >= 8 and max(nx, ny, nz) <= (8 if kind == "mixed" else 24) * min(nx, ny, nz):
            break
    c = _case(kind, nx, ny, nz, stretched=rng.random() < 0.7, wait=rng.random() < 0.5)
    if kind == "projection":
        c["tension"] = rng.random() < 0.4
    if kind == "mg":
        c["levels"] = levels
    if kind in ("momentum", "substep"):
        c["scheme"] = rng.randrange(6)
    if kind == "substep":
        c["tension"] = rng.random() < 0.5
    if kind == "ensemble":
        c["members"] = rng.choice((3, 8, 16))
        c["by"] = 1
        for n, q in (("nx", 16), ("nz", 8)):  # the smaller members need lengths 2^a or 3*2^a as well
            while c[n] % 3 == 0 or c[n] & (c[n] - 1):
                c[n] = 1 << (c[n].bit_length() - 1)
            c[n] = max(c[n], q)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _grid(case, nx=None, ny=None, nz=None):
    return Grid(nx or case["nx"], ny or case["ny"], nz or case["nz"], LX, LY, LZ, case["stretched"], 1.5)


class _Space:
    """Coordinates and spacings of the channel, plain formulas (index 0 of each array is Fortran index -1)."""

    def __init__(self, nx, ny, nz, stretched, dev):
        self.n = (nx, ny, nz)
        self.d = (LX / nx, None, LZ / nz)
        f = lambda q: torch.tensor(q, dtype=torch.float64, device=dev)  # noqa: E731
        s = np.arange(-1, ny + 2, dtype=np.float64)
        hyper = lambda q: 0.5 * LY * (1.0 + np.tanh(-1.5 + 3.0 * q / ny) / math.tanh(1.5))  # noqa: E731
        line = lambda q: LY * q / ny  # noqa: E731
        pos = hyper if stretched else line
        yf, yc = pos(s), pos(s - 0.5)
        self.yf, self.yc = f(yf), f(yc)                                   # yf(-1..ny+1), yc(-1..ny+1)
        self.dyf = f(np.concatenate([[yf[1] - pos(-1.0)], np.diff(yf)]))  # dyf(-1..): [0] unused, dyf(j) = yf(j)-yf(j-1)
        self.dyc = f(np.concatenate([[np.nan], np.diff(yc)]))             # dyc(j) = yc(j) - yc(j-1)

    def at(self, t, j0, j1):
        return t[j0 + 1:j1 + 2][None, :, None]

    def df(self, d, box, o=0):
        return self.d[d] if d != 1 else self.at(self.dyf, box[2] + o, box[3] + o)

    def dc(self, d, box, o=0):
        return self.d[d] if d != 1 else self.at(self.dyc, box[2] + o, box[3] + o)


def _space(case, dev, size=None):
    return _Space(*(size or (case["nx"], case["ny"], case["nz"])), case["stretched"], dev)


_LO = {"cl": (1, 1, 1), "sx": (0, 1, 1), "sy": (1, 0, 1), "sz": (1, 1, 0)}


def _cut(a, kind, hd, box, s=(0, 0, 0)):
    """View of the Fortran index box (i0, i1, j0, j1, k0, k1) of a field array, shifted by s."""
    li, lj, lk = (q - hd for q in _LO[kind])
    return a[box[4] + s[2] - lk:box[5] + s[2] - lk + 1, box[2] + s[1] - lj:box[3] + s[1] - lj + 1,
             box[0] + s[0] - li:box[1] + s[0] - li + 1]


def _ghosts(a, n, hd=1):
    """Cell field: zero-gradient walls (first ghost row), then periodic halos in x and z."""
    nx, ny, nz = n
    o = hd
    a[:, o - 1] = a[:, o]
    a[:, o + ny] = a[:, o + ny - 1]
    a[:, :, o + nx:] = a[:, :, o:2 * o]
    a[:, :, :o] = a[:, :, nx:nx + o]
    a[o + nz:] = a[o:2 * o]
    a[:o] = a[nz:nz + o]


def _velocity_ghosts(u, sp, hd=2):
    """Velocity triple: no-slip walls (one ghost row), periodic halos and duplicate faces in x and z."""
    nx, ny, nz = sp.n
    y = lambda t, j: float(t[j + 1])  # noqa: E731
    for kind, a in zip(CELL[1:], u):
        lo = _LO[kind]
        if kind == "sy":
            ends = ((-1, 1, y(sp.dyf, 0), y(sp.dyf, 0) + y(sp.dyf, 1)),
                    (ny + 1, ny - 1, y(sp.dyf, ny + 1), y(sp.dyf, ny) + y(sp.dyf, ny + 1)))
        else:
            ends = ((0, 1, y(sp.yf, 0) - y(sp.yc, 0), y(sp.dyc, 1)),
                    (ny + 1, ny, y(sp.yc, ny + 1) - y(sp.yf, ny), y(sp.dyc, ny + 1)))
        oj = lo[1] - hd
        inner = (slice(hd, hd + nz + 1 - lo[2]), slice(hd, hd + nx + 1 - lo[0]))
        for g, b, hb, hi in ends:
            a[inner[0], g - oj, inner[1]] = a[inner[0], b - oj, inner[1]] * hb / (hb - hi)
        for ax, n, stag in ((2, nx, lo[0] == 0), (0, nz, lo[2] == 0)):
            first, last = lo[2 - ax], n                 # interior range first..last, n cells per period
            o = first - hd
            v = a.movedim(ax, 0)
            for h in range(1, hd + 1):
                v[last + h - o] = v[last + h - n - o].clone()
                v[first - h - o] = v[first - h + n - o].clone()
            if stag:
                v[-o] = v[n - o].clone()


def _fields(case, seed, dev, size=None):
    """Seeded fields: volume fraction with by rows of bubbles, smoothed properties, velocity, two pressure levels."""
    sp = _space(case, dev, size)
    nx, ny, nz = n = sp.n
    gen = torch.Generator(device=dev).manual_seed(1000003 * (seed % (1 << 32)) + 17 * nx + 5 * ny + nz)
    rand = lambda *shape: torch.rand(*shape, generator=gen, dtype=torch.float64, device=dev)  # noqa: E731
    by = case["by"]
    nb = (max(1, round(by * LX / LY / 2)), by, max(1, round(by * LZ / LY / 1.5)))
    blk = [L / b for L, b in zip((LX, LY, LZ), nb)]
    R = 0.25 * min(blk)
    y = sp.yc[2:ny + 2]
    pos = [(torch.arange(nx, device=dev, dtype=torch.float64) + 0.5) * sp.d[0], y,
           (torch.arange(nz, device=dev, dtype=torch.float64) + 0.5) * sp.d[2]]
    site = [torch.clamp((p / b).long(), max=m - 1) for p, b, m in zip(pos, blk, nb)]
    jit = [0.8 * (0.5 * b - R) * (2.0 * rand(nb[2], nb[1], nb[0]) - 1.0) for b in blk]
    idx = (site[2][:, None, None], site[1][None, :, None], site[0][None, None, :])
    off = []
    for d, shape in ((0, (1, 1, -1)), (1, (1, -1, 1)), (2, (-1, 1, 1))):
        centre = ((site[d] + 0.5) * blk[d]).reshape(shape)
        off.append(pos[d].reshape(shape) - centre - jit[d][idx])
    dist = (off[0] ** 2 + off[1] ** 2 + off[2] ** 2).sqrt_()
    h = [sp.d[0], sp.at(sp.dyf, 1, ny), sp.d[2]]
    # width of the cell along the bubble's normal: the fraction falls linearly across it
    width = sum(o.abs() * w for o, w in zip(off, h)) / dist.clamp_min(1e-12)
    del off
    cell = lambda v: _padded(v, n)  # noqa: E731
    dist -= R
    f = {"c": cell((0.5 - dist / width).clamp_(0.0, 1.0))}
    cs = cell((0.5 - dist / (3.0 * width)).clamp_(0.0, 1.0))
    del dist, width
    f["rho"] = RHOG * cs + (1.0 - cs) * RHOL
    f["mu"] = MUG * cs + (1.0 - cs) * MUL
    del cs
    for kind in CELL[1:]:
        a = torch.zeros(field_shape(kind, 2, nx, ny, nz), dtype=torch.float64, device=dev)
        lo = _LO[kind]
        inner = _cut(a, kind, 2, (lo[0], nx, lo[1], ny, lo[2], nz))
        inner.copy_(rand(*inner.shape).sub_(0.5).mul_(0.1))
        if kind == "sx":
            inner += (1.5 * y * (LY - y))[None, :, None]
        if kind == "sy":
            inner[:, 0] = 0.0
            inner[:, -1] = 0.0
        f[kind] = a
    u = [f[k] for k in CELL[1:]]
    _velocity_ghosts(u, sp)
    wave = lambda m, p: torch.cos(m * p)  # noqa: E731
    ph = 2.0 * math.pi * rand(2)
    smooth = (wave(1, pos[0] + ph[0])[None, None, :] * wave(math.pi / LY, y)[None, :, None]
              * wave(2, pos[2] + ph[1])[:, None, None])
    f["pn"] = cell(0.05 * smooth + 0.01 * rand(nz, ny, nx))
    f["pnm1"] = cell(0.045 * smooth + 0.01 * rand(nz, ny, nx))
    return f, sp


def _padded(v, n, hd=1):
    a = torch.zeros(field_shape("cl", hd, *n), dtype=torch.float64, device=v.device)
    a[hd:-hd, hd:-hd, hd:-hd] = v
    _ghosts(a, n, hd)
    return a


def _old_tension(f, sp):
    """An earlier level of the surface tension: sigma * 2/R * grad c with a constant curvature."""
    nx, ny, nz = n = sp.n
    out = []
    for d, kind in enumerate(CELL[1:]):
        lo = _LO[kind]
        box = (lo[0], nx, 1, ny - (d == 1), lo[2], nz)
        a = torch.zeros(field_shape(kind, 1, *n), dtype=torch.float64, device=f["c"].device)
        e = [int(d == q) for q in range(3)]
        _cut(a, kind, 1, box).copy_(10.0 * SIGMA * (_cut(f["c"], "cl", 1, box, e) - _cut(f["c"], "cl", 1, box))
                                    / sp.dc(d, box, 1))
        out.append(a)
    return out


def _vfield(arrays, hd, n):
    return VField(*[Field(k, hd, *n, a) for k, a in zip(CELL[1:], arrays)])


def _vzeros(n, hd, dev="cuda"):
    return _vfield([torch.zeros(field_shape(k, hd, *n), dtype=torch.float64, device=dev) for k in CELL[1:]], hd, n)


@functools.lru_cache(maxsize=1)
def _stream():
    """The one stream that the program drives its solvers on."""
    return torch.cuda.Stream()


def prepare(case, seed):
    kind, dev = case["kind"], torch.device("cuda")
    s = {"kind": kind}
    if kind == "ensemble":
        s["meshes"], s["members"] = [], []
        for m in range(case["members"]):
            size = _member_size(case, m)
            f, sp = _fields(case, seed + 7919 * m, dev, size)
            cl = lambda a: Field("cl", 1, *size, a)  # noqa: B023,E731
            s["meshes"].append(_grid(case, *size))
            s["members"].append((cl(torch.zeros_like(f["pn"])), cl(f["pn"]), cl(f["pnm1"]), cl(f["rho"]),
                                 _vfield([f[k] for k in CELL[1:]], 2, size), _vzeros(size, 2)))
        torch.cuda.synchronize()
        s["ens"] = Ensemble(s["meshes"], nstreams=len(s["meshes"]))
        return s
    f, sp = _fields(case, seed, dev)
    n, g = sp.n, _grid(case)
    for k in ("c", "rho", "mu", "pn", "pnm1"):
        s[k] = Field("cl", 1, *n, f[k])
    s["u"] = _vfield([f[k] for k in CELL[1:]], 2, n)
    s["psi"] = Field("cl", 1, *n, torch.zeros_like(f["pn"]))
    s["wait"] = case["wait"]
    how = {"asynchronous": not case["wait"], "stream": _stream().cuda_stream}
    if kind in ("projection", "mixed", "substep"):
        s["out"] = _vzeros(n, 2)
        s["eqn"] = PoissonEqn(g, RHOL, RHOG, precision="mixed" if kind == "mixed" else "fp64", tol=TOL_ITER,
                              **how)
    s["st"] = s["sto"] = None
    if case.get("tension"):
        s["sto"] = list(_vfield(_old_tension(f, sp), 1, n).components())
        s["st"] = list(_vfield([a.a * 1.05 for a in s["sto"]], 1, n).components())
    if kind == "solve":
        s["fps"] = FastPoissonSolver(g, **how)
    if kind == "mg":
        s["out"] = _vzeros(n, 2)
        s["pcg"] = PCG(g, n_levels=case["levels"], tol_pcg=TOL_ITER, max_iter_pcg=400, stream=how["stream"])
    if kind == "surface":
        s["fps"] = FastPoissonSolver(g, **how)
        s["st"] = _vzeros(n, 1)
    if kind in ("momentum", "substep"):
        solver = s["eqn"].solver if kind == "substep" else FastPoissonSolver(g, **how)
        s["fps"] = solver
        s["mom"] = MomentumEqn(solver, scheme=case["scheme"], gch=GCH)
        s["ustar"] = _vzeros(n, 2)
        torch.cuda.synchronize()
        if kind == "substep":
            s["vof"] = VOF(solver, RHOL, RHOG, MUL, MUG)
            s["flow"] = FlowControl(solver, 1, ret=RET)
            s["cs"] = Field("cl", 1, *n, torch.zeros_like(f["pn"]))
            s["vof"].update_material_props(s["c"], s["cs"], s["rho"], s["mu"])
        # the step before this one leaves its fluxes in the handle
        s["mom"].predictor(s["u"], s["c"], s["mu"], s["rho"], DT, ALPHA, GAMMA, XI, RHOG, u_out=s["ustar"])
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind in ("projection", "mixed"):
        s["eqn"].projection(s["psi"], s["pn"], s["pnm1"], s["rho"], s["u"], DT, ALPHA, s["st"], s["sto"],
                            u_out=s["out"], want_stats=s["wait"])
        return [s["psi"].a] + [c.a for c in s["out"].components()]
    if kind == "solve":
        s["fps"].solve_fps(s["psi"], s["pn"])
        return s["psi"].a
    if kind == "mg":
        with torch.cuda.stream(_stream()):
            s["psi"].a.zero_()  # the guess
        s["pcg"].projection(s["psi"], s["rho"], s["u"], DT, ALPHA, u_out=s["out"])
        return [s["psi"].a] + [c.a for c in s["out"].components()]
    if kind == "surface":
        compute_surface_tension(s["fps"], s["c"], SIGMA, s["st"])
        return [c.a for c in s["st"].components()]
    if kind == "momentum":
        s["mom"].solve(s["u"], s["c"], s["mu"], s["rho"], DT, ALPHA, GAMMA, XI, RHOG, fs=0.1, u_out=s["ustar"])
        return [c.a for c in s["ustar"].components()]
    if kind == "substep":
        if s["st"] is not None:
            compute_surface_tension(s["fps"], s["c"], SIGMA, VField(*s["st"]))
        s["vof"].update_material_props(s["c"], s["cs"], s["rho"], s["mu"])
        fs = s["flow"].set_press_grad(s["rho"], RHOL, MUL, GCH)
        s["mom"].solve(s["u"], s["c"], s["mu"], s["rho"], DT, ALPHA, GAMMA, XI, RHOG, fs=fs, st=s["st"],
                       u_out=s["ustar"])
        s["eqn"].projection(s["psi"], s["pn"], s["pnm1"], s["rho"], s["ustar"], DT, ALPHA, s["st"], s["sto"],
                            u_out=s["out"], want_stats=s["wait"])
        s["mom"].update_boundaries_v(s["out"])
        return [s["psi"].a, s["cs"].a, s["rho"].a, s["mu"].a] + [c.a for c in s["out"].components()]
    s["ens"].projection(s["members"], DT, ALPHA, RHOG)
    return [[m[0].a] + [c.a for c in m[5].components()] for m in s["members"]]


def work(case):
    """Bytes: every input field read once, every output written once, 8 bytes a cell and field, and for the
    transforms, whose lines run in three directions, nothing more.  Flops: the arithmetic of the stencils and
    transforms."""
    kind = case["kind"]
    sizes = [_member_size(case, m) for m in range(case["members"])] if kind == "ensemble" else \
        [(case["nx"], case["ny"], case["nz"])]
    b = f = 0.0
    for nx, ny, nz in sizes:
        N = float(nx) * ny * nz
        fft = 5.0 * math.log2(nx * nz) * N + 12.0 * N
        tension = 48.0 * N if case.get("tension") else 0.0
        if kind in ("projection", "ensemble", "mixed"):   # u*, rho, psi^n, psi^n-1 -> u, psi
            b, f = b + 80.0 * N + tension, f + fft + 100.0 * N
        elif kind == "solve":
            b, f = b + 16.0 * N, f + fft
        elif kind == "mg":                                # u*, rho, guess -> u, psi
            b, f = b + 72.0 * N, f + 20 * 100.0 * N
        elif kind == "surface":
            b, f = b + 32.0 * N, f + 30.0 * N
        elif kind == "momentum":                          # u, c, mu, rho, fluxes -> u*, fluxes
            b, f = b + 120.0 * N, f + 400.0 * N
        elif kind == "substep":                           # c, u, fluxes, psi^n, psi^n-1 -> cs, rho, mu, fluxes, u, psi
            b, f = b + 152.0 * N + tension, f + fft + 560.0 * N
    return {"bytes": b, "flops": f}


def tolerance(case):
    """FP64 throughout, each about four times what the paths are seen to be off exact(), where sums in another order
    or other roundings show.  The iterative solvers leave what their stopping rule of 1e-10 leaves: the multigrid
    solver's pressure has its residual times the operator's condition, and may stop an iteration earlier or later."""
    return {"mg": {"rel": 1e-7, "max": 1e-5}, "mixed": {"rel": 1e-9, "max": 1e-7},
            "momentum": {"rel": 1e-14, "max": 1e-11}, "surface": {"rel": 1e-12, "max": 1e-9}}.get(
        case["kind"], {"rel": 4e-11, "max": 1e-8})


# ---------------------------------------------------------------------------
# the same outputs in plain torch
# ---------------------------------------------------------------------------
def _solve_y(spec, sp):
    """Thomas sweeps along y of the spectrum spec[k, j, kx] (in place); the (0, 0) system keeps its last unknown 0."""
    nx, ny, nz = sp.n
    dev = spec.device
    ang = lambda n, m: 2.0 * (torch.cos(2.0 * math.pi * torch.arange(m, device=dev, dtype=torch.float64) / n) - 1.0)  # noqa: E731
    lam = ang(nz, nz)[:, None] / sp.d[2] ** 2 + ang(nx, nx // 2 + 1)[None, :] / sp.d[0] ** 2
    df, dc = sp.dyf[2:ny + 2].tolist(), sp.dyc[2:ny + 3].tolist()
    am = [0.0] + [1.0 / (dc[j] * df[j]) for j in range(1, ny)]
    ap = [1.0 / (dc[j + 1] * df[j]) for j in range(ny - 1)] + [0.0]
    cp = []
    for j in range(ny):
        diag = lam - (am[j] + ap[j])
        if j:
            diag = diag - am[j] * cp[-1]
            spec[:, j] -= am[j] * spec[:, j - 1]
        if j == ny - 1:
            diag[0, 0] = 1.0
            spec[0, j, 0] = 0.0
        inv = 1.0 / diag
        cp.append(ap[j] * inv)
        spec[:, j] *= inv
    for j in range(ny - 2, -1, -1):
        spec[:, j] -= cp[j] * spec[:, j + 1]


def _direct(s, sp):
    """L^{-1} s of the constant-coefficient operator, zero mean over the volume; s[k, j, i]."""
    nx, ny, nz = sp.n
    spec = torch.fft.fft(torch.fft.rfft(s, dim=2), dim=0)
    _solve_y(spec, sp)
    p = torch.fft.irfft(torch.fft.ifft(spec, dim=0), n=nx, dim=2)
    p -= (p * sp.at(sp.dyf, 1, ny)).sum() / (nx * nz * LY)
    return p


def _divergence(u, sp):
    nx, ny, nz = sp.n
    box = (1, nx, 1, ny, 1, nz)
    out = 0.0
    for d, kind in enumerate(CELL[1:]):
        e = [-int(d == q) for q in range(3)]
        out = out + (_cut(u[d], kind, 2, box) - _cut(u[d], kind, 2, box, e)) / sp.df(d, box)
    return out


def _faces(d, n, walls=False):
    """Index box of the faces of direction d that the equations act on (walls: with the y wall faces)."""
    box = [1, n[0], 1, n[1], 1, n[2]]
    box[2 * d] = 0 if d != 1 or walls else 1
    if d == 1 and not walls:
        box[3] = n[1] - 1
    return tuple(box)


def _unit(d):
    return [int(d == q) for q in range(3)]


def _face_grad(p, d, box, sp):
    return (_cut(p, "cl", 1, box, _unit(d)) - _cut(p, "cl", 1, box)) / sp.dc(d, box, 1)


def _face_irho(rho, d, box):
    return 0.5 * (1.0 / _cut(rho, "cl", 1, box, _unit(d)) + 1.0 / _cut(rho, "cl", 1, box))


def _old_grad(f, d, box, sp, st, sto):
    """Extrapolated old pressure gradient 2 p^n - p^n-1 on faces, less its surface tension."""
    g = 2.0 * _face_grad(f["pn"], d, box, sp) - _face_grad(f["pnm1"], d, box, sp)
    if st is not None:
        kind = CELL[1 + d]
        g = g - 2.0 * _cut(st[d], kind, 1, box) + _cut(sto[d], kind, 1, box)
    return g


def _projected(f, sp, st=None, sto=None):
    n = sp.n
    s = _divergence([f[k] for k in CELL[1:]], sp) * (RHOG / (ALPHA * DT))
    for d in range(3):
        box = _faces(d, n)
        t = (1.0 - RHOG * _face_irho(f["rho"], d, box)) * _old_grad(f, d, box, sp, st, sto)
        if d == 1:  # nothing through the walls
            t = torch.nn.functional.pad(t, (0, 0, 1, 1))
        s += t.diff(dim=2 - d) / sp.df(d, (1, n[0], 1, n[1], 1, n[2]))
        del t
    psi = _padded(_direct(s, sp), n)
    del s
    out = []
    for d, kind in enumerate(CELL[1:]):
        box = _faces(d, n)
        a = torch.zeros_like(f[kind])
        whole = _faces(d, n, walls=True)
        _cut(a, kind, 2, whole).copy_(_cut(f[kind], kind, 2, whole))
        grad = _face_grad(psi, d, box, sp) / RHOG
        grad += (_face_irho(f["rho"], d, box) - 1.0 / RHOG) * _old_grad(f, d, box, sp, st, sto)
        _cut(a, kind, 2, box).sub_(grad.mul_(DT * ALPHA))
        out.append(a)
        del grad
    return psi, out


def _variable(f, sp):
    """MG_MODE: div((dt alpha / rho) grad psi) = div u* by conjugate gradients preconditioned with the direct solver."""
    n = sp.n
    cells = (1, n[0], 1, n[1], 1, n[2])
    vol = sp.at(sp.dyf, 1, n[1])
    beta = [DT * ALPHA * _face_irho(f["rho"], d, _faces(d, n)) for d in range(3)]

    def apply(p):
        a, out = _padded(p, n), 0.0
        for d in range(3):
            box = _faces(d, n)
            t = beta[d] * _face_grad(a, d, box, sp)
            if d == 1:
                t = torch.nn.functional.pad(t, (0, 0, 1, 1))
            out = out + t.diff(dim=2 - d) / sp.df(d, cells)
        return out

    r = _divergence([f[k] for k in CELL[1:]], sp)
    p, rz, d = torch.zeros_like(r), None, None
    stop = 1e-13 * float(r.norm())
    for _ in range(400):
        z = _direct(r, sp)
        new = float((r * z * vol).sum())
        d = z if d is None else z + (new / rz) * d
        rz = new
        q = apply(d)
        a = rz / float((d * q * vol).sum())
        p += a * d
        r -= a * q
        if float(r.norm()) < stop:
            break
    psi = _padded(p - p.mean(), n)
    out = []
    for d, kind in enumerate(CELL[1:]):
        box, whole = _faces(d, n), _faces(d, n, walls=True)
        a = torch.zeros_like(f[kind])
        _cut(a, kind, 2, whole).copy_(_cut(f[kind], kind, 2, whole))
        _cut(a, kind, 2, box).sub_(beta[d] * _face_grad(psi, d, box, sp))
        out.append(a)
    return psi, out


def _limiter(num, den, scheme, sharp):
    r = num / torch.where(den == 0.0, 1e-50, den)
    if scheme == 2:
        return (r + 3.0) / 4.0
    r = r.clamp_min(0.0)
    if scheme == 3:
        return 2.0 * r / (1.0 + r)
    sb = torch.maximum((2.0 * r).clamp_max(1.0), r.clamp_max(2.0))
    return sb if scheme == 4 else torch.where(sharp, sb, 1.0)


def _momentum(f, sp, scheme, fs, st=None):
    """The predictor's velocity with its boundaries: u + dt (gamma + xi) phi(u) + sources."""
    n, out = sp.n, []
    vel = [f[k] for k in CELL[1:]]
    for d, kind in enumerate(CELL[1:]):
        box = _faces(d, n)
        ed = _unit(d)
        sh = lambda *vs: [sum(q) for q in zip(*vs)]  # noqa: E731
        U = lambda s=(0, 0, 0): _cut(vel[d], kind, 2, box, s)  # noqa: B023,E731
        M = lambda s=(0, 0, 0): _cut(f["mu"], "cl", 1, box, s)  # noqa: B023,E731
        C = lambda s: _cut(f["c"], "cl", 1, box, s)  # noqa: B023,E731
        neg = lambda s: [-q for q in s]  # noqa: E731
        sharp = False
        if scheme == 5:
            for e in range(3):
                sharp = sharp | ((C(_unit(e)) - C([0, 0, 0] if e == d else neg(_unit(e)))) > np.finfo(np.float64).eps)
        phi, visc = 0.0, 0.0
        for e in range(3):
            ee, me = _unit(e), neg(_unit(e))
            W = lambda s=(0, 0, 0): _cut(vel[e], CELL[1 + e], 2, box, s)  # noqa: B023,E731
            div = sp.dc(d, box, 1) if e == d else sp.df(e, box)
            for side, lo, hi in ((1, [0, 0, 0], ee), (-1, me, [0, 0, 0])):
                if e == d:
                    q = 0.5 * (U(lo) + U(hi))
                else:
                    at = [0, 0, 0] if side > 0 else me
                    q = (W(sh(at, ed)) * sp.df(1, box, 1) + W(at) * sp.df(1, box)) * 0.5 / sp.dc(1, box, 1) \
                        if d == 1 else 0.5 * (W(sh(at, ed)) + W(at))
                a, b = U(lo), U(hi)
                if scheme == 0:
                    A, B = 0.5 * (a + b), 0.5 * (a + b)
                elif scheme == 1:
                    A, B = a, b
                else:
                    A = a + 0.5 * _limiter(a - U(sh(lo, me)), b - a, scheme, sharp) * (b - a)
                    B = b + 0.5 * _limiter(U(sh(hi, ee)) - b, b - a, scheme, sharp) * (a - b)
                phi = phi - side * (q.clamp_min(0.0) * A + q.clamp_max(0.0) * B) / div
                del A, B, q
                if e == d:
                    t = 2.0 * M(hi) * (b - a) / sp.df(d, box, 1 if side > 0 else 0)
                else:
                    to = ee if side > 0 else me
                    m = 0.25 * (M() + M(ed) + M(to) + M(sh(to, ed)))
                    at = [0, 0, 0] if side > 0 else me
                    t = m * ((b - a) / sp.dc(e, box, 1 if side > 0 else 0)
                             + (W(sh(at, ed)) - W(at)) / sp.dc(d, box, 1))
                visc = visc + side * t / div
                del t
        irho = _face_irho(f["rho"], d, box)
        phi = phi + visc * irho
        new = vel[d].clone()
        t = _cut(new, kind, 2, box)
        t += DT * (GAMMA + XI) * phi
        if st is not None:
            t += DT * ALPHA / RHOG * _cut(st[d], kind, 1, box)
        if d == 0:
            t += DT * ALPHA * (irho * fs + GCH)
        out.append(new)
        del phi, visc
    _velocity_ghosts(out, sp)
    return out


def _smoothed(c, sp):
    """Cell -> vertex -> cell twice, linear in each direction."""
    nx, ny, nz = n = sp.n
    dev = c.device
    a = c
    for _ in range(2):
        for ax, m, d in ((2, nx, 0), (1, ny, 1), (0, nz, 2)):
            if d == 1:
                xc, xf = sp.yc[1:ny + 3], sp.yf[1:ny + 2]
            else:
                r = torch.arange(m + 2, device=dev, dtype=torch.float64)
                xc, xf = (r - 0.5) * sp.d[d], r[:m + 1] * sp.d[d]
            shape = [1, 1, 1]
            shape[ax] = -1
            w = ((xf - xc[:-1]) / (xc[1:] - xc[:-1])).reshape(shape)
            v = (1.0 - w) * a.narrow(ax, 0, m + 1) + w * a.narrow(ax, 1, m + 1)
            w = ((xc[1:-1] - xf[:-1]) / (xf[1:] - xf[:-1])).reshape(shape)
            a = (1.0 - w) * v.narrow(ax, 0, m) + w * v.narrow(ax, 1, m)
        a = _padded(a, n)
    return a


def _tension(c, sp):
    """Height-function surface tension on the faces (halos: periodic images, zero outside the walls)."""
    nx, ny, nz = n = sp.n
    eps, reach, dev = 1e-12, 6, c.device
    cc = c[1:-1, 1:-1, 1:-1]
    cls = lambda a: ((a >= eps) & (a <= 1.0 - eps), a >= 1.0 - eps)  # noqa: E731
    m0, full0 = cls(c)
    empty = ~(m0 | full0)
    near = empty[1:-1, 1:-1, :-2] | empty[1:-1, 1:-1, 2:] | empty[1:-1, :-2, 1:-1] | empty[1:-1, 2:, 1:-1] \
        | empty[:-2, 1:-1, 1:-1] | empty[2:, 1:-1, 1:-1]
    promote = full0[1:-1, 1:-1, 1:-1] & near
    cp = torch.where(promote, 1.0 - 2.0 * eps, cc).contiguous()
    mixed = m0[1:-1, 1:-1, 1:-1] | promote
    full = full0[1:-1, 1:-1, 1:-1] & ~promote
    none = ~(mixed | full)
    del m0, full0, empty, near, promote
    k, j, i = torch.nonzero(mixed, as_tuple=True)
    P = [i, j, k]
    flat = lambda x: (x[2] % nz) * (ny * nx) + x[1].clamp(0, ny - 1) * nx + x[0] % nx  # noqa: E731
    val, fl, em = cp.view(-1), full.reshape(-1), none.reshape(-1)
    dyf, dyc, yf = sp.dyf[2:ny + 2], sp.dyc[2:ny + 3], sp.yf[1:ny + 2]

    def moved(base, *steps):
        x = list(base)
        for d, t in steps:
            x[d] = x[d] + t
        return x

    nv = []
    for d in range(3):
        t1, t2 = [q for q in range(3) if q != d]
        tot = 0.0
        for a in (-1, 0, 1):
            for b in (-1, 0, 1):
                w = (2 - abs(a)) * (2 - abs(b))
                tot = tot + w * (val[flat(moved(P, (d, 1), (t1, a), (t2, b)))] - val[flat(moved(P, (d, -1), (t1, a), (t2, b)))])
        if d == 1:
            yc = sp.yc[2:ny + 2]
            tot = tot / (yc[(j + 1).clamp_max(ny - 1)] - yc[(j - 1).clamp_min(0)])
        else:
            tot = tot / (2.0 * sp.d[d])
        nv.append(tot)
    mag = torch.stack([q.abs() for q in nv], 1)
    order = torch.sort(mag, dim=1, descending=True, stable=True).indices
    kap, done = torch.zeros_like(nv[0]), torch.zeros_like(mixed[k, j, i])
    for rank in range(3):
        for d in range(3):
            sel = torch.nonzero((order[:, rank] == d) & ~done).flatten()
            if not sel.numel():
                continue
            base = [q[sel] for q in P]
            s = torch.where(nv[d][sel] >= 0.0, 1, -1)
            t1, t2 = [q for q in range(3) if q != d]
            F, ok = {}, torch.ones_like(s, dtype=torch.bool)
            for a in (-1, 0, 1):
                for b in (-1, 0, 1):
                    st0 = moved(base, (t1, a), (t2, b))
                    ok &= (st0[1] >= 0) & (st0[1] < ny)

                    def walk(flags, sign):
                        end, alive = torch.full_like(s, -1), torch.ones_like(ok)  # noqa: B023
                        for t in range(reach + 1):
                            x = moved(st0, (d, sign * t * s))  # noqa: B023
                            alive = alive & (x[1] >= 0) & (x[1] < ny)
                            hit = alive & flags[flat(x)] & (end < 0)
                            end = torch.where(hit, t, end)
                        return end

                    tf, te = walk(fl, 1), walk(em, -1)
                    ok &= (tf >= 0) & (te >= 0)
                    hs = torch.zeros_like(kap[sel])
                    for t in range(-reach, reach + 1):
                        x = moved(st0, (d, t * s))
                        wd = dyf[x[1].clamp(0, ny - 1)] if d == 1 else sp.d[d]
                        hs += torch.where((t >= -te) & (t <= tf), val[flat(x)] * wd, 0.0)
                    q = st0[d] + s * tf + (s > 0)
                    F[a, b] = (yf[q.clamp(0, ny)] if d == 1 else q.double() * sp.d[d]) - s * hs
            h = []
            for t in (t1, t2):
                h.append((dyc[base[1]], dyc[base[1] + 1]) if t == 1 else (sp.d[t], sp.d[t]))
            (am, ap), (bm, bp) = h
            d1 = (am * am * F[1, 0] - ap * ap * F[-1, 0] + (ap * ap - am * am) * F[0, 0]) / (ap * am * (ap + am))
            d11 = 2.0 * (am * F[1, 0] - (ap + am) * F[0, 0] + ap * F[-1, 0]) / (ap * am * (ap + am))
            d2 = (bm * bm * F[0, 1] - bp * bp * F[0, -1] + (bp * bp - bm * bm) * F[0, 0]) / (bp * bm * (bp + bm))
            d22 = 2.0 * (bm * F[0, 1] - (bp + bm) * F[0, 0] + bp * F[0, -1]) / (bp * bm * (bp + bm))
            d12 = (F[1, 1] - F[1, -1] - F[-1, 1] + F[-1, -1]) / ((ap + am) * (bp + bm))
            g = 1.0 + d1 * d1 + d2 * d2
            v = s * (d11 * (1.0 + d2 * d2) + d22 * (1.0 + d1 * d1) - 2.0 * d1 * d2 * d12) / (g * g.sqrt())
            kap[sel] = torch.where(ok, v, 0.0)
            done[sel] = ok
    K = torch.zeros_like(cp)
    K[k, j, i] = kap
    out = []
    for d, kind in enumerate(CELL[1:]):
        ax = 2 - d
        nxt = lambda t: torch.roll(t, -1, ax)  # noqa: B023,E731
        kq, mq = nxt(K), nxt(mixed)
        kf = torch.where(mixed & mq, 0.5 * (K + kq), torch.where(mq, kq, torch.where(mixed, K, 0.0)))
        diff = nxt(cp) - cp
        if d == 1:
            diff[:, -1] = 0.0
            v = SIGMA * kf * (diff / dyc[1:][None, :, None])      # face j between cells j and j+1
        else:
            v = SIGMA * kf * (diff / sp.d[d])
        shape = field_shape(kind, 1, *n)
        a = torch.zeros(shape, dtype=torch.float64, device=dev)
        lo = [_LO[kind][q] - 1 for q in range(3)]
        gi = (torch.arange(shape[2], device=dev) + lo[0] - 1) % nx
        gk = (torch.arange(shape[0], device=dev) + lo[2] - 1) % nz
        j1 = 1 - lo[1]
        a[:, j1:j1 + ny] = v[gk][:, :, gi]
        out.append(a)
    return out


def exact(case, seed):
    kind, dev = case["kind"], torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if kind == "ensemble":
        out = []
        for m in range(case["members"]):
            f, sp = _fields(case, seed + 7919 * m, dev, _member_size(case, m))
            psi, u = _projected(f, sp)
            out.append([psi] + u)
        return out
    f, sp = _fields(case, seed, dev)
    if kind in ("projection", "mixed"):
        st = sto = None
        if case.get("tension"):
            sto = _old_tension(f, sp)
            st = [1.05 * a for a in sto]
        psi, u = _projected(f, sp, st, sto)
        return [psi] + u
    if kind == "solve":
        return _padded(_direct(f["pn"][1:-1, 1:-1, 1:-1], sp), sp.n)
    if kind == "mg":
        psi, u = _variable(f, sp)
        return [psi] + u
    if kind == "surface":
        return _tension(f["c"], sp)
    if kind == "momentum":
        return _momentum(f, sp, case["scheme"], 0.1)
    st = sto = None
    if case["tension"]:
        st, sto = _tension(f["c"], sp), _old_tension(f, sp)
    cs = _smoothed(f["c"], sp)
    f["rho"] = RHOG * cs + (1.0 - cs) * RHOL
    f["mu"] = MUG * cs + (1.0 - cs) * MUL
    nx, ny, nz = sp.n
    # the volume sum of rho on the x faces is that of the cells, its two neighbours averaged
    box = (0, nx - 1, 1, ny, 1, nz)
    face = 0.5 * (_cut(f["rho"], "cl", 1, box, (1, 0, 0)) + _cut(f["rho"], "cl", 1, box))
    rho_av = float((face * sp.at(sp.dyf, 1, ny)).sum()) * sp.d[0] * sp.d[2] / (LX * LY * LZ)
    fs = (RET * MUL / RHOL) ** 2 - rho_av * GCH
    for k, a in zip(CELL[1:], _momentum(f, sp, case["scheme"], fs, st)):
        f[k] = a
    psi, u = _projected(f, sp, st, sto)
    _velocity_ghosts(u, sp)
    return [psi, cs, f["rho"], f["mu"]] + u
