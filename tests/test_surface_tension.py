"""Surface tension (computeSurfaceTension, VOF.f90:1872-2002): the oracle's
grid-wide height-function curvature pinned by analytic interfaces on the CPU,
and the CUDA kernels through the C ABI against the oracle on the GPU.

Bars: on a sphere of radius 10 cells the mean curvature of the interface cells
is within 1 % of 2/R and 90 % of the cells within 15 % (height functions from a
volume fraction sampled on 8^3 sub-cells); a plane gives zero curvature; the
CUDA curvature and face force match the oracle within 1e-12 relative to the
field's maximum, on a uniform box and on the tanh-stretched channel with
bubbles touching the wall region; a projection fed with that force matches the
oracle's projection with the same force within 1e-12.
"""
import numpy as np
import pytest

from oracle import tbfp_oracle as O
from tbfsolver_b200 import synth
from tbfsolver_b200.fields import Field, VField
from tbfsolver_b200.grid import Grid
from tests._helpers import mesh_of, rel_linf


def _sphere(n=48, R_cells=10.0, nref=8, off=(0.13, -0.21, 0.07)):
    L = 2 * np.pi
    h = L / n
    R = R_cells * h
    cen = np.array([L / 2 + off[0] * h, L / 2 + off[1] * h, L / 2 + off[2] * h])
    sub = (np.arange(nref) + 0.5) / nref
    c = np.zeros((n, n, n))
    for a in sub:
        for b in sub:
            for d in sub:
                xs, ys, zs = (np.arange(n) + a) * h, (np.arange(n) + b) * h, (np.arange(n) + d) * h
                r2 = (xs[None, None, :] - cen[0]) ** 2 + (ys[None, :, None] - cen[1]) ** 2 + \
                    (zs[:, None, None] - cen[2]) ** 2
                c += r2 <= R * R
    return c / nref ** 3, h, R


def test_sphere_curvature_is_two_over_r():
    c, h, R = _sphere()
    n = c.shape[0]
    kap, stx, sty, stz = O.surface_tension(c, 1.0, h, h, np.full(n, h), np.full(n + 1, h))
    _, mixed, _ = O.st_classify(c)
    k = kap[mixed]
    valid = k != 0.0
    assert valid.mean() > 0.97
    ratio = k[valid] * R / 2.0
    assert abs(ratio.mean() - 1.0) < 0.01
    assert np.mean(np.abs(ratio - 1.0) < 0.15) > 0.9
    # the cells without a valid direction (under 3 %) are thin slivers of the sphere
    assert np.max(c[mixed][~valid]) < 0.3
    # the force points into the bubble: on x faces left of the centre c grows with x
    assert np.sum(stx[:, :, : n // 2 - 2]) > 0.0 and np.sum(stx[:, :, n // 2 + 3:]) < 0.0


def test_plane_has_zero_curvature():
    """A tilted plane y = y0 + 0.3 x on a uniform grid, exact volume fractions
    (the clipped linear profile integrated over each cell): the heights are
    linear, so every second difference vanishes to rounding."""
    n = 32
    h = 1.0 / n
    x = (np.arange(n * 512) + 0.5) * (h / 512)  # fine x quadrature of each cell
    y_int = 0.37 + 0.3 * (x - 0.5)
    c = np.zeros((n, n, n))
    for j in range(n):
        frac = np.clip((y_int - j * h) / h, 0.0, 1.0)  # fraction of the cell's height under the plane
        c[:, j, :] = frac.reshape(n, 512).mean(axis=1)[None, :]
    kap, *_ = O.surface_tension(c, 1.0, h, h, np.full(n, h), np.full(n + 1, h))
    _, mixed, _ = O.st_classify(c)
    assert mixed.sum() > 0
    assert np.max(np.abs(kap)) < 1e-6 / h


def _gpu_vs_oracle(c_field: Field, g: Grid, sigma=5e-3):
    import torch

    from tbfsolver_b200.solver import FastPoissonSolver, compute_surface_tension

    nx, ny, nz = g.nx, g.ny, g.nz
    m = mesh_of(g)
    dyf, dyc = np.ascontiguousarray(g.dyf.r(1, ny)), np.ascontiguousarray(g.dyc.r(1, ny + 1))
    ci = Field.like(c_field, c_field.a).interior()
    kap, stx, sty, stz = O.surface_tension(np.ascontiguousarray(ci), sigma, g.dx_fft, g.dz_fft, dyf, dyc)
    with FastPoissonSolver(g) as fps:
        cd = Field.like(c_field, torch.from_numpy(np.ascontiguousarray(c_field.a)).cuda())
        st = VField(*[Field(k, 1, nx, ny, nz, torch.full(Field(k, 1, nx, ny, nz).a.shape, 7.0, dtype=torch.float64,
                                                         device="cuda")) for k in ("sx", "sy", "sz")])
        kd = Field("cl", 1, nx, ny, nz, torch.full(c_field.a.shape, 7.0, dtype=torch.float64, device="cuda"))
        compute_surface_tension(fps, cd, sigma, st, kappa=kd)
        torch.cuda.synchronize()
        got = [Field.like(f, f.a.cpu().numpy()) for f in st.components()]
        gk = Field.like(kd, kd.a.cpu().numpy())
    assert rel_linf(gk.interior(), kap) < 1e-12
    # interiors of the staggered fields: x faces 0..nx, y faces 0..ny, z faces 0..nz
    assert rel_linf(got[0].v(0, nx, 1, ny, 1, nz), stx) < 1e-12
    assert rel_linf(got[1].v(1, nx, 0, ny, 1, nz), sty) < 1e-12
    assert rel_linf(got[2].v(1, nx, 1, ny, 0, nz), stz) < 1e-12
    # halos: periodic images in x, zero y ghost rows and wall faces
    assert np.array_equal(got[0].v(-1, -1, 1, ny, 1, nz), got[0].v(nx - 1, nx - 1, 1, ny, 1, nz))
    assert np.all(got[1].v(1, nx, 0, 0, 1, nz) == 0.0) and np.all(got[1].v(1, nx, ny, ny, 1, nz) == 0.0)
    assert np.max(np.abs(kap)) > 0.0 and np.max(np.abs(stx)) > 0.0
    return got, m


@pytest.mark.gpu
def test_gpu_surface_tension_uniform_sphere():
    c, h, R = _sphere(n=32, R_cells=7.0)
    n = c.shape[0]
    g = Grid(n, n, n, 2 * np.pi, 2 * np.pi, 2 * np.pi, False, 1.5)
    f = Field("cl", 1, n, n, n)
    f.interior()[...] = c
    _gpu_vs_oracle(f, g)


@pytest.mark.gpu
def test_gpu_surface_tension_stretched_channel_and_projection():
    import torch

    from tbfsolver_b200.solver import PoissonEqn

    spec = synth.small_spec(64, 48, 32, stretched=True, nbubbles=3, radius=0.35, rhog=0.05)
    g = spec.grid()
    c = synth.vof_field(spec, synth.bubble_centres(spec, 7), hd=1).numpy().copy()
    cf = Field("cl", 1, g.nx, g.ny, g.nz, c)
    st, m = _gpu_vs_oracle(cf, g)
    # a projection fed with the force (both levels) against the oracle's
    inp = synth.make_inputs(spec, seed=3)
    ost = [O.FField(f.kind, 1, g.nx, g.ny, g.nz, f.a.copy()) for f in st]
    to = lambda f: O.FField(f.kind, f.hd, g.nx, g.ny, g.nz, f.a.numpy().copy())  # noqa: E731
    ref = O.projection(m, to(inp.u.ux), to(inp.u.uy), to(inp.u.uz), to(inp.rho), to(inp.psi_n), to(inp.psi_nm1),
                       inp.dt, inp.alpha, inp.rho0, ost, ost)
    eqn = PoissonEqn(g, spec.rhol, spec.rhog)
    try:
        cu = lambda f: Field.like(f, torch.from_numpy(np.ascontiguousarray(f.a)).cuda())  # noqa: E731
        u = VField(*[cu(f) for f in inp.u.components()])
        std = [cu(f) for f in st]
        psi = cu(Field("cl", 1, g.nx, g.ny, g.nz))
        res = eqn.projection(psi, cu(inp.psi_n), cu(inp.psi_nm1), cu(inp.rho), u, inp.dt, inp.alpha, std, std)
        assert rel_linf(psi.a.cpu().numpy(), ref.psi.a) < 1e-12
        for f, r in zip(u.components(), (ref.ux, ref.uy, ref.uz)):
            assert rel_linf(f.a.cpu().numpy(), r.a) < 1e-12
        assert abs(res.max_div - ref.max_div) < 1e-12
    finally:
        eqn.close()


def _speckled(nx, ny, nz, seed):
    """Random volume fractions: empty, full and mixed cells side by side, so that
    promoted cells, walls, wrapped columns and invalid directions all occur."""
    rng = np.random.default_rng(seed)
    c = rng.random((nz, ny, nx))
    kind = rng.random((nz, ny, nx))
    c[kind < 0.4] = 0.0
    c[kind > 0.6] = 1.0
    x = np.arange(nx)[None, None, :] + 3.0 * rng.random()
    c[:, :, :] = np.where(np.sin(2 * np.pi * x / nx) + 0.3 * np.arange(ny)[None, :, None] / ny > 0.9, 1.0,
                          np.where(np.sin(2 * np.pi * x / nx) < -0.8, 0.0, c))
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("n, hd_st, stretched", [((8, 4, 4), 0, False), ((12, 9, 6), 1, True), ((8, 7, 24), 3, True),
                                                 ((96, 5, 8), 1, False), ((1024, 4, 4), 1, True)])
def test_gpu_surface_tension_shapes(n, hd_st, stretched):
    """Rows of one and many 32-cell chunks with and without a remainder, row
    counts that leave a block's last warps idle, columns that wrap more than
    once, every st halo width, an interface without and with mixed cells.  Bar:
    the decisions are the oracle's bit for bit, the rest is rounding of a few
    second differences of heights (1e-12 of the largest curvature)."""
    import torch

    from tbfsolver_b200.solver import FastPoissonSolver, compute_surface_tension

    nx, ny, nz = n
    g = Grid(nx, ny, nz, 2 * np.pi, 2.0, np.pi, stretched, 1.5)
    dyf, dyc = np.ascontiguousarray(g.dyf.r(1, ny)), np.ascontiguousarray(g.dyc.r(1, ny + 1))
    with FastPoissonSolver(g, hd_st=hd_st) as fps:
        for c in (_speckled(nx, ny, nz, 5), np.zeros((nz, ny, nx)), np.ones((nz, ny, nx)), np.full((nz, ny, nx), 0.5)):
            kap, *st_ref = O.surface_tension(c, 0.07, g.dx_fft, g.dz_fft, dyf, dyc)
            f = Field("cl", 1, nx, ny, nz)
            f.interior()[...] = c
            cd = Field.like(f, torch.from_numpy(f.a).cuda())
            st = VField(*[Field(k, hd_st, nx, ny, nz, torch.full(Field(k, hd_st, nx, ny, nz).a.shape, 7.0,
                                                                dtype=torch.float64, device="cuda"))
                          for k in ("sx", "sy", "sz")])
            kd = Field.like(cd, torch.full_like(cd.a, 7.0))
            torch.cuda.synchronize()
            compute_surface_tension(fps, cd, 0.07, st, kappa=kd)
            assert rel_linf(Field.like(kd, kd.numpy()).interior(), kap) < 1e-12
            boxes = [(0, nx, 1, ny, 1, nz), (1, nx, 0, ny, 1, nz), (1, nx, 1, ny, 0, nz)]
            for fd, ref, b in zip(st.components(), st_ref, boxes):
                a = Field.like(fd, fd.numpy())
                assert rel_linf(a.v(*b), ref) < 1e-12
                # halos: periodic images of the interior in x and z, zero rows beyond the walls
                lo = a.lb
                ii = [(i - b[0]) % nx for i in range(lo[0], lo[0] + a.a.shape[2])]
                kk = [(k - b[4]) % nz for k in range(lo[2], lo[2] + a.a.shape[0])]
                whole = np.zeros_like(a.a)
                j0 = b[2] - lo[1]
                whole[:, j0:j0 + b[3] - b[2] + 1, :] = a.v(*b)[kk][:, :, ii]
                assert np.array_equal(a.a, whole)


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_gpu_surface_tension_carries_non_finite_cells(bad):
    """A cell that is not finite makes the force of its own faces non-finite, also
    away from every interface."""
    import torch

    from tbfsolver_b200.solver import FastPoissonSolver, compute_surface_tension

    nx, ny, nz = 16, 12, 8
    g = Grid(nx, ny, nz, 2 * np.pi, 2.0, np.pi, True, 1.5)
    f = Field("cl", 1, nx, ny, nz)
    if bad == np.inf:  # counts as full: among empty cells it would be promoted to a finite value
        f.a[...] = 1.0
    f.v(7, 7, 5, 5, 4, 4)[...] = bad
    cd = Field.like(f, torch.from_numpy(f.a).cuda())
    with FastPoissonSolver(g) as fps:
        st = VField(*[Field(k, 1, nx, ny, nz, torch.zeros(Field(k, 1, nx, ny, nz).a.shape, dtype=torch.float64,
                                                         device="cuda")) for k in ("sx", "sy", "sz")])
        torch.cuda.synchronize()
        compute_surface_tension(fps, cd, 0.07, st)
        for fd, (di, dj, dk) in zip(st.components(), ((1, 0, 0), (0, 1, 0), (0, 0, 1))):
            a = Field.like(fd, fd.numpy())
            assert not np.isfinite(a.v(7, 7, 5, 5, 4, 4)).any()
            assert not np.isfinite(a.v(7 - di, 7 - di, 5 - dj, 5 - dj, 4 - dk, 4 - dk)).any()
            assert np.isnan(a.a).sum() + np.isinf(a.a).sum() == 2
