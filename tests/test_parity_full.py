"""Parity at the benchmarked sizes.

The 3-call projection chain (computeSource -> solveFPS -> makeVelocityDivFree
-> computeContinuityError, with the pressure history rotated between calls as
updatePressure does) of the 512x384x256 tanh-stretched workload and of the
256x256x128 workload runs on the GPU through the C ABI.  It is compared at
every call with the C restatement of the reference path (oracle/tbfp_oracle.c).
That oracle uses the reference's own rule for the singular (0,0) system: the
LAPACK-style elimination with the epsilon pivot of fastPoissonSolver.f90:318-322,
then zeroAveragePressure (:388-423).  The library gauges that system exactly.
Bar: psi and u within 1e-12 relative (L-infinity over the field's maximum),
max|div u| within 1e-12 absolute.

The CPU test at the end runs the numpy oracle with the literal epsilon pivot
and with the exact gauge on the 128x128x64 chain.  It records how far the two
rules sit apart on projection sources.
"""
import numpy as np
import pytest
import torch

from oracle import cref
from oracle import tbfp_oracle as O
from tbfsolver_b200 import synth
from tbfsolver_b200.fields import Field, VField
from tests._helpers import mesh_of, rel_linf, to_oracle

TOL_P = 1e-12
TOL_DIV = 1e-12


def _chain_inputs(name, seed=2024):
    spec = synth.CONFIGS[name]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return spec, synth.make_inputs(spec, seed=seed, device=dev)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["c2", "c5"])
def test_projection_chain_against_the_c_oracle(name):
    from tbfsolver_b200.solver import PoissonEqn

    spec, inp = _chain_inputs(name)
    g = inp.grid
    host = lambda f: f.a.detach().cpu().numpy().copy()  # noqa: E731
    hu = [host(f) for f in inp.u.components()]
    hrho, hpn, hpnm1 = host(inp.rho), host(inp.psi_n), host(inp.psi_nm1)
    eqn = PoissonEqn(g, spec.rhol, spec.rhog)
    try:
        pn, pnm1 = inp.psi_n, inp.psi_nm1
        for call in range(3):
            # oracle: u* restored for every call, psi from zero
            wu = [a.copy() for a in hu]
            hpsi = np.zeros_like(hpn)
            md_ref = cref.projection(g, *wu, hrho, hpn, hpnm1, inp.dt, inp.alpha, inp.rho0, hpsi)
            psi = Field.like(pn, torch.zeros_like(pn.a))
            uo = VField(*[Field.like(f, torch.empty_like(f.a)) for f in inp.u.components()])
            st = eqn.projection(psi, pn, pnm1, inp.rho, inp.u, inp.dt, inp.alpha, u_out=uo)
            assert rel_linf(host(psi), hpsi) < TOL_P, (name, call)
            for f, want in zip(uo.components(), wu):
                got = Field.like(f, host(f)).interior()
                assert rel_linf(got, Field.like(f, want).interior()) < TOL_P, (name, call, f.kind)
            assert abs(st.max_div - md_ref) < TOL_DIV, (name, call, st.max_div, md_ref)
            hpnm1, hpn = hpn, hpsi
            pnm1, pn = pn, psi
    finally:
        eqn.close()


def test_epsilon_pivot_against_exact_gauge_on_the_projection_chain():
    """The reference's epsilon pivot against the exact gauge (numpy oracle,
    LAPACK zgttrf/zgttrs) on the 128x128x64 chain.  The two rules differ only
    in the (0,0) system, and only by the compatibility defect of the source:
    sum s V, which a projection source has at rounding level.  So psi agrees
    to 1e-12 relative at every call."""
    spec = synth.CONFIGS["c1"]
    inp = synth.make_inputs(spec, seed=2024)
    g = inp.grid
    m = mesh_of(g)
    ou = [to_oracle(f, g) for f in inp.u.components()]
    orho, opn, opnm1 = to_oracle(inp.rho, g), to_oracle(inp.psi_n, g), to_oracle(inp.psi_nm1, g)
    worst = 0.0
    for call in range(3):
        lit = O.projection(m, *ou, orho, opn, opnm1, inp.dt, inp.alpha, inp.rho0, tridiag="lapack")
        pin = O.projection(m, *ou, orho, opn, opnm1, inp.dt, inp.alpha, inp.rho0, tridiag="lapack-pinned")
        d = rel_linf(lit.psi.a, pin.psi.a)
        worst = max(worst, d)
        assert d < TOL_P, (call, d)
        for a, b in ((lit.ux, pin.ux), (lit.uy, pin.uy), (lit.uz, pin.uz)):
            assert rel_linf(a.a, b.a) < TOL_P, call
        assert abs(lit.max_div - pin.max_div) < TOL_DIV
        opnm1, opn = opn, pin.psi
    print(f"epsilon pivot vs exact gauge, 128x128x64 chain: max rel psi difference {worst:.2e}")


@pytest.mark.gpu
@pytest.mark.parametrize("nx", [768, 1024])
def test_long_x_rows_against_the_c_oracle(nx):
    """nx = 768 and 1024 (half-length transforms of 384 and 512 points): the
    right-hand side runs apart from the x transform there, and the x transforms
    at two CTAs per SM.  One projection on a thin channel against the C
    restatement, same bar as the benchmarked sizes."""
    from tbfsolver_b200.solver import PoissonEqn

    spec = synth.small_spec(nx, 24, 8, stretched=True, nbubbles=2, radius=0.3, rhog=0.05)
    inp = synth.make_inputs(spec, seed=31, device="cuda")
    g = inp.grid
    host = lambda f: f.a.detach().cpu().numpy().copy()  # noqa: E731
    wu = [host(f) for f in inp.u.components()]
    hpsi = np.zeros_like(host(inp.psi_n))
    md_ref = cref.projection(g, *wu, host(inp.rho), host(inp.psi_n), host(inp.psi_nm1), inp.dt, inp.alpha,
                             inp.rho0, hpsi)
    eqn = PoissonEqn(g, spec.rhol, spec.rhog)
    try:
        psi = Field.like(inp.psi_n, torch.zeros_like(inp.psi_n.a))
        uo = VField(*[Field.like(f, torch.empty_like(f.a)) for f in inp.u.components()])
        st = eqn.projection(psi, inp.psi_n, inp.psi_nm1, inp.rho, inp.u, inp.dt, inp.alpha, u_out=uo)
    finally:
        eqn.close()
    assert rel_linf(host(psi), hpsi) < TOL_P
    for f, want in zip(uo.components(), wu):
        assert rel_linf(Field.like(f, host(f)).interior(), Field.like(f, want).interior()) < TOL_P, f.kind
    assert abs(st.max_div - md_ref) < TOL_DIV


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(512, 25, 8), (768, 25, 8), (1024, 7, 4), (1024, 33, 64)])
@pytest.mark.parametrize("tension", [False, True])
def test_long_x_rows_and_both_forms_of_the_right_hand_side(dims, tension):
    """nx = 512, where a thread of the fused right-hand side marches two columns, and the lengths from 768 on, where
    it runs apart: rows per block of one, two and the full 32, each with a remainder, with and without surface
    tension.  One projection against the oracle, same bar."""
    from tbfsolver_b200.fields import VField
    from tbfsolver_b200.solver import PoissonEqn

    nx, ny, nz = dims
    spec = synth.small_spec(nx, ny, nz, stretched=True, nbubbles=2, radius=0.3, rhog=0.05)
    inp = synth.make_inputs(spec, seed=32)
    g, rng = inp.grid, np.random.default_rng(nx + ny)
    st = [[O.FField(k, 1, nx, ny, nz, 0.01 * rng.standard_normal(Field(k, 1, nx, ny, nz).a.shape))
           for k in ("sx", "sy", "sz")] for _ in range(2)] if tension else [None, None]
    if tension:
        for f in st:
            O.equate_periodic_bc(f[0], f[2])             # periodic duplicate faces
            f[1].a[:, 1, :] = f[1].a[:, -2, :] = 0.0  # no force on the wall faces
    ref = O.projection(mesh_of(g), *[to_oracle(f, g) for f in (*inp.u.components(), inp.rho, inp.psi_n, inp.psi_nm1)],
                       inp.dt, inp.alpha, inp.rho0, *st)
    cu = lambda f: Field(f.kind, f.hd, nx, ny, nz, torch.as_tensor(f.a).cuda())  # noqa: E731
    eqn = PoissonEqn(g, spec.rhol, spec.rhog)
    try:
        psi = cu(inp.psi_n)
        u = VField(*[cu(f) for f in inp.u.components()])
        uo = VField(*[Field.like(f, torch.zeros_like(f.a)) for f in u.components()])
        extra = [[cu(f) for f in fs] for fs in st] if tension else []
        torch.cuda.synchronize()
        eqn.projection(psi, cu(inp.psi_n), cu(inp.psi_nm1), cu(inp.rho), u, inp.dt, inp.alpha, *extra, u_out=uo)
    finally:
        eqn.close()
    assert rel_linf(psi.a.cpu().numpy(), ref.psi.a) < TOL_P
    for f, r in zip(uo.components(), (ref.ux, ref.uy, ref.uz)):
        assert rel_linf(Field.like(f, f.a.cpu().numpy()).interior(), r.interior()) < TOL_P
