"""The cut-cell CN solve on the GPU: the one-pass viscous operator on packed vectors against the flux
form of the same operator (compute_momentum_rhs), and step graphs that hold a fixed number of gated
Arnoldi steps.

Both forms sum the same terms (up to some two hundred for a face near the body, merged or owning covered
volumes) in another order: they differ by a few hundred roundings of the largest term, below 1e-12 of
max |L q|; H q = q - dt/2 L q carries the same bound.

A system that needs more Arnoldi steps than the graph holds repeats its step with more: six at first, beyond
30 restart cycles.  A second run on the same handle starts with enough, and steps that converge early
skip the rest, so both runs are equal bit for bit."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu
QUIET = dict(perturb_transient=False, save_artifacts=False, verbose=False)


def make(pkg, nx, ny, nu=0.01, h=0.1, slip=False, shift=0.013):
    return pkg.MAC_CylinderFlow(boundary='cut_cell', time_scheme='ab2_cn', nx=nx, ny=ny, Lx=nx * h, Ly=ny * h, D=1.0,
                                xc=nx * h * 0.3, yc=ny * h * 0.5 + shift, nu=nu, slip_walls=slip, verbose=False)


@pytest.mark.parametrize('nx,ny,h,slip,shift', [(40, 20, 0.1, False, 0.013), (40, 20, 0.1, True, 0.0),
                                                (64, 39, 0.1, False, 0.031), (30, 13, 0.25, True, 0.07),
                                                (200, 101, 0.05, False, 0.0)])
def test_operator_against_fluxes(nx, ny, h, slip, shift):
    pkg = load_package()
    s = make(pkg, nx, ny, 0.01, h, slip, shift)
    q = np.random.default_rng(nx + ny).standard_normal(s.cc.qsize)
    for inlet, got in ((s.u_inlet, s.cc.diffusion(q)), (np.zeros(ny), None)):
        u, v = s.cc.unpack(q, inlet)
        au, av, _, _ = s.cc.compute_momentum_rhs(u, v, s.nu, s.rho, transport='centered', include_advection=False)
        want = s.cc.pack(au, av)
        if got is None:
            dt = 0.004
            got, want = s.cc.H_matvec(q, dt), q - 0.5 * dt * want
        assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want))


@pytest.mark.parametrize('nu,least', [(0.01, 1), (0.1, 7), (0.3, 13), (1.0, 21), (1.5, 31)])
def test_repeated_steps_equal_first_time_steps(nu, least):
    pkg = load_package()
    s = make(pkg, 64, 39, nu)
    start = s.u.copy(), s.v.copy(), s.p.copy()
    runs = []
    for _ in range(2):
        for field, value in zip((s.u, s.v, s.p), start):
            field[...] = value
        s.time = 0.0
        s.cc.set_history(None, None, None)
        t, cd, cl = s.solve(n_steps=4, dt=0.01, **QUIET)
        d = s.last_step_diagnostics
        runs.append((s.u.copy(), s.v.copy(), s.p.copy(), cd, cl, d['momentum_iterations'], d['max_divergence'],
                     d['coupled_momentum_residual_linf'], *s.cc.history()))
        assert d['momentum_iterations'] >= least
        assert d['momentum_residual_linf'] <= 1e-10
    for a, b in zip(*runs):
        assert np.array_equal(a, b)
