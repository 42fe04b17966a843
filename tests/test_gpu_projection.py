"""The projection kernels (k_proj_rhs, k_proj_update, k_proj_tail, k_step_tail) against the same
quantities composed from the single operators, which fill every ghost value first: the points next
to the body read ghost rows formed inside the kernels.  Both forms are the same few operations in
FP64 up to the contraction of products, so a value may differ by a few eps of its terms; the
pressure solve's right-hand side then differs by that, and phi by the solve's own 1e-11."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


@pytest.mark.parametrize('nx,ny,h,ext,interp,inflow', [
    (40, 31, 0.125, 'neumann', 'bilinear', 'uniform'), (64, 48, 0.1, 'quadratic', 'biquadratic', 'parabolic'),
    (96, 61, 0.08, 'neumann', 'biquadratic', 'uniform'), (128, 77, 0.05, 'quadratic', 'bilinear', 'uniform')])
def test_projection_matches_operators(nx, ny, h, ext, interp, inflow):
    pkg = load_package()
    s = pkg.MAC_CylinderFlow(nx=nx, ny=ny, Lx=nx * h, Ly=ny * h, D=1.0, xc=nx * h / 4, yc=ny * h / 2, nu=0.02,
                             boundary='ghost_cell', time_scheme='ab2_cn', verbose=False, inflow=inflow,
                             ghost_pressure_extension=ext, ghost_velocity_interpolation=interp)
    g, dt = s.gg, 0.004
    rng = np.random.default_rng(nx)
    q = rng.standard_normal(g.qsize)
    qo, phi = g.project(q, dt)
    rhs = g.divergence(q) / dt
    ref = g.pressure_solve(rhs)
    assert np.max(np.abs(phi - ref)) <= 1e-11 * np.max(np.abs(ref))
    grad = g.gradient(phi)
    # the ghost rows' weights are of order one to a few: 64 eps of the largest term covers their sums
    assert np.max(np.abs(qo - (q - dt * grad))) <= 64 * EPS * (np.max(np.abs(q)) + dt * np.max(np.abs(grad)))
    assert np.max(np.abs(g.divergence(qo))) < 1e-10


@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
@pytest.mark.parametrize('steps', [1, 2, 3, 7])
def test_step_record_matches_state(precision, steps):
    """The step's end: forces, maxima and divergence of the record are those of the state, whether
    the steps run in one call or several (ghost values of the half pressure carried or rebuilt)."""
    pkg = load_package()
    kw = dict(nx=64, ny=45, Lx=8.0, Ly=5.625, D=1.0, xc=2.0, yc=2.8, nu=0.02, boundary='ghost_cell',
              time_scheme='ab2_cn', verbose=False, precision=precision)
    quiet = dict(dt=0.004, perturb_transient=False, save_artifacts=False, verbose=False)
    one, many = pkg.MAC_CylinderFlow(**kw), pkg.MAC_CylinderFlow(**kw)
    t, cd, cl = one.solve(n_steps=steps, **quiet)
    for k in range(steps):
        many.solve(n_steps=1, **quiet)
        if k == 1:  # the AB2 history through the host: its half pressure comes without ghost values
            many.gg.set_history(*many.gg.history())
    for name in ('u', 'v', 'p'):
        assert np.array_equal(getattr(one, name), getattr(many, name))
    d = one.last_step_diagnostics
    f = one.gg.surface_forces(one.u, one.v, one.p, one.nu * one.rho)
    assert abs(d['cd'] - f[0] / 0.5) <= 4 * EPS * abs(d['cd']) and abs(d['cl'] - f[1] / 0.5) <= 4 * EPS * (abs(f[3]) + abs(f[5]) + abs(d['cl']))
    cfl = 0.004 * (np.max(np.abs(one.u)) / one.dx + np.max(np.abs(one.v)) / one.dy)
    assert abs(d['cfl'] - cfl) <= 4 * EPS * cfl
    assert abs(d['max_divergence'] - one.divergence_stats()[0]) <= 1e-13
