"""The legacy loops' queued steps (one library call without host checks in between) and the divides by
known divisors of their kernels.

Every kernel repeats the reference's arithmetic without contraction, so the corrector equals NumPy's bit for
bit on any operands, and n steps in one call equal n calls of one step bit for bit."""
import sys

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu
QUIET = dict(dt=0.002, perturb_transient=False, save_artifacts=False, verbose=False)


@pytest.mark.parametrize('seed', range(6))
def test_divides_are_exact(seed):
    pkg = load_package()
    __import__(pkg.__name__ + '.mac_engine')
    M = sys.modules[pkg.__name__ + '.mac_engine']
    rng = np.random.default_rng(seed)
    nx, ny = 64, 48
    mask, inlet = np.zeros((ny, nx), bool), np.zeros(ny)
    for dx in (0.05, 1 / 3, 0.1 * (1 + rng.random()), 2.0 ** -7, np.nextafter(1.0, 2.0), np.nextafter(1.0, 0.0), 1e-120, 1e120,
               float(np.exp(rng.uniform(-8, 8)))):
        phi = rng.standard_normal((ny, nx))
        if seed % 2:  # the whole exponent range, zeros of both signs, infinities and NaN
            phi *= 10.0 ** rng.integers(-323, 300, phi.shape)
            phi[rng.random(phi.shape) < 0.2] = 0.0
            phi[rng.random(phi.shape) < 0.1] = -0.0
            phi[5, 5:8] = np.inf, -np.inf, np.nan
        us, vs = rng.standard_normal((ny, nx + 1)) * (seed % 3), np.zeros((ny + 1, nx))
        u, v = np.zeros_like(us), np.zeros_like(vs)
        dt, rho = 0.003, 1.7
        M.corrector_cpp(u, v, us, vs, phi, mask, inlet, dx, dx, dt, rho, False)
        with np.errstate(all='ignore'):
            c = dt / rho
            wu = us[:, 1:nx] - (c * (phi[:, 1:] - phi[:, :-1])) / dx
            wv = vs[1:ny] - (c * (phi[1:] - phi[:-1])) / dx
        assert np.array_equal(u[:, 1:nx], wu, equal_nan=True)
        assert np.array_equal(v[1:ny], wv, equal_nan=True)


def make(pkg, boundary, transport, nx=50, ny=27):
    return pkg.MAC_CylinderFlow(nx=nx, ny=ny, Lx=nx * 0.1, Ly=ny * 0.1, D=1.0, xc=1.3, yc=1.3, nu=0.02, boundary=boundary,
                                time_scheme='legacy', transport=transport, pressure_solver='direct', verbose=False)


@pytest.mark.parametrize('boundary,transport', [('staircase', 'centered'), ('staircase', 'upwind'), ('ghost_cell', 'centered'),
                                                ('ghost_cell', 'upwind')])
def test_queue_equals_single_steps(boundary, transport):
    pkg = load_package()
    a, b = make(pkg, boundary, transport), make(pkg, boundary, transport)
    ta, cda, cla = a.solve(n_steps=7, **QUIET)
    rows = [b.solve(n_steps=1, **QUIET) for _ in range(7)]
    assert np.array_equal(cda, [r[1][0] for r in rows]) and np.array_equal(cla, [r[2][0] for r in rows])
    for name in ('u', 'v', 'p'):
        assert np.array_equal(getattr(a, name), getattr(b, name))


@pytest.mark.parametrize('boundary', ['staircase', 'ghost_cell'])
def test_failed_solve_keeps_state(boundary):
    pkg = load_package()
    s = make(pkg, boundary, 'upwind')
    s.solve(n_steps=2, **QUIET)
    s._d['p'][3, 4] = float('nan')
    before = {k: s._d[k].clone() for k in ('u', 'v', 'p')}
    with pytest.raises((RuntimeError, ValueError, FloatingPointError)):
        s._steps(0.002, 3)
    for k, value in before.items():
        assert np.array_equal(s._d[k].cpu().numpy(), value.cpu().numpy(), equal_nan=True)
