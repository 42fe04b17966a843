"""FGMRES in the boundary rows' space (plain FP64, csrc/kernels.cu k_cg_cycle) where it can go wrong:
right-hand sides on the boundary rows alone (no part off them), off them alone and of one point,
zero; grids with few and with odd numbers of rows; a body with more rows than the kernel takes (the
grid iteration runs).  Against the host-controlled grid iteration (the same Krylov space, so the same
iteration count up to a tie at the tolerance) and the direct solver: GMRES stops at a residual of
1e-12 ||b||, and the reference asserts 1e-9 between its backends."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu

GRIDS = [dict(nx=40, ny=31, Lx=5.0, Ly=3.875, D=1.0, xc=1.5, yc=1.9),
         dict(nx=96, ny=48, Lx=9.6, Ly=4.8, D=1.0, xc=2.4, yc=2.4, ghost_pressure_extension='quadratic'),
         dict(nx=160, ny=131, Lx=4.0, Ly=3.275, D=1.0, xc=1.5, yc=1.6),
         dict(nx=384, ny=360, Lx=2.0, Ly=1.875, D=1.0, xc=0.9, yc=0.93)]


@pytest.mark.parametrize('kw', GRIDS, ids=['40x31', '96x48', '160x131', '384x360'])
def test_right_hand_sides(monkeypatch, kw):
    pkg = load_package()
    make = lambda solver: pkg.MAC_CylinderFlow(boundary='ghost_cell', time_scheme='ab2_cn', verbose=False, nu=0.02,
                                               pressure_solver=solver, **kw)
    direct, compact = make('direct'), make('iterative')
    pi = direct.gg.pi
    rows = np.isin(pi, direct.gg.schur_rows(0))  # the active boundary rows
    rng = np.random.default_rng(kw['nx'])
    b = rng.standard_normal(len(pi))
    one = np.zeros(len(pi))
    one[len(pi) // 3] = 1.0
    sides = dict(all=b, on=np.where(rows, b, 0.0), off=np.where(rows, 0.0, b), one=one, small=1e-3 * b)
    got = {}
    for name, r in sides.items():
        x = compact.gg.pressure_solve(r)
        got[name] = x, compact.gg.pressure_inverse_info['last_solve']['iterations']
        ref = direct.gg.pressure_solve(r)
        assert np.max(np.abs(x - ref)) < 1e-9 * max(1.0, np.max(np.abs(ref))), name
    assert not compact.gg.pressure_solve(np.zeros(len(pi))).any()
    monkeypatch.setenv('GHOSTMAC_GMRES_HOST', '1')
    host = make('iterative')
    for name, r in sides.items():
        host.gg.pressure_solve(r)
        its = host.gg.pressure_inverse_info['last_solve']['iterations']
        assert abs(got[name][1] - its) <= 1, (name, got[name][1], its)
