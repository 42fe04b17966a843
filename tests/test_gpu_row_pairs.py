"""FP64 type-IV row passes with two lines a thread group (k_xpass<.., true>, picked by timing on grids of many
rows; GHOSTMAC_SHAPES sets it) against one line a group: the same butterflies on each line, so the same
bits, also where an odd number of rows leaves the last group one line, for every radix."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu
QUIET = dict(dt=0.002, perturb_transient=False, save_artifacts=False, verbose=False)


@pytest.mark.parametrize('shape', ['64,1,4', '128,2,4', '512,1,8'])
@pytest.mark.parametrize('nx,ny', [(60, 31), (84, 33), (88, 32), (104, 47), (122, 35), (128, 63), (200, 121)])
def test_two_lines_equal_one(monkeypatch, nx, ny, shape):
    pkg = load_package()
    h, out = 0.1, []
    for two in '01':
        monkeypatch.setenv('GHOSTMAC_SHAPES', f'{shape},{two}')
        s = pkg.MAC_CylinderFlow(boundary='ghost_cell', time_scheme='ab2_cn', nx=nx, ny=ny, Lx=nx * h, Ly=ny * h, D=1.0,
                                 xc=nx * h * 0.3, yc=ny * h * 0.5, nu=0.05, verbose=False)
        s.u += 0.01 * np.random.default_rng(nx).standard_normal(s.u.shape)
        s.solve(n_steps=4, **QUIET)
        out.append((s.u.copy(), s.v.copy(), s.p.copy(), s.last_step_diagnostics['pressure_residual_linf']))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
