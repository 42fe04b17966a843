"""Held sweeps and Arnoldi steps of the cut-cell and the legacy loops: set by the first step, raised by a step
that needs more, lowered when later steps do not use them; a legacy step that goes on with a sweep more,
and a gate that fails behind good queued steps."""
import ctypes as C

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu
QUIET = dict(dt=0.002, perturb_transient=False, save_artifacts=False, verbose=False)


def cut_cell(pkg):
    return pkg.MAC_CylinderFlow(boundary='cut_cell', time_scheme='ab2_cn', nx=96, ny=48, Lx=9.6, Ly=4.8, D=1.0, xc=2.4, yc=2.4,
                                nu=0.01, verbose=False)


def held_cc(pkg, s):
    n, rep = (C.c_int32 * 6)(), C.c_int64()
    assert pkg._lib.lib.gm_cc_held_sweeps(s._h, n, C.byref(rep)) == 0
    return list(n), rep.value


def test_cut_cell_counts():
    """One call of many steps and one call a step, with counts that differ on the way, are the same
    computation."""
    pkg = load_package()
    a, b = cut_cell(pkg), cut_cell(pkg)
    a.solve(n_steps=4, **QUIET)
    n, repeats = held_cc(pkg, a)
    assert repeats == 0 and n[5] == a.last_step_diagnostics['momentum_iterations']
    a.solve(n_steps=140, **QUIET)
    calm = held_cc(pkg, a)
    assert calm[0][3:5] == [0, 0]
    for _ in range(4):
        b.solve(n_steps=1, **QUIET)
    for n in (100, 40):
        b.solve(n_steps=n, **QUIET)
    rng = np.random.default_rng(1)
    q = 0.1 * rng.standard_normal(a.cc.pack(a.u, a.v).size)
    for s in (a, b):
        s.u[:], s.v[:] = s.cc.unpack(s.cc.pack(s.u, s.v) + q)
    a.solve(n_steps=5, **QUIET)
    assert held_cc(pkg, a)[1] > calm[1]
    for _ in range(5):
        b.solve(n_steps=1, **QUIET)
    for name in ('u', 'v', 'p'):
        assert np.array_equal(getattr(a, name), getattr(b, name))


def legacy(pkg, boundary, transport, nx, ny, h):
    return pkg.MAC_CylinderFlow(nx=nx, ny=ny, Lx=nx * h, Ly=ny * h, D=1.0, xc=nx * h / 4, yc=ny * h / 2, nu=0.02, boundary=boundary,
                                time_scheme='legacy', transport=transport, pressure_solver='direct', verbose=False)


def held_legacy(pkg, s):
    n, rep = C.c_int32(), C.c_int64()
    assert pkg._lib.lib.gm_poisson_held_sweeps(s._poisson, C.byref(n), C.byref(rep)) == 0
    return n.value, rep.value


@pytest.mark.parametrize('boundary', ['staircase', 'ghost_cell'])
def test_legacy_goes_on_with_a_sweep_more(boundary):
    pkg = load_package()
    a, b = (legacy(pkg, boundary, 'centered', 50, 27, 0.1) for _ in range(2))
    for s in (a, b):
        s.solve(n_steps=1, **QUIET)
    assert held_legacy(pkg, a)[1] == 0
    for s in (a, b):
        for _ in range(3):
            s.solve(n_steps=100, **QUIET)
    calm = held_legacy(pkg, a)
    assert calm[0] == 0
    noise = np.random.default_rng(0).standard_normal(a.u.shape)
    for s in (a, b):
        s.u[:] += noise
    one = a.solve(n_steps=9, **QUIET)
    assert held_legacy(pkg, a)[1] > calm[1]
    rows = [b.solve(n_steps=1, **QUIET) for _ in range(9)]
    for q in (1, 2):
        assert np.array_equal(one[q], [r[q][0] for r in rows])
    for name in ('u', 'v', 'p'):
        assert np.array_equal(getattr(a, name), getattr(b, name))


def test_legacy_gate_fails_behind_queued_steps():
    """A loop that blows up stops at the same step with the same state, queued or step by step."""
    pkg = load_package()
    a, b = (legacy(pkg, 'ghost_cell', 'upwind', 200, 121, 0.05) for _ in range(2))
    for s in (a, b):
        s.solve(n_steps=1, **QUIET)
    with pytest.raises((RuntimeError, ValueError, FloatingPointError)) as ea:
        a._steps(0.002, 95)
    done = 0
    with pytest.raises((RuntimeError, ValueError, FloatingPointError)) as eb:
        while done < 95:
            b._steps(0.002, 1)
            done += 1
    assert done > 5 and str(ea.value) == str(eb.value)
    for k in ('u', 'v', 'p'):
        assert np.array_equal(a._d[k].cpu().numpy(), b._d[k].cpu().numpy(), equal_nan=True)
