"""How many refinement sweeps the steps' graphs hold, and how often a step had to be repeated for one more
(gm_held_sweeps): alone and in a batch."""
import ctypes as C

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu
QUIET = dict(dt=0.002, perturb_transient=False, save_artifacts=False, verbose=False)


def make(pkg, nx=200, ny=121, precision='fp64'):
    return pkg.MAC_CylinderFlow(boundary='ghost_cell', time_scheme='ab2_cn', nx=nx, ny=ny, Lx=nx * 0.05, Ly=ny * 0.05, D=1.0,
                                xc=nx * 0.0125, yc=ny * 0.025, nu=0.02, verbose=False, precision=precision)


def shake(s, amp, seed):
    q = s.gg.pack(s.u, s.v)
    q += amp * np.random.default_rng(seed).standard_normal(q.size)
    u, v = s.gg.unpack(q)
    s.u[:], s.v[:] = u, v


def held(pkg, s):
    n, rep = (C.c_int32 * 5)(), C.c_int64()
    assert pkg._lib.lib.gm_held_sweeps(s._h, n, C.byref(rep)) == 0
    return list(n), rep.value


def test_batch_replays_no_graph_of_fewer_sweeps():
    """A case that has step graphs of its own and whose solves need more sweeps in a batch repeats its
    steps as often, and holds as many sweeps after it, as the same case stepped alone."""
    pkg = load_package()
    out = []
    for batch in (False, True):
        cases = [make(pkg), make(pkg, 160, 100)]
        for s in cases:
            s.solve(n_steps=6, **QUIET)
        calm = [held(pkg, s) for s in cases]
        for k, s in enumerate(cases):
            shake(s, 0.3, k)
        if batch:
            b = pkg.CylinderBatch(cases)
            b.solve(5, dt=0.002)
            b.close()
        else:
            for s in cases:
                s.solve(n_steps=5, **QUIET)
        out.append([held(pkg, s) for s in cases] + [s.u.copy() for s in cases])
        assert all(h[1] > c[1] for h, c in zip(out[-1][:2], calm))
    assert out[0][:2] == out[1][:2]
    for a, b in zip(out[0][2:], out[1][2:]):
        assert np.array_equal(a, b)


def test_first_step_sets_and_later_steps_lower(monkeypatch):
    """From rest the FP32 mode's pressure solves need two sweeps for some twenty steps and one from there
    on: the first step sets the counts, so no step is repeated, and 64 steps that use one lower them."""
    pkg = load_package()
    a = make(pkg, precision='fp32')
    a.solve(n_steps=5, **QUIET)
    assert held(pkg, a) == ([1, 1, 1, 2, 2], 0)
    a.solve(n_steps=160, **QUIET)
    assert held(pkg, a) == ([1, 1, 1, 1, 1], 0)
    monkeypatch.setenv('GHOSTMAC_NO_GRAPHS', '1')
    b = make(pkg, precision='fp32')
    b.solve(n_steps=165, **QUIET)
    for name in ('u', 'v', 'p'):
        assert np.array_equal(getattr(a, name), getattr(b, name))


@pytest.mark.parametrize('batch', [False, True])
def test_one_hard_step_is_not_kept(batch):
    """A perturbed FP64 state needs a sweep that later steps do not: the count goes up and down again."""
    pkg = load_package()
    cases = [make(pkg), make(pkg, 96, 48)]
    b = pkg.CylinderBatch(cases)
    step = (lambda n: b.solve(n, dt=0.002)) if batch else (lambda n: [s.solve(n_steps=n, **QUIET) for s in cases])
    step(4)
    assert [held(pkg, s) for s in cases] == [([0] * 5, 0)] * 2
    for k, s in enumerate(cases):
        shake(s, 0.3, k)
    step(3)
    assert [held(pkg, s) for s in cases] == [([0, 0, 0, 1, 1], 2)] * 2
    step(130)
    assert [held(pkg, s) for s in cases] == [([0] * 5, 2)] * 2
    b.close()
