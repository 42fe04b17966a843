"""A batch whose FP32 cases refine in loops (WHILE nodes; large batches of large grids) against held, gated
sweeps and against the cases stepped alone: the same kernels, so the same bits."""
import time

import numpy as np
import pytest

from conftest import load_package
from test_gpu_held_sweeps import QUIET, held, make, shake

pytestmark = pytest.mark.gpu
CALLS = (1, 3, 9, 2)


@pytest.mark.parametrize('loops', ['0', '1'])
def test_loops_and_held_sweeps_equal_single_cases(monkeypatch, loops):
    pkg = load_package()
    monkeypatch.setenv('GHOSTMAC_BATCH_LOOPS', loops)
    specs = [(200, 121, 'fp32', 0.3), (160, 100, 'fp32', 1e-3), (128, 90, 'fp64', 0.1), (96, 48, 'fp32', 0.3)]
    batch, alone = [make(pkg, *x[:3]) for x in specs], [make(pkg, *x[:3]) for x in specs]
    for group in (batch, alone):
        for k, (s, x) in enumerate(zip(group, specs)):
            shake(s, x[3], k)
    b = pkg.CylinderBatch(batch)
    for n in CALLS:
        series = b.solve(n, dt=0.002)
        for s, t, got in zip(batch, alone, series):
            for p, q in zip(got, t.solve(n_steps=n, **QUIET)):
                assert np.array_equal(p, q)
            for name in ('u', 'v', 'p'):
                assert np.array_equal(getattr(s, name), getattr(t, name))
            key = 'pressure_refinement_iterations'
            assert s.last_step_diagnostics[key] == t.last_step_diagnostics[key]
    b.close()


def test_loops_never_repeat_a_step(monkeypatch):
    """A state that needs more sweeps than are held repeats no step in loops; a failed gate still stops
    its case alone at the step that it fails."""
    pkg = load_package()
    monkeypatch.setenv('GHOSTMAC_BATCH_LOOPS', '1')
    cases = [make(pkg, precision='fp32'), make(pkg, 96, 48, 'fp32')]
    b = pkg.CylinderBatch(cases)
    b.solve(140, dt=0.002)
    before = [held(pkg, s) for s in cases]
    for k, s in enumerate(cases):
        shake(s, 0.3, k)
    b.solve(4, dt=0.002)
    assert [held(pkg, s)[1] for s in cases] == [h[1] for h in before]
    good = cases[1].u.copy()
    cases[0].v[40, 50] = np.nan
    with pytest.raises((ValueError, RuntimeError, FloatingPointError)):
        b.solve(3, dt=0.002)
    assert np.isfinite(cases[1].u).all() and not np.array_equal(cases[1].u, good)
    b.close()


def test_case_stepped_alone_in_between():
    """After one step of one case alone the batch pairs its cases' buffers anew and captures its two graphs
    again, once: its steps then replay them (a step that captures eight cases takes many times as long)."""
    pkg = load_package()
    cases = [make(pkg, 96, 48) for _ in range(8)]
    b = pkg.CylinderBatch(cases)

    def fastest():
        times = []
        for _ in range(6):
            t0 = time.perf_counter()
            rc, _, _ = b.step_raw(0.002, 1)
            times.append(time.perf_counter() - t0)
            b._check(rc)
        return min(times)

    fastest()
    before = fastest()
    rc, _ = cases[3].step_raw(0.002, 1)
    pkg._lib.check(rc, cases[3]._h)
    after = fastest()
    b.close()
    assert after < 3 * before
