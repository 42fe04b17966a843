"""Step graphs with a fixed number of gated refinement sweeps: solves that need more than the graph
holds repeat their step with one more.  A perturbed FP32 flow needs two and three pressure sweeps in
its first steps and one later; steps launched one by one (every sweep gated, no graph) are the same
kernels, so states and diagnostics are equal bit for bit, alone and in a batch."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu
QUIET = dict(dt=0.002, perturb_transient=False, save_artifacts=False, verbose=False)


def make(pkg, nx, ny, precision, amp, seed):
    s = pkg.MAC_CylinderFlow(boundary='ghost_cell', time_scheme='ab2_cn', nx=nx, ny=ny, Lx=nx * 0.05, Ly=ny * 0.05, D=1.0,
                             xc=nx * 0.0125, yc=ny * 0.025, nu=0.02, verbose=False, precision=precision)
    q = s.gg.pack(s.u, s.v)
    q += amp * np.random.default_rng(seed).standard_normal(q.size)
    u, v = s.gg.unpack(q)
    s.u[:], s.v[:] = u, v
    return s


def history(s, calls):
    out = []
    for n in calls:
        t, cd, cl = s.solve(n_steps=n, **QUIET)
        d = s.last_step_diagnostics
        out.append((t, cd, cl, d['pressure_refinement_iterations'], d['pressure_residual_linf'], d['max_divergence']))
    return out


@pytest.mark.parametrize('precision,amp', [('fp32', 0.3), ('fp32', 1e-3), ('fp64', 0.3)])
def test_graph_equals_launches(monkeypatch, precision, amp):
    pkg = load_package()
    calls = (2, 1, 7, 3)
    a = make(pkg, 200, 121, precision, amp, 3)
    ha = history(a, calls)
    monkeypatch.setenv('GHOSTMAC_NO_GRAPHS', '1')
    b = make(pkg, 200, 121, precision, amp, 3)
    hb = history(b, calls)
    for name in ('u', 'v', 'p'):
        assert np.array_equal(getattr(a, name), getattr(b, name))
    for x, y in zip(ha, hb):
        for p, q in zip(x, y):
            assert np.array_equal(p, q)


def test_batch_equals_alone():
    pkg = load_package()
    specs = [(200, 121, 'fp32', 0.3, 1), (160, 100, 'fp32', 1e-3, 2), (128, 90, 'fp64', 0.1, 3), (200, 121, 'fp32', 0.1, 4)]
    batch, alone = [make(pkg, *x) for x in specs], [make(pkg, *x) for x in specs]
    b = pkg.CylinderBatch(batch)
    series = [b.solve(n, dt=0.002) for n in (3, 9, 4)]
    refined = 0
    for k, s in enumerate(alone):
        for got, n in zip(series, (3, 9, 4)):
            want = s.solve(n_steps=n, **QUIET)
            for p, q in zip(got[k], want):
                assert np.array_equal(p, q)
            refined = max(refined, s.last_step_diagnostics['pressure_refinement_iterations'])
        for name in ('u', 'v', 'p'):
            assert np.array_equal(getattr(batch[k], name), getattr(s, name))
    b.close()
    assert refined > 0
