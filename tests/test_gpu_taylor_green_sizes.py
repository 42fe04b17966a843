"""The periodic solver's packed transforms (csrc/periodic.cu) at the sizes where they can go wrong:
the smallest grid, odd sizes (a last unpaired row, no Nyquist mode), sizes with generic radices,
sizes around the groups of 32 threads, against the CPU oracle in float64; and the state after a
failed gate in the middle of a queued call."""
import numpy as np
import pytest

import ghost_oracle as go
from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [8, 9, 14, 15, 21, 26, 49, 63, 64, 100, 129, 196, 250])
def test_sizes_match_oracle(n):
    """Six steps; the oracle solves the CN system with GMRES to rtol 1e-12, so fields agree to
    1e-11 of their maxima (velocity) and 1e-10 (pressure), as on the reference's own runs."""
    tg = load_package().taylor_green
    dt, nu = 2e-3, 0.05
    ref = go.taylor_green_run(n, dt, end_time=6 * dt, nu=nu)
    _, q, p = tg.run(n, dt, 6 * dt, nu)
    assert np.max(np.abs(q - ref[1])) < 1e-11 * np.max(np.abs(ref[1]))
    assert np.max(np.abs(p - ref[2])) < 1e-10 * np.max(np.abs(ref[2]))


@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
def test_general_field_matches_small_steps_of_itself(precision):
    """n steps in one call and one call a step are the same computation."""
    tg = load_package().taylor_green
    n, rng = 45, np.random.default_rng(3)
    q0, p0 = tg.exact(n, 0.02, 0.0)
    q0[:n * n] += 0.1 * np.repeat(rng.standard_normal(n), n)
    out = []
    for calls, steps in ((1, 5), (5, 1)):
        case = tg.TaylorGreen(n, 0.02, precision)
        case.set_state(q0, p0)
        md = max(case.step(1e-3, steps) for _ in range(calls))
        out.append((*case.state(), md))
        case.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
@pytest.mark.parametrize('steps', [1, 2, 5])
def test_failed_gate_keeps_state(precision, steps):
    tg = load_package().taylor_green
    n = 24
    q0, p0 = tg.exact(n, 0.02, 0.0)
    case = tg.TaylorGreen(n, 0.02, precision)
    bad = q0.copy()
    bad[5] = np.nan
    case.set_state(bad, p0)
    with pytest.raises(RuntimeError, match='CN momentum solve failed'):
        case.step(1e-3, steps)
    q, half, _ = case.state()
    assert np.array_equal(q, bad, equal_nan=True) and np.array_equal(half, p0)
    case.set_state(q0, p0)
    case.step(1e-3, 3)
    again = case.state()
    fresh = tg.TaylorGreen(n, 0.02, precision)
    fresh.set_state(q0, p0)
    fresh.step(1e-3, 3)
    for a, b in zip(again, fresh.state()):
        assert np.array_equal(a, b)
