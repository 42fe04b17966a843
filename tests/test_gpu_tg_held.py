"""The periodic solver's held refinement sweeps (FP32 mode): set by the first step, raised by a step that needs
more, lowered when later steps do not use them; the values do not depend on them."""
import ctypes as C

import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


def held(pkg, case):
    n, rep = (C.c_int32 * 4)(), C.c_int64()
    assert pkg._lib.lib.gm_tg_held_sweeps(case._t, n, C.byref(rep)) == 0
    return list(n), rep.value


@pytest.mark.parametrize('n', [45, 64])
def test_counts_follow_the_need(n):
    pkg = load_package()
    tg = pkg.taylor_green
    smooth = tg.exact(n, 0.02, 0.0)
    rough = (smooth[0] + 0.2 * np.random.default_rng(3).standard_normal(2 * n * n), smooth[1])
    tiny = (1e-7 * smooth[0], 1e-14 * smooth[1])
    cases = [tg.TaylorGreen(n, 0.02, 'fp32') for _ in range(2)]
    for calls in ((1, 3), (130,), (2, 7)):
        one, single = cases
        for state in (tiny, rough):
            for c in cases:
                c.set_state(*state)
            md = max(one.step(1e-3, k) for k in calls)
            ms = max(single.step(1e-3, 1) for _ in range(sum(calls)))
            assert md == ms
            for a, b in zip(one.state(), single.state()):
                assert np.array_equal(a, b)
    fresh = tg.TaylorGreen(n, 0.02, 'fp32')
    fresh.set_state(*rough)
    fresh.step(1e-3, 9)
    for a, b in zip(one.state(), fresh.state()):
        assert np.array_equal(a, b)
    assert held(pkg, fresh)[1] == 0 and held(pkg, one)[1] > 0
