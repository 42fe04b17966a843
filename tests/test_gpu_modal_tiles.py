"""The POD kernels' tiles and slices (csrc/modal.cu) at their edges: snapshot counts around the
16-wide Gram tiles and the 32-wide coefficient tiles, point counts around the staged chunks and the
slice length, mode counts around the groups of eight, against numpy in float64.  Every entry is a
dot product of n terms summed in another order, so it may differ by twice the a priori bound
(n + 2) eps sum |a| |b| of either sum (the subtraction of the mean is the same single rounding
on both sides)."""
import ctypes as C

import numpy as np
import pytest

from conftest import load_package

EPS = np.finfo(np.float64).eps


@pytest.mark.gpu
@pytest.mark.parametrize('m,n,k', [(1, 1, 1), (2, 63, 2), (15, 64, 8), (16, 65, 9), (17, 511, 17), (31, 513, 5),
                                   (33, 1024, 3), (48, 40001, 6), (65, 2047, 16), (96, 20000, 10), (130, 777, 7)])
def test_gram_modes_coefficients(m, n, k):
    pkg = load_package()
    lib, ptr = pkg._lib.lib, pkg._lib.ptr
    rng = np.random.default_rng(1000 * m + n)
    x = rng.standard_normal((m, n)) + 3.0
    v, sigma = rng.standard_normal((m, k)), rng.uniform(0.5, 2.0, k)
    sigma[k // 2] = 1e-13 if k > 2 else sigma[k // 2]  # a null mode gives zeros
    h = C.c_void_p()
    assert lib.gm_pod_create(m, n, C.byref(h)) == 0
    try:
        mean, gram = np.empty(n), np.empty((m, m))
        assert lib.gm_pod_gram(h, ptr(x), ptr(mean), ptr(gram), None) == 0
        modes, coef = np.empty((k, n)), np.empty((k, m))
        assert lib.gm_pod_modes(h, ptr(v), ptr(sigma), k, ptr(modes), ptr(coef), None) == 0
    finally:
        lib.gm_pod_destroy(h)
    ref_mean = np.zeros(n)
    for row in x:  # the snapshots in order
        ref_mean = ref_mean + row
    ref_mean = ref_mean / m
    assert np.array_equal(mean, ref_mean)
    d = x - ref_mean
    assert np.array_equal(gram, gram.T)
    assert np.all(np.abs(gram - d @ d.T / m) <= 2 * (n + 2) * EPS * (np.abs(d) @ np.abs(d).T) / m)
    inv = np.where(sigma > 1e-12, 1.0 / sigma, 0.0)
    assert np.all(np.abs(modes - (d.T @ v * inv).T) <= 2 * (m + 2) * EPS * (np.abs(d).T @ np.abs(v) * inv).T)
    assert np.all(np.abs(coef - modes @ d.T) <= 2 * (n + 2) * EPS * (np.abs(modes) @ np.abs(d).T))
