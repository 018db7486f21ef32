"""Accuracy of the digit products on data whose parts differ in size: rows of two
sublattices, and configurations that the weights take out or nearly so.

The reference is numpy's long double (64 or 113 bits) on the same inputs, and errors are
measured against the part in question, not against the largest part."""
import numpy as np
import pytest

from tdscha_gb300 import _native as nat

pytestmark = pytest.mark.gpu

LD = np.longdouble


@pytest.mark.parametrize("ratio", [1.0, 1e2, 1e4, 1e8])
def test_projection_of_two_sublattices(gpu_lib, ratio):
    """Light atoms with forces `ratio` times larger, modes on one sublattice each.  An
    element carries three roundings before the product (scale, mean, mass) and one after:
    4 2^-53 sum|a b| <= 4 2^-53 sqrt(n) rms(a) = 3.4e-15 rms(a) for n = 60; the entries of
    a column are normal with about that rms, the largest of 300 x 60 above 3 times it.
    2e-15 of the largest entry of a sublattice's modes, for either sublattice."""
    from tdscha_gb300.preprocessing import project_modes
    rng = np.random.default_rng(8)
    N, n = 300, 60
    light = np.arange(2 * n) // 3 % 2 == 0               # every other atom
    masses = np.where(light, 1.0, 200.0) * 911.444
    u = rng.standard_normal((N, 2 * n)) / np.sqrt(masses)
    f = rng.standard_normal((N, 2 * n)) * np.where(light, ratio, 1.0)
    u[:, light] *= ratio
    pols = np.zeros((2 * n, 2 * n))
    pols[np.ix_(light, np.arange(n))] = np.linalg.qr(rng.standard_normal((n, n)))[0]
    pols[np.ix_(~light, n + np.arange(n))] = np.linalg.qr(rng.standard_normal((n, n)))[0]
    X, Y = project_modes(u, f, masses, pols, f.mean(0), u_scale=0.5, f_scale=2.0)
    root, p = np.sqrt(masses).astype(LD), pols.astype(LD)
    f_mean = f.mean(0).astype(LD)
    for got, a in ((X, u.astype(LD) * LD(0.5) * root), (Y, (f.astype(LD) * 2 - f_mean * 2) / root)):
        ref = a @ p
        for part in (slice(0, n), slice(n, 2 * n)):
            assert np.abs(got[:, part] - ref[:, part]).max() <= 2e-15 * np.abs(ref[:, part]).max()
