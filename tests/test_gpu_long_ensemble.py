"""A float64 context of more rows than 65535 blocks of 128 hold, the limit of a grid's
second dimension."""
import numpy as np
import pytest

import oracle
from tdscha_gb300 import _native as nat
from tdscha_gb300.synthetic import random_R1, random_sym

pytestmark = pytest.mark.gpu


def test_averages(gpu_lib):
    """8.4 million configurations, 3 modes (41 GB of digits).  The oracle adds up N terms in
    float64: sqrt(8.4e6) 30 2^-53 = 1e-11 of the largest entry."""
    M, N = 3, 65535 * 128 + 11
    rng = np.random.default_rng(1)
    X = rng.standard_normal((N, M))
    Y = 1e-3 * (rng.standard_normal((N, M)) + 0.1 * X ** 2)
    w, rho = np.array([1e-3, 1.7e-3, 2.1e-3]), rng.uniform(0.5, 1.5, N)
    tables = oracle.identity_symmetries(M)
    R1, Y1 = random_R1(M, 1), random_sym(M, 2, scale=1e-3)
    ref = oracle.perturb_averages(X, Y, w, rho, R1, Y1, 300.0, 1, *tables, n_threads=8)
    ctx = nat.Context(X, Y, w, rho, 300.0, *tables)
    f, d2v = np.zeros(M), np.zeros((M, M))
    nat.check(nat.load().tdscha_perturb_averages(ctx.handle, nat.dp(R1), nat.dp(Y1), 1, nat.PREC_FP64,
                                                 nat.dp(f), nat.dp(d2v), 0, None))
    ctx.close()
    nat.check(nat.load().tdscha_release_cached_memory(None))
    for a, b in zip((f, d2v), ref):
        assert np.abs(a - b).max() <= 1e-11 * np.abs(b).max()
