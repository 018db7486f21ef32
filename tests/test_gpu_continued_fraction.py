"""The continued fraction on the GPU (csrc/lanczos.cu) at the edges of its chunks of
levels and blocks of frequencies, against the oracle.

Tolerance: with |b c| <= 1 and every level's denominator above 2.5 an error of a level
reaches the next one divided by six, so that of G is about that of one level, at most
ten roundings on either side: 20 2^-53 1.2 = 3e-15 of |G|.  1e-14."""
import numpy as np
import pytest

import oracle
from tdscha_gb300 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_w", [(1, 1), (2, 63), (3, 64), (24, 500), (256, 65), (257, 128),
                                   (258, 129), (600, 7)])
@pytest.mark.parametrize("wigner", [0, 1])
@pytest.mark.parametrize("term,ramp,nonsym", [(0, 0, 0), (1, 0, 1), (1, 3, 1)])
def test_matches_oracle(gpu_lib, n, n_w, wigner, term, ramp, nonsym):
    rng = np.random.default_rng(n + n_w)
    if term and n == 1:
        pytest.skip("the terminator needs b coefficients")
    a = 4.5 + rng.random(n)
    b = 0.5 + 0.5 * rng.random(n - 1)
    c = 0.5 + 0.5 * rng.random(n - 1) if nonsym else b
    w = np.linspace(0, 1, n_w)
    out = np.zeros(2 * n_w)
    last = min(5, n - 1) if term else 1
    nat.check(nat.load().tdscha_continued_fraction(
        nat.dp(a), n, nat.dp(b), n - 1, nat.dp(c), n - 1, nat.dp(w), n_w, wigner, 1.7, 0, 0.0, term,
        last, 0.02, ramp, nat.dp(out)))
    ref = oracle.continued_fraction(a, b, c, w, use_wigner=bool(wigner), modulus=1.7,
                                    use_terminator=bool(term), last_average=last, smearing=0.02,
                                    smooth_ramp=ramp)
    got = out[0::2] + 1j * out[1::2]
    assert np.abs(got - ref).max() <= 1e-14 * np.abs(ref).max()
