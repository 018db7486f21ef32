"""Stage A of the mixed averages with symmetry images (csrc/perturb_mixed.cu, up to 192
modes): edges of its column tiles and row tiles, and blocks that take a single image of
a row tile, an odd number of them, or more images than a row tile has.

Tolerance: that of the mixed averages against the float64 ones (tests/test_gpu_mixed.py).
Both sides run on the GPU, so the ensembles can be long."""
import numpy as np
import pytest

from tdscha_gb300 import _native as nat
from tdscha_gb300.synthetic import make_ensemble, random_R1, random_sym

pytestmark = pytest.mark.gpu

TOL_CALL = 2e-5


def _rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("M,N,S", [(6, 1, 8), (24, 129, 8), (63, 640, 24), (66, 2600, 8),
                                   (126, 5000, 24), (129, 127, 48), (132, 2433, 8), (189, 128, 8),
                                   (192, 385, 48), (192, 1500, 24)])
def test_images(gpu_lib, M, N, S):
    ens = make_ensemble(M, N, seed=M + N, n_syms=S, rho_sigma=0.1)
    R1, Y1 = random_R1(M, 8), random_sym(M, 9, scale=1e-3)
    ctx = nat.Context(ens["X"], ens["Y"], ens["w"], ens["rho"], ens["T"], ens["symmetries"],
                      ens["degenerate_space"], ens["sym_block_id"], with_mixed=True)
    out = []
    for precision in (nat.PREC_FP64, nat.PREC_MIXED, nat.PREC_MIXED):
        f, d2v = np.zeros(M), np.zeros((M, M))
        nat.check(nat.load().tdscha_perturb_averages(ctx.handle, nat.dp(R1), nat.dp(Y1), 1, precision,
                                                     nat.dp(f), nat.dp(d2v), 0, None))
        out.append((f, d2v))
    for a, b, c in zip(*out):
        assert _rel(b, a) <= TOL_CALL
        assert np.array_equal(b, c)
    ctx.close()
