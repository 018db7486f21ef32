"""Float64 averages with more symmetry images than one pass of the digit products takes
(64): a full pass, then what is left, with and without the row scalars and forces as
products of their own.

Tolerance: the oracle adds up N S <= 2e5 float64 terms one after the other, of up to about
30 times their rms: sqrt(2e5) 30 2^-53 = 1.5e-12 of the largest entry."""
import numpy as np
import pytest

import oracle
from tdscha_gb300 import _native as nat
from tdscha_gb300.synthetic import make_ensemble, random_R1, random_sym

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,S", [(24, 300, 65), (24, 300, 100), (63, 1400, 64), (63, 1400, 65),
                                   (63, 1400, 130), (66, 1000, 127)])
def test_more_images_than_a_pass(gpu_lib, M, N, S):
    ens = make_ensemble(M, N, seed=M + S, n_syms=48, rho_sigma=0.1)
    which = np.arange(S) % 48
    tables = ([s[which] for s in ens["symmetries"]], ens["degenerate_space"], ens["sym_block_id"])
    R1, Y1 = random_R1(M, 1), random_sym(M, 2, scale=1e-3)
    ref = oracle.perturb_averages(ens["X"], ens["Y"], ens["w"], ens["rho"], R1, Y1, ens["T"], 1,
                                  *tables, n_threads=8)
    ctx = nat.Context(ens["X"], ens["Y"], ens["w"], ens["rho"], ens["T"], *tables)
    assert ctx.layout()[0] == S
    f, d2v = np.zeros(M), np.zeros((M, M))
    for _ in range(2):
        nat.check(nat.load().tdscha_perturb_averages(ctx.handle, nat.dp(R1), nat.dp(Y1), 1,
                                                     nat.PREC_FP64, nat.dp(f), nat.dp(d2v), 0, None))
        for a, b in zip((f, d2v), ref):
            assert np.abs(a - b).max() <= 1.5e-12 * max(np.abs(b).max(), 1e-300)
    ctx.close()
