"""Tensor-core kernels whose bounded waits give up at once (TDSCHA_WAIT_BUDGET_CYCLES=0):
no copy outlives its block and no thread waits for one that has left, so the call ends with
ERR_TIMEOUT (or, where nothing had to be waited for, with the right averages) and the GPU
serves the next context.

Shapes: fewer K blocks than a ring has slots, so that a producer has issued everything when
another role gives up; and rings that wrap."""
import numpy as np
import pytest

import oracle
from tdscha_gb300 import _native as nat
from tdscha_gb300.synthetic import make_ensemble, random_R1, random_sym

pytestmark = pytest.mark.gpu

# of the largest entry: N S <= 4e5 float64 terms in the oracle; the mixed averages
TOL = {nat.PREC_FP64: 3e-12, nat.PREC_MIXED: 2e-5}


def _call(ctx, R1, Y1, precision):
    f, d2v = np.zeros(R1.size), np.zeros(Y1.shape)
    nat.check(nat.load().tdscha_perturb_averages(ctx.handle, nat.dp(R1), nat.dp(Y1), 1, precision,
                                                 nat.dp(f), nat.dp(d2v), 0, None))
    return f, d2v


@pytest.mark.parametrize("M,N,S,precision", [
    (20, 100, 1, nat.PREC_FP64), (66, 700, 1, nat.PREC_FP64), (129, 9000, 1, nat.PREC_FP64),
    (24, 400, 48, nat.PREC_FP64), (63, 1400, 48, nat.PREC_FP64), (189, 2000, 8, nat.PREC_FP64),
    (20, 100, 1, nat.PREC_MIXED), (66, 700, 1, nat.PREC_MIXED), (129, 9000, 1, nat.PREC_MIXED),
    # blocks with a single image of a row tile, so that one epilogue set has none
    (24, 130, 24, nat.PREC_MIXED), (63, 1400, 48, nat.PREC_MIXED), (189, 2000, 8, nat.PREC_MIXED)])
def test_averages(gpu_lib, monkeypatch, M, N, S, precision):
    ens = make_ensemble(M, N, seed=M + S, n_syms=S)
    tables = ((ens["symmetries"], ens["degenerate_space"], ens["sym_block_id"]) if S > 1
              else oracle.identity_symmetries(M))
    R1, Y1 = random_R1(M, 1), random_sym(M, 2, scale=1e-3)
    ref = oracle.perturb_averages(ens["X"], ens["Y"], ens["w"], ens["rho"], R1, Y1, ens["T"], 1,
                                  *tables, n_threads=8)
    args = (ens["X"], ens["Y"], ens["w"], ens["rho"], ens["T"], *tables,
            precision == nat.PREC_MIXED)

    def right(got):
        for a, b in zip(got, ref):
            assert np.abs(a - b).max() <= TOL[precision] * max(np.abs(b).max(), 1e-300)

    monkeypatch.setenv("TDSCHA_AUTOTUNE", "0")
    monkeypatch.setenv("TDSCHA_WAIT_BUDGET_CYCLES", "0")
    ctx = nat.Context(*args)
    monkeypatch.delenv("TDSCHA_WAIT_BUDGET_CYCLES")
    for _ in range(3):
        try:
            right(_call(ctx, R1, Y1, precision))
        except nat.TdschaError as e:
            assert e.code == nat.ERR_TIMEOUT
    ctx.close()
    ctx = nat.Context(*args)
    right(_call(ctx, R1, Y1, precision))
    ctx.close()
