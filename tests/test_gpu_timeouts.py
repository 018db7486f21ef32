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


@pytest.mark.parametrize("M,N,S", [(48, 5000, 1), (129, 9000, 1), (24, 400, 48), (189, 2000, 8)])
def test_device_pointers_get_nan(gpu_lib, monkeypatch, M, N, S):
    """A call on device pointers returns before its kernels have run: after a wait that gave
    up every result is NaN, and tdscha_ctx_sync says so once."""
    import torch
    ens = make_ensemble(M, N, seed=M + S, n_syms=S)
    tables = ((ens["symmetries"], ens["degenerate_space"], ens["sym_block_id"]) if S > 1
              else oracle.identity_symmetries(M))
    monkeypatch.setenv("TDSCHA_WAIT_BUDGET_CYCLES", "0")
    ctx = nat.Context(ens["X"], ens["Y"], ens["w"], ens["rho"], ens["T"], *tables)
    monkeypatch.delenv("TDSCHA_WAIT_BUDGET_CYCLES")
    R1 = torch.tensor(random_R1(M, 1), device="cuda")
    Y1 = torch.tensor(random_sym(M, 2, scale=1e-3), device="cuda")
    f, d2v = torch.zeros_like(R1), torch.zeros_like(Y1)
    st = torch.cuda.current_stream().cuda_stream
    nat.check(nat.load().tdscha_perturb_averages(ctx.handle, R1.data_ptr(), Y1.data_ptr(), 1,
                                                 nat.PREC_FP64, f.data_ptr(), d2v.data_ptr(), 1, st))
    with pytest.raises(nat.TdschaError) as e:
        nat.check(nat.load().tdscha_ctx_sync(ctx.handle, st))
    assert e.value.code == nat.ERR_TIMEOUT
    assert torch.isnan(f).all() and torch.isnan(d2v).all()
    nat.check(nat.load().tdscha_ctx_sync(ctx.handle, st))
    ctx.close()


@pytest.mark.parametrize("batch", [False, True])
def test_run_reports_the_wait(gpu_lib, monkeypatch, batch):
    """A run whose averages are NaN after such a wait reports the wait, not the NaN."""
    from tdscha_gb300.DynamicalLanczos import Lanczos
    from tdscha_gb300.batch import run_batch
    M, N = 70, 4000
    ens = make_ensemble(M, N, seed=1)
    lanc = Lanczos.from_arrays(ens["X"], ens["Y"], ens["w"], ens["rho"], ens["T"], use_wigner=True)
    lanc.init(use_symmetries=False)
    lanc.prepare_perturbation(random_R1(M, 1), masses_exp=0)
    monkeypatch.setenv("TDSCHA_WAIT_BUDGET_CYCLES", "0")
    with pytest.raises(nat.TdschaError) as e:
        run_batch([lanc], 4) if batch else lanc.run_FT(4, verbose=False)
    assert e.value.code == nat.ERR_TIMEOUT


@pytest.mark.parametrize("call", ["averages", "averages on device pointers", "apply", "run", "batch",
                                  "moments"])
def test_bloch_space(gpu_lib, monkeypatch, call):
    """Every way into the Bloch-space averages reports the wait, once, and leaves nothing of
    it to the next call."""
    import torch
    from tdscha_gb300.batch import run_batch
    from tdscha_gb300.QSpaceKPM import QSpaceKPM
    from tdscha_gb300.synthetic import make_qspace_ensemble
    e = make_qspace_ensemble((4, 2, 1), 12, 9000, seed=2, dispersion=0.2)
    ql = QSpaceKPM.from_arrays(e["X_q"], e["Y_q"], e["w_q"], e["rho"], e["T"], q_points=e["q"])
    ql.init(use_symmetries=False)
    ql.prepare_mode_q(1, 2)
    rng = np.random.default_rng(1)
    R1 = rng.standard_normal(12) + 0j
    alpha = [rng.standard_normal((12, 12)) + 0j for _ in ql.unique_pairs]
    monkeypatch.setenv("TDSCHA_WAIT_BUDGET_CYCLES", "0")
    ctx = ql._qcontext()
    st = torch.cuda.current_stream().cuda_stream
    if call == "averages on device pointers":
        a, b = (torch.tensor(v, device="cuda") for v in (R1, np.stack(alpha)))
        f, d2v = torch.zeros_like(a), torch.zeros_like(b)
        nat.check(nat.load().tdscha_qperturb_averages(ctx.handle, a.data_ptr(), b.data_ptr(), 1,
                                                      f.data_ptr(), d2v.data_ptr(), 1, st))
    with pytest.raises(nat.TdschaError) as err:
        if call == "averages":
            ql.get_perturb_averages_q(R1, alpha)
        elif call == "apply":
            ql.apply_full_L()
        elif call == "run":
            ql.run_FT(3, verbose=False)
        elif call == "batch":
            run_batch([ql], 3)
        elif call == "moments":
            ql.run_KPM(8, lambda_min=0.0, lambda_max=1e-4, verbose=False)
        else:
            nat.check(nat.load().tdscha_qctx_sync(ctx.handle, st))
    assert err.value.code == nat.ERR_TIMEOUT
    nat.check(nat.load().tdscha_qctx_sync(ctx.handle, st))
    if call == "averages on device pointers":
        assert torch.isnan(f.real).all() and torch.isnan(d2v.real).all()
