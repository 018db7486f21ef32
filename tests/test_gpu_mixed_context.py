"""Float64 calls of contexts with mixed operands (with_mixed=True): their digit operands are
made at the first of them, not with the context."""
import numpy as np
import pytest

import oracle
from tdscha_gb300 import _native as nat
from tdscha_gb300.synthetic import make_ensemble, random_R1, random_sym

pytestmark = pytest.mark.gpu

M, N = 96, 20000


def _setup():
    ens = make_ensemble(M, N, seed=3, rho_sigma=0.1)
    tables = oracle.identity_symmetries(M)
    R1, Y1 = random_R1(M, 1), random_sym(M, 2, scale=1e-3)
    return (ens["X"], ens["Y"], ens["w"], ens["rho"], ens["T"], *tables), R1, Y1


def _call(ctx, R1, Y1):
    f, d2v = np.zeros(M), np.zeros((M, M))
    nat.check(nat.load().tdscha_perturb_averages(ctx.handle, nat.dp(R1), nat.dp(Y1), 1, nat.PREC_FP64,
                                                 nat.dp(f), nat.dp(d2v), 0, None))
    return f, d2v


def test_digits_at_the_first_call(gpu_lib):
    import torch
    args, R1, Y1 = _setup()
    plain = nat.Context(*args)
    ref = _call(plain, R1, Y1)
    plain.close()
    nat.check(nat.load().tdscha_release_cached_memory(None))
    ctx = nat.Context(*args, with_mixed=True)
    before = torch.cuda.mem_get_info()[0]
    got = _call(ctx, R1, Y1)
    held = before - torch.cuda.mem_get_info()[0]
    assert held >= 44 * M * N           # x, g and the digits of x, once in rows and once in columns
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)
    before = torch.cuda.mem_get_info()[0]
    _call(ctx, R1, Y1)
    assert torch.cuda.mem_get_info()[0] == before
    ctx.close()


@pytest.mark.parametrize("entry", ["averages", "apply", "static"])
def test_first_call_in_a_capture(gpu_lib, entry):
    """Nothing may be allocated there.  Tolerance of two float64 sums over N terms of up to
    about 30 times their rms: 2 sqrt(2e4) 30 2^-53 = 1e-12 of the largest entry."""
    import torch
    args, R1, Y1 = _setup()
    lib = nat.load()
    ctx = nat.Context(*args, with_mixed=True)
    ctx.set_options(True, False, False, False, False, 0.0)
    n = {"averages": M + M * M, "apply": ctx.P, "static": M + M * (M + 1) // 2}[entry]
    rng = np.random.default_rng(5)
    psi = torch.tensor(np.concatenate([R1, Y1.ravel()]) if entry == "averages"
                       else rng.standard_normal(n), device="cuda")
    out = torch.zeros(n, dtype=torch.float64, device="cuda")

    def call():
        st = torch.cuda.current_stream().cuda_stream
        a, b = psi.data_ptr(), out.data_ptr()
        if entry == "averages":
            nat.check(lib.tdscha_perturb_averages(ctx.handle, a, a + 8 * M, 1, nat.PREC_FP64, b, b + 8 * M,
                                                  1, st))
        elif entry == "apply":
            nat.check(lib.tdscha_apply_full_L(ctx.handle, a, b, 0, nat.PREC_FP64, st))
        else:
            nat.check(lib.tdscha_static_L(ctx.handle, 1, a, b, 2, 1.0, nat.PREC_FP64, st))

    if entry == "static":               # its own tables, made at the first call of any kind
        nat.check(lib.tdscha_static_L(ctx.handle, 1, psi.data_ptr(), out.data_ptr(), 1, 1.0, nat.PREC_FP64,
                                      None))
        torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    graph.replay()
    torch.cuda.synchronize()
    captured = out.cpu().numpy().copy()
    call()
    torch.cuda.synchronize()
    ref = out.cpu().numpy().copy()
    assert np.abs(captured - ref).max() <= 1e-12 * np.abs(ref).max()
    graph.replay()                      # the captured kernels' buffers are still there
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), captured)
    ctx.close()
