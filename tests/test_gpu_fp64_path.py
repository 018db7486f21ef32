"""Which kernels serve float64 averages, and that the choice counts idle blocks of the
library's cache as free memory."""
import numpy as np
import pytest

import oracle
from tdscha_gb300 import _native as nat
from tdscha_gb300.QSpaceLanczos import QSpaceLanczos
from tdscha_gb300.synthetic import make_ensemble, make_qspace_ensemble, random_R1, random_sym

pytestmark = pytest.mark.gpu


def test_paths(gpu_lib, monkeypatch):
    ens = make_ensemble(12, 300, seed=1)
    args = (ens["X"], ens["Y"], ens["w"], ens["rho"], ens["T"], *oracle.identity_symmetries(12))
    R1, Y1, f, d2v = random_R1(12, 1), random_sym(12, 2), np.zeros(12), np.zeros((12, 12))

    def path(with_mixed, call=False):
        ctx = nat.Context(*args, with_mixed=with_mixed)
        if call:
            nat.check(nat.load().tdscha_perturb_averages(ctx.handle, nat.dp(R1), nat.dp(Y1), 1, nat.PREC_FP64,
                                                         nat.dp(f), nat.dp(d2v), 0, None))
        p = ctx.fp64_path()
        ctx.close()
        return p

    assert path(False) == "tensor cores"
    assert path(True) == "pending" and path(True, True) == "tensor cores"
    assert path("fp32") == "none"
    e = make_qspace_ensemble((2, 1, 1), 3, 50, seed=1)
    lz = QSpaceLanczos.from_arrays(e["X_q"], e["Y_q"], e["w_q"], e["rho"], e["T"], q_points=e["q"])
    lz.init(use_symmetries=False)
    lz.build_q_pair_map(0)
    assert lz._qcontext().fp64_path() == "tensor cores"
    monkeypatch.setenv("TDSCHA_FP64_DIGITS", "0")
    assert path(False) == "CUDA cores" and path(True, True) == "CUDA cores"
    lz._invalidate()
    assert lz._qcontext().fp64_path() == "CUDA cores"


def test_memory_rule(gpu_lib):
    """4.2 GiB of digits: with 15 GiB free and 8 GiB idle they are within a quarter, with 15
    alone they are not.  The oracle adds up N terms: sqrt(9e5) 30 2^-53 = 3e-12."""
    import torch
    lib = nat.load()
    M, N = 64, 900000
    rng = np.random.default_rng(1)
    X = rng.standard_normal((N, M))
    Y = 1e-3 * (rng.standard_normal((N, M)) + 0.1 * X ** 2)
    w, rho = np.linspace(1e-3, 3e-3, M), rng.uniform(0.5, 1.5, N)
    args = (X, Y, w, rho, 300.0, *oracle.identity_symmetries(M))
    R1, Y1 = random_R1(M, 1), random_sym(M, 2, scale=1e-3)
    ref = oracle.perturb_averages(X, Y, w, rho, R1, Y1, 300.0, 1, *args[5:], n_threads=8)

    def make():
        ctx = nat.Context(*args)
        f, d2v = np.zeros(M), np.zeros((M, M))
        nat.check(lib.tdscha_perturb_averages(ctx.handle, nat.dp(R1), nat.dp(Y1), 1, nat.PREC_FP64,
                                              nat.dp(f), nat.dp(d2v), 0, None))
        for a, b in zip((f, d2v), ref):
            assert np.abs(a - b).max() <= 3e-12 * np.abs(b).max()
        p = ctx.fp64_path()
        ctx.close()
        return p

    nat.check(lib.tdscha_release_cached_memory(None))
    assert make() == "tensor cores"
    gib = 1 << 30
    other = nat.Context(X[: N // 2], Y[: N // 2], w, rho[: N // 2], *args[4:])     # other blocks
    other.close()
    held = []
    try:
        held.append(torch.empty(torch.cuda.mem_get_info()[0] - 15 * gib, dtype=torch.uint8, device="cuda"))
        assert make() == "tensor cores"
        nat.check(lib.tdscha_release_cached_memory(None))
        held.append(torch.empty(torch.cuda.mem_get_info()[0] - 15 * gib, dtype=torch.uint8, device="cuda"))
        assert make() == "CUDA cores"
    finally:
        held.clear()
        torch.cuda.empty_cache()
        nat.check(lib.tdscha_release_cached_memory(None))
