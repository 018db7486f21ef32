"""Float64 averages by exact digit products on the tensor cores
(csrc/perturb_digits.cu) at the edges of its tiles, against the oracle, and
over the forms a context accepts, against the CUDA-core kernels.

Tolerance: the oracle adds up to N S terms one after the other in float64; with
N S <= 2e4 and terms of up to about 30 times their rms that is at most
sqrt(2e4) 30 2^-53 = 5e-13 of the largest entry.  The digit products leave out
less than 2^-60 of it.  1e-12 for either."""
import numpy as np
import pytest

import oracle
from tdscha_gb300 import _native as nat
from tdscha_gb300.synthetic import make_ensemble, random_R1, random_sym

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _rel(got, ref):
    return np.abs(np.asarray(got) - ref).max() / max(np.abs(ref).max(), 1e-300)


def _tables(ens, M):
    if "symmetries" in ens:
        return ens["symmetries"], ens["degenerate_space"], ens["sym_block_id"]
    return oracle.identity_symmetries(M)


def _context(ens, monkeypatch=None, cores=False):
    if cores:
        monkeypatch.setenv("TDSCHA_FP64_DIGITS", "0")
    try:
        return nat.Context(ens["X"], ens["Y"], ens["w"], ens["rho"], ens["T"],
                           *_tables(ens, ens["X"].shape[1]))
    finally:
        if cores:
            monkeypatch.delenv("TDSCHA_FP64_DIGITS")


def _call(ctx, R1, Y1, d4=1):
    """Device pointers, so that non-finite input reaches the kernels."""
    import torch
    M = R1.size
    a, b = torch.tensor(R1, device="cuda"), torch.tensor(Y1, device="cuda")
    f = torch.empty(M, dtype=torch.float64, device="cuda")
    d2v = torch.empty((M, M), dtype=torch.float64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    nat.check(nat.load().tdscha_perturb_averages(ctx.handle, a.data_ptr(), b.data_ptr(), d4,
                                                 nat.PREC_FP64, f.data_ptr(), d2v.data_ptr(), 1, st))
    nat.check(nat.load().tdscha_ctx_sync(ctx.handle, st))
    return f.cpu().numpy(), d2v.cpu().numpy()


@pytest.mark.parametrize("M,N,S,T", [(1, 5, 1, 300.0), (1, 193, 1, 0.0), (63, 127, 1, 300.0),
                                     (64, 128, 1, 0.0), (65, 129, 1, 700.0), (192, 192, 1, 300.0),
                                     (193, 385, 1, 120.0), (257, 1000, 1, 300.0),
                                     (24, 400, 48, 300.0), (66, 257, 8, 300.0), (129, 150, 24, 0.0)])
@pytest.mark.parametrize("d4", [0, 1])
def test_edges_against_oracle(gpu_lib, M, N, S, T, d4):
    ens = make_ensemble(M, N, seed=M + N + S, T=T, n_syms=S, rho_sigma=0.1)
    R1, Y1 = random_R1(M, 3), random_sym(M, 4, scale=1e-5)
    ctx = _context(ens)
    f, d2v = _call(ctx, R1, Y1, d4)
    ctx.close()
    f_ref, d_ref = oracle.perturb_averages(ens["X"], ens["Y"], ens["w"], ens["rho"], R1, Y1,
                                           ens["T"], d4, *_tables(ens, M), n_threads=8)
    assert _rel(f, f_ref) <= TOL and _rel(d2v, d_ref) <= TOL


def _forms():
    rng = np.random.default_rng(5)
    M, N = 70, 900
    ens = make_ensemble(M, N, seed=21, rho_sigma=0.1)
    R1, Y1 = random_R1(M, 3), random_sym(M, 4, scale=1e-5)
    z = 2 * rng.standard_normal((M, M))
    yield "wide", ens, R1, Y1 * np.exp(z + z.T)
    yield "asymmetric", ens, R1, Y1 + 1e-5 * rng.standard_normal((M, M))
    yield "no Y1", ens, R1, 0 * Y1
    yield "no R1", ens, 0 * R1, Y1
    yield "one entry", ens, R1, np.where(np.arange(M * M).reshape(M, M) == 3 * M + 3, 1.0, 0.0)
    yield "tiny", ens, 1e-120 * R1, 1e-120 * Y1
    yield "huge", ens, 1e120 * R1, 1e120 * Y1
    rho = ens["rho"].copy()
    rho[::3] = 0
    yield "weights", dict(ens, rho=rho), R1, Y1
    X, Y = ens["X"].copy(), ens["Y"].copy()
    X[:, 7], Y[:, 9], X[11], Y[11] = 0, 0, 0, 0
    yield "zero rows", dict(ens, X=X, Y=Y), R1, Y1
    X = ens["X"].copy()
    X[5] *= 1e3
    yield "outlier", dict(ens, X=X), R1, Y1
    # every digit of every element at the same value: the largest sums there are
    one = np.full((N, M), float.fromhex("0x1.7f7f7f7f7f7f7p+0"))
    yield "coherent", dict(ens, X=one, Y=one * 1e-6), R1, np.full((M, M), 1e-5)


@pytest.mark.parametrize("name", [f[0] for f in _forms()])
def test_forms_against_cuda_cores(gpu_lib, monkeypatch, name):
    _, ens, R1, Y1 = next(f for f in _forms() if f[0] == name)
    digits, cores = _context(ens), _context(ens, monkeypatch, cores=True)
    a, b = _call(digits, R1, Y1), _call(cores, R1, Y1)
    again = _call(digits, R1, Y1)
    digits.close()
    cores.close()
    assert _rel(a[0], b[0]) <= TOL and _rel(a[1], b[1]) <= TOL
    assert np.array_equal(a[0], again[0]) and np.array_equal(a[1], again[1])


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("S", [1, 8])
def test_non_finite_perturbation_gives_nan(gpu_lib, bad, S):
    M, N = 66, 300
    ens = make_ensemble(M, N, seed=4, n_syms=S)
    ctx = _context(ens)
    R1, Y1 = random_R1(M, 3), random_sym(M, 4, scale=1e-5)
    Y1b, R1b = Y1.copy(), R1.copy()
    Y1b[3, 4] = Y1b[4, 3] = bad
    R1b[5] = bad
    assert np.isnan(_call(ctx, R1, Y1b)[1]).any()
    assert np.isnan(_call(ctx, R1b, Y1)[1]).any()
    f, d2v = _call(ctx, R1, Y1)                       # nothing is left of it
    assert np.isfinite(f).all() and np.isfinite(d2v).all()
    ctx.close()


def test_stored_image_rows(gpu_lib, monkeypatch):
    M, N, S = 24, 130, 8
    ens = make_ensemble(M, N, seed=6, n_syms=S, rho_sigma=0.1)
    monkeypatch.setenv("TDSCHA_SYMMETRY_IMAGES", "rows")
    rows = _context(ens)
    monkeypatch.delenv("TDSCHA_SYMMETRY_IMAGES")
    assert rows.layout() == (1, N * S)
    images = _context(ens)
    R1, Y1 = random_R1(M, 3), random_sym(M, 4, scale=1e-5)
    a, b = _call(rows, R1, Y1), _call(images, R1, Y1)
    rows.close()
    images.close()
    assert _rel(a[0], b[0]) <= TOL and _rel(a[1], b[1]) <= TOL


def test_bounded_wait_reports_timeout(gpu_lib, monkeypatch):
    M, N = 66, 700
    ens = make_ensemble(M, N, seed=5)
    R1, Y1 = random_R1(M, 1), random_sym(M, 2, scale=1e-5)
    monkeypatch.setenv("TDSCHA_WAIT_BUDGET_CYCLES", "0")
    ctx = _context(ens)
    monkeypatch.delenv("TDSCHA_WAIT_BUDGET_CYCLES")
    with pytest.raises(nat.TdschaError) as e:
        _call(ctx, R1, Y1)
    assert e.value.code == nat.ERR_TIMEOUT
    ctx.close()
    ctx = _context(ens)
    f, d2v = _call(ctx, R1, Y1)
    ctx.close()
    f_ref, d_ref = oracle.perturb_averages(ens["X"], ens["Y"], ens["w"], ens["rho"], R1, Y1,
                                           ens["T"], 1, *_tables(ens, M))
    assert _rel(f, f_ref) <= TOL and _rel(d2v, d_ref) <= TOL


@pytest.mark.parametrize("N,n,M", [(1, 3, 1), (127, 63, 60), (128, 64, 64), (129, 66, 65),
                                   (300, 195, 190), (65541, 9, 6)])
def test_projection_edges_against_oracle(gpu_lib, N, n, M):
    """X and Y of the mode projection; the oracle's products round n <= 195 terms in
    float64, at most 195 2^-53 = 2e-14 of the largest entry."""
    from tdscha_gb300.preprocessing import project_modes
    rng = np.random.default_rng(N + n)
    u, f = rng.standard_normal((N, n)), 1e-3 * rng.standard_normal((N, n))
    masses, mean = rng.uniform(1e3, 2e5, n), f.mean(0)
    pols = np.linalg.qr(rng.standard_normal((n, max(M, 1))))[0][:, :M]
    got = project_modes(u, f, masses, pols, mean, u_scale=0.5, f_scale=2.0)
    ref = oracle.project_modes(u, f, masses, pols, mean, 0.5, 2.0)
    for a, b in zip(got, ref):
        assert _rel(a, b) <= 1e-13
    u[0, 1] = np.nan
    X, Y = project_modes(u, f, masses, pols, mean, u_scale=0.5, f_scale=2.0)
    assert np.isnan(X[0]).all() and np.isfinite(X[1:]).all() and np.isfinite(Y).all()


@pytest.mark.parametrize("M,N,S", [(189, 460, 48), (192, 900, 24), (252, 2100, 8), (129, 1300, 24)])
@pytest.mark.parametrize("d4", [0, 1])
def test_many_images(gpu_lib, M, N, S, d4):
    """From 8 images and 4 million elements on: the row scalars and the forces as
    products of their own.  N S <= 3.2e4 here: 7e-13 by the estimate above."""
    ens = make_ensemble(M, N, seed=M, n_syms=S, rho_sigma=0.1)
    assert min(S, 64) * M * N >= 4e6
    R1, Y1 = random_R1(M, 1), random_sym(M, 2, scale=1e-3)
    ref = oracle.perturb_averages(ens["X"], ens["Y"], ens["w"], ens["rho"], R1, Y1, ens["T"], d4,
                                  *_tables(ens, M), n_threads=8)
    ctx = _context(ens)
    got = _call(ctx, R1, Y1, d4)
    ctx.close()
    assert _rel(got[1], ref[1]) < TOL
    assert np.abs(got[0] - ref[0]).max() < TOL * max(np.abs(ref[0]).max(), 1e-300)


def test_many_images_matches_core_kernels(gpu_lib, monkeypatch):
    """Zero and non-finite perturbations, a scaled ensemble, a repeated call."""
    ens = make_ensemble(63, 1400, seed=3, n_syms=48, rho_sigma=0.1)
    R1, Y1 = random_R1(63, 1), random_sym(63, 2, scale=1e-3)
    ctx, cores = _context(ens), _context(ens, monkeypatch, cores=True)
    for r, y in ((R1, Y1), (R1 * 0, Y1), (R1, Y1 * 0), (R1 * 1e100, Y1), (R1, Y1 * 1e-200), (R1, Y1)):
        a, b = _call(ctx, r, y), _call(cores, r, y)
        for u, v in zip(a, b):
            assert np.abs(u - v).max() <= 3e-12 * np.abs(v).max()     # N S = 6.7e4 on both sides
    for bad in (np.nan, np.inf):
        y = Y1.copy()
        y[3, 5] = y[5, 3] = bad
        a, b = _call(ctx, R1, y), _call(cores, R1, y)
        for u, v in zip(a, b):
            assert (np.isfinite(u) == np.isfinite(v)).all()
    ctx.close()
    cores.close()


@pytest.mark.parametrize("M,N", [(16, 100), (17, 300), (32, 129), (33, 700), (48, 2500), (64, 4800),
                                 (64, 9800)])
def test_column_parts(gpu_lib, M, N):
    """Up to 64 modes and few rows: several work items share a tile (stage A), blocks of
    32 modes (W), slabs of two rows (the end)."""
    ens = make_ensemble(M, N, seed=M + N, rho_sigma=0.1)
    R1, Y1 = random_R1(M, 3), random_sym(M, 4, scale=1e-5)
    ctx = _context(ens)
    got = _call(ctx, R1, Y1)
    ctx.close()
    ref = oracle.perturb_averages(ens["X"], ens["Y"], ens["w"], ens["rho"], R1, Y1, ens["T"], 1,
                                  *_tables(ens, M), n_threads=8)
    assert _rel(got[0], ref[0]) <= TOL and _rel(got[1], ref[1]) <= TOL
