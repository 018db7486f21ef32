"""Float64 Bloch-space averages by digit products (csrc/qspace_digits.cu) at the
edges of their tiles, against the oracle, and over the forms a context accepts,
against the CUDA-core kernels (csrc/qspace.cu).

Tolerance: both sides of a comparison add up to N S terms in float64; with
N S <= 1e3 and terms of up to about 30 times their rms that is at most
sqrt(1e3) 30 2^-53 = 1e-13 of the largest entry of a block.  The digit products
leave out less than 2^-60 of it.  1e-12 for either."""
import numpy as np
import pytest

import oracle.qspace as oq
from tdscha_gb300 import _native as nat
from tdscha_gb300.QSpaceLanczos import QSpaceLanczos
from tdscha_gb300.synthetic import make_qspace_ensemble

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _rel(got, ref):
    return np.abs(np.asarray(got) - ref).max() / max(np.abs(ref).max(), 1e-300)


def _setup(dims, nb, N, iq=0, syms=False, pairing="sum", scale=None):
    e = make_qspace_ensemble(dims, nb, N, seed=nb + N, T=250.0, dispersion=0.3, rho_sigma=0.2)
    if scale is not None:
        e["Y_q"] = e["Y_q"] * scale
    lz = QSpaceLanczos.from_arrays(e["X_q"], e["Y_q"], e["w_q"], e["rho"], e["T"],
                                   q_points=e["q"], pairing=pairing)
    valid = np.ones((nb, e["n_q"]), dtype=bool)
    valid[0, 0] = nb == 1
    lz.valid_modes_q = valid
    symmetries = None
    if syms:
        symmetries = [np.diag(np.repeat(np.exp(-2j * np.pi * (e["q"] @ t)), nb)) for t in e["cells"]]
    lz.prepare_symmetrization(symmetries=symmetries)
    lz.build_q_pair_map(iq)
    o = oq.OracleQSpaceLanczos(e["X_q"], e["Y_q"], e["w_q"], e["rho"], e["T"], lz.q_pair_map, iq,
                               symmetries=symmetries, valid=valid)
    rng = np.random.default_rng(3)
    R1 = rng.standard_normal(nb) + 1j * rng.standard_normal(nb)
    alpha = [rng.standard_normal((nb, nb)) + 1j * rng.standard_normal((nb, nb))
             for _ in lz.unique_pairs]
    return e, lz, o, R1, alpha


def _check(got, ref):
    assert _rel(got[0], ref[0]) < TOL
    for a, b in zip(got[1], ref[1]):
        assert _rel(a, b) < TOL


@pytest.mark.parametrize("dims,nb,N,iq,syms,pairing", [
    ((1, 1, 1), 1, 1, 0, False, "sum"), ((2, 1, 1), 1, 64, 1, False, "sum"),
    ((2, 1, 1), 7, 65, 0, False, "difference"), ((2, 1, 1), 8, 128, 1, False, "sum"),
    ((2, 1, 1), 9, 129, 0, False, "sum"), ((3, 1, 1), 15, 191, 2, False, "sum"),
    ((3, 1, 1), 16, 193, 0, False, "difference"), ((2, 1, 1), 17, 256, 1, False, "sum"),
    ((2, 1, 1), 31, 127, 0, False, "sum"), ((2, 2, 1), 32, 257, 3, False, "sum"),
    ((2, 2, 2), 3, 120, 5, True, "sum"), ((4, 2, 1), 6, 1000, 3, False, "sum")])
@pytest.mark.parametrize("d4", [True, False])
def test_averages(gpu_lib, dims, nb, N, iq, syms, pairing, d4):
    e, lz, o, R1, alpha = _setup(dims, nb, N, iq, syms, pairing)
    ref = oq.perturb_averages_qspace(e["X_q"], e["Y_q"], e["w_q"], e["rho"], R1, alpha, e["T"], d4,
                                     iq, o.pairs, o.symmetries, o.valid)
    _check(lz.get_perturb_averages_q(R1, alpha, d4), ref)


@pytest.mark.parametrize("form", ["plain", "scaled", "zero_R1", "zero_alpha", "zero_Y", "huge_alpha",
                                  "column"])
def test_matches_core_kernels(gpu_lib, monkeypatch, form):
    """Scaled operands, zeros, one large element: what the kernels of qspace.cu give."""
    _, lz, _, R1, alpha = _setup((3, 1, 1), 5, 300, 1,
                                 scale={"scaled": 2.0 ** 90, "zero_Y": 0.0}.get(form))
    if form == "zero_R1":
        R1 = R1 * 0
    if form == "zero_alpha":
        alpha = [a * 0 for a in alpha]
    if form == "huge_alpha":
        alpha = [a * 1e150 for a in alpha]
    if form == "column":
        alpha[0][:, 2] *= 1e12
    got = lz.get_perturb_averages_q(R1, alpha, True)
    monkeypatch.setenv("TDSCHA_FP64_DIGITS", "0")
    lz._invalidate()
    ref = lz.get_perturb_averages_q(R1, alpha, True)
    _check(got, ref)


@pytest.mark.parametrize("where", ["R1", "alpha"])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_non_finite(gpu_lib, monkeypatch, where, value):
    """What a non-finite perturbation reaches is not finite, as with the CUDA cores."""
    import torch
    _, lz, _, R1, alpha = _setup((3, 1, 1), 5, 150, 1)
    a = np.stack(alpha)
    if where == "R1":
        R1[2] = value
    else:
        a[1, 0, 3] = value
    out = []
    for cores in (False, True):
        if cores:
            monkeypatch.setenv("TDSCHA_FP64_DIGITS", "0")
            lz._invalidate()
        ctx = lz._qcontext()
        dev = [torch.tensor(v, device="cuda") for v in (R1, a)]
        f = torch.empty(R1.size, dtype=torch.complex128, device="cuda")
        d2v = torch.empty(a.shape, dtype=torch.complex128, device="cuda")
        st = torch.cuda.current_stream().cuda_stream
        nat.check(nat.load().tdscha_qperturb_averages(ctx.handle, dev[0].data_ptr(),
                                                      dev[1].data_ptr(), 1, f.data_ptr(),
                                                      d2v.data_ptr(), 1, st))
        out.append((np.isfinite(f.cpu().numpy()), np.isfinite(d2v.cpu().numpy())))
    assert not out[1][1].any()
    for x, y in zip(*out):
        assert (x == y).all()


def test_precision_and_perturbation_change(gpu_lib):
    """One context through both precisions and several perturbations."""
    e, lz, o, R1, alpha = _setup((2, 2, 1), 4, 150, 0)
    first = lz.get_perturb_averages_q(R1, alpha, True)
    lz.precision = "mixed"
    lz.get_perturb_averages_q(R1, alpha, True)
    lz.build_q_pair_map(3)
    lz.get_perturb_averages_q(R1, [alpha[0]] * len(lz.unique_pairs), True)
    lz.precision = "fp64"
    lz.get_perturb_averages_q(R1, [alpha[0]] * len(lz.unique_pairs), True)
    lz.build_q_pair_map(0)
    again = lz.get_perturb_averages_q(R1, alpha, True)
    assert (first[0] == again[0]).all()
    assert all((x == y).all() for x, y in zip(first[1], again[1]))


@pytest.mark.parametrize("dims,nb,N", [((1, 1, 1), 1, 40), ((2, 1, 1), 7, 60), ((2, 2, 1), 8, 60),
                                       ((4, 2, 2), 22, 30), ((4, 2, 2), 23, 30)])
@pytest.mark.parametrize("reorth", [False, True])
def test_lanczos_vector_lengths(gpu_lib, dims, nb, N, reorth):
    """The step in one launch (csrc/lanczos.cu, up to 16384 elements) and in several, on
    both sides of its limit: the coefficients of the oracle up to a near-breakdown, to
    1e-8: 1e-12 of an average, magnified by at most 1e4 = max|b| / b of the steps kept."""
    _, lz, o, _, _ = _setup(dims, nb, N)
    assert (2 * lz.get_psi_size() > 16384) == (nb == 23)
    lz.prepare_mode_q(0, nb - 1)
    o.psi[nb - 1] = 1.0
    lz.run_FT(5, verbose=False, reorthogonalize=reorth)
    o.run_FT(5, reorthogonalize=reorth)
    b = np.abs(np.array(o.b_coeffs))
    small = np.where(b < 1e-4 * b.max())[0] if len(b) else []
    k = int(small[0]) + 1 if len(small) else len(b)
    assert k >= min(5, len(o.b_coeffs)) - (nb == 1) * 4
    for name in ("a_coeffs", "b_coeffs", "c_coeffs"):
        np.testing.assert_allclose(getattr(lz, name)[:k], getattr(o, name)[:k], rtol=1e-8, atol=1e-14)
