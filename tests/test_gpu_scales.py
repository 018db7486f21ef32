"""Accuracy of the digit products on data whose parts differ in size: rows of two
sublattices, and configurations that the weights take out or nearly so.

The reference is numpy's long double (64 or 113 bits) on the same inputs, and errors are
measured against the part in question, not against the largest part."""
import numpy as np
import pytest

import oracle
from tdscha_gb300 import _native as nat
from tdscha_gb300.synthetic import make_ensemble, random_R1, random_sym

pytestmark = pytest.mark.gpu

LD = np.longdouble


@pytest.mark.parametrize("ratio", [1.0, 1e2, 1e4, 1e8])
def test_projection_of_two_sublattices(gpu_lib, ratio):
    """Light atoms with forces `ratio` times larger, modes on one sublattice each.  An
    element carries three roundings before the product (scale, mean, mass) and one after:
    4 2^-53 sum|a b| <= 4 2^-53 sqrt(n) rms(a) = 3.4e-15 rms(a) for n = 60; the entries of
    a column are normal with about that rms, the largest of 300 x 60 above 3 times it.
    2e-15 of the largest entry of a sublattice's modes, for either sublattice."""
    from tdscha_gb300.preprocessing import project_modes
    rng = np.random.default_rng(8)
    N, n = 300, 60
    light = np.arange(2 * n) // 3 % 2 == 0               # every other atom
    masses = np.where(light, 1.0, 200.0) * 911.444
    u = rng.standard_normal((N, 2 * n)) / np.sqrt(masses)
    f = rng.standard_normal((N, 2 * n)) * np.where(light, ratio, 1.0)
    u[:, light] *= ratio
    pols = np.zeros((2 * n, 2 * n))
    pols[np.ix_(light, np.arange(n))] = np.linalg.qr(rng.standard_normal((n, n)))[0]
    pols[np.ix_(~light, n + np.arange(n))] = np.linalg.qr(rng.standard_normal((n, n)))[0]
    X, Y = project_modes(u, f, masses, pols, f.mean(0), u_scale=0.5, f_scale=2.0)
    root, p = np.sqrt(masses).astype(LD), pols.astype(LD)
    f_mean = f.mean(0).astype(LD)
    for got, a in ((X, u.astype(LD) * LD(0.5) * root), (Y, (f.astype(LD) * 2 - f_mean * 2) / root)):
        ref = a @ p
        for part in (slice(0, n), slice(n, 2 * n)):
            assert np.abs(got[:, part] - ref[:, part]).max() <= 2e-15 * np.abs(ref[:, part]).max()


@pytest.mark.parametrize("what", ["row", "element", "noise", "zeros"])
def test_projection_of_outliers_and_noise(gpu_lib, what):
    """One configuration, or one element of it, 1e6 times the others: each of the others
    keeps its accuracy; coordinates of rounding noise over 40 decades, and of zeros beside
    small numbers: all do.  2e-15 of the largest entry of X, Y in ordinary configurations,
    as above."""
    from tdscha_gb300.preprocessing import project_modes
    rng = np.random.default_rng(9)
    N, n, M = 2000, 60, 57
    u, f = rng.standard_normal((N, n)), rng.standard_normal((N, n))
    masses = rng.uniform(1.0, 10.0, n)
    pols = np.linalg.qr(rng.standard_normal((n, n)))[0][:, :M]
    ordinary = np.ones(N, dtype=bool)
    for a in (u, f):
        if what == "noise":
            a[:, 6:9] *= 10.0 ** rng.uniform(-57, -17, (N, 3))
        elif what == "zeros":
            a *= 2.0 ** -40
            a[:, 6:9] = 0
        else:
            a[37, slice(None) if what == "row" else 5] *= 1e6
            ordinary[37] = False
    X, Y = project_modes(u, f, masses, pols, None, u_scale=0.5, f_scale=2.0)
    root, p = np.sqrt(masses).astype(LD), pols.astype(LD)
    for got, a in ((X, u.astype(LD) * LD(0.5) * root), (Y, f.astype(LD) * 2 / root)):
        ref = a @ p
        assert np.abs(got - ref)[ordinary].max() <= 2e-15 * np.abs(ref[ordinary]).max()
        assert np.abs(got - ref)[37].max() <= 2e-15 * np.abs(ref[37]).max()


def _outlier(a, what, size):
    a = a.copy()
    if what == "row":
        a[37] *= size
    elif what == "element":
        a[37, 5] *= size
    return a


@pytest.mark.parametrize("S", [1, 48])
@pytest.mark.parametrize("x,y", [("row", "row"), ("row", ""), ("", "row"), ("element", "element"),
                                 ("element", ""), ("", "element")])
@pytest.mark.parametrize("weight,size", [(0.0, 1e3), (0.0, 1e6), (0.0, 1e8), (1e-40, 1e6),
                                         (1e-24, 1e6), (1e-12, 1e3)])
def test_outlier_of_little_weight(gpu_lib, x, y, weight, size, S):
    """One configuration far out in displacements, forces or one of their elements, with a
    weight of zero, one that makes it vanish, or one that leaves it a part in the sums.  The
    oracle adds up N S <= 2e4 float64 terms: 5e-13 of the largest entry (as for ordinary
    ensembles, tests/test_gpu_digits.py)."""
    M, N = (63, 2000) if S == 1 else (24, 400)
    ens = make_ensemble(M, N, seed=12, n_syms=S, rho_sigma=0.1)
    tables = ((ens["symmetries"], ens["degenerate_space"], ens["sym_block_id"]) if S > 1
              else oracle.identity_symmetries(M))
    X, Y, rho = _outlier(ens["X"], x, size), _outlier(ens["Y"], y, size), ens["rho"].copy()
    rho[37] = weight
    R1, Y1 = random_R1(M, 3), random_sym(M, 4, scale=1e-5)
    ref = oracle.perturb_averages(X, Y, ens["w"], rho, R1, Y1, ens["T"], 1, *tables, n_threads=8)
    ctx = nat.Context(X, Y, ens["w"], rho, ens["T"], *tables)
    f, d2v = np.zeros(M), np.zeros((M, M))
    nat.check(nat.load().tdscha_perturb_averages(ctx.handle, nat.dp(R1), nat.dp(Y1), 1, nat.PREC_FP64,
                                                 nat.dp(f), nat.dp(d2v), 0, None))
    ctx.close()
    for a, b in zip((f, d2v), ref):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


@pytest.mark.parametrize("S", [1, 48])
@pytest.mark.parametrize("x,y", [(True, False), (False, True), (True, True)])
def test_mode_of_noise(gpu_lib, x, y, S):
    """Modes that symmetry holds at zero, up to rounding noise over 40 decades: the others
    keep their accuracy.  Tolerance as above."""
    M, N = (63, 2000) if S == 1 else (24, 400)
    ens = make_ensemble(M, N, seed=13, n_syms=S, rho_sigma=0.1)
    tables = ((ens["symmetries"], ens["degenerate_space"], ens["sym_block_id"]) if S > 1
              else oracle.identity_symmetries(M))
    rng = np.random.default_rng(2)
    X, Y = ens["X"].copy(), ens["Y"].copy()
    for a, on in ((X, x), (Y, y)):
        if on:
            a[:, 3:6] = rng.standard_normal((N, 3)) * 10.0 ** rng.uniform(-57, -17, (N, 3))
    R1, Y1 = random_R1(M, 3), random_sym(M, 4, scale=1e-5)
    ref = oracle.perturb_averages(X, Y, ens["w"], ens["rho"], R1, Y1, ens["T"], 1, *tables, n_threads=8)
    ctx = nat.Context(X, Y, ens["w"], ens["rho"], ens["T"], *tables)
    f, d2v = np.zeros(M), np.zeros((M, M))
    nat.check(nat.load().tdscha_perturb_averages(ctx.handle, nat.dp(R1), nat.dp(Y1), 1, nat.PREC_FP64,
                                                 nat.dp(f), nat.dp(d2v), 0, None))
    ctx.close()
    for a, b in zip((f, d2v), ref):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


@pytest.mark.parametrize("S", [1, 48])
@pytest.mark.parametrize("x,y", [(True, False), (False, True)])
@pytest.mark.parametrize("scale", [2.0 ** -40, 2.0 ** 40])
def test_mode_of_zeros(gpu_lib, x, y, scale, S):
    """Modes without displacements, or without forces, in ensembles of small and of large
    numbers (multiplied by a power of two).  Tolerance as above."""
    M, N = (63, 2000) if S == 1 else (24, 400)
    ens = make_ensemble(M, N, seed=14, n_syms=S, rho_sigma=0.1)
    tables = ((ens["symmetries"], ens["degenerate_space"], ens["sym_block_id"]) if S > 1
              else oracle.identity_symmetries(M))
    X, Y = scale * ens["X"], scale * ens["Y"]
    if x:
        X[:, 3:6] = 0
    if y:
        Y[:, 3:6] = 0
    R1, Y1 = random_R1(M, 3), random_sym(M, 4, scale=1e-5)
    ref = oracle.perturb_averages(X, Y, ens["w"], ens["rho"], R1, Y1, ens["T"], 1, *tables, n_threads=8)
    ctx = nat.Context(X, Y, ens["w"], ens["rho"], ens["T"], *tables)
    f, d2v = np.zeros(M), np.zeros((M, M))
    nat.check(nat.load().tdscha_perturb_averages(ctx.handle, nat.dp(R1), nat.dp(Y1), 1, nat.PREC_FP64,
                                                 nat.dp(f), nat.dp(d2v), 0, None))
    ctx.close()
    for a, b in ((f, ref[0]), (d2v, ref[1]), (d2v[3:6], ref[1][3:6])):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


def _bloch_averages(e, rho, iq):
    """f and the blocks of d2v, from the GPU and from the oracle."""
    import oracle.qspace as oq
    from tdscha_gb300.QSpaceLanczos import QSpaceLanczos
    nb = e["X_q"].shape[2]
    lz = QSpaceLanczos.from_arrays(e["X_q"], e["Y_q"], e["w_q"], rho, e["T"], q_points=e["q"])
    valid = np.ones((nb, 3), dtype=bool)
    valid[0, 0] = False
    lz.valid_modes_q = valid
    lz.prepare_symmetrization(symmetries=None)
    lz.build_q_pair_map(iq)
    o = oq.OracleQSpaceLanczos(e["X_q"], e["Y_q"], e["w_q"], rho, e["T"], lz.q_pair_map, iq, valid=valid)
    rng = np.random.default_rng(3)
    R1 = rng.standard_normal(nb) + 1j * rng.standard_normal(nb)
    alpha = [rng.standard_normal((nb, nb)) + 1j * rng.standard_normal((nb, nb)) for _ in o.pairs]
    got = lz.get_perturb_averages_q(R1, alpha, True)
    ref = oq.perturb_averages_qspace(e["X_q"], e["Y_q"], e["w_q"], rho, R1, alpha, e["T"], True, iq,
                                     o.pairs, o.symmetries, o.valid)
    return [(got[0], ref[0]), *zip(got[1], ref[1])]


@pytest.mark.parametrize("what", ["X", "Y", "XY", "X element", "Y element", "XY element"])
@pytest.mark.parametrize("weight,size", [(0.0, 1e3), (0.0, 1e6), (0.0, 1e8), (1e-40, 1e6),
                                         (1e-24, 1e6), (1e-12, 1e3), (1.0, 1e3), (1.0, 1e6)])
@pytest.mark.parametrize("nb", [5, 20])
def test_bloch_space_outlier(gpu_lib, what, weight, size, nb):
    """The same in Bloch space, against the oracle: N <= 300 float64 terms, 1e-13 of the
    largest entry of a block (tests/test_gpu_qspace_digits.py); an element of one q-point
    takes nothing from the blocks of the others."""
    from tdscha_gb300.synthetic import make_qspace_ensemble
    e = make_qspace_ensemble((3, 1, 1), nb, 300, seed=nb, T=250.0, dispersion=0.3, rho_sigma=0.2)
    at = (1, 37, 3) if "element" in what else (slice(None), 37)
    for k in "XY":
        if k in what.split()[0]:
            e[k + "_q"] = e[k + "_q"].copy()
            e[k + "_q"][at] *= size
    rho = e["rho"].copy()
    rho[37] *= weight
    for a, b in _bloch_averages(e, rho, 1):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


@pytest.mark.parametrize("what", ["real", "noise"])
@pytest.mark.parametrize("scale", [2.0 ** -40, 1.0, 2.0 ** 40])
@pytest.mark.parametrize("iq", [0, 1])
def test_bloch_space_at_gamma(gpu_lib, what, scale, iq):
    """Imaginary parts at Gamma that are zero, or rounding noise over 40 decades, in
    ensembles of small and of large numbers.  Tolerance as above."""
    from tdscha_gb300.synthetic import make_qspace_ensemble
    e = make_qspace_ensemble((3, 1, 1), 5, 300, seed=3, T=250.0, dispersion=0.3, rho_sigma=0.2)
    rng = np.random.default_rng(4)
    for k in ("X_q", "Y_q"):
        e[k] = scale * e[k]
        re = e[k][0].real
        e[k][0] = re + (1j * re * 10.0 ** rng.uniform(-57, -17, re.shape) if what == "noise" else 0)
    for a, b in _bloch_averages(e, e["rho"], iq):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
