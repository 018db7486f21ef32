"""What a user of this framework has it compute, as cases that can be timed.

The Lanczos linear response spends its time in the ensemble-averaged D3/D4
operator; around it stand the Krylov recurrence, the static (free-energy
Hessian) form, the Bloch-space form and the mode projection of a new ensemble.
Every case below is one of these through its public entry point, in the
precision that it is used in: float64, which is the default of every class, or
the mixed tensor-core path of long runs.

Ensembles are the seeded synthetic ones of tdscha_gb300/synthetic.py, drawn
on the GPU: Gaussian displacements with the covariance of their modes, cubic
and quartic forces in symmetric CP form, log-normal weights.
"""
import ctypes
import itertools
import math
import os

import numpy as np
import torch

# The tuner of the tensor-core path times its candidates, so two processes may
# settle on kernels that add in another order.  A user who needs the same bits
# from every process fixes the rule-based shape, as these cases do.
os.environ.setdefault("TDSCHA_AUTOTUNE", "0")

from tdscha_gb300 import _native as nat  # noqa: E402
from tdscha_gb300 import preprocessing  # noqa: E402
from tdscha_gb300.DynamicalLanczos import Lanczos  # noqa: E402

RY_TO_K = 157887.32400374097
RY_TO_CM = 109691.40235
CUDA = torch.device("cuda")
F64 = torch.float64

# one application at the largest ensemble: configurations x images x modes^2
MOST_WORK = 50000 * 573 ** 2


def listed():
    return [
        # the averages of a two-atom cell with a small ensemble: what a first
        # trial or a test runs, a matter of launches
        dict(name="averages fp64 m21 n1k", kind="averages", M=21, N=1000, S=1, T=300.0,
             precision="fp64"),
        # L^T of the non-symmetric recurrence on a middling, ragged ensemble
        dict(name="apply fp64 m97 n4999 Lt", kind="apply", M=97, N=4999, S=1, T=120.0,
             precision="fp64", wigner=False, transpose=True),
        # the headline ensemble (192-atom supercell) in the default precision
        dict(name="averages fp64 m573 n50k", kind="averages", M=573, N=50000, S=1, T=300.0,
             precision="fp64"),
        # a cubic crystal with its 48 images in the default precision
        dict(name="averages fp64 m189 n10k s48", kind="averages", M=189, N=10000, S=48, T=300.0,
             precision="fp64"),
        # the default run of the reference: symmetric Lanczos in the Wigner
        # representation, float64, through the class
        dict(name="run_FT fp64 wigner m48 n2k", kind="run_FT", M=48, N=2000, S=1, T=300.0,
             precision="fp64", wigner=True, steps=16),
        # a complete short bi-Lanczos run and its Green function through the
        # class on a small ensemble: launches and host work
        dict(name="run_FT mixed m21 n1k", kind="run_FT", M=21, N=1000, S=1, T=300.0,
             precision="mixed", wigner=False, steps=24),
        # the headline run: bi-Lanczos with re-biorthogonalisation, mixed
        dict(name="lanczos mixed m573 n50k", kind="lanczos", M=573, N=50000, S=1, T=300.0,
             precision="mixed", wigner=False, steps=12),
        # the same on the symmetric crystal
        dict(name="lanczos mixed m189 n10k s48", kind="lanczos", M=189, N=10000, S=48, T=300.0,
             precision="mixed", wigner=False, steps=6),
        # the anharmonic part of the free-energy Hessian's matvec: a batch of
        # static vectors
        dict(name="static fp64 m60 n5k", kind="static", M=60, N=5000, S=1, T=300.0,
             precision="fp64", nvec=24),
        # Hermitian Lanczos of a 2x2x2 supercell in Bloch space
        dict(name="q lanczos fp64 222 nb6 n2k", kind="qlanczos", d1=2, d2=2, d3=2, nb=6, N=2000,
             iq=0, T=300.0, precision="fp64", steps=12),
        # the Bloch-space averages of a 4x4x4 supercell of a four-atom cell
        dict(name="q averages fp64 444 nb12 n10k", kind="qaverages", d1=4, d2=4, d3=4, nb=12, N=10000,
             iq=0, T=300.0, precision="fp64"),
        # a new ensemble from Cartesian displacements and forces on the host
        dict(name="project n10k 576 to 573", kind="project", n_cart=576, M=573, N=10000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["averages", "averages", "averages", "apply", "apply", "lanczos", "lanczos",
                       "run_FT", "static", "qaverages", "qlanczos", "project"])
    if kind in ("qaverages", "qlanczos"):
        while True:
            dims = [rng.randint(1, 4) for _ in range(3)]
            nb, N = rng.randint(3, 12), _log(rng, 200, 10000)
            n_q = dims[0] * dims[1] * dims[2]
            steps = rng.randint(4, 12)
            runs = steps if kind == "qlanczos" else 1
            if n_q >= 2 and n_q * nb >= 12 and runs * N * n_q * nb * nb <= 10000 * 64 * 144:
                break
        c = dict(kind=kind, d1=dims[0], d2=dims[1], d3=dims[2], nb=nb, N=N, iq=rng.randrange(n_q),
                 T=float(rng.choice([0, 100, 300, 600])),
                 precision=rng.choice(["fp64", "fp64", "mixed"]))
        if kind == "qlanczos":
            c["steps"] = steps
        return c
    if kind == "project":
        M = _log(rng, 12, 573)
        return dict(kind=kind, n_cart=3 * -(-M // 3) + 3, M=M, N=_log(rng, 200, 10000))
    while True:
        S = rng.choice([1, 1, 1, 8, 24, 48]) if kind in ("averages", "apply", "lanczos") else 1
        M = _log(rng, 12, 573)
        M += -M % 3 if S > 1 else 0
        N = _log(rng, 300, 50000)
        c = dict(kind=kind, M=M, N=N, S=S, T=float(rng.choice([0, 120, 300, 700])),
                 precision=rng.choice(["fp64", "mixed"] if kind != "static" else ["fp64"]))
        runs = 1
        if kind in ("apply", "lanczos", "run_FT"):
            c["wigner"] = rng.random() < 0.5
        if kind == "apply":
            c["transpose"] = not c["wigner"] and rng.random() < 0.5
        if kind in ("lanczos", "run_FT"):
            c["steps"] = rng.randint(3, 6) if S > 1 else rng.randint(4, 16)
            runs = c["steps"] * (1 if c["wigner"] else 2)
        if kind == "static":
            c["nvec"] = runs = rng.randint(2, 32)
        # float64 rates are far below the tensor cores': a mixed run may do more
        if runs * N * S * M * M <= MOST_WORK * (12 if c["precision"] == "mixed" and S == 1 else 1):
            return c


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=CUDA)
    g.manual_seed(seed)
    return g


def _bose(w, T):
    return 1.0 / torch.expm1(w * RY_TO_K / T) if T > 0 else torch.zeros_like(w)


def _f_ups(w, T):
    return 2 * w / (1 + 2 * _bose(w, T))


def _f_psi(w, T):
    return (1 + 2 * _bose(w, T)) / (2 * w)


def _forces(x, scale, g):
    """-1/2 Phi3 xx - 1/6 Phi4 xxx of random symmetric CP tensors, each of the given rms."""
    M = x.shape[1]
    rank = max(8, min(M, 64))
    out = torch.zeros_like(x)
    for order, fact in ((3, 2.0), (4, 6.0)):
        G = torch.randn(rank, M, generator=g, device=CUDA, dtype=F64) / math.sqrt(M)
        c = torch.randn(rank, generator=g, device=CUDA, dtype=F64)
        f = -(((x @ G.T) ** (order - 1)) * c) @ G / fact
        out += f * (scale / f.square().mean().sqrt())
    return out


def _oh_group():
    mats = []
    for perm in itertools.permutations(range(3)):
        for signs in itertools.product((1.0, -1.0), repeat=3):
            m = np.zeros((3, 3))
            for r, c in enumerate(perm):
                m[r, c] = signs[r]
            mats.append(m)
    return np.array(mats)


def _ensemble(case, seed):
    """X, Y, w, rho on the GPU and the symmetry tables (lists as the classes take them)."""
    M, N, S, T = case["M"], case["N"], case["S"], case["T"]
    g = _gen(seed)
    nblock = M // 3 if S > 1 else M
    w = torch.rand(nblock, generator=g, device=CUDA, dtype=F64) * 450 + 50
    w = torch.sort(w).values / RY_TO_CM
    w = w.repeat_interleave(M // nblock)
    X = torch.randn(N, M, generator=g, device=CUDA, dtype=F64) * _f_psi(w, T).sqrt()
    Y = _forces(X, 0.05 * (X * w ** 2).square().mean().sqrt(), g)
    rho = torch.exp(0.1 * torch.randn(N, generator=g, device=CUDA, dtype=F64))
    Y -= (rho[:, None] * Y).sum(0) / rho.sum()
    if S == 1:
        syms, spaces = [np.ones((1, 1, 1))] * M, [np.array([i], dtype=np.intc) for i in range(M)]
    else:
        group = _oh_group()
        order = np.random.default_rng(seed).permutation(np.arange(1, len(group)))[:S - 1]
        group = group[[0] + list(order)]
        pseudo = group * np.linalg.det(group)[:, None, None]
        syms = [np.ascontiguousarray(pseudo if b % 2 else group) for b in range(nblock)]
        spaces = [np.arange(3 * b, 3 * b + 3, dtype=np.intc) for b in range(nblock)]
    return X, Y, w, rho, syms, spaces


def _perturbation(case, seed):
    """A unit vector of the modes and a symmetric matrix of the pairs' size."""
    M = case["M"]
    g = _gen(seed + 1000003)
    R1 = torch.randn(M, generator=g, device=CUDA, dtype=F64)
    R1 /= R1.norm()
    Y1 = torch.randn(M, M, generator=g, device=CUDA, dtype=F64) * 1e-6
    return R1, (Y1 + Y1.T) / 2


def _psi(case, seed, size):
    """A vector in the middle of a run: every sector filled."""
    g = _gen(seed + 2000003)
    v = torch.randn(size, generator=g, device=CUDA, dtype=F64)
    return v / v.norm()


def _dims(case):
    return (case["d1"], case["d2"], case["d3"])


def _q_ensemble(case, seed):
    """X_q, Y_q (n_q, N, nb) complex, w_q (nb, n_q), rho of a supercell's real ensemble."""
    dims, nb, N, T = _dims(case), case["nb"], case["N"], case["T"]
    n_q = dims[0] * dims[1] * dims[2]
    g = _gen(seed)
    wb = torch.sort(torch.rand(nb, generator=g, device=CUDA, dtype=F64) * 450 + 50).values / RY_TO_CM
    q = torch.tensor(list(itertools.product(*(np.arange(d) / d for d in dims))), dtype=F64,
                     device=CUDA)
    w_q = wb[:, None] * (1 + 0.15 * (1 - torch.cos(2 * math.pi * q).mean(1)))
    white = torch.randn(N, nb, *dims, generator=g, device=CUDA, dtype=F64)
    X = torch.fft.fftn(white, dim=(2, 3, 4), norm="ortho").reshape(N, nb, n_q)
    X = X * _f_psi(w_q, T).sqrt()
    real = torch.fft.ifftn(X.reshape(N, nb, *dims), dim=(2, 3, 4), norm="ortho").real
    real = real.reshape(N, nb * n_q)
    wr = wb.repeat_interleave(n_q)
    F = _forces(real, 0.05 * (real * wr ** 2).square().mean().sqrt(), g)
    rho = torch.exp(0.1 * torch.randn(N, generator=g, device=CUDA, dtype=F64))
    F -= (rho[:, None] * F).sum(0) / rho.sum()
    Y = torch.fft.fftn(F.reshape(N, nb, *dims), dim=(2, 3, 4), norm="ortho").reshape(N, nb, n_q)
    return X.permute(2, 0, 1).contiguous(), Y.permute(2, 0, 1).contiguous(), w_q, rho


def _q_pairs(case):
    """q2 = q_pert - q1 on the grid."""
    d = np.array(_dims(case))
    cells = np.array(list(itertools.product(*(range(k) for k in d))))
    index = {tuple(c): i for i, c in enumerate(cells)}
    return np.array([index[tuple((cells[case["iq"]] - c) % d)] for c in cells], dtype=np.int32)


def _q_layout(case):
    """(pairs, psi length) of the reference's layout [R | a' blocks | b' blocks]."""
    m, nb = _q_pairs(case), case["nb"]
    pairs = [(a, int(b)) for a, b in enumerate(m) if a <= b]
    size = [nb * nb if a < b else nb * (nb + 1) // 2 for a, b in pairs]
    return pairs, size, nb + 2 * sum(size)


def _q_mask(case):
    pairs, _, P = _q_layout(case)
    nb = case["nb"]
    tri = [1.0 if j == i else 2.0 for i in range(nb) for j in range(i, nb)]
    m = [1.0] * nb
    for _ in range(2):
        for a, b in pairs:
            m += [2.0] * (nb * nb) if a < b else tri
    return torch.tensor(m, dtype=F64, device=CUDA)


def _q_vector(case, seed):
    """A unit vector of the bands at the perturbation's q."""
    v = torch.randn(case["nb"], 2, generator=_gen(seed + 1000003), device=CUDA, dtype=F64)
    return torch.view_as_complex(v / v.norm())


def _q_start(case, seed):
    """psi of a one-phonon perturbation."""
    v = torch.zeros(_q_layout(case)[2], dtype=torch.complex128, device=CUDA)
    v[:case["nb"]] = _q_vector(case, seed)
    return v


def _q_blocks(case, seed):
    """alpha1 of every pair, Hermitian where a q is paired with itself."""
    nb, g = case["nb"], _gen(seed + 2000003)
    pairs = _q_layout(case)[0]
    a = torch.view_as_complex(torch.randn(len(pairs), nb, nb, 2, generator=g, device=CUDA,
                                          dtype=F64)) * 1e-6
    own = [p for p, (q1, q2) in enumerate(pairs) if q1 == q2]
    if own:
        a[own] = (a[own] + a[own].conj().transpose(1, 2)) / 2
    return a


def _cartesian(case, seed):
    g = _gen(seed)
    n, M, N = case["n_cart"], case["M"], case["N"]
    masses = torch.rand(n // 3, generator=g, device=CUDA, dtype=F64).repeat_interleave(3) * 2e5 + 1e3
    pols = torch.linalg.qr(torch.randn(n, M, generator=g, device=CUDA, dtype=F64)).Q
    u = torch.randn(N, n, generator=g, device=CUDA, dtype=F64) * 0.05
    f = torch.randn(N, n, generator=g, device=CUDA, dtype=F64) * 1e-3
    return u, f, masses, pols, f.mean(0)


# ------------------------------------------------------------ the program
def _context(case, ens):
    X, Y, w, rho, syms, spaces = ens
    bid = np.empty(case["M"], dtype=np.intc)
    for b, s in enumerate(spaces):
        bid[s] = b
    ctx = nat.Context(X.cpu().numpy(), Y.cpu().numpy(), w.cpu().numpy(), rho.cpu().numpy(),
                      case["T"], syms, spaces, bid,
                      with_mixed="fp32" if case["precision"] == "mixed" else False)
    ctx.set_options(case.get("wigner", True), False, False, False, False, 0.0)
    return ctx


def _prec(case):
    return nat.PREC_MIXED if case["precision"] == "mixed" else nat.PREC_FP64


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind, case=case)
    if kind == "project":
        s["host"] = [t.cpu().numpy() for t in _cartesian(case, seed)]
        return s
    if kind in ("qaverages", "qlanczos"):
        X, Y, w_q, rho = _q_ensemble(case, seed)
        ctx = nat.QContext(X.cpu().numpy(), Y.cpu().numpy(), w_q.cpu().numpy(), rho.cpu().numpy(),
                           case["T"])
        ctx.set_precision(case["precision"])
        ctx.set_pert(case["iq"], _q_pairs(case))
        s["ctx"] = ctx
        if kind == "qaverages":
            s["in"] = [torch.view_as_real(v).contiguous() for v in (_q_vector(case, seed),
                                                                    _q_blocks(case, seed))]
            s["out"] = [torch.empty_like(v) for v in s["in"]]
        else:
            s["psi"] = torch.view_as_real(_q_start(case, seed)).reshape(-1)
            cap = case["steps"] + 2
            s["Q"] = torch.zeros(cap, s["psi"].numel(), dtype=F64, device=CUDA)
            s["P"] = torch.zeros_like(s["Q"])
        return s
    ens = _ensemble(case, seed)
    R1, Y1 = _perturbation(case, seed)
    if kind == "run_FT":
        X, Y, w, rho, syms, spaces = ens
        lanc = Lanczos.from_arrays(X.cpu().numpy(), Y.cpu().numpy(), w.cpu().numpy(),
                                   rho.cpu().numpy(), case["T"], use_wigner=case["wigner"],
                                   precision=case["precision"])
        lanc.fp32_storage = case["precision"] == "mixed"
        lanc.init(use_symmetries=False)
        s["lanc"], s["vector"] = lanc, R1.cpu().numpy()
        s["grid"] = np.linspace(20, 600, 500) / RY_TO_CM
        lanc.get_perturb_averages(s["vector"], Y1.cpu().numpy())     # the ensemble resident from here on
        return s
    ctx = s["ctx"] = _context(case, ens)
    M = case["M"]
    if kind == "averages":
        s["in"] = (R1, Y1.contiguous())
        s["out"] = (torch.empty(M, dtype=F64, device=CUDA), torch.empty(M, M, dtype=F64, device=CUDA))
    elif kind == "apply":
        s["psi"] = _psi(case, seed, ctx.P)
        s["out"] = torch.empty_like(s["psi"])
    elif kind == "static":
        n = M + M * (M + 1) // 2
        s["psi"] = torch.stack([_psi(case, seed + 17 * v, n) for v in range(case["nvec"])])
        s["out"] = torch.empty_like(s["psi"])
    else:
        s["ld"] = ctx.basis_ld()
        ctx.set_basis_ld(s["ld"])
        s["Q"] = torch.zeros(case["steps"] + 2, s["ld"], dtype=F64, device=CUDA)
        s["P"] = torch.zeros_like(s["Q"])
        s["first"] = torch.zeros(ctx.P, dtype=F64, device=CUDA)
        s["first"][:M] = R1
    return s


def _krylov(s, first, call):
    """A run of `steps` steps from `first` into the caller's basis buffers."""
    n, size = s["case"]["steps"], first.numel()
    cap = n + 2
    s["Q"][0, :size].copy_(first)
    s["P"][0, :size].copy_(first)
    hist = np.zeros(4 * cap)
    hist[3] = 1.0
    done, conv = ctypes.c_int(0), ctypes.c_int(0)
    nat.check(call(s["Q"].data_ptr(), s["P"].data_ptr(), cap, n, nat.dp(hist), ctypes.byref(done),
                   ctypes.byref(conv), torch.cuda.current_stream().cuda_stream))
    h = hist.reshape(cap, 4)
    return dict(a=h[:n, 0].copy(), b=h[:n, 1].copy(), c=h[:n, 2].copy(), Q=s["Q"][:n + 1, :size],
                P=s["P"][:n + 1, :size])


def run(s):
    kind, case, lib = s["kind"], s["case"], nat.load()
    if kind == "project":
        return preprocessing.project_modes(*s["host"])
    if kind == "run_FT":
        lanc = s["lanc"]
        lanc.prepare_perturbation(s["vector"], masses_exp=0)
        lanc.run_FT(case["steps"], verbose=False, n_rep_orth=1)
        G = lanc.get_green_function_continued_fraction(s["grid"], smearing=10 / RY_TO_CM)
        return dict(a=np.array(lanc.a_coeffs), b=np.array(lanc.b_coeffs),
                    c=np.array(lanc.c_coeffs), G=G)
    st = torch.cuda.current_stream().cuda_stream
    if kind == "qaverages":
        (R1, alpha), (f, d2v) = s["in"], s["out"]
        nat.check(lib.tdscha_qperturb_averages(s["ctx"].handle, R1.data_ptr(), alpha.data_ptr(), 1,
                                               f.data_ptr(), d2v.data_ptr(), 1, st))
        return dict(f=f, d2v=d2v)
    if kind == "qlanczos":
        return _krylov(s, s["psi"], lambda Q, P, cap, n, h, d, c, st: lib.tdscha_qlanczos_run(
            s["ctx"].handle, Q, P, cap, 0, n, 1, h, d, c, st))
    h = s["ctx"].handle
    if kind == "averages":
        (R1, Y1), (f, d2v) = s["in"], s["out"]
        nat.check(lib.tdscha_perturb_averages(h, R1.data_ptr(), Y1.data_ptr(), 1, _prec(case),
                                              f.data_ptr(), d2v.data_ptr(), 1, st))
        return dict(f=f, d2v=d2v)
    if kind == "apply":
        nat.check(lib.tdscha_apply_full_L(h, s["psi"].data_ptr(), s["out"].data_ptr(),
                                          1 if case["transpose"] else 0, _prec(case), st))
        return s["out"]
    if kind == "static":
        nat.check(lib.tdscha_static_L(h, case["nvec"], s["psi"].data_ptr(), s["out"].data_ptr(), 2,
                                      1.0, _prec(case), st))
        return s["out"]
    return _krylov(s, s["first"], lambda Q, P, cap, n, hist, d, c, st: lib.tdscha_lanczos_run(
        h, Q, P, cap, 0, n, 1 if case["wigner"] else 0, _prec(case), 1, hist, d, c, st))


def work(case):
    kind = case["kind"]
    if kind == "project":
        n, M, N = case["n_cart"], case["M"], case["N"]
        return dict(bytes=8.0 * (2 * N * (n + M) + n * M), flops=4.0 * N * n * M)
    steps = case.get("steps", 1)
    if kind in ("qaverages", "qlanczos"):
        pairs, _, P = _q_layout(case)
        n_q, nb, N = _dims(case)[0] * _dims(case)[1] * _dims(case)[2], case["nb"], case["N"]
        item = 8 if case["precision"] == "mixed" else 16
        flops = N * (8.0 * n_q * nb * nb + 16.0 * n_q * nb + 16.0 * len(pairs) * nb * nb)
        sweeps = 2.0 * 16 * P * steps * (steps + 1) / 2 if kind == "qlanczos" else 0.0
        return dict(bytes=steps * (2.0 * N * n_q * nb * item + 32.0 * P) + sweeps, flops=steps * flops)
    M, N, S = case["M"], case["N"], case["S"]
    P = M + M * (M + 1)
    item = 4 if case["precision"] == "mixed" else 8
    calls = case.get("nvec", steps * (1 if case.get("wigner", True) else 2))
    if kind in ("averages", "apply"):
        calls = 1
    reads = 1 if kind == "static" else steps     # one reading serves the vectors of a step
    sweeps = 2.0 * 16 * P * steps * (steps + 1) / 2 if kind in ("lanczos", "run_FT") else 0.0
    return dict(bytes=reads * 2.0 * N * M * item + calls * 16.0 * M * M + sweeps,
                flops=calls * 4.0 * N * S * M * M)


# -------------------------------------------------- the same in 64 bits
def _images(X, syms, spaces, j):
    """The image S_j of every row; triplets of modes share a block."""
    if len(spaces) == X.shape[1]:
        return X
    G = torch.tensor(np.stack([b[j] for b in syms]), device=CUDA)
    return torch.einsum("bmn,ibn->ibm", G, X.reshape(X.shape[0], -1, 3)).reshape(X.shape)


def _exact_averages(case, ens, R1, Y1):
    X, Y, w, rho, syms, spaces = ens
    fY, fp, S = _f_ups(w, case["T"]), _f_psi(w, case["T"]), case["S"]
    f, G = torch.zeros_like(R1), torch.zeros_like(Y1)
    for j in range(S):
        x, y = (X, Y) if S == 1 else (_images(X, syms, spaces, j), _images(Y, syms, spaces, j))
        v, u = x @ Y1, x * fY
        q, p = (x * v).sum(1), ((y * fp) * v).sum(1)
        s, t = u @ R1, y @ R1
        f += -((rho * q / 6) @ y + (rho * p / 3) @ u)
        W = (rho * (s / 3 - q / 8))[:, None] * y + (rho * (t / 3 - p / 4) / 2)[:, None] * u
        G += u.T @ W
    norm = S * rho.sum()
    return f / norm, -(G + G.T) / norm


class _Exact:
    """L, L^T and the Wigner form on psi = [R | pairs | pairs]."""

    def __init__(self, case, ens):
        self.case, self.ens = case, ens
        w, T, M = ens[2], case["T"], case["M"]
        self.M, self.w = M, w
        self.i, self.j = torch.triu_indices(M, M, device=CUDA)
        self.h = len(self.i)
        n = _bose(w, T)
        self.Yw, self.Aw = 2 * w / (2 * n + 1), 2 * w * n * (n + 1) / (2 * n + 1)
        wa, wb, na, nb = w[self.j], w[self.i], n[self.j], n[self.i]
        self.wa, self.wb = wa, wb
        den = (2 * na + 1) * (2 * nb + 1)
        occ = 2 * na * nb + na + nb
        self.X = wa ** 2 + wb ** 2 + 2 * wa * wb / den
        self.Y = 8 * wa * wb / den
        self.X1 = occ * (occ + 1) * 2 * wa * wb / den
        self.Y1 = wa ** 2 + wb ** 2 - 2 * wa * wb / den
        self.cm = (-0.5 * (wa - wb) * (na - nb) / (2 * wa * wb)).clamp_min(0).sqrt()
        self.cp = (0.5 * (wa + wb) * (1 + na + nb) / (2 * wa * wb)).sqrt()
        self.wx = wa * wb * 8 / den
        self.mask = torch.ones(M + 2 * self.h, dtype=F64, device=CUDA)
        self.mask[M:] += (self.i != self.j).to(F64).repeat(2)

    def full(self, v):
        A = torch.zeros(self.M, self.M, dtype=F64, device=CUDA)
        A[self.i, self.j] = v
        A[self.j, self.i] = v
        return A

    def __call__(self, psi, transpose=False):
        M, h, i, j = self.M, self.h, self.i, self.j
        R, a, b = psi[:M], psi[M:M + h], psi[M + h:]
        if self.case["wigner"]:
            Y1 = self.full(self.wx * (self.cm * a - self.cp * b))
            f, d2v = _exact_averages(self.case, self.ens, R, Y1)
            d = d2v[i, j]
            return torch.cat([-R * self.w ** 2 + f, -(self.wa - self.wb) ** 2 * a + self.cm * d,
                              -(self.wa + self.wb) ** 2 * b - self.cp * d])
        Yw, Aw = self.Yw, self.Aw
        if transpose:
            half = torch.where(i == j, 1.0, 0.5)
            cY = 2 * Yw[i] * Yw[j] * (Yw[i] + Yw[j])
            cA = 2 * Yw[i] * Yw[j] * (Aw[i] + Aw[j])
            Y1 = self.full(half * (a * cY + b * cA))
            ha, hb = self.X * a + self.X1 * b, self.Y * a + self.Y1 * b
        else:
            Y1 = self.full(a)
            ha, hb = self.X * a + self.Y * b, self.X1 * a + self.Y1 * b
        f, d2v = _exact_averages(self.case, self.ens, R, Y1)
        d = d2v[i, j]
        if transpose:
            return torch.cat([R * self.w ** 2 - f, ha - d / (2 * half * Yw[i] * Yw[j]), hb])
        return torch.cat([R * self.w ** 2 - f, ha - d * (Yw[i] + Yw[j]), hb - d * (Aw[i] + Aw[j])])


def _exact_krylov(op, first, mask, symmetric, steps, hermitian=False):
    """The recurrence with one pass of re-biorthogonalisation against every stored pair."""
    dot = lambda x, y: torch.real((x.conj() * y * mask).sum())  # noqa: E731
    Q, P, sn, al, be, ce = [first], [first], [1.0], [], [], []
    for k in range(steps):
        q, p = Q[-1], P[-1]
        Lq = op(q, False)
        pL = Lq if symmetric else op(p, True)
        pn = sn[-1] / (ce[-1] if ce else 1.0)
        a = dot(p, Lq) * pn
        r, s = Lq - a * q, pL - a * p
        if k:
            r = r - ce[-1] * Q[-2]
            old = sn[-2] / ce[-2] if len(ce) > 1 else sn[-2]
            s = s - be[-1] * (old / pn) * P[-2]
        raw, b = dot(s, s).sqrt(), dot(r, r).sqrt()
        c = dot(s / raw, r / b) * raw * pn
        q, p = r / b, s / raw
        if hermitian:
            q = q - sum(dot(x, q) * x for x in Q)
            q = q / dot(q, q).sqrt()
            p = q
        else:
            pq = [dot(y, x) for x, y in zip(Q, P)]
            q, p = (q - sum(dot(y, q) / t * x for x, y, t in zip(Q, P, pq)),
                    p - sum(dot(x, p) / t * y for x, y, t in zip(Q, P, pq)))
        al, be, ce = al + [a], be + [b], ce + [c]
        Q, P, sn = Q + [q], P + [p], sn + [c if hermitian else raw * pn]
    return al, be, ce, Q, P


def _exact_fraction(a, b, c, grid, smearing, wigner, modulus):
    w2, sgn = grid ** 2, (1.0 if wigner else -1.0)
    d = a[-1] + sgn * w2
    root = np.sqrt(d ** 2 - 4 * b[-1] * c[-1] + 0j)
    up, dn = (d + root) / (2 * b[-1] * c[-1]), (d - root) / (2 * b[-1] * c[-1])
    G = np.where(np.abs(up) < np.abs(dn), up, dn)
    for k in range(len(a) - 2, -1, -1):
        G = 1 / (a[k] + sgn * w2 + 2j * grid * smearing - b[k] * c[k] * G)
    return (-G.real + 1j * G.imag if wigner else G) * modulus


def _exact_static(case, ens, psi):
    op, M = _Exact(dict(case, wigner=False), ens), case["M"]
    out = []
    for v in psi:
        Y1 = -2 * op.full(v[M:]) * op.Yw[:, None] * op.Yw[None, :]
        f, d2v = _exact_averages(case, ens, v[:M], Y1)
        out.append(torch.cat([-f, d2v[op.i, op.j]]))
    return torch.stack(out)


class _ExactQ:
    """The Wigner operator in Bloch space."""

    def __init__(self, case, ens):
        self.case, self.ens = case, ens
        self.pairs, self.size, self.P = _q_layout(case)
        nb = case["nb"]
        self.iu = torch.triu_indices(nb, nb, device=CUDA)

    def blocks(self, v):
        nb, out, off = self.case["nb"], [], 0
        for (a, b), s in zip(self.pairs, self.size):
            raw = v[off:off + s]
            if a < b:
                m = raw.reshape(nb, nb)
            else:
                m = torch.zeros(nb, nb, dtype=v.dtype, device=CUDA)
                m[self.iu[1], self.iu[0]] = raw.conj()
                m[self.iu[0], self.iu[1]] = raw
            out.append(m)
            off += s
        return out

    def pack(self, mats):
        return torch.cat([m.reshape(-1) if a < b else m[self.iu[0], self.iu[1]]
                          for (a, b), m in zip(self.pairs, mats)])

    def averages(self, R, alpha):
        case, (X, Y, w_q, rho) = self.case, self.ens
        fY, fp, iq = _f_ups(w_q, case["T"]), _f_psi(w_q, case["T"]), case["iq"]
        u, tot = torch.zeros_like(X), torch.zeros_like(X[0, :, 0])
        for (a, b), al in zip(self.pairs, alpha):
            u[a] += X[b] @ al.T
            if a != b:
                u[b] += X[a] @ al.conj()
            lw = (X[a].conj() * (X[b] @ al.T)).sum(1)
            tot += lw + lw.conj() if a < b else lw
        bfw = sum((u[q].conj() * (Y[q] * fp[:, q])).sum(1) for q in range(X.shape[0]))
        xp, yp = X[iq] * fY[:, iq], Y[iq]
        cross = rho * ((xp @ R.conj()) / 3 - tot / 8)
        diag = rho * ((yp @ R.conj()) / 3 - bfw / 4)
        f = -((rho * tot / 6) @ yp + (rho * bfw / 3) @ xp) / rho.sum()
        d2v = []
        for a, b in self.pairs:
            u1, u2, f1, f2 = X[a] * fY[:, a], X[b] * fY[:, b], Y[a], Y[b]
            d2v.append(-((cross[:, None] * u1).T @ f2.conj()
                         + (cross[:, None] * f1 + diag[:, None] * u1).T @ u2.conj()) / rho.sum())
        return f, d2v

    def __call__(self, psi, transpose=False):
        case, w_q = self.case, self.ens[2]
        nb, iq, n, half = case["nb"], case["iq"], _bose(w_q, case["T"]), sum(self.size)
        R, A, B = psi[:nb], self.blocks(psi[nb:nb + half]), self.blocks(psi[nb + half:])
        alpha, fac = [], []
        for (a, b), ma, mb in zip(self.pairs, A, B):
            w1, w2, n1, n2 = w_q[:, a, None], w_q[None, :, b], n[:, a, None], n[None, :, b]
            cm = (-0.5 * (w1 - w2) * (n1 - n2) / (2 * w1 * w2)).clamp_min(0).sqrt()
            cp = (0.5 * (w1 + w2) * (1 + n1 + n2) / (2 * w1 * w2)).sqrt()
            fac.append((w1, w2, cm, cp))
            alpha.append(8 * w1 * w2 / ((1 + 2 * n1) * (1 + 2 * n2)) * (cm * ma - cp * mb))
        f, d2v = self.averages(R, alpha)
        oa = [-(w1 - w2) ** 2 * m + cm * d for (w1, w2, cm, _), m, d in zip(fac, A, d2v)]
        ob = [-(w1 + w2) ** 2 * m - cp * d for (w1, w2, _, cp), m, d in zip(fac, B, d2v)]
        return torch.cat([-w_q[:, iq] ** 2 * R + f, self.pack(oa), self.pack(ob)])


def _stack(values):
    return np.array([float(v) for v in values])


def _real(v):
    return torch.view_as_real(v).reshape(-1) if v.is_complex() else v


def exact(case, seed):
    kind = case["kind"]
    if kind == "project":
        u, f, masses, pols, mean = _cartesian(case, seed)
        bohr = preprocessing.BOHR
        return ((u / bohr * masses.sqrt()) @ pols).cpu().numpy(), \
            (((f - mean) * bohr / masses.sqrt()) @ pols).cpu().numpy()
    if kind in ("qaverages", "qlanczos"):
        op = _ExactQ(case, _q_ensemble(case, seed))
        if kind == "qaverages":
            f, d2v = op.averages(_q_vector(case, seed), _q_blocks(case, seed))
            return dict(f=torch.view_as_real(f), d2v=torch.view_as_real(torch.stack(d2v)))
        a, b, c, Q, P = _exact_krylov(op, _q_start(case, seed), _q_mask(case), True, case["steps"], hermitian=True)
        return dict(a=_stack(a), b=_stack(b), c=_stack(c), Q=torch.stack([_real(v) for v in Q]),
                    P=torch.stack([_real(v) for v in P]))
    ens = _ensemble(case, seed)
    R1, Y1 = _perturbation(case, seed)
    if kind == "averages":
        f, d2v = _exact_averages(case, ens, R1, Y1)
        return dict(f=f, d2v=d2v)
    M = case["M"]
    if kind == "static":
        n = M + M * (M + 1) // 2
        return _exact_static(case, ens, [_psi(case, seed + 17 * v, n) for v in range(case["nvec"])])
    op = _Exact(case, ens)
    if kind == "apply":
        return op(_psi(case, seed, M + M * (M + 1)), case["transpose"])
    first = torch.zeros(M + M * (M + 1), dtype=F64, device=CUDA)
    first[:M] = R1
    mask = op.mask if case["wigner"] else torch.ones_like(op.mask)
    a, b, c, Q, P = _exact_krylov(op, first, mask, case["wigner"], case["steps"])
    a, b, c = _stack(a), _stack(b), _stack(c)
    if kind == "lanczos":
        return dict(a=a, b=b, c=c, Q=torch.stack(Q), P=torch.stack(P))
    grid = np.linspace(20, 600, 500) / RY_TO_CM
    return dict(a=a, b=b, c=c,
                G=_exact_fraction(a, b, c, grid, 10 / RY_TO_CM, case["wigner"], float(R1 @ R1)))
