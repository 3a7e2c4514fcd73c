"""The workloads this solver is timed on, through its public entry points.

Each case is one call pattern of a spin-wave program: a batch of Hermitian-definite pencils
H u = lambda S u (complex128) of one size, the metric form Sigma u = lambda S u, the metric form
with S(q) assembled on the device and reduced to spectra, or a batch of mixed sizes.

  kind "solve"      Solver.launch (or run_kernel where `alloc` is set: outputs allocated by the call)
  kind "mixed"      Solver(kernel="mixed").launch
  kind "sigma"      Solver.launch_sigma: H = diag(I, -I) implied
  kind "intensity"  Solver.launch_sigma_intensity: metric solve reduced to S(q, E)
  kind "fourier"    Solver.launch_fourier_sigma_intensity: S(q) from Fourier terms, then S(q, E)
  kind "uneven"     UnevenSolver.launch: up to seven sizes in one call

Inputs follow the benchmark's distributions: H of the BdG block structure shifted positive definite
(odd n: a Hermitian matrix of the same element distribution), S a dense positive-definite matrix
with cond(S) near 100 (a Wishart matrix with 1.5 n samples).

An eigenvector is defined up to a phase factor, so the programs that return eigenvectors end with
the convention that the sum of a vector's components is real and positive.
"""
import math

import torch

from sunny_gen_eigensolver_b200 import Solver, UnevenSolver, lswt

DEV = "cuda:0"
FWHM = 0.15
MIX = "12:30,24:20,54:25,72:10,108:8,162:5,216:2"   # size:percent of the mixed-size benchmark


def listed():
    return [
        # a handful of small cells, one call at a time (an interactive look at a few q-points): latency
        {"name": "few_n12", "kind": "solve", "n": 12, "batch": 8, "alloc": True},
        # one line through the zone of a 27-site cell: less than one pencil per SM
        {"name": "path_n54", "kind": "sigma", "n": 54, "batch": 100},
        # dense q-grid of an 8-site cell
        {"name": "grid_n16", "kind": "solve", "n": 16, "batch": 65536, "alloc": False},
        # an odd size and a batch that divides by nothing
        {"name": "odd_n33", "kind": "solve", "n": 33, "batch": 9001, "alloc": False},
        # the headline: a powder shell of a 27-site cell
        {"name": "shell_n54", "kind": "solve", "n": 54, "batch": 16384, "alloc": False},
        # just above the shared-memory sizes, odd
        {"name": "odd_n77", "kind": "solve", "n": 77, "batch": 1501, "alloc": False},
        # 54-, 108- and 192-site cells
        {"name": "cell_n108", "kind": "solve", "n": 108, "batch": 2048, "alloc": False},
        {"name": "cell_n216", "kind": "solve", "n": 216, "batch": 444, "alloc": False},
        {"name": "cell_n384", "kind": "solve", "n": 384, "batch": 74, "alloc": False},
        # powder spectra: S(q) assembled from the exchange terms, solved and reduced to S(q, E)
        {"name": "spectra_n54", "kind": "fourier", "n": 54, "batch": 8192, "ne": 200, "bonds": 120},
        # requests of many sizes packed into one call
        {"name": "uneven", "kind": "uneven", "total": 4000, "mix": MIX},
        # the mixed-precision form
        {"name": "mixed_n54", "kind": "mixed", "n": 54, "batch": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "sigma", "intensity", "fourier", "uneven", "mixed"])
    if kind == "uneven":
        sizes = sorted(rng.sample([12, 18, 24, 31, 45, 54, 60, 72, 85, 108, 130, 162, 216], rng.randint(2, 7)))
        w = [rng.uniform(0.5, 1.5) / n for n in sizes]
        pct = [max(1, int(100 * x / sum(w))) for x in w]
        top = 3.0e10 / _flops(max(sizes))
        return {"kind": kind, "total": _log_int(rng, 200, max(400, min(4000, top))),
                "mix": ",".join("%d:%d" % p for p in zip(sizes, pct))}
    if kind == "solve":
        n = _log_int(rng, 4, 384)
        most = 5.0e10
    elif kind == "mixed":
        n = _log_int(rng, 16, 128)
        most = 1.2e10
    else:
        n = 2 * _log_int(rng, 3, 30)
        most = 3.0e10
    batch = _log_int(rng, 1, max(2, min(40000, int(most / _flops(n)))))
    case = {"kind": kind, "n": n, "batch": batch}
    if kind == "solve":
        case["alloc"] = rng.random() < 0.25
    if kind in ("intensity", "fourier"):
        case["ne"] = _log_int(rng, 20, 500)
    if kind == "fourier":
        case["bonds"] = _log_int(rng, n, 4 * n)
    return case


# ---------------------------------------------------------------- inputs
def _cn(gen, *shape):
    return torch.view_as_complex(torch.randn(*shape, 2, generator=gen, dtype=torch.float64, device=DEV))


def _bdg(gen, n, batch):
    """Hermitian, unit-variance off-diagonal elements, shifted so that lambda_min is near 0.1 ||H||."""
    if n % 2:
        H = _cn(gen, batch, n, n)
        H = 0.5 * (H + H.mH)
    else:
        m = n // 2
        G = _cn(gen, batch, m, m)
        A = 0.5 * (G + G.mH)
        G = _cn(gen, batch, m, m)
        B = 0.5 * (G + G.mT)
        H = torch.cat([torch.cat([A, B], 2), torch.cat([B.conj(), A.conj()], 2)], 1)
    H.diagonal(dim1=-2, dim2=-1).add_(2.45 * math.sqrt(n) + 1.0)
    return H


def _overlap(gen, n, batch):
    p = -(-3 * n // 2) + 4
    X = _cn(gen, batch, n, p)
    S = (X @ X.mH) / (2.0 * p)
    return 0.5 * (S + S.mH)


def _gen(seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    return gen


def _mix(case):
    """{n: count}: the mix's shares of `total`, at least one problem each."""
    parts = [p.split(":") for p in case["mix"].split(",")]
    tot = sum(int(w) for _, w in parts)
    return {int(n): max(1, case["total"] * int(w) // tot) for n, w in parts}


def _inputs(case, seed):
    """The call's inputs in natural layout (matrix b is [b, i, j])."""
    gen = _gen(seed)
    kind = case["kind"]
    if kind == "uneven":
        out = {}
        for n, c in _mix(case).items():
            out[n] = (_bdg(gen, n, c), _overlap(gen, n, c))
        return out
    n, batch = case["n"], case["batch"]
    if kind in ("solve", "mixed"):
        return {"H": _bdg(gen, n, batch), "S": _overlap(gen, n, batch)}
    x = {}
    if kind in ("sigma", "intensity"):
        x["S"] = _bdg(gen, n, batch)
    if kind == "fourier":
        model = lswt.random_model(n // 2, case["bonds"], seed=seed)
        x["terms"] = lswt.pack_terms(n, *lswt.fourier_terms(model))
        x["q"] = torch.rand(batch, 3, generator=gen, dtype=torch.float64, device=DEV)
    if kind in ("intensity", "fourier"):
        x["O"] = _cn(gen, batch, n, 3)
        q = torch.randn(batch, 3, generator=gen, dtype=torch.float64, device=DEV)
        x["qhat"] = q / q.norm(dim=1, keepdim=True)
        # the magnon energies are 1 / lambda: the eigenvalues of diag(I, -I) S lie within the norm of S
        top = 5.5 * math.sqrt(n) if kind == "intensity" else 2.0 + 4.0 * case["bonds"] / n
        x["E"] = torch.linspace(0.0, top, case["ne"], dtype=torch.float64, device=DEV)
    return x


def prepare(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "uneven":
        s = {"kind": kind, "solver": UnevenSolver(list(x)), "H": {}, "S": {}, "W": {}, "U": {}, "info": {}}
        for n, (H, S) in x.items():
            s["H"][n], s["S"][n] = H.mT.contiguous(), S.mT.contiguous()
            s["W"][n], s["U"][n], s["info"][n] = _outputs(n, H.shape[0])
        return s
    n, batch = case["n"], case["batch"]
    s = {"kind": kind, "alloc": case.get("alloc", False),
         "solver": Solver(n, kernel="mixed") if kind == "mixed" else Solver(n)}
    for k in ("H", "S"):
        if k in x:
            s[k] = x[k].mT.contiguous()          # column-major buffers
    if not s["alloc"]:
        s["W"], s["U"], s["info"] = _outputs(n, batch, vectors=kind not in ("intensity", "fourier"))
    if kind in ("intensity", "fourier"):
        s.update(O=x["O"], qhat=x["qhat"], E=x["E"])
        s["spec"] = torch.empty((batch, case["ne"]), dtype=torch.float64, device=DEV)
    if kind == "fourier":
        s["q"] = x["q"]
        s["terms"] = s["solver"].device_terms(*x["terms"])
    return s


def _outputs(n, batch, vectors=True):
    return (torch.empty((batch, n), dtype=torch.float64, device=DEV),
            torch.empty((batch, n, n), dtype=torch.complex128, device=DEV) if vectors else None,
            torch.empty((batch,), dtype=torch.int32, device=DEV))


def _fixed_phase(U):
    """U[b, k] is eigenvector k of problem b: the sum of its components made real and positive."""
    return U.div_(U.sum(-1, keepdim=True).sgn_())


# ---------------------------------------------------------------- one pass
def run(s):
    kind, solver = s["kind"], s["solver"]
    if kind == "uneven":
        solver.launch(s["H"], s["S"], s["W"], s["U"], s["info"])
        return [[s["W"][n], _fixed_phase(s["U"][n]), s["info"][n]] for n in s["H"]]
    if kind == "intensity":
        solver.launch_sigma_intensity(s["S"], s["O"], s["qhat"], s["E"], FWHM, s["W"], s["spec"], s["info"])
        return [s["W"], s["spec"], s["info"]]
    if kind == "fourier":
        solver.launch_fourier_sigma_intensity(s["terms"], s["q"], s["O"], s["qhat"], s["E"], FWHM, s["W"],
                                              s["spec"], s["info"])
        return [s["W"], s["spec"], s["info"]]
    if s["alloc"]:
        W, U, info = solver.run_kernel(s["H"], s["S"])
    elif kind == "sigma":
        W, U, info = s["W"], s["U"], s["info"]
        solver.launch_sigma(s["S"], W, U, info)
    else:
        W, U, info = s["W"], s["U"], s["info"]
        solver.launch(s["H"], s["S"], W, U, info)
    return [W, _fixed_phase(U), info]


# ---------------------------------------------------------------- work and exact values
def _flops(n, vectors=True):
    """Real FP64 operations of one solve: Cholesky, reduction to standard form, tridiagonalisation and,
    where eigenvectors come back, the two back-transforms. Without vectors (spectra) the reduction of
    the diagonal metric and the tridiagonalisation are what is left at order n^3."""
    return 68.0 / 3.0 * n ** 3 if vectors else 28.0 / 3.0 * n ** 3


def work(case):
    kind = case["kind"]
    if kind == "uneven":
        m = _mix(case)
        return {"bytes": sum(c * (48 * n * n + 8 * n + 4) for n, c in m.items()),
                "flops": sum(c * _flops(n) for n, c in m.items())}
    n, batch = case["n"], case["batch"]
    if kind in ("intensity", "fourier"):
        per = 8 * n + 4 + 48 * n + 24 + 8 * case["ne"] + (24 if kind == "fourier" else 16 * n * n)
        return {"bytes": batch * per, "flops": batch * _flops(n, vectors=False)}
    mats = 2 if kind == "sigma" else 3
    return {"bytes": batch * (16 * mats * n * n + 8 * n + 4), "flops": batch * _flops(n)}


def _eig(H, S):
    L = torch.linalg.cholesky(S)
    Y = torch.linalg.solve_triangular(L, H, upper=False)
    C = torch.linalg.solve_triangular(L, Y.mH, upper=False)
    W, V = torch.linalg.eigh(0.5 * (C + C.mH))
    return W, torch.linalg.solve_triangular(L.mH, V, upper=True)


def _exact_pencils(H, S):
    Ws, Us = [], []
    for i in range(0, H.shape[0], 2048):
        W, U = _eig(H[i:i + 2048], S[i:i + 2048])
        Ws.append(W)
        Us.append(U.mT.contiguous())
    W, U = torch.cat(Ws), torch.cat(Us)
    return [W, _fixed_phase(U), torch.zeros(W.shape[0], dtype=torch.int32, device=DEV)]


def _assembled(n, terms, q):
    start, coef, disp = (torch.as_tensor(t).to(DEV) for t in terms)
    entry = torch.repeat_interleave(torch.arange(n * n, device=DEV), start.long().diff())
    ph = torch.exp(2j * math.pi * (q @ disp.T).to(torch.complex128)) * coef
    S = torch.zeros((q.shape[0], n * n), dtype=torch.complex128, device=DEV)
    S.index_add_(1, entry, ph)
    S = S.reshape(-1, n, n).mT                # entry e = row + n col
    low = torch.tril(S, -1)
    return low + low.mH + torch.diag_embed(torch.diagonal(S, dim1=-2, dim2=-1).real.to(torch.complex128))


def exact(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "uneven":
        return [_exact_pencils(H, S) for H, S in x.values()]
    if kind in ("solve", "mixed"):
        return _exact_pencils(x["H"], x["S"])
    n, batch = case["n"], case["batch"]
    sig = torch.ones(n, dtype=torch.complex128, device=DEV)
    sig[n // 2:] = -1.0
    Sigma = torch.diag(sig).expand(batch, n, n)
    S = _assembled(n, x["terms"], x["q"]) if kind == "fourier" else x["S"]
    W, U, info = _exact_pencils(Sigma, S)
    if kind == "sigma":
        return [W, U, info]
    # t = u / sqrt(lambda) per positive eigenvalue, omega = 1 / lambda, intensity |Y|^2 - |q . Y|^2
    Y = torch.einsum("bia,bki->bka", x["O"], U)
    qy = (Y * x["qhat"][:, None, :]).sum(-1)
    inten = (Y.abs().square().sum(-1) - qy.abs().square()) / W
    pos = W > 0
    inten = torch.where(pos, inten, torch.zeros_like(inten))
    omega = torch.where(pos, 1.0 / W, torch.full_like(W, 1.0e9))
    sd = FWHM / (2.0 * math.sqrt(2.0 * math.log(2.0)))
    spec = torch.zeros((batch, case["ne"]), dtype=torch.float64, device=DEV)
    for k in range(n):
        d = (x["E"][None, :] - omega[:, k:k + 1]) / sd
        spec += inten[:, k:k + 1] * torch.exp(-0.5 * d * d)
    return [W, spec / (sd * math.sqrt(2.0 * math.pi)), info]
