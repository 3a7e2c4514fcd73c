"""Householder columns whose squares leave the range of FP64: matrices of rank
one, which leave columns of ever smaller rounding residues (1e-16, 1e-32, ...),
couplings of 1e-155 to 1e-310 between decoupled levels, and whole matrices
scaled by 1e+-160 and 1e+-200. Shared-memory kernel and tiled kernel (N = 130,
and by name), against LAPACK zhegv with the parity tests' bars (1e-12)."""
import numpy as np
import pytest

from oracle import zhegv_batch
from sunny_gen_eigensolver_b200 import accuracy

pytestmark = pytest.mark.gpu


def _pencils(n):
    rng = np.random.default_rng(60 + n)

    def cn(*s):
        return rng.standard_normal(s) + 1j * rng.standard_normal(s)
    G, X, v = cn(n, n), cn(n, 2 * n), cn(n, 1)
    herm, spd, one = 0.5 * (G + G.conj().T), X @ X.conj().T / (4 * n), np.eye(n, dtype=complex)
    off = herm - np.diag(np.diag(herm))
    levels = np.diag(rng.integers(-1, 2, n)).astype(complex)
    out = [(np.ones((n, n), dtype=complex), one), (v @ v.conj().T, one)]
    out += [(levels + x * off, one) for x in (1e-155, 1e-158, 1e-161, 1e-162, 1e-200, 1e-310)]
    scaled = [(herm * f, spd * g) for f, g in ((1e-160, 1), (1e160, 1), (1, 1e160), (1, 1e-160), (1e200, 1), (1, 1e200))]
    return out, scaled, herm, spd


@pytest.mark.parametrize("n,kw", [(n, {}) for n in (2, 3, 8, 16, 17, 27, 33, 54, 72, 108, 130)] +
                         [(n, {"regime": "l2-slot", "slots_per_sm": 2}) for n in (2, 33, 72)])
def test_columns_out_of_square_range(cuda, n, kw):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, solve
    plain, scaled, herm, spd = _pencils(n)
    H, S = (np.stack(x) for x in zip(*(plain + scaled)))
    with Solver(n, **kw) as s:
        W, U, info = solve(torch.from_numpy(H).cuda(), torch.from_numpy(S).cuda(), solver=s)
    W, U = W.cpu().numpy(), U.cpu().numpy()
    assert np.all(info.cpu().numpy() == 0)
    k = len(plain)
    Wr, _, ir = zhegv_batch(H[:k], S[:k])
    assert np.all(ir == 0)
    assert accuracy.eig_err_rel(H[:k], W[:k], Wr).max() <= 1e-12
    assert accuracy.residual(H[:k], S[:k], W[:k], U[:k]).max() <= 1e-12
    assert accuracy.s_orth(S[:k], U[:k]).max() <= 1e-12
    # scaled pencils: the solution of the unscaled one, W f / g and U / sqrt(g)
    Wr, _, _ = zhegv_batch(herm[None], spd[None])
    for i in range(k, len(H)):
        f, g = np.abs(H[i]).max() / np.abs(herm).max(), np.abs(S[i]).max() / np.abs(spd).max()
        Wi, Ui = (W[i] / f) * g, U[i] * np.sqrt(g)
        assert accuracy.eig_err_rel(herm[None], Wi[None], Wr).max() <= 1e-12
        assert accuracy.residual(herm[None], spd[None], Wi[None], Ui[None]).max() <= 1e-12
        assert accuracy.s_orth(spd[None], Ui[None]).max() <= 1e-12
