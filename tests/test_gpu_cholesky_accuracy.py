"""S-orthonormality of the shared-memory kernel's vectors for ill-conditioned S:
||U^H S U - I||_F in extended precision, the mean over many pencils, against
LAPACK zhegv's on the same pencils. It measures the Cholesky factor's error
amplified by cond(S); both factor by elimination in FP64, so their means agree
to the statistics of rounding: 1.25 times zhegv's is allowed. (Panels multiplied
by the explicit inverse of their diagonal tile without a correction have 1.8
times zhegv's at N = 12 and cond(S) = 1e10.)"""
import numpy as np
import pytest

from oracle import zhegv_batch

pytestmark = pytest.mark.gpu


def _spread(n, batch, cond):
    rng = np.random.default_rng(500 + n)
    G, Q = rng.standard_normal((2, batch, n, n)) + 1j * rng.standard_normal((2, batch, n, n))
    Q = np.linalg.qr(Q)[0]
    S = (Q * np.exp(np.linspace(0.0, -np.log(cond), n))) @ np.conj(np.swapaxes(Q, 1, 2))
    return G + np.conj(np.swapaxes(G, 1, 2)), 0.5 * (S + np.conj(np.swapaxes(S, 1, 2)))


def _mean_error(S, U):
    U = U.astype(np.clongdouble)
    R = np.conj(np.swapaxes(U, 1, 2)) @ S.astype(np.clongdouble) @ U - np.eye(S.shape[1])
    return float(np.mean(np.sqrt((np.abs(R) ** 2).sum((1, 2)))))


@pytest.mark.parametrize("cond", [1e6, 1e10])
@pytest.mark.parametrize("n,batch", [(9, 400), (12, 400), (16, 300), (24, 150), (33, 100), (54, 40)])
def test_vectors_as_orthonormal_as_zhegvs(cuda, n, batch, cond):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, solve
    H, S = _spread(n, batch, cond)
    with Solver(n) as s:
        _, U, info = solve(torch.from_numpy(H).cuda(), torch.from_numpy(S).cuda(), solver=s)
    _, Ur, ir = zhegv_batch(H, S)
    assert np.all(ir == 0) and np.all(info.cpu().numpy() == 0)
    assert _mean_error(S, U.cpu().numpy()) <= 1.25 * _mean_error(S, Ur)
