"""The smem-wide kernel at the sizes where the divide and conquer's leaves take
more room than a matrix (N = 1..13 and 17) and on both sides of them, asked for
by name and as a candidate of an autotuned create, against LAPACK zhegv with the
parity tests' bars (1e-12)."""
import numpy as np
import pytest

from oracle import zhegv_batch
from sunny_gen_eigensolver_b200 import accuracy

pytestmark = pytest.mark.gpu


def _check(n, **kw):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, solve
    rng = np.random.default_rng(40 + n)
    A, B = rng.standard_normal((2, 7, n, n)) + 1j * rng.standard_normal((2, 7, n, n))
    H = A + np.conj(np.swapaxes(A, -1, -2))
    S = B @ np.conj(np.swapaxes(B, -1, -2)) + n * np.eye(n)
    with Solver(n, **kw) as s:
        regime = s.regime
        W, U, info = solve(torch.from_numpy(H).cuda(), torch.from_numpy(S).cuda(), solver=s)
    W, U = W.cpu().numpy(), U.cpu().numpy()
    Wr, _, _ = zhegv_batch(H, S)
    assert np.all(info.cpu().numpy() == 0)
    assert accuracy.eig_err_rel(H, W, Wr).max() <= 1e-12
    assert accuracy.residual(H, S, W, U).max() <= 1e-12
    assert accuracy.s_orth(S, U).max() <= 1e-12
    return regime


@pytest.mark.parametrize("n", list(range(1, 20)))
def test_smem_wide_small(cuda, n):
    assert _check(n, regime="smem-wide") == "smem-wide"


@pytest.mark.parametrize("n", [2, 8, 12, 17])
def test_autotuned_small(cuda, n):
    _check(n, tuning="autotune", cache="nocache")
