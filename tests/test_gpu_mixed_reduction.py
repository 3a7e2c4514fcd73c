"""The mixed form's FP32 reduction, in shared memory up to N = 101 and on its
global-memory copy above: sizes at the edges of its row blocks of 32, of the
back-transform's strips of 8 columns and pairs of 16 reflectors, and on both
sides of the change-over, against zhegv with the FP64 forms' bars (the
refinement ends at FP64 rounding level)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 8, 16, 17, 18, 31, 32, 33, 34, 49, 50, 63, 64, 65, 96, 97, 101, 102, 110, 111])
def test_mixed_matches_zhegv(cuda, n):
    import torch
    from oracle import zhegv_batch
    from sunny_gen_eigensolver_b200 import Solver, accuracy, solve
    rng = np.random.default_rng(700 + n)
    A, B = rng.standard_normal((2, 5, n, n)) + 1j * rng.standard_normal((2, 5, n, n))
    H = A + np.conj(np.swapaxes(A, -1, -2))
    S = B @ np.conj(np.swapaxes(B, -1, -2)) + n * np.eye(n)
    with Solver(n, kernel="mixed") as s:
        W, U, info = solve(torch.from_numpy(H).cuda(), torch.from_numpy(S).cuda(), solver=s)
    W, U = W.cpu().numpy(), U.cpu().numpy()
    Wr, _, _ = zhegv_batch(H, S)
    assert np.all(info.cpu().numpy() == 0)
    assert accuracy.eig_err_rel(H, W, Wr).max() <= 1e-12
    assert accuracy.residual(H, S, W, U).max() <= 1e-12
    assert accuracy.s_orth(S, U).max() <= 1e-12
