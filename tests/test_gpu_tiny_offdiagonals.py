"""Off-diagonals far below the matrix's norm beside zero diagonals, where no
off-diagonal is negligible next to its neighbours and squares underflow: blocks
[[0, x], [x, 0]] and chains with zero diagonal, an entry of one in the last
corner (and two more, so that the chain is cut). S = I, real H, so that the
reduction to tridiagonal form leaves H as it is. Against LAPACK zhegv with the
parity tests' bars (1e-12)."""
import numpy as np
import pytest

from oracle import zhegv_batch
from sunny_gen_eigensolver_b200 import accuracy

pytestmark = pytest.mark.gpu

X = [1e-20, 1e-99, 1e-101, 1e-120, 1e-150, 1e-155, 1e-158, 1e-160, 3e-161, 1e-161, 1e-162, 1e-170, 1e-300, 1e-310]


def _family(n):
    out = []
    for x in X:
        blocks = np.zeros((n, n), dtype=complex)
        for i in range(0, n - 1, 2):
            blocks[i, i + 1] = blocks[i + 1, i] = x
        blocks[n - 1, n - 1] = 1.0
        chain = np.diag(np.full(n - 1, x + 0j), 1) + np.diag(np.full(n - 1, x + 0j), -1)
        chain[n - 1, n - 1] = 1.0
        cut = chain.copy()
        cut[0, 0], cut[n // 2, n // 2] = 1.0, -1.0
        out += [blocks, chain, cut]
    return np.stack(out)


@pytest.mark.parametrize("n", [3, 8, 9, 16, 27, 54, 72, 108, 130])
def test_tiny_offdiagonals(cuda, n):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, solve
    H = _family(n)
    S = np.broadcast_to(np.eye(n, dtype=complex), H.shape).copy()
    with Solver(n) as s:
        W, U, info = solve(torch.from_numpy(H).cuda(), torch.from_numpy(S).cuda(), solver=s)
    W, U = W.cpu().numpy(), U.cpu().numpy()
    Wr, _, ir = zhegv_batch(H, S)
    assert np.all(ir == 0) and np.all(info.cpu().numpy() == 0)
    assert accuracy.eig_err_rel(H, W, Wr).max() <= 1e-12
    assert accuracy.residual(H, S, W, U).max() <= 1e-12
    assert accuracy.s_orth(S, U).max() <= 1e-12
