"""The tiled kernel (matrices in a global-memory slot) where its splits change:
above the shared-memory class (N = 111), around the 128-row blocks that its
Householder product deals to the warps, around the 16-column panels, and at the
256-thread form that explicit requests take up to N = 110; and the uneven-size
solver with such sizes beside its persistent kernel. Tolerances as in the
parity tests (1e-12; a backward-stable FP64 solver stays near 1e-13 at N = 400:
n eps is 9e-14)."""
import numpy as np
import pytest

from oracle import zhegv_batch
from sunny_gen_eigensolver_b200 import accuracy

pytestmark = pytest.mark.gpu


def _random(n, batch, seed):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    B = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    return A + np.conj(np.swapaxes(A, -1, -2)), B @ np.conj(np.swapaxes(B, -1, -2)) + n * np.eye(n)


def _solve_and_check(n, batch, **kw):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, solve
    H, S = _random(n, batch, 500 + n)
    S[-1] = np.eye(n)
    S[-1, n // 2, n // 2] = 0.0                      # info = n + n/2 + 1
    with Solver(n, **kw) as s:
        assert s.regime == "l2-slot"
        W, U, info = solve(torch.from_numpy(H).cuda(), torch.from_numpy(S).cuda(), solver=s)
    W, U, info = W.cpu().numpy(), U.cpu().numpy(), info.cpu().numpy()
    Wr, _, ir = zhegv_batch(H, S)
    assert np.array_equal(info, ir) and ir[-1] == n + n // 2 + 1
    ok = ir == 0
    assert accuracy.eig_err_rel(H[ok], W[ok], Wr[ok]).max() <= 1e-12
    assert accuracy.residual(H[ok], S[ok], W[ok], U[ok]).max() <= 1e-12
    assert accuracy.s_orth(S[ok], U[ok]).max() <= 1e-12


@pytest.mark.parametrize("n", [111, 128, 129, 145, 255, 257, 385])
def test_block_edges(cuda, n):
    _solve_and_check(n, 3)


@pytest.mark.parametrize("n", [3, 16, 17, 33, 60, 110])
@pytest.mark.parametrize("slots", [1, 2])
def test_narrow_form(cuda, n, slots):
    _solve_and_check(n, 4, regime="l2-slot", slots_per_sm=slots)


def test_uneven_solver_with_large_sizes(cuda):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, UnevenSolver, to_colmajor
    sizes = [12, 130, 61, 260, 40]
    Hs, Ss, ref, W, U, info = {}, {}, {}, {}, {}, {}
    for n in sizes:
        H, S = _random(n, 5, n)
        Hs[n], Ss[n] = to_colmajor(torch.from_numpy(H).cuda()), to_colmajor(torch.from_numpy(S).cuda())
        with Solver(n) as s:
            ref[n] = s.run_kernel(Hs[n], Ss[n])
        W[n], U[n], info[n] = (torch.full_like(x, -7) for x in ref[n])
    with UnevenSolver(sizes) as us:
        assert [x[0] for x in us.shape] == sorted(sizes, reverse=True)
        for rep in range(2):
            us.launch(Hs, Ss, W, U, info, torch.cuda.Stream() if rep else None)
            torch.cuda.synchronize()
            for n in sizes:
                for x, r in zip((W[n], U[n], info[n]), ref[n]):
                    assert torch.equal(x, r), (n, rep)
                    x.fill_(-7)
