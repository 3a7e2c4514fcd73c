"""Sizes 61 to 110, solved with the matrix in one CTA's shared memory (one
pencil per CTA) although their regime is l2-slot: the edges of the row bounds
and of the class itself against LAPACK zhegv, the same results bit for bit from
the uneven-size solver (which runs them beside its persistent kernel) and from
the mixed form's FP64 fallback, and the allocation-free entry point above the
class. Tolerances as in the parity tests (1e-12; a backward-stable FP64 solver
stays below 1e-13 at these sizes)."""
import numpy as np
import pytest

from oracle import zhegv_batch
from sunny_gen_eigensolver_b200 import accuracy, generators

pytestmark = pytest.mark.gpu


def _random(n, batch, seed):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    B = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    return A + np.conj(np.swapaxes(A, -1, -2)), B @ np.conj(np.swapaxes(B, -1, -2)) + n * np.eye(n)


def _check(H, S, W, U, info):
    Wr, _, ir = zhegv_batch(H, S)
    assert np.array_equal(info, ir)
    ok = ir == 0
    assert accuracy.eig_err_rel(H[ok], W[ok], Wr[ok]).max() <= 1e-12
    assert accuracy.residual(H[ok], S[ok], W[ok], U[ok]).max() <= 1e-12
    assert accuracy.s_orth(S[ok], U[ok]).max() <= 1e-12


@pytest.mark.parametrize("n", [61, 64, 65, 72, 73, 79, 80, 81, 96, 97, 105, 110, 111])
def test_edges_of_the_class(cuda, n):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, solve
    H, S = _random(n, 4, 900 + n)
    S[2] = np.eye(n)
    S[2, n - 1, n - 1] = -1.0                           # info = 2n
    with Solver(n) as s:
        assert s.regime == "l2-slot"
        W, U, info = solve(torch.from_numpy(H).cuda(), torch.from_numpy(S).cuda(), solver=s)
    assert int(info[2]) == 2 * n
    _check(H, S, W.cpu().numpy(), U.cpu().numpy(), info.cpu().numpy())


@pytest.mark.parametrize("sizes", [[60, 61, 110, 111], [64, 96], [12, 72, 112]])
def test_uneven_solver_matches_per_size_launches(cuda, sizes):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, UnevenSolver, to_colmajor
    Hs, Ss, ref, W, U, info = {}, {}, {}, {}, {}, {}
    for n in sizes:
        H, S = _random(n, 7, n)
        Hs[n], Ss[n] = to_colmajor(torch.from_numpy(H).cuda()), to_colmajor(torch.from_numpy(S).cuda())
        with Solver(n) as s:
            ref[n] = s.run_kernel(Hs[n], Ss[n])
        W[n], U[n], info[n] = (torch.full_like(x, -7) for x in ref[n])
    with UnevenSolver(sizes) as us:
        for rep in range(2):
            us.launch(Hs, Ss, W, U, info)
            torch.cuda.synchronize()
            for n in sizes:
                for x, r in zip((W[n], U[n], info[n]), ref[n]):
                    assert torch.equal(x, r), (n, rep)
                    x.fill_(-7)
        g = torch.cuda.CUDAGraph()
        st = torch.cuda.Stream()
        with torch.cuda.graph(g, stream=st):
            us.launch(Hs, Ss, W, U, info, st)
        g.replay()
        torch.cuda.synchronize()
        for n in sizes:
            assert all(torch.equal(x, r) for x, r in zip((W[n], U[n], info[n]), ref[n])), n
        del g


@pytest.mark.parametrize("n", [16, 61, 110, 111])
def test_mixed_fallback_equals_plain(cuda, monkeypatch, n):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, to_colmajor
    H, S = generators.baseline_problems(n - n % 2, 5, seed=n, kappa=1e5)
    Hc, Sc = to_colmajor(torch.from_numpy(H).cuda()), to_colmajor(torch.from_numpy(S).cuda())
    n = H.shape[-1]
    with Solver(n) as sp:
        ref = sp.run_kernel(Hc, Sc)
    monkeypatch.setenv("SUNNY_GENEIG_MIXED_REFINE_MAX", "0")
    with Solver(n, kernel="mixed") as sm:
        got = sm.run_kernel(Hc, Sc)
    torch.cuda.synchronize()
    assert all(torch.equal(x, r) for x, r in zip(got, ref))


@pytest.mark.parametrize("n", [16, 72])
def test_mixed_fallback_with_U_over_H(cuda, monkeypatch, n):
    """The fallback then works from what its kernel still holds (H is gone)."""
    import torch
    from sunny_gen_eigensolver_b200 import Solver, to_colmajor
    H, S = generators.baseline_problems(n, 5, seed=n)
    Hc, Sc = to_colmajor(torch.from_numpy(H).cuda()), to_colmajor(torch.from_numpy(S).cuda())
    W = torch.empty((5, n), dtype=torch.float64, device="cuda")
    info = torch.empty((5,), dtype=torch.int32, device="cuda")
    monkeypatch.setenv("SUNNY_GENEIG_MIXED_REFINE_MAX", "0")
    with Solver(n, kernel="mixed") as sm:
        sm.launch(Hc, Sc, W, Hc, info)
        torch.cuda.synchronize()
    _check(H, S, W.cpu().numpy(), Hc.transpose(-1, -2).cpu().numpy(), info.cpu().numpy())


def test_noalloc_above_the_class(cuda):
    import torch
    from sunny_gen_eigensolver_b200 import _native as nat, to_colmajor
    n = 128
    H, S = _random(n, 9, 1)
    Hc, Sc = to_colmajor(torch.from_numpy(H).cuda()), to_colmajor(torch.from_numpy(S).cuda())
    W = torch.empty((9, n), dtype=torch.float64, device="cuda")
    U = torch.empty_like(Hc)
    info = torch.empty((9,), dtype=torch.int32, device="cuda")
    st = nat.load().sunny_geneig_launch_noalloc(n, Hc.data_ptr(), Sc.data_ptr(), W.data_ptr(), U.data_ptr(),
                                                info.data_ptr(), 9, torch.cuda.current_stream().cuda_stream)
    assert st == nat.STATUS_OK, nat.last_error()
    torch.cuda.synchronize()
    _check(H, S, W.cpu().numpy(), U.transpose(-1, -2).cpu().numpy(), info.cpu().numpy())
