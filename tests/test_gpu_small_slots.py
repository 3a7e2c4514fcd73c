"""The tiled kernel below its default sizes, asked for by name: both sides of the
change between its two Householder reductions (N = 95 / 96), edges of the row
blocks of 32, one and two slots per SM, and inside the uneven-size kernel; and the
mixed form at the edge of its FP32 copy in shared memory (N = 103 / 104), with U
apart from H and over it, where no pencil needs the FP64 fallback and where all do.
Against LAPACK zhegv with the parity tests' bars (1e-12)."""
import numpy as np
import pytest

from oracle import zhegv_batch
from sunny_gen_eigensolver_b200 import accuracy

pytestmark = pytest.mark.gpu


def _random(n, batch, seed):
    rng = np.random.default_rng(seed)
    A, B = rng.standard_normal((2, batch, n, n)) + 1j * rng.standard_normal((2, batch, n, n))
    return A + np.conj(np.swapaxes(A, -1, -2)), B @ np.conj(np.swapaxes(B, -1, -2)) + n * np.eye(n)


def _check(H, S, W, U, info):
    Wr, _, _ = zhegv_batch(H, S)
    W, U = W.cpu().numpy(), U.cpu().numpy()
    assert np.all(info.cpu().numpy() == 0)
    assert accuracy.eig_err_rel(H, W, Wr).max() <= 1e-12
    assert accuracy.residual(H, S, W, U).max() <= 1e-12
    assert accuracy.s_orth(S, U).max() <= 1e-12


@pytest.mark.parametrize("slots", [1, 2])
@pytest.mark.parametrize("n", [1, 2, 3, 8, 31, 32, 33, 60, 64, 65, 80, 95, 96, 97, 110])
def test_tiled_kernel_by_name(cuda, n, slots):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, solve
    H, S = _random(n, 5, 1000 + n)
    with Solver(n, regime="l2-slot", slots_per_sm=slots) as s:
        _check(H, S, *solve(torch.from_numpy(H).cuda(), torch.from_numpy(S).cuda(), solver=s))


def test_uneven_l2_slot_sizes_match_the_tiled_kernel(cuda):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, UnevenSolver, to_colmajor
    sizes = [5, 33, 60]
    Hs, Ss, ref, out = {}, {}, {}, {}
    for n in sizes:
        H, S = _random(n, 9, n)
        Hs[n], Ss[n] = to_colmajor(torch.from_numpy(H).cuda()), to_colmajor(torch.from_numpy(S).cuda())
        with Solver(n, regime="l2-slot", slots_per_sm=2) as s:
            ref[n] = s.run_kernel(Hs[n], Ss[n])
        out[n] = tuple(torch.full_like(x, -7) for x in ref[n])
    with UnevenSolver(sizes, regimes={n: "l2-slot" for n in sizes}) as us:
        us.launch(Hs, Ss, *({n: out[n][k] for n in sizes} for k in range(3)))
    torch.cuda.synchronize()
    for n in sizes:
        assert all(torch.equal(a, b) for a, b in zip(out[n], ref[n]))


@pytest.mark.parametrize("alias", [False, True])
@pytest.mark.parametrize("refine", ["8", "0"])
@pytest.mark.parametrize("n", [33, 95, 96, 103, 104, 110, 111])
def test_mixed_form_at_the_edges(cuda, monkeypatch, n, refine, alias):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, to_colmajor
    monkeypatch.setenv("SUNNY_GENEIG_MIXED_REFINE_MAX", refine)
    H, S = _random(n, 4, 2000 + n)
    Ht, St = to_colmajor(torch.from_numpy(H).cuda()), to_colmajor(torch.from_numpy(S).cuda())
    U = Ht if alias else torch.empty_like(Ht)
    W = torch.empty((4, n), dtype=torch.float64, device="cuda")
    info = torch.full((4,), -7, dtype=torch.int32, device="cuda")
    with Solver(n, kernel="mixed") as s:
        s.launch(Ht, St, W, U, info)
        torch.cuda.synchronize()
    _check(H, S, W, U.transpose(-1, -2), info)
