"""The mixed form where its FP32 reduction leaves FP32's range: couplings of
1e-20 and 1e-30 between levels (squares underflow, their reciprocal overflows), a
graded matrix, rank one, and whole matrices scaled by 1e+-100. Such pencils are
solved by the FP64 reduction, in the shared-memory kernel or, with U over H, in
the same kernel; input that is not finite still reports zhegv's info. Bars as in
the FP64 form (1e-12)."""
import numpy as np
import pytest

from oracle import zhegv_batch
from sunny_gen_eigensolver_b200 import accuracy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alias", [False, True])
@pytest.mark.parametrize("n", [2, 5, 17, 54, 108, 130])
def test_fp32_out_of_range(cuda, n, alias):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, to_colmajor
    rng = np.random.default_rng(80 + n)
    G = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    herm = 0.5 * (G + G.conj().T)
    levels = np.diag(rng.integers(-1, 2, n)).astype(complex)
    off = herm - np.diag(np.diag(herm))
    d = 10.0 ** (-16.0 * np.arange(n) / n)
    v = G[:, :1]
    H = np.stack([herm, levels + 1e-20 * off, levels + 1e-30 * off, herm * np.outer(d, d), v @ v.conj().T,
                  herm * 1e100, herm * 1e-100, np.full((n, n), np.nan + 0j)])
    S = np.broadcast_to(np.eye(n, dtype=complex), H.shape).copy()
    Ht, St = to_colmajor(torch.from_numpy(H).cuda()), to_colmajor(torch.from_numpy(S).cuda())
    U = Ht if alias else torch.empty_like(Ht)
    W = torch.empty((len(H), n), dtype=torch.float64, device="cuda")
    info = torch.full((len(H),), -7, dtype=torch.int32, device="cuda")
    with Solver(n, kernel="mixed") as s:
        s.launch(Ht, St, W, U, info)
        torch.cuda.synchronize()
    W, U, info = W.cpu().numpy(), U.transpose(-1, -2).cpu().numpy(), info.cpu().numpy()
    assert np.all(info[:-1] == 0) and info[-1] == (n - 1 if n >= 3 else 0)
    assert np.isnan(W[-1]).all() and np.isnan(U[-1]).all()
    H, S, W, U = H[:-1], S[:-1], W[:-1], U[:-1]
    Wr, _, _ = zhegv_batch(H, S)
    assert accuracy.eig_err_rel(H, W, Wr).max() <= 1e-12
    assert accuracy.residual(H, S, W, U).max() <= 1e-12
    assert accuracy.s_orth(S, U).max() <= 1e-12
