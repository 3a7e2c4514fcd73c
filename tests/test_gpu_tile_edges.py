"""Sizes and structures where the tiled shared-memory solver can go wrong:
row counts one below, at and one above its 8-row tiles and row bounds, tears
of the divide and conquer that are exactly zero, equal poles on both sides of
a tear (rotated and deflated columns), the intensity form at its smallest and
largest sizes, and Fourier term tables longer than the staging triangle.

Tolerances: those of the parity tests (eigenvalues within 1e-12 ||H||_2 of
LAPACK zhegv, residual and S-orthonormality 1e-12, spectra within 1e-9 of
their largest value). A backward-stable FP64 solver is at c n eps with a
modest c, below 1e-13 at these sizes.
"""
import numpy as np
import pytest

from oracle import fourier, zhegv_batch
from oracle.intensity import sigma_intensities
from sunny_gen_eigensolver_b200 import accuracy, generators, lswt

pytestmark = pytest.mark.gpu


def _random(n, batch, seed):
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    B = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    return A + np.conj(np.swapaxes(A, -1, -2)), B @ np.conj(np.swapaxes(B, -1, -2)) + n * np.eye(n)


def _check(H, S, **kw):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, solve
    with Solver(H.shape[-1], **kw) as s:
        W, U, info = solve(torch.from_numpy(np.ascontiguousarray(H)).cuda(),
                           torch.from_numpy(np.ascontiguousarray(S)).cuda(), solver=s)
    W, U, info = W.cpu().numpy(), U.cpu().numpy(), info.cpu().numpy()
    Wr, _, ir = zhegv_batch(H, S)
    assert np.array_equal(info, ir) and (ir == 0).all()
    assert accuracy.eig_err_rel(H, W, Wr).max() <= 1e-12
    assert accuracy.residual(H, S, W, U).max() <= 1e-12
    assert accuracy.s_orth(S, U).max() <= 1e-12
    assert (np.diff(W, axis=-1) >= 0).all()


@pytest.mark.parametrize("n", [8, 9, 15, 16, 17, 23, 25, 31, 34, 41, 47, 49, 56, 57, 59])
def test_tile_and_row_bound_edges(cuda, n):
    _check(*_random(n, 3, 700 + n))


@pytest.mark.parametrize("n", [61, 63, 64])
def test_largest_sizes_in_shared_memory(cuda, n):
    _check(*_random(n, 3, 800 + n), regime="smem-cta")


@pytest.mark.parametrize("n", [16, 20, 40, 52, 72])
def test_zero_tears_and_equal_poles(cuda, n):
    """H = blockdiag of equal 4 x 4 blocks (zero off-diagonals of T, every
    eigenvalue n/4 times), the same with one entry coupling two blocks, and a
    diagonal H; S = I."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4))
    H = np.zeros((3, n, n), dtype=np.complex128)
    H[0] = np.kron(np.eye(n // 4), A + A.conj().T)
    H[1] = H[0]
    H[1, n // 2, n // 2 - 1] = H[1, n // 2 - 1, n // 2] = 1e-9
    H[2] = np.diag(np.arange(n) % 3)
    _check(H, np.broadcast_to(np.eye(n, dtype=np.complex128), H.shape).copy())


@pytest.mark.parametrize("n", [2, 4, 16, 34, 60])
def test_intensity_sizes(cuda, n):
    import torch
    from sunny_gen_eigensolver_b200 import Solver, to_colmajor
    _, D = generators.sigma_metric_problems(n, 5, seed=40 + n)
    rng = np.random.default_rng(n)
    O = rng.standard_normal((5, 3, n)) + 1j * rng.standard_normal((5, 3, n))
    q = rng.standard_normal((5, 3))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    _, om, _, _, _ = sigma_intensities(D, O, q, np.linspace(0.0, 1.0, 4), 0.1)
    E = np.linspace(0.0, om.max() * 1.2, 61)
    fwhm = om.max() / 30
    Wr, _, _, ref, _ = sigma_intensities(D, O, q, E, fwhm)
    dev = torch.device("cuda")
    W = torch.empty((5, n), dtype=torch.float64, device=dev)
    spec = torch.empty((5, 61), dtype=torch.float64, device=dev)
    info = torch.empty((5,), dtype=torch.int32, device=dev)
    with Solver(n) as s:
        s.launch_sigma_intensity(to_colmajor(torch.from_numpy(D).to(dev)),
                                 torch.from_numpy(np.ascontiguousarray(np.swapaxes(O, 1, 2))).to(dev),
                                 torch.from_numpy(q).to(dev), torch.from_numpy(E).to(dev), fwhm, W, spec, info)
        torch.cuda.synchronize()
    assert (info.cpu().numpy() == 0).all()
    assert np.abs(W.cpu().numpy() - Wr).max() <= 1e-12
    assert (np.abs(spec.cpu().numpy() - ref) / np.abs(ref).max(axis=1, keepdims=True)).max() <= 1e-9


@pytest.mark.parametrize("m,bonds", [(1, 3), (4, 60), (7, 90), (20, 1500)])
def test_fourier_terms_beyond_the_staging_triangle(cuda, m, bonds):
    import torch
    from sunny_gen_eigensolver_b200 import Solver
    n = 2 * m
    model = lswt.random_model(m, bonds, seed=m)
    rows, cols, coef, disp = lswt.fourier_terms(model)
    packed = lswt.pack_terms(n, rows, cols, coef, disp)
    assert m == 1 or packed[1].shape[0] > n * (n - 1) // 2
    q = np.random.default_rng(m).uniform(-0.5, 0.5, size=(9, 3))
    S = fourier.assemble(n, rows, cols, coef, disp, q)
    H = np.broadcast_to(np.diag(np.r_[np.ones(m), -np.ones(m)]).astype(np.complex128), S.shape).copy()
    Wr, _, ir = zhegv_batch(H, S)
    assert (ir == 0).all()
    dev = torch.device("cuda")
    W = torch.empty((9, n), dtype=torch.float64, device=dev)
    U = torch.empty((9, n, n), dtype=torch.complex128, device=dev)
    info = torch.empty((9,), dtype=torch.int32, device=dev)
    with Solver(n) as s:
        s.launch_fourier_sigma(s.device_terms(*packed), torch.from_numpy(q).to(dev), W, U, info)
        torch.cuda.synchronize()
    assert (info.cpu().numpy() == 0).all()
    W, U = W.cpu().numpy(), U.transpose(-1, -2).cpu().numpy()
    assert np.abs(W - Wr).max() <= 1e-12
    assert accuracy.residual(H, S, W, U).max() <= 1e-12
    assert accuracy.s_orth(S, U).max() <= 1e-12
