"""Dense steps at the edges of their tiles and dispatch: Jacobi pairs (odd sizes,
one 2 x 2 block, the largest projected problem), block orthonormalisation (one warp
to 16 and 32 columns), FP64 products (32-column tiles, K splits) and the FP32 Gram's
paired loads (m odd, even, a multiple of four) and tiled mirror.

Bounds: the eigensolver stops at residuals of 1e-12 of the largest eigenvalue (4 of
them allowed); a product of length K rounds within K 2^-53 of |A|^T |B|; the split
FP32 products as in test_dense_gpu.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-60, 1e60])
@pytest.mark.parametrize("dim", [1, 2, 3, 4, 31, 32, 33, 63, 64, 65, 95, 96, 97])
def test_syevd_sizes(gpu, dim, scale):
    rng = np.random.default_rng(dim)
    B = rng.standard_normal((dim, dim))
    A = B @ B.T * scale
    A[dim // 2:, :dim // 2] = A[:dim // 2, dim // 2:].T
    r = min(dim, 16)
    U = gpu.matrix.syevd(A, dim, r)
    w = np.linalg.eigvalsh(A)
    assert np.linalg.norm(U.T @ U - np.eye(r)) < 1e-12
    lam = np.sort(np.einsum("ij,ij->j", U, A @ U))
    assert np.all(np.abs(lam - w[-r:]) <= 4e-12 * w[-1])
    assert np.all(np.linalg.norm(A @ U - U * np.einsum("ij,ij->j", U, A @ U), axis=0) <= 4e-12 * w[-1])


def test_syevd_ties(gpu):
    dim, r = 48, 6
    Q, _ = np.linalg.qr(np.random.default_rng(1).standard_normal((dim, dim)))
    w = np.r_[[3.0, 3.0, 3.0, 2.0, 2.0, 1.0], np.zeros(dim - 6)]
    A = (Q * w) @ Q.T
    A = (A + A.T) / 2
    U = gpu.matrix.syevd(A, dim, r)
    assert np.linalg.norm(U.T @ U - np.eye(r)) < 1e-12
    assert np.allclose(np.sort(np.einsum("ij,ij->j", U, A @ U)), np.sort(w[:r]), rtol=0, atol=4e-12 * 3)


@pytest.mark.parametrize("nc", [1, 2, 3, 7, 8, 9, 15, 16, 17, 31, 32])
def test_orthonormal_columns(gpu, nc):
    A = np.random.default_rng(nc).standard_normal((301, nc)) + 0.1
    U = gpu.matrix.leftsvd(A, 301, nc, nc)
    assert np.linalg.norm(U.T @ U - np.eye(nc)) < 1e-12
    assert np.linalg.norm(A - U @ (U.T @ A)) < 1e-10 * np.linalg.norm(A)


@pytest.mark.parametrize("arow", [1, 15, 16, 17, 255, 1025, 5003])
@pytest.mark.parametrize("acol,bcol", [(1, 1), (31, 33), (32, 32), (64, 17), (65, 65), (96, 96), (200, 31)])
def test_products(gpu, arow, acol, bcol):
    rng = np.random.default_rng(arow + acol + bcol)
    A, B = rng.standard_normal((arow, acol)), rng.standard_normal((arow, bcol))
    C = gpu.matrix.gemmtn(A, B, arow, acol, bcol)
    bound = (arow + 4) * 2.0**-53 * (np.abs(A).T @ np.abs(B)) * 2  # numpy's own rounding too
    assert np.all(np.abs(C - A.T @ B) <= bound)
    s = rng.uniform(0.5, 2.0, arow)
    D = gpu.matrix.symgemm(np.ascontiguousarray(A.T), np.ascontiguousarray(B.T), s, acol, bcol)
    bound = (arow + 8) * 2.0**-53 * (np.abs(A).T @ (s[:, None] * np.abs(B))) * 2
    assert np.all(np.abs(D - A.T @ (s[:, None] * B)) <= bound)


@pytest.mark.parametrize("n,m", [(1, 1), (65, 3), (129, 31), (200, 33), (333, 126), (512, 129), (700, 257), (1000, 516)])
def test_gram_f32(gpu, n, m):
    import torch
    Y = torch.randn(n, m, generator=torch.Generator().manual_seed(n)).cuda()
    s = (torch.rand(m, generator=torch.Generator().manual_seed(m)) + 0.5).cuda()
    G = torch.empty(m, m, dtype=torch.float64, device="cuda")
    gpu.gram_device(Y.data_ptr(), n, m, s.data_ptr(), G.data_ptr(), gpu.FP32)
    Z = Y.double() * s.double()
    E = Z.T @ Z
    bound = (3 * (n + 63) / 16 * 2.0**-24 + 1e-5) * (Z.abs().T @ Z.abs())
    assert bool(((G - E).abs() <= bound).all())
    assert bool((G == G.T).all())
