"""The multi-SM Jacobi kernels at the edges of their dispatch, against LAPACK.

Up to 200 KB of vectors and rotations: four warps per vector pair, one cluster up to 96
vectors and one CTA per pair above, with the vectors held in registers up to 128 and 256
elements and re-read beyond.  Above 200 KB: one CTA per pair after a Householder QR, held up
to 256 elements.  Tolerances as for the other exact SVD tests: singular values to 1e-13 of
s_0, orthonormal factors to 1e-12, reconstruction to 1e-13 of the largest entry times the
rank's square root.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2), (3, 2), (2, 3), (31, 33), (64, 64), (65, 64), (96, 96), (97, 97), (96, 129), (113, 113),
          (4, 257), (300, 4), (2, 700), (114, 114), (256, 120), (257, 200)]


def _matrix(m, n):
    rng = np.random.default_rng(1000 * m + n)
    k = min(m, n)
    U, _ = np.linalg.qr(rng.standard_normal((m, k)))
    V, _ = np.linalg.qr(rng.standard_normal((n, k)))
    return (U * np.exp(-6.0 * np.arange(k) / k)) @ V.T


@pytest.mark.parametrize("m,n", SHAPES)
def test_svd_trunc_edges(ctx, m, n):
    import chemtensor_mojo_gb300 as ct
    M = _matrix(m, n)
    U, S, Vt, c = ct.dense_tensor_svd_trunc(ct.create_dense_tensor_from_data(ctx, M, M.shape), ctx, 1 << 30, 0.0)
    u, s, vt = U.to_numpy(), S.to_numpy(), Vt.to_numpy()
    ref = np.linalg.svd(M, compute_uv=False)
    assert c == min(m, n)
    assert np.abs(s - ref).max() <= 1e-13 * ref[0]
    assert np.abs(u.T @ u - np.eye(c)).max() < 1e-12
    assert np.abs(vt @ vt.T - np.eye(c)).max() < 1e-12
    assert np.abs((u * s) @ vt - M).max() <= 1e-13 * np.sqrt(c)


@pytest.mark.parametrize("left", [True, False])
@pytest.mark.parametrize("Dl,Dr", [(1, 1), (16, 48), (48, 49), (8, 100), (64, 57)])
def test_split_edges(ctx, Dl, Dr, left):
    import chemtensor_mojo_gb300 as ct
    M = _matrix(2 * Dl, 2 * Dr)
    th = M.reshape(Dl, 2, 2, Dr)
    A, B, disc, S = ct.split_two_site_theta_svd(ct.create_dense_tensor_from_data(ctx, th, th.shape), 1 << 20, 0.0, ctx,
                                                left, return_spectrum=True)
    k = min(M.shape)
    a, b = A.tensor.to_numpy().reshape(2 * Dl, k), B.tensor.to_numpy().reshape(k, 2 * Dr)
    ref = np.linalg.svd(M, compute_uv=False)
    q = a.T @ a if left else b @ b.T
    assert np.abs(q - np.eye(k)).max() < 1e-12
    assert np.abs(a @ b - M).max() <= 1e-13 * np.sqrt(k)
    assert np.abs(S - ref).max() <= 1e-13 * ref[0]


def test_svd_scaled_and_rank_deficient(ctx):
    """Entries far from 1 (the exponent ranges of the fast division and square root) and exactly
    dependent rows."""
    import chemtensor_mojo_gb300 as ct
    M = _matrix(40, 40)
    ref = np.linalg.svd(M, compute_uv=False)
    for scale in (2.0 ** 200, 2.0 ** -200):
        U, S, Vt, c = ct.dense_tensor_svd_trunc(ct.create_dense_tensor_from_data(ctx, M * scale, M.shape), ctx, 1 << 30,
                                                0.0)
        assert np.abs(S.to_numpy() / scale - ref).max() <= 1e-13 * ref[0]
    R = M.copy()
    R[20:] = R[:20]
    U, S, Vt, c = ct.dense_tensor_svd_trunc(ct.create_dense_tensor_from_data(ctx, R, R.shape), ctx, 1 << 30, 0.0)
    s = S.to_numpy()
    ref = np.linalg.svd(R, compute_uv=False)
    assert np.abs(s - ref).max() <= 1e-13 * ref[0]
    assert np.abs((U.to_numpy() * s) @ Vt.to_numpy() - R).max() <= 1e-13 * np.sqrt(c)
