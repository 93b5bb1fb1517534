"""The FP64 GEMM of small products at its edges: 8 x 16 tiles, K blocks of 32, K split into one
cluster (2 to 8 pieces) or through scratch memory (more), and the boundary to 64 x 64 tiles.

Integer operands: every sum is below 2^53 and the products are exact in any order.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (7, 15, 31), (8, 16, 32), (9, 17, 33), (16, 33, 64), (40, 70, 97), (64, 16, 80), (33, 31, 255),
          (32, 32, 256), (32, 32, 288), (96, 96, 2048), (5, 4100, 70), (1095, 1095, 9), (1153, 1153, 9)]


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
def test_small_fp64_products(ctx, m, n, k, ta, tb):
    import chemtensor_mojo_gb300 as ct
    if not ta and not tb and n == k:
        pytest.skip("B's side would be inferred as leading")
    rng = np.random.default_rng(m + n + k)
    A = rng.integers(-1000, 1000, (k, m) if ta else (m, k)).astype(float)
    B = rng.integers(-1000, 1000, (k, n) if tb else (n, k)).astype(float)
    a, b = (ct.create_dense_tensor_from_data(ctx, x, x.shape) for x in (A, B))
    c = ct.create_dense_tensor_from_data(ctx, np.full((m, n), np.nan), (m, n))
    ct.dense_tensor_dot(c, a, b, ctx, 1, ta, tb)
    assert np.array_equal(c.to_numpy(), (A.T if ta else A) @ (B if tb else B.T))
