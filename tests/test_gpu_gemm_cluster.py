"""Small FP64 products whose K is split over a cluster, with pieces that have no K of their own (the
piece length is rounded up to 16): such a CTA hands its sum to the first one at once.

Integer operands: every sum is below 2^53 and the products are exact in any order.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# pieces of 48 of K, the last two of 8 or 7 empty (on 152 SMs); the last one with K has 20, 30, 38, 33
@pytest.mark.parametrize("m,n,k", [(608, 32, 260), (601, 29, 270), (700, 31, 230), (611, 30, 225)])
def test_empty_pieces(ctx, m, n, k):
    import chemtensor_mojo_gb300 as ct
    rng = np.random.default_rng(m + k)
    A, B = rng.integers(-1000, 1000, (m, k)).astype(float), rng.integers(-1000, 1000, (n, k)).astype(float)
    a, b = (ct.create_dense_tensor_from_data(ctx, x, x.shape) for x in (A, B))
    outs = [ct.create_dense_tensor_from_data(ctx, np.full((m, n), np.nan), (m, n)) for _ in range(64)]
    for c in outs:   # back to back: a launch's CTAs start beside those of the one before
        ct.dense_tensor_dot(c, a, b, ctx, 1, False, False)
    torch.cuda.synchronize()
    ref = A @ B.T
    for c in outs:
        assert np.array_equal(c.to_numpy(), ref)
