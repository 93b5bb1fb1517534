"""The FP64 -> split-TF32 packs at the edges of their 32 x 64 tiles, in both source orders.

Integers below 2^10 are exact in TF32 and their sums below 2^24 exact in FP32, so those products
must be exact.  Values over the whole FP32 exponent range times one: the split keeps 22 bits of
the FP32 value, itself rounded once, so 2^-20 bounds the relative error.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dot(ctx, A, B, ta, tb):
    import chemtensor_mojo_gb300 as ct
    a, b = (ct.create_dense_tensor_from_data(ctx, x, x.shape) for x in (A, B))
    m, n = A.shape[1 if ta else 0], B.shape[1 if tb else 0]
    c = ct.create_dense_tensor_from_data(ctx, np.zeros((m, n)), (m, n))
    ct.dense_tensor_dot(c, a, b, ctx, 1, ta, tb, prec="tf32x3")
    return c.to_numpy()


@pytest.mark.parametrize("m,n,k", [(1, 2, 1), (31, 33, 31), (32, 34, 32), (33, 31, 63), (95, 64, 64), (128, 65, 65),
                                   (129, 257, 97)])
@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False), (True, True)])
def test_pack_edges(ctx, m, n, k, ta, tb):
    if not ta and not tb and n == k:
        pytest.skip("B's side would be inferred as leading")
    rng = np.random.default_rng(m + n + k)
    A = rng.integers(-200, 200, (k, m) if ta else (m, k)).astype(float)
    B = rng.integers(-200, 200, (k, n) if tb else (n, k)).astype(float)
    assert np.array_equal(_dot(ctx, A, B, ta, tb), (A.T if ta else A) @ (B if tb else B.T))


def test_pack_rounding_over_the_exponent_range(ctx):
    rng = np.random.default_rng(1)
    A = np.ldexp(rng.uniform(1.0, 2.0, (300, 1)) * rng.choice([-1.0, 1.0], (300, 1)), rng.integers(-100, 120, (300, 1)))
    A[0], A[1], A[2] = 0.0, 1.0 + 2.0**-24, 1.0 + 3.0 * 2.0**-24   # ties
    got = _dot(ctx, A, np.ones((1, 2)), False, True)
    assert (np.abs(got - A) <= 2.0**-20 * np.abs(A)).all()
