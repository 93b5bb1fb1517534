"""FP64-form products on the tensor cores by residues.

With operands of a few bits each product sum is an integer below 2^53 (times powers of two), so
the scheme, which rounds once, must give it exactly: any wrong residue, accumulator reduction
or reconstruction shows.  Random operands fill all bits; there the reference, an FP64 matmul,
is itself off by at most K 2^-53 |A||B|, and the scheme by 2^-53 |C| plus K 2^-62 of the
rows' largest entries.
"""
import numpy as np
import pytest

from oracle import dmrg as od

pytestmark = pytest.mark.gpu


def _dt(ctx, a):
    import chemtensor_mojo_gb300 as ct
    return ct.create_dense_tensor_from_data(ctx, a, a.shape)


def _product(ctx, A, B, launches=None):
    """A @ B through build_two_site_theta; the residue route takes 3 launches up to K = 256, else 4."""
    import chemtensor_mojo_gb300 as ct
    from chemtensor_mojo_gb300 import _lib
    a = ct.MPSSite(_dt(ctx, A.reshape(A.shape[0] // 2, 2, A.shape[1])))
    b = ct.MPSSite(_dt(ctx, B.reshape(B.shape[0], 2, B.shape[1] // 2)))
    n0 = _lib.launch_count()
    out = ct.build_two_site_theta(a, b, ctx)
    if launches != 0:
        assert _lib.launch_count() - n0 == (3 if A.shape[1] <= 256 else 4)
    return out.to_numpy().reshape(A.shape[0], B.shape[1])


# tile edges in M and N (128), in K (64 per block, 1024 per exact chunk) and in the packs
SHAPES = [(254, 256, 256), (256, 258, 257), (258, 254, 255), (256, 256, 319), (256, 256, 321), (130, 386, 1023),
          (256, 384, 1024), (384, 256, 1025), (130, 130, 4097), (2, 4098, 2048), (4098, 2, 2049)]


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_residue_products(ctx, m, n, k):
    rng = np.random.default_rng(m + 3 * n + 7 * k)
    A = rng.integers(-(1 << 20), 1 << 20, (m, k)).astype(float)
    B = rng.integers(-(1 << 20), 1 << 20, (k, n)).astype(float)
    A[m // 2] = 0.0
    A[-1] = 1.0 * (1 << 20)           # the largest sums
    B[:, -1] = -1.0 * (1 << 20)
    ea = rng.integers(-400, 400, (m, 1))
    eb = rng.integers(-400, 400, (1, n))
    ref = np.ldexp(A @ B, ea + eb)
    small = min(m, n) == 2            # too few tiles: FP64 FMAs, exact all the same
    got = _product(ctx, np.ldexp(A, ea), np.ldexp(B, eb), 0 if small else None)
    assert np.array_equal(got, ref)
    A = rng.standard_normal((m, k)) * np.exp(-8.0 * np.arange(k) / k)
    B = rng.standard_normal((k, n)) * np.exp(8.0 * np.arange(k) / k)[:, None]
    got = _product(ctx, A, B, 0 if small else None)
    bound = 2.0 * k * 2.0**-53 * (np.abs(A) @ np.abs(B)) + \
        k * 2.0**-62 * np.abs(A).max(1, keepdims=True) * np.abs(B).max(0, keepdims=True)
    assert (np.abs(got - A @ B) <= bound).all()


def test_residue_nonfinite_rows_and_extreme_scales(ctx):
    rng = np.random.default_rng(5)
    m, n, k = 260, 300, 300
    A = rng.integers(-99, 99, (m, k)).astype(float)
    B = rng.integers(-99, 99, (k, n)).astype(float)
    A[3, 5], A[200, 1], B[7, 9], B[0, 299] = np.inf, np.nan, -np.inf, np.nan
    with np.errstate(invalid="ignore"):
        ref = A @ B
    assert np.array_equal(_product(ctx, A, B), ref, equal_nan=True)
    A = np.ldexp(rng.integers(-99, 99, (m, k)).astype(float), -1074)   # subnormal operands
    B = np.ldexp(rng.integers(-99, 99, (k, n)).astype(float), 1000)
    assert np.array_equal(_product(ctx, A, B), A @ B)
    with np.errstate(over="ignore"):
        ref = np.ldexp(np.ldexp(A, 1074) @ np.ldexp(B, -1000), 1020)   # overflows to infinity
    assert np.array_equal(_product(ctx, np.ldexp(A, 1074 + 600), np.ldexp(B, 420 - 1000)), ref)


def test_residue_workspace_limit_falls_back(ctx):
    import chemtensor_mojo_gb300 as ct
    rng = np.random.default_rng(6)
    A = rng.integers(-999, 999, (256, 256)).astype(float)
    B = rng.integers(-999, 999, (256, 256)).astype(float)
    h2 = ct.DeviceContext(0)
    h2.set_workspace_limit(1 << 20)
    a = ct.MPSSite(_dt(h2, A.reshape(128, 2, 256)))
    b = ct.MPSSite(_dt(h2, B.reshape(256, 2, 128)))
    got = ct.build_two_site_theta(a, b, h2).to_numpy().reshape(256, 256)
    assert np.array_equal(got, A @ B)


# the chains' two-level row and column indexing, unequal sides, with small-integer tensors: exact
@pytest.mark.parametrize("Dl,d,Dr,wl,wr", [(129, 2, 130, 5, 4), (96, 3, 140, 3, 1), (140, 4, 61, 1, 6)])
def test_residue_chains(ctx, Dl, d, Dr, wl, wr):
    import chemtensor_mojo_gb300 as ct
    rng = np.random.default_rng(Dl + Dr)
    ints = lambda *s: rng.integers(-4, 5, s).astype(float)  # noqa: E731
    th, L, R, A = ints(Dl, d, d, Dr), ints(wl, Dl, Dl), ints(wr, Dr, Dr), ints(Dl, d, Dr)
    W1, W2, W = ints(wl, d, d, 3), ints(3, d, d, wr), ints(wl, d, d, wr)
    mpo = lambda w: ct.MPOSite(_dt(ctx, w))                 # noqa: E731
    out = ct.apply_two_site_heff(_dt(ctx, th), _dt(ctx, L), _dt(ctx, R), mpo(W1), mpo(W2), ctx)
    assert np.array_equal(out.to_numpy(), od.apply_two_site_heff(th, L, R, W1, W2))
    left = ct.update_left_environment(_dt(ctx, L), ct.MPSSite(_dt(ctx, A)), mpo(W), ctx)
    assert np.array_equal(left.to_numpy(), od.update_left_environment(L, A, W))
    right = ct.update_right_environment(_dt(ctx, R), ct.MPSSite(_dt(ctx, A)), mpo(W), ctx)
    assert np.array_equal(right.to_numpy(), od.update_right_environment(R, A, W))
