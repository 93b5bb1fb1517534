"""FP64-form products of graded operands keep FP64 accuracy element by element.

One operand falls along the contraction and the other rises (a gauge X, X^-1 between two
tensors), or rows hold entries many orders apart.  An FP64 product is off by about sqrt(K) 2^-53
(|A| |B|) of each element, whatever the rows' largest entries are; the bound is three times that.
Exact products come from double-double sums on the host.
"""
import numpy as np
import pytest

from oracle import dmrg as od

pytestmark = pytest.mark.gpu
U = 2.0**-53


def _dt(ctx, a):
    import chemtensor_mojo_gb300 as ct
    return ct.create_dense_tensor_from_data(ctx, a, a.shape)


def _split(x):
    c = 134217729.0 * x
    hi = c - (c - x)
    return hi, x - hi


def exact_matmul(A, B):
    """A @ B rounded from double-double sums."""
    hi, lo = np.zeros((A.shape[0], B.shape[1])), np.zeros((A.shape[0], B.shape[1]))
    (ah, al), (bh, bl) = _split(A), _split(B)
    for k in range(A.shape[1]):
        p = A[:, k, None] * B[k]
        e = ((ah[:, k, None] * bh[k] - p) + ah[:, k, None] * bl[k] + al[:, k, None] * bh[k]) + al[:, k, None] * bl[k]
        s = hi + p
        t = s - hi
        lo += ((hi - (s - t)) + (p - t)) + e
        hi = s
    return hi + lo


def product(ctx, A, B):
    """A @ B through build_two_site_theta, on the tensor cores (3 launches up to K = 256, else 4)."""
    import chemtensor_mojo_gb300 as ct
    from chemtensor_mojo_gb300 import _lib
    a = ct.MPSSite(_dt(ctx, np.ascontiguousarray(A).reshape(A.shape[0] // 2, 2, A.shape[1])))
    b = ct.MPSSite(_dt(ctx, np.ascontiguousarray(B).reshape(B.shape[0], 2, B.shape[1] // 2)))
    n0 = _lib.launch_count()
    out = ct.build_two_site_theta(a, b, ctx)
    assert _lib.launch_count() - n0 == (3 if A.shape[1] <= 256 else 4)
    return out.to_numpy().reshape(A.shape[0], B.shape[1])


def check(ctx, A, B):
    err = np.abs(product(ctx, A, B) - exact_matmul(A, B))
    bound = 3.0 * np.sqrt(A.shape[1]) * U * (np.abs(A) @ np.abs(B))
    assert (err <= bound).all(), (err / np.maximum(bound, 1e-300)).max()


@pytest.mark.parametrize("fall", [1e2, 1e4, 1e6, 1e8, 1e10, 1e12])
@pytest.mark.parametrize("m,n,k", [(256, 256, 256), (270, 398, 300), (258, 260, 1100)])
@pytest.mark.parametrize("positive", [False, True])
def test_opposite_grading(ctx, fall, m, n, k, positive):
    rng = np.random.default_rng(int(np.log10(fall)) + m + n)
    g = fall ** (np.arange(k) / k)
    A, B = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    if positive:
        A, B = np.abs(A), np.abs(B)
    check(ctx, A / g, B * g[:, None])


@pytest.mark.parametrize("part", [0.02, 0.5])
def test_opposite_grading_in_some_columns(ctx, part):
    rng = np.random.default_rng(11)
    A, B = rng.standard_normal((300, 280)), rng.standard_normal((280, 320))
    g = 1e9 ** (np.arange(280) / 280)
    A[:int(300 * part)] /= g
    B[:, :int(320 * part)] *= g[:, None]
    check(ctx, A, B)


def test_rows_with_entries_far_apart(ctx):
    # every row of A has a 1 where B has nothing; what is left is 2^-70 and less
    rng = np.random.default_rng(3)
    A, B = rng.standard_normal((256, 256)), rng.standard_normal((256, 256))
    A *= 2.0 ** rng.integers(-90, -70, A.shape)
    A[:, 17], B[17] = 1.0, 0.0
    check(ctx, A, B)
    # an environment's identity with noise next to it, times columns that decay
    L = np.eye(256) + 1e-17 * rng.standard_normal((256, 256))
    th = rng.standard_normal((256, 512)) * np.exp(-12.0 * np.arange(256) / 256)[:, None]
    check(ctx, np.concatenate([L, rng.standard_normal((256, 256))]), th)
    # blocks: nothing between them
    A, B = rng.standard_normal((256, 256)), rng.standard_normal((256, 256)) * 1e-3
    A[:128, 128:] = A[128:, :128] = B[:128, 128:] = B[128:, :128] = 0.0
    check(ctx, A, B)
    # both all but one entry small
    A, B = rng.standard_normal((256, 256)) * 1e-13, rng.standard_normal((256, 256)) * 1e-13
    A[:, 0], B[0], A[:, 1], B[1] = 1.0, 0.0, 0.0, 1.0
    check(ctx, A, B)


# the deepest products: fewer bits per operand
@pytest.mark.parametrize("k", [2048, 2049, 32768, 40000, 131072])
def test_deep_products(ctx, k):
    rng = np.random.default_rng(k)
    m, n = (256, 256) if k < 30000 else (128, 256)
    A = rng.integers(-(1 << 17), 1 << 17, (m, k)).astype(float)
    B = rng.integers(-(1 << 17), 1 << 17, (k, n)).astype(float)
    A[0], B[:, 0] = float(1 << 17), float(1 << 17)       # the largest sums, of both signs: 2^34 k <= 2^51
    A[-1] = -float(1 << 17)
    assert np.array_equal(product(ctx, A, B), A @ B)
    A, B = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    g = 1e5 ** (np.arange(k) / k)
    if k < 30000:
        check(ctx, A, B)
        check(ctx, A / g, B * g[:, None])


GAUGES = [1e4, 1e6, 1e8, 1e12]


# a gauge between the environment and the site (or theta), entries of H_eff and of both updates
@pytest.mark.parametrize("fall", GAUGES)
def test_gauge_in_heff_and_environments(ctx, fall):
    import chemtensor_mojo_gb300 as ct
    rng = np.random.default_rng(int(np.log10(fall)))
    D, d, w = 130, 2, 4
    x = fall ** (np.arange(D) / D)
    rnd = lambda *s: rng.standard_normal(s)              # noqa: E731
    th, L, R, A, W = rnd(D, d, d, D), rnd(w, D, D), rnd(w, D, D), rnd(D, d, D), rnd(w, d, d, w)
    mpo = ct.MPOSite(_dt(ctx, W))
    L = L * x[:, None] * x
    R = R / x[:, None] / x
    th = th / x[:, None, None, None] * x
    A = A / x[:, None, None] * x
    tol = 3.0 * 3.0 * np.sqrt(4 * D * d) * U             # three contractions, K up to 4 D d
    cases = [(ct.apply_two_site_heff(_dt(ctx, th), _dt(ctx, L), _dt(ctx, R), mpo, mpo, ctx), od.apply_two_site_heff,
              (th, L, R, W, W)),
             (ct.update_left_environment(_dt(ctx, L), ct.MPSSite(_dt(ctx, A)), mpo, ctx), od.update_left_environment,
              (L, A, W)),
             (ct.update_right_environment(_dt(ctx, R), ct.MPSSite(_dt(ctx, A)), mpo, ctx), od.update_right_environment,
              (R, A, W))]
    for got, f, args in cases:
        ref, size = f(*args), f(*[np.abs(a) for a in args])
        err = np.abs(got.to_numpy() - ref) / size        # (the reference has the same error)
        assert err.max() <= 2.0 * tol


@pytest.mark.parametrize("fall", GAUGES)
def test_gauge_in_gradient(ctx, fall):
    """A power-of-two gauge at every bond is exact, and the gradient takes its inverse transpose."""
    import torch
    import chemtensor_mojo_gb300 as ct
    from chemtensor_mojo_gb300.autograd import energy_and_gradient
    from chemtensor_mojo_gb300.hamiltonians import bose_hubbard_arrays
    rng = np.random.default_rng(7)
    L, d, chi = 8, 4, 160
    mpo = ct.mpo_from_arrays(ctx, bose_hubbard_arrays(L, d, 1.0, 4.0, 0.5))
    dims = [min(d**i, d ** (L - i), chi) for i in range(L + 1)]
    sites = [rng.standard_normal((dims[i], d, dims[i + 1])) / np.sqrt(dims[i] * d) for i in range(L)]
    gauge = [2.0 ** np.round(np.log2(fall) * np.arange(n) / n) for n in dims]
    moved = [s / gauge[i][:, None, None] * gauge[i + 1] for i, s in enumerate(sites)]

    def grad(s):
        e, g = energy_and_gradient(mpo, [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in s], ctx=ctx)
        return float(e), [x.cpu().numpy() for x in g]
    e0, g0 = grad(sites)
    e1, g1 = grad(moved)
    assert abs(e1 - e0) <= 1e-11 * max(1.0, abs(e0))
    for i in range(L):
        back = g1[i] / gauge[i][:, None, None] * gauge[i + 1]
        assert np.abs(back - g0[i]).max() <= 1e-11 * np.abs(g0[i]).max()
