"""The mixed form's MPO leg: listed non-zero weights or all of them, rows in one or several
blocks, odd sizes, outputs along either side, non-finite operands.

Tensors of -1, 0, 1 keep every intermediate an integer that the split TF32 planes hold exactly
(below 2^21) and every sum below 2^24, so the chain must be exact.
"""
import numpy as np
import pytest

from oracle import dmrg as od

pytestmark = pytest.mark.gpu


# Dl, d, Dr, w, share of non-zero weights
@pytest.mark.parametrize("Dl,d,Dr,w,fill", [
    (33, 2, 31, 5, 0.1), (32, 2, 64, 5, 1.0), (40, 3, 35, 4, 0.1), (34, 4, 38, 6, 0.02), (33, 4, 41, 6, 0.02),
    (35, 4, 37, 6, 1.0), (65, 4, 33, 6, 0.0), (9, 4, 7, 12, 0.05), (5, 6, 6, 9, 0.5)])
@pytest.mark.parametrize("bad", [False, True])
def test_mixed_mpo_leg(ctx, Dl, d, Dr, w, fill, bad):
    import chemtensor_mojo_gb300 as ct
    rng = np.random.default_rng(Dl + 10 * d + 100 * Dr)
    dt = lambda a: ct.create_dense_tensor_from_data(ctx, a, a.shape)      # noqa: E731
    ints = lambda *s: rng.integers(-1, 2, s).astype(float)                # noqa: E731
    mpo = lambda: ints(w, d, d, w) * (rng.random((w, d, d, w)) < fill)    # noqa: E731
    th, L, R, A, W1, W2 = ints(Dl, d, d, Dr), ints(w, Dl, Dl), ints(w, Dr, Dr), ints(Dl, d, Dr), mpo(), mpo()
    W1[0, :, :, 0] = W2[0, :, :, 0] = np.eye(d)
    if bad:
        th[0, 0, 0, Dr // 2], L[0, 0, Dl // 2], A[0, 0, Dr - 1] = np.inf, np.nan, -np.inf
    with np.errstate(invalid="ignore"):
        refs = (od.apply_two_site_heff(th, L, R, W1, W2), od.update_left_environment(L, A, W1),
                od.update_right_environment(R, A, W1))
    m1, m2, site = ct.MPOSite(dt(W1)), ct.MPOSite(dt(W2)), ct.MPSSite(dt(A))
    got = (ct.apply_two_site_heff(dt(th), dt(L), dt(R), m1, m2, ctx, prec="tf32x3"),
           ct.update_left_environment(dt(L), site, m1, ctx, prec="tf32x3"),
           ct.update_right_environment(dt(R), site, m1, ctx, prec="tf32x3"))
    for g, ref in zip(got, refs):
        x = g.to_numpy()
        assert not np.isfinite(x[~np.isfinite(ref)]).any()
        ok = np.isfinite(x)
        assert bad or ok.all()
        assert np.array_equal(x[ok], ref[ok])
