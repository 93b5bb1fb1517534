"""The FP64 MPO leg over listed non-zero weights: column tiles of 32 that cross slabs, rows in one
or several chunks, the wide form beyond K = 192, dense, zero and non-finite operands.

Small-integer tensors: the chain is exact in FP64, so the comparison is too.
"""
import numpy as np
import pytest

from oracle import dmrg as od

pytestmark = pytest.mark.gpu


def _dt(ctx, a):
    import chemtensor_mojo_gb300 as ct
    return ct.create_dense_tensor_from_data(ctx, a, a.shape)


# Dl, d, Dr, w, share of non-zero weights: K = d^2 w of the two-site leg from 4 to 576
@pytest.mark.parametrize("Dl,d,Dr,w,fill", [
    (1, 2, 1, 1, 1.0), (5, 2, 7, 5, 0.1), (16, 2, 2, 5, 0.0), (3, 2, 33, 5, 0.1), (9, 4, 11, 6, 0.02),
    (7, 4, 5, 12, 1.0), (6, 5, 5, 9, 0.3), (4, 8, 5, 9, 0.1)])
@pytest.mark.parametrize("bad", [False, True])
def test_mpo_leg_matches_oracle(ctx, Dl, d, Dr, w, fill, bad):
    import chemtensor_mojo_gb300 as ct
    rng = np.random.default_rng(Dl + 10 * d + 100 * Dr)
    ints = lambda *s: rng.integers(-4, 5, s).astype(float)   # noqa: E731
    mpo = lambda: ints(w, d, d, w) * (rng.random((w, d, d, w)) < fill)   # noqa: E731
    th, L, R, A, W1, W2 = ints(Dl, d, d, Dr), ints(w, Dl, Dl), ints(w, Dr, Dr), ints(Dl, d, Dr), mpo(), mpo()
    W1[0, :, :, 0] = W2[0, :, :, 0] = np.eye(d)
    if bad:
        th[0, 0, 0, Dr // 2], L[0, 0, Dl // 2], A[0, 0, Dr - 1] = np.inf, np.nan, -np.inf
    with np.errstate(invalid="ignore"):
        refs = (od.apply_two_site_heff(th, L, R, W1, W2), od.update_left_environment(L, A, W1),
                od.update_right_environment(R, A, W1))
    m1, m2, site = ct.MPOSite(_dt(ctx, W1)), ct.MPOSite(_dt(ctx, W2)), ct.MPSSite(_dt(ctx, A))
    got = (ct.apply_two_site_heff(_dt(ctx, th), _dt(ctx, L), _dt(ctx, R), m1, m2, ctx),
           ct.update_left_environment(_dt(ctx, L), site, m1, ctx),
           ct.update_right_environment(_dt(ctx, R), site, m1, ctx))
    for g, ref in zip(got, refs):
        ok = np.isfinite(ref)
        assert np.array_equal(np.isfinite(g.to_numpy()), ok)
        assert np.array_equal(g.to_numpy()[ok], ref[ok])
