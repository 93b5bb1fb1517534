"""Work that runs in clusters of up to 16 CTAs, where clusters have to be smaller or are not to be had
(CTDMRG_MAX_CLUSTER): the Lanczos step in separate launches, the exact SVD in smaller clusters or one
CTA.  The arithmetic is the same, so every bit is.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lanczos(ctx, Dl, d, Dr, form, symmetric=True, iters=10):
    import chemtensor_mojo_gb300 as ct
    rng = np.random.default_rng(Dl + d + Dr)
    dt = lambda a: ct.create_dense_tensor_from_data(ctx, a, a.shape)   # noqa: E731
    th, L, R = (rng.standard_normal(s) for s in ((Dl, d, d, Dr), (3, Dl, Dl), (3, Dr, Dr)))
    W = rng.standard_normal((3, d, d, 3))
    if symmetric:
        L, R, W = L + L.transpose(0, 2, 1), R + R.transpose(0, 2, 1), W + W.transpose(0, 2, 1, 3)
    info = ct.dmrg.LanczosInfo(0, [], [])
    E, v = ct.lanczos_two_site_optimize(dt(th), dt(L), dt(R), ct.MPOSite(dt(W)), ct.MPOSite(dt(W)), ctx, max_iter=iters,
                                        tol=1e-10, prec="tf32x3" if form == "mixed" else "fp64", max_rotations=0,
                                        reorth=form != "plain", info=info)
    return (E, info.numiter, list(info.alpha), list(info.beta), v.to_numpy()), (th, L, R, W)


def same(a, b):
    return all(np.array_equal(np.asarray(x), np.asarray(y)) for x, y in zip(a, b))


@pytest.mark.parametrize("Dl,d,Dr", [(16, 2, 33), (33, 3, 31), (64, 2, 128)])   # 2, 5 and 16 blocks
@pytest.mark.parametrize("form", ["plain", "reorth", "mixed"])
def test_lanczos_without_large_clusters(ctx, monkeypatch, Dl, d, Dr, form):
    ref, _ = lanczos(ctx, Dl, d, Dr, form)
    for most in ("8", "1"):
        monkeypatch.setenv("CTDMRG_MAX_CLUSTER", most)
        got, _ = lanczos(ctx, Dl, d, Dr, form)
        assert same(got, ref)


@pytest.mark.parametrize("m,n", [(2, 3), (31, 33), (64, 64), (96, 96), (96, 129), (4, 257), (300, 40)])
def test_exact_svd_without_large_clusters(ctx, monkeypatch, m, n):
    import chemtensor_mojo_gb300 as ct
    M = np.random.default_rng(m + n).standard_normal((m, n))

    def run():
        U, S, Vt, _ = ct.dense_tensor_svd_trunc(ct.create_dense_tensor_from_data(ctx, M, M.shape), ctx, 1 << 30, 0.0)
        return U.to_numpy(), S.to_numpy(), Vt.to_numpy()
    ref = run()
    for most in ("8", "3", "1"):
        monkeypatch.setenv("CTDMRG_MAX_CLUSTER", most)
        assert same(run(), ref)
