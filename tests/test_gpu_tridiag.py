"""The Lanczos matrix's lowest eigenpair: bracket in scaled FP32 and minors, last steps by pivots.

Against LAPACK on the same alpha and beta: bisection and dstev each err by a few n eps |T|, so
1e-13 |T| for up to 64 steps.  Powers of two scale the problem, up to where the bracket is not used.
"""
import numpy as np
import pytest

from oracle import dmrg as od

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 2, 3, 20, 32, 33, 64])
@pytest.mark.parametrize("exp", [0, 60, 480])
def test_lowest_eigenpair(ctx, steps, exp):
    import chemtensor_mojo_gb300 as ct
    rng = np.random.default_rng(steps)
    dt = lambda a: ct.create_dense_tensor_from_data(ctx, a, a.shape)   # noqa: E731
    sym = lambda a: a + a.transpose(0, 2, 1)                           # noqa: E731
    th, L, R = rng.standard_normal((8, 2, 2, 8)), sym(rng.standard_normal((3, 8, 8))), sym(rng.standard_normal((3, 8, 8)))
    W = rng.standard_normal((3, 2, 2, 3))
    W = np.ldexp(W + W.transpose(0, 2, 1, 3), exp // 2)
    info = ct.dmrg.LanczosInfo(0, [], [])
    E, v = ct.lanczos_two_site_optimize(dt(th), dt(L), dt(R), ct.MPOSite(dt(W)), ct.MPOSite(dt(W)), ctx,
                                        max_iter=steps, tol=0.0, max_rotations=0, reorth=True, info=info)
    n = info.numiter
    assert n == steps
    T = np.diag(np.ldexp(info.alpha[:n], -exp)) + np.diag(np.ldexp(info.beta[:n - 1], -exp), 1)
    T = T + np.triu(T, 1).T
    ev = np.linalg.eigvalsh(T)
    assert abs(np.ldexp(E, -exp) - ev[0]) <= 1e-13 * np.abs(ev).max()
    x = v.to_numpy()
    assert abs(np.linalg.norm(x) - 1.0) < 1e-12
    Wu = np.ldexp(W, -(exp // 2))
    assert abs((x * od.apply_two_site_heff(x, L, R, Wu, Wu)).sum() - ev[0]) <= 1e-10 * np.abs(ev).max()
