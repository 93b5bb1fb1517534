"""The Lanczos step's vector work in one launch (up to 32768 elements, 16 blocks) and in separate
ones beyond, odd and even lengths, in the three forms, against the oracle.

Tolerances as for the other Lanczos tests: FP64 alpha and beta to 1e-9 of the largest, the energy
to 1e-10; the mixed form's energy to 1e-6.
"""
import numpy as np
import pytest

from oracle import dmrg as od

pytestmark = pytest.mark.gpu


# N = 1, 2 blocks, odd, the last fused and the first separate length
@pytest.mark.parametrize("Dl,d,Dr", [(16, 2, 32), (16, 2, 33), (33, 3, 31), (64, 2, 128), (64, 2, 129)])
@pytest.mark.parametrize("form", ["plain", "reorth", "mixed"])
def test_lanczos_step_lengths(ctx, Dl, d, Dr, form):
    import chemtensor_mojo_gb300 as ct
    rng = np.random.default_rng(Dl + d + Dr)
    dt = lambda a: ct.create_dense_tensor_from_data(ctx, a, a.shape)   # noqa: E731
    sym = lambda a: a + a.transpose(0, 2, 1)                           # noqa: E731
    th, L, R = rng.standard_normal((Dl, d, d, Dr)), sym(rng.standard_normal((3, Dl, Dl))), sym(rng.standard_normal((3, Dr, Dr)))
    W = rng.standard_normal((3, d, d, 3))
    W = W + W.transpose(0, 2, 1, 3)
    reorth = form != "plain"
    tr = od.LanczosTrace()
    E_ref, v_ref = od.lanczos_two_site_optimize(th, L, R, W, W, 10, 1e-10, eig="exact", trace=tr, reorth=reorth)
    info = ct.dmrg.LanczosInfo(0, [], [])
    E, v = ct.lanczos_two_site_optimize(dt(th), dt(L), dt(R), ct.MPOSite(dt(W)), ct.MPOSite(dt(W)), ctx, max_iter=10,
                                        tol=1e-10, prec="tf32x3" if form == "mixed" else "fp64", max_rotations=0,
                                        reorth=reorth, info=info)
    assert info.numiter == tr.numiter
    if form == "mixed":
        assert abs(E - E_ref) <= 1e-6 * max(1.0, abs(E_ref))
        return
    scale = np.abs(tr.alpha).max()
    assert np.allclose(info.alpha, tr.alpha, rtol=1e-9, atol=1e-9 * scale)
    assert np.allclose(info.beta, tr.beta, rtol=1e-9, atol=1e-9 * scale)
    assert abs(E - E_ref) <= 1e-10 * max(1.0, abs(E_ref))
    assert abs(abs(v.to_numpy().reshape(-1) @ v_ref.reshape(-1)) - 1.0) < 1e-8
