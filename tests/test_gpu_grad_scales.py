"""Environments renormalised on the device: site tensors scaled by powers of two.

Scaling site i by 2^e_i leaves the energy alone and divides its gradient by 2^e_i; powers of two
commute with every rounding on the way, so both must come out the same to the last bit, however
far the unnormalised chain over- or underflows.
"""
import numpy as np
import pytest
import torch

from oracle import hamiltonians as oh
from oracle import rng as orng

pytestmark = pytest.mark.gpu


def _sites(L, chi):
    mps, _ = orng.create_random_mps_c_compatible(L, 2, chi, 3)
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in mps]


@pytest.mark.parametrize("L,chi,ckpt", [(2, 2, 0), (9, 8, 0), (9, 8, 4), (12, 16, 3)])
def test_gradient_of_scaled_sites(ctx, L, chi, ckpt):
    import chemtensor_mojo_gb300 as ct
    from chemtensor_mojo_gb300.autograd import energy_and_gradient
    mpo = ct.mpo_from_arrays(ctx, oh.heisenberg_xxz(L, J=1.0, D=0.7, h=0.1))
    sites = _sites(L, chi)
    E, grads = energy_and_gradient(mpo, sites, checkpoint_every=ckpt, ctx=ctx)
    exps = np.random.default_rng(L).integers(-150, 150, L)
    scaled = [torch.from_numpy(np.ldexp(s.cpu().numpy(), int(e))).cuda() for s, e in zip(sites, exps)]
    E2, grads2 = energy_and_gradient(mpo, scaled, checkpoint_every=ckpt, ctx=ctx)
    assert E2 == E
    for g, g2, e in zip(grads, grads2, exps):
        assert np.array_equal(np.ldexp(g2.cpu().numpy(), int(e)), g.cpu().numpy())


@pytest.mark.parametrize("site", [0, 4, 8])
def test_nonfinite_site_is_an_error(ctx, site):
    import chemtensor_mojo_gb300 as ct
    from chemtensor_mojo_gb300 import _lib
    from chemtensor_mojo_gb300.autograd import energy_and_gradient
    mpo = ct.mpo_from_arrays(ctx, oh.heisenberg_xxz(9, J=1.0, D=0.7, h=0.1))
    sites = _sites(9, 8)
    good = energy_and_gradient(mpo, sites, ctx=ctx)[0]
    bad = [s.clone() for s in sites]
    bad[site].view(-1)[0] = float("nan")
    with pytest.raises(ct.CTDMRGError) as err:
        energy_and_gradient(mpo, bad, ctx=ctx)
    assert err.value.status == _lib.CT_ERR_NONFINITE
    assert energy_and_gradient(mpo, sites, ctx=ctx)[0] == good   # the handle is usable again
