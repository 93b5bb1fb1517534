"""Scratch of the FP64-form products on the tensor cores: reported, kept within the workspace limit
beside the arena, given back, grown in few steps, and the same products with and without a capture.

Small-integer operands: the products are exact on either path.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ints(ctx, seed, *shape):
    import chemtensor_mojo_gb300 as ct
    a = np.random.default_rng(seed).integers(-9, 10, shape).astype(float)
    return a, ct.create_dense_tensor_from_data(ctx, a, a.shape)


def _theta(ctx, m, n, k):
    import chemtensor_mojo_gb300 as ct
    a, da = _ints(ctx, m + k, m // 2, 2, k)
    b, db = _ints(ctx, n + k, k, 2, n // 2)
    got = ct.build_two_site_theta(ct.MPSSite(da), ct.MPSSite(db), ctx).to_numpy().reshape(m, n)
    assert np.array_equal(got, a.reshape(m, k) @ b.reshape(k, n))


def _heff(ctx, D, prec="fp64"):
    import chemtensor_mojo_gb300 as ct
    (_, th), (_, L), (_, R), (_, W) = [_ints(ctx, D + i, *s) for i, s in
                                       enumerate([(D, 2, 2, D), (5, D, D), (5, D, D), (5, 2, 2, 5)])]
    return ct.apply_two_site_heff(th, L, R, ct.MPOSite(W), ct.MPOSite(W), ctx, prec=prec).to_numpy()


def test_scratch_is_reported_and_given_back():
    import chemtensor_mojo_gb300 as ct
    ctx = ct.DeviceContext(0)
    _theta(ctx, 256, 256, 256)                       # no arena, residue planes of 2 x 256 x 256
    used = ctx.workspace_bytes()
    assert used >= 2 * 16 * 256 * 256 * 2
    ctx.set_workspace_limit(used)
    _theta(ctx, 256, 256, 256)
    assert ctx.workspace_bytes() == used             # still within the limit
    ctx.set_workspace_limit(used // 2)
    assert ctx.workspace_bytes() <= used // 2
    _theta(ctx, 256, 256, 256)                       # on FP64 FMAs
    assert ctx.workspace_bytes() <= used // 2
    ctx.set_workspace_limit(0)
    _theta(ctx, 256, 256, 256)
    assert ctx.workspace_bytes() >= 2 * 16 * 256 * 256 * 2


def test_arena_has_the_limit_to_itself():
    import chemtensor_mojo_gb300 as ct
    probe = ct.DeviceContext(0)
    probe.set_workspace_limit(1)                     # refuses the arena, so nothing is reserved
    with pytest.raises(ct.CTDMRGError):
        _heff(probe, 128)
    probe.set_workspace_limit(0)
    ref = _heff(probe, 128)
    limit = 12 << 20                                 # room for the apply's arena (5.3 MB) or for the residues' scratch (8.3)
    ctx = ct.DeviceContext(0)
    ctx.set_workspace_limit(limit)
    _theta(ctx, 256, 256, 200)
    assert 0 < ctx.workspace_bytes() <= limit
    assert np.array_equal(_heff(ctx, 128), ref)      # as with no residues before it
    assert ctx.workspace_bytes() <= limit


def test_growing_bonds_grow_the_scratch_in_few_steps():
    import chemtensor_mojo_gb300 as ct
    ctx = ct.DeviceContext(0)
    sizes = set()
    for k in range(160, 330, 6):
        _theta(ctx, 2 * (k // 2), 2 * (k // 2), k)
        sizes.add(ctx.workspace_bytes())
    assert len(sizes) <= 8                           # 4.3 times as much in steps of a quarter


@pytest.mark.parametrize("D", [160])
def test_captured_apply_without_scratch_computes_as_the_eager_one(D):
    import chemtensor_mojo_gb300 as ct
    gen = torch.Generator(device="cuda").manual_seed(D)
    rnd = lambda *s: ct.DenseTensor(torch.randn(s, dtype=torch.float64, device="cuda", generator=gen), list(s))  # noqa: E731
    th, L, R, W = rnd(D, 2, 2, D), rnd(5, D, D), rnd(5, D, D), ct.MPOSite(rnd(5, 2, 2, 5))
    ref = ct.apply_two_site_heff(th, L, R, W, W, ct.DeviceContext(0)).storage.clone()
    ctx = ct.DeviceContext(0)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        ct.apply_two_site_heff(th, L, R, W, W, ctx, prec="tf32x3")   # the arena alone
        s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            out = ct.apply_two_site_heff(th, L, R, W, W, ctx).storage
        for n in (512, 768):                         # eager products outgrow the graph's scratch (no arena here)
            _theta(ctx, n, n, n)
            out.fill_(float("nan"))
            graph.replay()
            s.synchronize()
            assert torch.equal(out, ref)
