"""Applies captured into a CUDA graph: launches that overlap their predecessors keep stream order
when replayed, and a scratch buffer outgrown after the capture stays valid for the graph.

Replays must repeat the captured arithmetic: bit-identical to the eager call on the same inputs.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,D", [("fp64", 24), ("fp64", 160), ("tf32x3", 64), ("tf32x3", 65)])
def test_captured_heff_apply(prec, D):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import chemtensor_mojo_gb300 as ct
    ctx = ct.DeviceContext(0)
    gen = torch.Generator(device="cuda").manual_seed(D)
    rnd = lambda *s: ct.DenseTensor(torch.randn(s, dtype=torch.float64, device="cuda", generator=gen), list(s))  # noqa: E731
    th, L, R, W = rnd(D, 2, 2, D), rnd(5, D, D), rnd(5, D, D), ct.MPOSite(rnd(5, 2, 2, 5))
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        ref = ct.apply_two_site_heff(th, L, R, W, W, ctx, prec=prec).storage.clone()
        s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            out = ct.apply_two_site_heff(th, L, R, W, W, ctx, prec=prec).storage
        # a larger product afterwards outgrows the residues' scratch buffer
        a = ct.MPSSite(rnd(256, 2, 512))
        ct.build_two_site_theta(a, ct.MPSSite(rnd(512, 2, 256)), ctx)
        for _ in range(3):
            out.fill_(float("nan"))
            graph.replay()
            s.synchronize()
            assert torch.equal(out, ref)
    assert np.isfinite(ref.cpu().numpy()).all()
