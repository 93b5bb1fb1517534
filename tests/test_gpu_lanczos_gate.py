"""The mixed Lanczos step's second Gram-Schmidt pass, in one launch and in separate ones.

With operands that are not symmetric the recurrence leaves w with components along the whole basis, as
large as beta, so the pass is due after every step but the first two: against the FP32 copy of the
basis, or against the FP64 one with CTDMRG_LANCZOS_REDO32=0.  That each of them ran shows in the
results: the two settings must differ.  In one launch the FP64 pass reads w under another mapping of
elements to threads than the pass that wrote it (lengths that are multiples of four, even, odd).  Both
forms do the same arithmetic, so their bits are the same.  Against the oracle, which reorthogonalises
in FP64: 1e-5 of the largest coefficient (TF32x3 products of K up to 384, 1e-6 each over ten steps).
"""
import numpy as np
import pytest

from oracle import dmrg as od
from test_gpu_clusters import lanczos, same

pytestmark = pytest.mark.gpu


# blocks and N mod 4: 1 / 0, 3 / 0, 4 / 2, 5 / 3, 16 / 0
@pytest.mark.parametrize("Dl,d,Dr", [(16, 2, 32), (23, 2, 61), (22, 3, 31), (33, 3, 31), (64, 2, 128)])
def test_second_pass(ctx, monkeypatch, Dl, d, Dr):
    results = []
    for redo32 in ("1", "0"):
        monkeypatch.setenv("CTDMRG_LANCZOS_REDO32", redo32)
        monkeypatch.delenv("CTDMRG_MAX_CLUSTER", raising=False)
        fused, (th, L, R, W) = lanczos(ctx, Dl, d, Dr, "mixed", symmetric=False)
        monkeypatch.setenv("CTDMRG_MAX_CLUSTER", "0")
        separate, _ = lanczos(ctx, Dl, d, Dr, "mixed", symmetric=False)
        assert same(fused, separate)
        results.append(fused)
    assert not same(*results)
    tr = od.LanczosTrace()
    od.lanczos_two_site_optimize(th, L, R, W, W, 10, 1e-10, eig="exact", trace=tr, reorth=True)
    for r in results:
        assert r[1] == tr.numiter == 10
        scale = max(np.abs(tr.alpha).max(), np.abs(tr.beta).max())
        assert np.abs(np.array(r[2]) - tr.alpha).max() <= 1e-5 * scale
        assert np.abs(np.array(r[3]) - tr.beta).max() <= 1e-5 * scale
