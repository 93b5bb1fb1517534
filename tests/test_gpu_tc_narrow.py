"""64-wide tensor-core tiles: the last product that fills the SMs with them and the first beyond, one
tile, ragged edges and K from less than a chunk to many.

Operands of -2 .. 2: exact in TF32, sums below 2^24, so the product must be exact.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [64, 65, 448, 512, 513])
@pytest.mark.parametrize("rows,k", [(1, 1), (128, 64), (129, 65), (0, 160)])
def test_narrow_tiles(ctx, rows, cols, k):
    import chemtensor_mojo_gb300 as ct
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    m = rows or 128 * (sms // 8)   # 512 columns: one 64-wide tile per SM (8 per row of tiles)
    rng = np.random.default_rng(m + cols + k)
    A, B = (rng.integers(-2, 3, s).astype(float) for s in ((m, k), (k, cols)))
    a, b, c = (ct.create_dense_tensor_from_data(ctx, x, x.shape) for x in (A, B, np.zeros((m, cols))))
    ctx.call("ct_gemm", 1, 0, 0, m, cols, k, 1.0, a.storage.data_ptr(), k, b.storage.data_ptr(), cols, 0.0,
             c.storage.data_ptr(), cols)
    assert np.array_equal(c.to_numpy(), A @ B)
