"""The paired tensor-core GEMM (two CTAs on one 256-row tile): ragged rows, columns and K, one and
several tiles per pair, both orientations.

Operands of -2 .. 2 are exact in TF32 and every sum is below 2^24, so the product must be exact.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(4096, 1024, 1024), (4070, 1010, 1030), (4864, 1024, 1056), (4740, 1000, 2000),
                                   (5120, 3192, 1024)])
@pytest.mark.parametrize("alpha_beta", [False, True])
def test_paired_products(ctx, m, n, k, alpha_beta):
    import chemtensor_mojo_gb300 as ct
    from chemtensor_mojo_gb300 import _lib
    import torch
    plan = (C.c_int64 * 8)()
    _lib.check(_lib.load().ct_tc_gemm_plan(m, n, k, torch.cuda.get_device_properties(0).multi_processor_count, plan),
               "ct_tc_gemm_plan")
    rows = n if plan[1] else m
    assert plan[0] >= 224 and plan[4] == 0 and -(-rows // 128) % 2 == 0   # the paired kernel's shapes
    rng = np.random.default_rng(m + n + k)
    A, B, X = (rng.integers(-2, 3, s).astype(float) for s in ((m, k), (k, n), (m, n)))
    a, b, c = (ct.create_dense_tensor_from_data(ctx, x, x.shape) for x in (A, B, X))
    alpha, beta = (-0.5, 2.0) if alpha_beta else (1.0, 0.0)
    ctx.call("ct_gemm", 1, 0, 0, m, n, k, alpha, a.storage.data_ptr(), k, b.storage.data_ptr(), n, beta,
             c.storage.data_ptr(), n)
    assert np.array_equal(c.to_numpy(), alpha * (A @ B) + beta * X)
