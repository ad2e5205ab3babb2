"""GPU test of the tensor-core contraction's tail split: outputs whose last,
partly filled wave of 128 x 144 tiles is cut along K (more than 148 tiles, a
remainder, K of several 512-element chunks), with ragged M, N and K, either
side the smaller one (tile order) and beta 0, 1 and general.

Tolerance: that of the split products, |C - C_fp64| <= 4e-5 (|A| |B|)_ij (each
product within 2^-16, FP32 sums of at most 512 K elements); the FP64 sums over
slices add nothing at that scale.
"""
import pytest
import torch

import acesb200 as ab

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    lib = ab.load()
    lib.init(0)
    return lib


@pytest.mark.parametrize("m,n,k", [(1300, 2200, 4000), (2561, 1297, 4099), (20000, 150, 9000),
                                   (150, 20000, 9001), (2433, 1153, 40001)])
@pytest.mark.parametrize("beta", [0.0, 1.0, 0.5])
def test_tail_split_error_bound(lib, m, n, k, beta):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    A = torch.randn((m, k), generator=g, dtype=torch.float64, device="cuda")
    B = torch.randn((n, k), generator=g, dtype=torch.float64, device="cuda")
    C0 = torch.randn((n, m), generator=g, dtype=torch.float64, device="cuda")
    C = C0.clone() if beta else torch.full_like(C0, float("nan"))
    lib.xgemm("T", "N", m, n, k, 0.9, A.data_ptr(), k, B.data_ptr(), k, beta, C.data_ptr(), m,
              precision=ab.PREC_BF16X3)
    ref = 0.9 * (B @ A.T) + (beta * C0 if beta else 0.0)
    bound = 4e-5 * 0.9 * (B.abs() @ A.abs().T) + 1e-12
    assert bool(((C - ref).abs() <= bound).all())
    again = C0.clone()
    lib.xgemm("T", "N", m, n, k, 0.9, A.data_ptr(), k, B.data_ptr(), k, beta, again.data_ptr(), m,
              precision=ab.PREC_BF16X3)
    assert torch.equal(again, C)   # the slices are added in a fixed order
