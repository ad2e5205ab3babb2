"""GPU test of the FP64 contraction kernel's tiles through aces_xgemm: outputs
just below, at and above the tile edges (16, 32, 64), short sides of 1 to 33,
K at and around the 16-wide k tile and long enough for split K, odd leading
dimensions (8-byte copies), both output orientations.

Tolerance: a sum of K products in any order has an error of at most
K u sum |a||b| (u = 2^-53), the reference product the same, and alpha, beta
and the two roundings of the update add 4 u (|result| + |beta C|).
"""
import numpy as np
import pytest
import torch

import acesb200 as ab

pytestmark = pytest.mark.gpu

SHAPES = [(33, 257, 33), (64, 129, 48), (65, 127, 47), (96, 97, 100), (128, 64, 1000),
          (129, 191, 17 * 16 + 1), (257, 255, 64), (1000, 33, 129), (4097, 3, 600),
          (4095, 7, 601), (2049, 8, 40), (31, 3000, 50), (16, 5000, 2000), (17, 700, 33),
          (1, 9000, 100), (9001, 1, 99), (32, 320, 5001), (130, 15, 20000), (640, 640, 500)]


@pytest.fixture(scope="module")
def lib():
    lib = ab.load()
    lib.init(0)
    return lib


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("ta,tb,alpha,beta", [("T", "N", 1.0, 0.0), ("N", "T", -0.7, 1.3)])
def test_tile_edges(lib, m, n, k, ta, tb, alpha, beta):
    g = torch.Generator().manual_seed(m * 7 + n * 3 + k)
    A = torch.randn((m, k), generator=g, dtype=torch.float64)
    B = torch.randn((k, n), generator=g, dtype=torch.float64)
    C0 = torch.randn((m, n), generator=g, dtype=torch.float64)
    dA = (A.T if ta == "N" else A).contiguous().cuda()
    dB = (B.T if tb == "N" else B).contiguous().cuda()
    dC = C0.T.contiguous().cuda()
    lib.xgemm(ta, tb, m, n, k, alpha, dA.data_ptr(), m if ta == "N" else k, dB.data_ptr(),
              k if tb == "N" else n, beta, dC.data_ptr(), m)
    ref = alpha * (A @ B) + beta * C0
    u = 2.0 ** -53
    tol = 2 * k * u * abs(alpha) * (A.abs() @ B.abs()) + 4 * u * (ref.abs() + abs(beta) * C0.abs())
    err = (dC.cpu().T - ref).abs()
    assert bool((err <= tol).all()), float((err / tol).max())
    if beta == 0.0:  # the output's old content must not matter
        dC.fill_(float("nan"))
        lib.xgemm(ta, tb, m, n, k, alpha, dA.data_ptr(), k, dB.data_ptr(), k, beta,
                  dC.data_ptr(), m)
        assert np.isfinite(dC.cpu().numpy()).all()


def test_a_nan_or_infinity_reaches_its_row_and_column_only(lib):
    m, n, k = 130, 70, 90
    A, B = torch.ones((m, k), dtype=torch.float64), torch.ones((n, k), dtype=torch.float64)
    A[65, 89] = float("nan")
    B[64, 0] = float("inf")
    dA, dB = A.cuda(), B.cuda()
    dC = torch.zeros((n, m), dtype=torch.float64, device="cuda")
    lib.xgemm("T", "N", m, n, k, 1.0, dA.data_ptr(), k, dB.data_ptr(), k, 0.0, dC.data_ptr(), m)
    np.testing.assert_array_equal(dC.cpu().numpy(), (A @ B.T).T.numpy())
