"""GPU test of the density's diagonal sums at sizes where the pair-block walk
has edges: one occupied orbital, fewer rows than warps, v just below, at and
above a warp's 32 columns -- against the autograd oracle (the tolerance of the
existing density test, 1e-10 on equations converged to 1e-11)."""
import numpy as np
import pytest

import acesb200 as ab
from oracle import ccsd, lambda_ad
from oracle.ccsd import Blocks
from oracle.hamiltonian import synthetic
from test_gpu_ccsd import setup_lists

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    lib = ab.load()
    lib.init(0)
    return lib


@pytest.mark.parametrize("o,v", [(1, 4), (2, 7), (3, 31), (2, 32), (2, 33)])
def test_density_matches_oracle(lib, o, v):
    ham = synthetic(o, v, 24, seed=o + v)
    setup_lists(lib, ham)
    lib.xvcc(cc_conv=11, cc_maxcyc=90, cc_exporder=6)
    lib.xlambda(cc_conv=11, cc_maxcyc=90, cc_exporder=6)
    lib.xdens()
    D = lib.getrec("DENSMAT", (o + v) ** 2).reshape(o + v, o + v)
    B = Blocks(ham)
    r = ccsd.run_ccsd(ham, cc_conv=12, maxcyc=120, exporder=6)
    l1, l2 = lambda_ad.solve_lambda(B, r["t1"], r["t2"])
    np.testing.assert_allclose(D, lambda_ad.density(B, r["t1"], r["t2"], l1, l2), atol=1e-10)
