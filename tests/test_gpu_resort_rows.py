"""Resorts whose rows keep unit stride but no multiple of four elements: a warp
per row from 64 elements and 2368 rows on.  CCSD amplitudes on both sides of
these limits (63..70 virtuals; 64 and 68 take the aligned kernel) against the
FP64 oracle after the same cycles: FP64 to 1e-11 (rounding), split precision to
1e-6 in the amplitudes (relative error 2^-17 of single operands)."""
import numpy as np
import pytest

import acesb200 as ab
from oracle import ccsd
from oracle.hamiltonian import synthetic
from test_gpu_ccsd import read_amplitudes, setup_lists

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("o,v", [(6, 65), (7, 63), (7, 65), (7, 67), (7, 70)])
def test_row_resorts_match_oracle(o, v):
    lib = ab.load()
    ham = synthetic(o, v, 40, seed=7 * v + o, bscale=0.5)
    _, dpd = setup_lists(lib, ham)
    ref = ccsd.run_ccsd(ham, cc_conv=8, maxcyc=60, exporder=5)
    for prec, tol in ((ab.PREC_FP64, 1e-11), (ab.PREC_BF16X3, 1e-6)):
        cfg = lib.xvcc(cc_conv=8, cc_maxcyc=60, cc_exporder=5, precision=prec)
        assert cfg.converged == 1
        t1, t2 = read_amplitudes(lib, dpd, o, v)
        np.testing.assert_allclose(t1, ref["t1"], atol=tol)
        np.testing.assert_allclose(t2, ref["t2"], atol=tol)
