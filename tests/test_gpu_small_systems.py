"""The smallest systems, and odd o v (copies between arrays at 8-byte offsets)
beside even ones: CCSD amplitudes against the FP64 oracle after the same
cycles, to the tolerance of the other oracle comparisons."""
import numpy as np
import pytest

import acesb200 as ab
from oracle import ccsd
from oracle.hamiltonian import synthetic
from test_gpu_ccsd import read_amplitudes, setup_lists

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("o,v", [(1, 1), (1, 2), (2, 1), (3, 5), (3, 34), (5, 33)])
def test_small_systems_match_oracle(o, v):
    lib = ab.load()
    ham = synthetic(o, v, 2 * (o + v), seed=17 * v + o, bscale=0.5)
    _, dpd = setup_lists(lib, ham)
    cfg = lib.xvcc(cc_conv=9, cc_maxcyc=60, cc_exporder=5)
    ref = ccsd.run_ccsd(ham, cc_conv=9, maxcyc=60, exporder=5)
    assert cfg.converged == 1
    assert abs(cfg.e_ccsd - ref["e_final"]) < 1e-11
    t1, t2 = read_amplitudes(lib, dpd, o, v)
    np.testing.assert_allclose(t1, ref["t1"], atol=1e-11)
    np.testing.assert_allclose(t2, ref["t2"], atol=1e-11)
