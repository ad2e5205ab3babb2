"""The ladder's U+/U- taken by pair irrep from the vvvv list's blocks.

Sizes at the edges of the kernel's 32 x 32 pair tiles: irreps with none, one,
31..33 and a little over 64 pairs, and irreps without antisymmetric pairs.
Amplitudes against the FP64 oracle after the same cycles, to the tolerance of
the other oracle comparisons (1e-11: rounding of some 10 cycles).
"""
import numpy as np
import pytest

import acesb200 as ab
from oracle import ccsd
from oracle.hamiltonian import synthetic
from test_gpu_ccsd import read_amplitudes, setup_lists

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("o,v,irreps", [(1, 2, 2), (2, 3, 8), (2, 11, 2), (3, 16, 4), (2, 22, 8)])
def test_symmetry_blocked_ladder_matches_oracle(o, v, irreps):
    lib = ab.load()
    ham = synthetic(o, v, 2 * (o + v), seed=31 * v + o, irreps=irreps, bscale=0.3)
    _, dpd = setup_lists(lib, ham)
    cfg = lib.xvcc(cc_conv=9, cc_maxcyc=60, cc_exporder=5)
    ref = ccsd.run_ccsd(ham, cc_conv=9, maxcyc=60, exporder=5)
    assert cfg.converged == 1
    assert abs(cfg.e_ccsd - ref["e_final"]) < 1e-11
    _, t2 = read_amplitudes(lib, dpd, o, v)
    np.testing.assert_allclose(t2, ref["t2"], atol=1e-11)
