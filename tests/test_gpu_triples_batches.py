"""GPU test of the batched FP64 (T): odd and even sizes (8- and 16-byte copies,
partial tiles, nocc below and above a k tile) against the oracle, and a
system whose triplets need more than one batch (364 slots of 17.6 MB against
the 4 GB budget) against its shards, which need one each.

Tolerances: those of the existing (T) tests: 1e-9 relative to the oracle on
amplitudes converged to 1e-10, 1e-11 relative between summation orders.
"""
import pytest

import acesb200 as ab
from oracle import ccsd
from oracle.hamiltonian import synthetic
from oracle.triples import triples
from test_gpu_ccsd import setup_lists

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    lib = ab.load()
    lib.init(0)
    return lib


@pytest.mark.parametrize("o,v", [(1, 5), (2, 33), (3, 32), (4, 19), (9, 8)])
def test_fp64_triples_match_the_oracle(lib, o, v):
    ham = synthetic(o, v, 30, seed=o * 10 + v)
    setup_lists(lib, ham)
    ref = ccsd.run_ccsd(ham, cc_conv=10, maxcyc=80, exporder=5)
    e4, e5 = triples(ham, ref["t1"], ref["t2"])
    c = lib.xvcc(cc_conv=10, cc_maxcyc=80, triples=1)
    assert abs(c.e_t4 - e4) < 1e-12 + 1e-9 * abs(e4)
    assert abs(c.e_st5 - e5) < 1e-13 + 1e-9 * abs(e5)


def test_two_batches_add_up(lib):
    ham = synthetic(12, 130, 60, seed=3, bscale=0.4)
    setup_lists(lib, ham)
    kw = dict(cc_conv=8, cc_maxcyc=60, triples=1)
    full = lib.xvcc(**kw)
    parts = [lib.xvcc(triples_rank=r, triples_nranks=2, **kw) for r in range(2)]
    assert abs(sum(p.e_t4 for p in parts) - full.e_t4) < 1e-13 + 1e-11 * abs(full.e_t4)
    assert abs(sum(p.e_st5 for p in parts) - full.e_st5) < 1e-14 + 1e-11 * abs(full.e_st5)
