"""GPU test of the wide tiles of the batched (T) class launches at the
edges of their range against the 144-wide tiles: v = 128 and 192 (one tile
across N, the narrowest and the widest), odd v (rows of W that start on
4-byte boundaries), v = 170 and 176 (8- and 16-byte boundaries), nocc with
partial K steps (3, 16, 17) and v^2 ragged against the tile rows.

Both widths do the same products in the same order per element; only the
order in which the three classes' FP32 sums reach W differs, so the energies
agree to the bound of the narrow/wide comparison at v = 160, 1e-9 relative.
"""
import pytest

import acesb200 as ab
from oracle.hamiltonian import synthetic
from test_gpu_ccsd import setup_lists

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    lib = ab.load()
    lib.init(0)
    return lib


@pytest.mark.parametrize("o,v", [(3, 128), (3, 129), (3, 145), (3, 151), (4, 170), (3, 176), (3, 192), (16, 146),
                                 (17, 145)])
def test_wide_tiles_match_narrow_tiles(lib, o, v):
    ham = synthetic(o, v, 40, seed=o + v, bscale=0.5)
    setup_lists(lib, ham)
    kw = dict(cc_conv=6, cc_maxcyc=60, triples=1, precision=ab.PREC_BF16X3)
    wide = lib.xvcc(**kw)
    lib.set_tc_wide(0)
    try:
        narrow = lib.xvcc(**kw)
    finally:
        lib.set_tc_wide(1)
    assert wide.e_ccsd == narrow.e_ccsd
    assert abs(wide.e_t4 - narrow.e_t4) < 1e-14 + 1e-9 * abs(narrow.e_t4)
    assert abs(wide.e_st5 - narrow.e_st5) < 1e-15 + 1e-9 * abs(narrow.e_st5)
