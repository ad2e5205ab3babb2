"""GPU test of the list producer on factors that are symmetric up to rounding,
as a transformation by matrix products leaves them: every list element is the
sum of products of the factors as given, B[L,r,p] B[L,s,q], to the rounding of
that sum alone (the tolerance of test_gpu_intprc_pairs.py without a term for
the asymmetry).  Elements far below the largest one show a difference of a few
units in the last place of the latter."""
import numpy as np
import pytest

import acesb200 as ab
from test_gpu_intprc_pairs import check, factors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("irreps", [1, 4])
@pytest.mark.parametrize("units", [1, 60])
def test_factors_symmetric_to_rounding_are_taken_as_given(irreps, units):
    lib = ab.load()
    lib.init(0)
    o, v, naux = 3, 34, 2
    B, irr = factors(o, v, naux, irreps, 11)
    B *= 1e-3
    B[0, 0, 0] = 1.0
    upper = np.triu(np.ones(B.shape[1:]), 1) * (B != 0)
    check(lib, B + units * 2.0 ** -52 * upper, irr, o, irreps)
