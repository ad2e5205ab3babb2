"""GPU test of the list producer's packed path (symmetric factors) and of its
dense path (factors that are not symmetric) against numpy: every list element
is <pq|rs> = sum_L B[L,r,p] B[L,s,q] of the factors as given.

Sizes: tile edges of the pair expansion (v = 31 .. 65, o = 1 .. 33), odd naux
(padded rows), 1, 2, 4 and 8 irreps with empty ones among them.  Tolerance: a
sum of naux products in any order is within naux u sum |B||B| (u = 2^-53) of
the exact value, the reference too; factors whose halves differ by d are off
by at most d sum |B| per side more.
"""
import numpy as np
import pytest

import acesb200 as ab
from acesb200 import INTEGRAL_LISTS

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    lib = ab.load()
    lib.init(0)
    return lib


def factors(o, v, naux, irreps, seed):
    rng = np.random.default_rng(seed)
    n = o + v
    B = rng.normal(0.0, 0.05, (naux, n, n))
    B = 0.5 * (B + B.transpose(0, 2, 1))
    irr = np.concatenate([np.sort(rng.integers(0, irreps, o)), np.sort(rng.integers(0, irreps, v))])
    aux = rng.integers(0, irreps, naux)
    B *= (irr[:, None] ^ irr[None, :])[None] == aux[:, None, None]
    return B, irr


def check(lib, B, irr, o, irreps, delta=0.0):
    n, naux = B.shape[1], B.shape[0]
    lib.init(0)
    lib.sym_init([int(np.sum(irr[:o] == h)) for h in range(irreps)],
                 [int(np.sum(irr[o:] == h)) for h in range(irreps)])
    lib.putrec("SCFEVALA", np.zeros(n))
    lib.intprc_df(B)
    orbs = {c: [[k for k in rng if irr[k] == h] for h in range(irreps)]
            for c, rng in (("o", range(o)), ("v", range(o, n)))}
    pairs = lambda a, b, h: [(p, q) for hq in range(irreps)  # noqa: E731
                             for q in orbs[b][hq] for p in orbs[a][hq ^ h]]
    spaces = {13: "oooo", 10: "ooov", 16: "vvoo", 25: "vovo", 30: "vvvo", 233: "vvvv"}
    u = 2.0 ** -53
    absB = np.abs(B)
    for lst in INTEGRAL_LISTS:
        a, b, c, d = spaces[lst]
        for h in range(irreps):
            rows, cols = pairs(a, b, h), pairs(c, d, h)
            assert lib.list_dims(h + 1, lst) == (len(rows), len(cols))
            if not rows or not cols:
                continue
            got = lib.getlst(1, len(cols), h + 1, lst)
            P, Q = np.array(rows).T
            R, S = np.array(cols).T
            ref, mag, one = np.zeros(got.shape), np.zeros(got.shape), np.zeros(got.shape)
            for L in range(naux):
                x, y = B[L][np.ix_(R, P)].T, B[L][np.ix_(S, Q)].T
                ref += x * y
                mag += np.abs(x * y)
                one += np.abs(x) + np.abs(y)
            tol = 2 * (naux + 2) * u * mag + delta * one + 4 * naux * delta * delta
            assert (np.abs(got - ref) <= tol).all(), (lst, h, np.abs(got - ref).max())


@pytest.mark.parametrize("o,v,naux,irreps", [(1, 31, 7, 1), (2, 33, 33, 1), (33, 5, 16, 1),
                                             (3, 65, 20, 1), (5, 32, 41, 2), (6, 21, 30, 4),
                                             (3, 37, 25, 8), (1, 3, 2, 8)])
def test_symmetric_factors(lib, o, v, naux, irreps):
    B, irr = factors(o, v, naux, irreps, 10 * o + v)
    check(lib, B, irr, o, irreps)


@pytest.mark.parametrize("irreps", [1, 8])
def test_factors_symmetric_to_rounding(lib, irreps):
    o, v, naux = 4, 33, 30
    B, irr = factors(o, v, naux, irreps, 3)
    d = 2.0 ** -47 * np.abs(B).max()
    rng = np.random.default_rng(1)
    B = np.where(B != 0, B + d * rng.uniform(-0.5, 0.5, B.shape), 0.0)
    check(lib, B, irr, o, irreps, delta=d)


@pytest.mark.parametrize("irreps", [1, 4])
def test_factors_that_are_not_symmetric(lib, irreps):
    o, v, naux = 3, 20, 19
    B, irr = factors(o, v, naux, irreps, 5)
    B[7] *= 1.0 + np.triu(np.ones(B.shape[1:]), 1) * 1e-9
    check(lib, B, irr, o, irreps)


def test_an_infinite_factor_takes_the_dense_path(lib):
    o, v, naux = 2, 9, 6
    B, irr = factors(o, v, naux, 1, 8)
    B[2, 4, 5] = B[2, 5, 4] = np.inf
    lib.init(0)
    lib.sym_init([o], [v])
    lib.intprc_df(B)
    got = lib.getlst(1, v * v, 1, 233)
    with np.errstate(invalid="ignore"):
        X = np.einsum("Lpr,Lqs->qpsr", B[:, o:, o:], B[:, o:, o:]).reshape(v * v, v * v)
    np.testing.assert_array_equal(np.isfinite(got), np.isfinite(X))
