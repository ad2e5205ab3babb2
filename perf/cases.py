"""Performance cases: the work that a user of the engine has it do, through its public
entry points (``acesb200``), over the range of sizes, precisions and options in use.

Kinds of case:

* ``xgemm``   the BLAS boundary on device operands (FP64 and split BF16x3, N/T, beta 0/1);
* ``lists``   MO density-fitting factors -> the six integral lists (``intprc_df``);
* ``ccsd``    factors -> lists -> ``xvcc`` to convergence, with (T), with Lambda and the
              one-particle density, or with EOM roots; the amplitudes are read from
              the list store.

The inputs are the synthetic closed-shell systems of ``acesb200.workloads`` made on the
GPU: orbital energies U[-1.5,-0.3] and U[0.2,3.0] Eh, symmetric Gaussian factors scaled
so that the CC iteration converges, orbitals dealt unevenly into 1, 4 or 8 irreps.
"""
import itertools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "aces-ii_b200"))
import acesb200 as ab  # noqa: E402

NAUX_PER_MO = 3


def listed():
    return [
        # a Fock-sized product: the many small XGEMM calls of a host program
        {"name": "xgemm_f64_small", "kind": "xgemm", "prec": "fp64", "ta": "N", "tb": "N",
         "m": 120, "n": 96, "k": 150, "beta": 1.0},
        # an ordinary FP64 DGEMM call of odd sizes, both operands as a Fortran caller has them
        {"name": "xgemm_f64_ragged", "kind": "xgemm", "prec": "fp64", "ta": "N", "tb": "N",
         "m": 2401, "n": 1519, "k": 2049, "beta": 0.0},
        # the o*v x o*v x o*v ring product in split precision, accumulated
        {"name": "xgemm_split_ring", "kind": "xgemm", "prec": "split", "ta": "N", "tb": "T",
         "m": 3600, "n": 3600, "k": 3600, "beta": 1.0},
        # the packed particle-particle ladder product of a 180-virtual system
        {"name": "xgemm_split_ladder", "kind": "xgemm", "prec": "split", "ta": "T", "tb": "N",
         "m": 16290, "n": 400, "k": 16290, "beta": 0.0},
        # the integral lists of the benchmark system from its factors
        {"name": "lists_o20_v180", "kind": "lists", "o": 20, "v": 180, "irreps": 1},
        # a small molecule in C2v (water in a double-zeta basis), FP64: launch bound
        {"name": "ccsd_f64_o5_v21_c2v", "kind": "ccsd", "prec": "fp64", "o": 5, "v": 21,
         "irreps": 4, "triples": 0, "lam": 0, "eom": 0},
        # CCSD(T) in FP64 without symmetry, ordinary size
        {"name": "ccsd_t_f64_o8_v70", "kind": "ccsd", "prec": "fp64", "o": 8, "v": 70,
         "irreps": 1, "triples": 1, "lam": 0, "eom": 0},
        # CCSD in split precision, the largest system of the 64-system batch without symmetry
        {"name": "ccsd_split_o24_v220", "kind": "ccsd", "prec": "split", "o": 24, "v": 220,
         "irreps": 1, "triples": 0, "lam": 0, "eom": 0},
        # CCSD(T) in split precision
        {"name": "ccsd_t_split_o14_v170", "kind": "ccsd", "prec": "split", "o": 14, "v": 170,
         "irreps": 1, "triples": 1, "lam": 0, "eom": 0},
        # a system of the 8-irrep batch in split precision
        {"name": "ccsd_split_o17_v151_d2h", "kind": "ccsd", "prec": "split", "o": 17, "v": 151,
         "irreps": 8, "triples": 0, "lam": 0, "eom": 0},
        # a property run: Lambda equations and the one-particle density
        {"name": "lambda_split_o16_v130", "kind": "ccsd", "prec": "split", "o": 16, "v": 130,
         "irreps": 1, "triples": 0, "lam": 1, "eom": 0},
        # excited states: the lowest singlet root of a small FP64 system
        {"name": "eom_f64_o6_v50", "kind": "ccsd", "prec": "fp64", "o": 6, "v": 50,
         "irreps": 1, "triples": 0, "lam": 0, "eom": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["xgemm", "xgemm", "lists", "ccsd", "ccsd", "ccsd"])
    if kind == "xgemm":
        prec = rng.choice(["fp64", "split"])
        top = 2600 if prec == "fp64" else 6000
        return {"kind": "xgemm", "prec": prec, "ta": rng.choice("NT"), "tb": rng.choice("NT"),
                "m": _log(rng, 40, top), "n": _log(rng, 40, top), "k": _log(rng, 40, top),
                "beta": rng.choice([0.0, 1.0])}
    if kind == "lists":
        return {"kind": "lists", "o": rng.randint(4, 20), "v": _log(rng, 30, 170),
                "irreps": rng.choice([1, 1, 4, 8])}
    prec = rng.choice(["fp64", "split", "split"])
    what = rng.choice(["ccsd", "ccsd", "triples", "lam", "eom"])
    if prec == "fp64" or what == "eom":
        o, v = rng.randint(4, 10), _log(rng, 20, 80)
    else:
        o, v = rng.randint(6, 18), _log(rng, 80, 180)
    irreps = rng.choice([1, 4, 8]) if what in ("ccsd", "triples") and o >= 5 else 1
    return {"kind": "ccsd", "prec": prec, "o": o, "v": v, "irreps": irreps,
            "triples": int(what == "triples"), "lam": int(what == "lam"),
            "eom": int(what == "eom")}


# ---- inputs ------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _split(n, g):
    """n orbitals dealt unevenly into g irreps, the first the largest."""
    if g == 1:
        return [n]
    w = [1.5 - h / (g - 1) for h in range(g)]
    c = [int(n * x / sum(w)) for x in w]
    c[0] += n - sum(c)
    return c


def _system(case, seed):
    """(pop, vrt, eps[nmo], B[naux, nmo, nmo]) in DPD order (by irrep inside each space)."""
    o, v, g = case["o"], case["v"], case["irreps"]
    dev = _device()
    gen = torch.Generator(device=dev).manual_seed(seed * 7919 + 1000 * o + v)
    n, naux = o + v, NAUX_PER_MO * (o + v)
    pop, vrt = _split(o, g), _split(v, g)
    u = torch.rand(n, generator=gen, device=dev, dtype=torch.float64)
    eps = torch.cat([-1.5 + 1.2 * u[:o], 0.2 + 2.8 * u[o:]]).cpu().numpy()
    for base, cnt in ((0, pop), (o, vrt)):
        at = base
        for c in cnt:
            eps[at:at + c] = np.sort(eps[at:at + c])
            at += c
    # entries N(0, sigma^2), the <ab|cd> coupling naux sigma^2 v held at 2.5 Eh or below
    # (the CC iteration then converges in about ten cycles)
    sigma = min(0.02, math.sqrt(2.5 * g / (naux * v)))
    B = torch.randn((naux, n, n), generator=gen, device=dev, dtype=torch.float64)
    B = (B + B.transpose(1, 2)).mul_(0.5 * sigma)
    if g > 1:
        irr = torch.tensor([h for h in range(g) for _ in range(pop[h])] +
                           [h for h in range(g) for _ in range(vrt[h])], device=dev)
        aux = torch.randint(0, g, (naux,), generator=gen, device=dev)
        B.mul_((irr[:, None] ^ irr[None, :])[None] == aux[:, None, None])
    return pop, vrt, eps, B.contiguous()


def _xgemm_inputs(case, seed):
    dev = _device()
    m, n, k = case["m"], case["n"], case["k"]
    gen = torch.Generator(device=dev).manual_seed(seed * 7919 + 31 * m + 17 * n + k)

    def mat(rows, cols):  # column-major rows x cols: a torch tensor [cols, rows]
        return torch.randn((cols, rows), generator=gen, device=dev, dtype=torch.float64)

    A = mat(m, k) if case["ta"] == "N" else mat(k, m)
    B = mat(k, n) if case["tb"] == "N" else mat(n, k)
    return A, B, mat(m, n)


def prepare(case, seed):
    lib = ab.load()
    lib.init(0)
    if case["kind"] == "xgemm":
        A, B, C0 = _xgemm_inputs(case, seed)
        return {"case": case, "lib": lib, "A": A, "B": B, "C0": C0, "C": torch.empty_like(C0)}
    pop, vrt, eps, B = _system(case, seed)
    return {"case": case, "lib": lib, "pop": pop, "vrt": vrt, "eps": eps, "B": B}


# ---- one pass ----------------------------------------------------------------------
class _Block:
    """A list block in the library's device memory, as torch takes it without a copy."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "version": 3,
                                         "data": (ptr, False)}


def _list(lib, lst, nirrep):
    out = []
    for h in range(1, nirrep + 1):
        nr, nc = lib.list_dims(h, lst)
        if nr * nc:
            out.append(torch.as_tensor(_Block(lib.h.aces_list_devptr(h, lst), (nc, nr)),
                                       device="cuda"))
    return out


def run(s):
    case, lib = s["case"], s["lib"]
    if case["kind"] == "xgemm":
        if case["beta"]:
            s["C"].copy_(s["C0"])
            torch.cuda.current_stream().synchronize()  # the call runs on its own stream
        m, n, k = case["m"], case["n"], case["k"]
        lib.xgemm(case["ta"], case["tb"], m, n, k, 1.0,
                  s["A"].data_ptr(), m if case["ta"] == "N" else k,
                  s["B"].data_ptr(), k if case["tb"] == "N" else n, case["beta"],
                  s["C"].data_ptr(), m,
                  precision=ab.PREC_BF16X3 if case["prec"] == "split" else ab.PREC_FP64)
        return s["C"]
    g = case["irreps"]
    lib.init(0)
    lib.sym_init(s["pop"], s["vrt"])
    lib.putrec("SCFEVALA", s["eps"])
    lib.intprc_df(s["B"])
    if case["kind"] == "lists":
        return {"list%d" % lst: _list(lib, lst, g) for lst in ab.INTEGRAL_LISTS}
    split = case["prec"] == "split"
    prec = ab.PREC_BF16X3 if split else ab.PREC_FP64
    cfg = lib.xvcc(cc_conv=7 if split else 9, cc_maxcyc=60, cc_exporder=6, precision=prec,
                   triples=case["triples"], use_graph=1 if split else 0)
    out = {"t1": _list(lib, 90, 1), "t2": _list(lib, 46, g), "e": cfg.e_ccsd}
    if case["triples"]:
        out["e_t4"], out["e_st5"] = cfg.e_t4, cfg.e_st5
    nmo = case["o"] + case["v"]
    if case["lam"]:
        lib.xlambda(cc_conv=7, cc_maxcyc=60, cc_exporder=6, precision=prec)
        lib.xdens()
        out["l1"], out["l2"] = _list(lib, 190, 1), _list(lib, 146, g)
        out["density"] = lib.getrec("DENSMAT", nmo * nmo).reshape(nmo, nmo)
    if case["eom"]:
        _, roots = lib.xvee([1], eom_conv=5, eom_maxcyc=80, precision=prec)
        out["omega"] = roots[0][0]
    return out


# ---- what a pass cannot do without --------------------------------------------------
def work(case):
    if case["kind"] == "xgemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 8.0 * (m * k + k * n + m * n * (2 if case["beta"] else 1)),
                "flops": 2.0 * m * n * k}
    o, v, g = case["o"], case["v"], case["irreps"]
    n, naux = o + v, NAUX_PER_MO * (o + v)
    factors = 8.0 * naux * n * n
    lists = 8.0 * (v ** 4 + o * v ** 3 + 2 * o * o * v * v + o ** 3 * v + o ** 4) / g
    pairs = n * (n + 1) // 2
    f_lists = 1.0 * naux * pairs * (pairs + 1) / g          # every distinct (pq|rs) once
    if case["kind"] == "lists":
        return {"bytes": factors + lists, "flops": f_lists}
    cycles = 9 if case["prec"] == "split" else 11
    ladder = 0.5 * 2.0 * o * o * float(v) ** 4               # packed pairs
    ring = 5 * 2.0 * o ** 3 * float(v) ** 3                  # W(mbej) and the ring products
    f = f_lists + cycles * (ladder + ring) / g
    b = factors + cycles * 4.0 * float(v) ** 4 / g           # packed <ab|cd> once a cycle
    b += cycles * 8.0 * 4 * o * o * v * v
    if case["triples"]:
        f += (2.0 * o ** 3 * float(v) ** 4 + 2.0 * o ** 4 * float(v) ** 3)
    if case["lam"]:
        f += 10 * 2 * (ladder / 2 + ring) / g
    if case["eom"]:
        f += 25 * 2 * (ladder / 2 + ring) / g
    return {"bytes": b, "flops": f}


# ---- the same values in plain 64-bit torch -------------------------------------------
def _orbs(cnt):
    """Irreps and first orbitals of a space laid out irrep by irrep."""
    first = [sum(cnt[:h]) for h in range(len(cnt))]
    return [list(range(first[h], first[h] + cnt[h])) for h in range(len(cnt))]


def _pairs(P, Q, h):
    """The (p, q) pairs of total irrep h in list order: by the irrep of q, p fastest."""
    return [(p, q) for hq in range(len(Q)) for q in Q[hq] for p in P[hq ^ h]]


def _blocks(dense, rows, cols, g):
    """Column-major list blocks [cols, rows] of dense[p, q, r, s], one per irrep."""
    out = []
    for h in range(g):
        r, c = _pairs(rows[0], rows[1], h), _pairs(cols[0], cols[1], h)
        if not r or not c:
            continue
        if g == 1:
            out.append(dense.permute(3, 2, 1, 0).reshape(len(c), len(r)))
            continue
        r, c = (torch.tensor(x, device=dense.device) for x in (r, c))
        out.append(dense[r[None, :, 0], r[None, :, 1], c[:, 0, None], c[:, 1, None]])
    return out


def _eri(B, o, spaces):
    """Physicists' <pq|rs> of the four spaces ('o' or 'v')."""
    sl = {"o": slice(0, o), "v": slice(o, None)}
    p, q, r, s = (sl[c] for c in spaces)
    L, R = B[:, p, r], B[:, q, s]
    X = L.reshape(L.shape[0], -1).T @ R.reshape(R.shape[0], -1)
    return X.reshape(L.shape[1:] + R.shape[1:]).permute(0, 2, 1, 3).contiguous()


def _ccsd(eps, B, o):
    """Closed-shell CCSD with canonical orbitals (Stanton-Gauss, spin-adapted), converged."""
    E = torch.einsum
    e = torch.from_numpy(eps).to(B.device)
    eo, ev = e[:o], e[o:]
    I = {k: _eri(B, o, k) for k in ("oooo", "ooov", "oovv", "ovov", "ovvo", "ovvv", "vvvv")}
    v = ev.numel()
    L = 2 * I["oovv"] - I["oovv"].transpose(2, 3)
    D1 = eo[:, None] - ev[None]
    D2 = D1[:, None, :, None] + D1[None, :, None, :]
    t1, t2 = torch.zeros_like(D1), I["oovv"] / D2
    VV = I["vvvv"].reshape(v * v, v * v)
    ooov, ovvv = I["ooov"], I["ovvv"]
    hist = []
    P = lambda x: x + x.permute(1, 0, 3, 2)  # noqa: E731
    for _ in range(80):
        tt = E("ia,jb->ijab", t1, t1)
        tau, tu = t2 + tt, t2 + 0.5 * tt
        Fae = 2 * E("mf,mafe->ae", t1, ovvv) - E("mf,maef->ae", t1, ovvv) \
            - E("mnaf,mnef->ae", tu, L)
        Fmi = 2 * E("ne,mnie->mi", t1, ooov) - E("ne,nmie->mi", t1, ooov) \
            + E("inef,mnef->mi", tu, L)
        Fme = E("nf,mnef->me", t1, L)
        W = E("je,mnie->mnij", t1, ooov)
        W = I["oooo"] + W + W.permute(1, 0, 3, 2) + E("ijef,mnef->mnij", tau, I["oovv"])
        X = 0.5 * t2 + E("jf,nb->jnfb", t1, t1)
        Wej = I["ovvo"] + E("jf,mbef->mbej", t1, ovvv) - E("nb,nmje->mbej", t1, ooov) \
            - E("jnfb,mnef->mbej", X, I["oovv"]) + 0.5 * E("njfb,mnef->mbej", t2, L)
        Wje = -I["ovov"] - E("jf,mbfe->mbje", t1, ovvv) + E("nb,mnje->mbje", t1, ooov) \
            + E("jnfb,mnfe->mbje", X, I["oovv"])
        Z = E("mbef,ijef->mbij", ovvv, tau)
        r1 = t1 @ Fae.T - Fmi.T @ t1 + 2 * E("imae,me->ia", t2, Fme) - E("imea,me->ia", t2, Fme)
        r1 = r1 + 2 * E("nf,nafi->ia", t1, I["ovvo"]) - E("nf,naif->ia", t1, I["ovov"])
        r1 = r1 + 2 * E("mief,maef->ia", t2, ovvv) - E("mife,maef->ia", t2, ovvv)
        r1 = r1 - 2 * E("mnae,mnie->ia", t2, ooov) + E("mnae,nmie->ia", t2, ooov)
        Y = E("ijae,be->ijab", t2, Fae - 0.5 * t1.T @ Fme)
        Y = Y - E("imab,mj->ijab", t2, Fmi + 0.5 * Fme @ t1.T)
        Y = Y - E("ma,mbij->ijab", t1, Z)
        Y = Y + E("imae,mbej->ijab", t2 - t2.transpose(2, 3), Wej) \
            + E("imae,mbej->ijab", t2, Wej + Wje.transpose(2, 3)) + E("mjae,mbie->ijab", t2, Wje)
        Y = Y - E("ie,ma,mbej->ijab", t1, t1, I["ovvo"]) - E("ie,mb,maje->ijab", t1, t1, I["ovov"])
        Y = Y + E("ie,jeba->ijab", t1, ovvv) - E("ma,ijmb->ijab", t1, ooov)
        r2 = I["oovv"] + P(Y) + E("mnab,mnij->ijab", tau, W)
        r2 = r2 + (tau.reshape(o * o, v * v) @ VV.T).reshape(o, o, v, v)
        n1, n2 = r1 / D1, r2 / D2
        new = torch.cat([n1.reshape(-1), n2.reshape(-1)])
        err = new - torch.cat([t1.reshape(-1), t2.reshape(-1)])
        hist = (hist + [(new, err)])[-8:]
        if float(err.abs().max()) < 1e-13:
            t1, t2 = n1, n2
            break
        n = len(hist)
        M = -torch.ones((n + 1, n + 1), dtype=torch.float64)
        M[n, n] = 0.0
        for i in range(n):
            for j in range(n):
                M[i, j] = float(hist[i][1] @ hist[j][1])
        M[:n, :n] /= M[:n, :n].diagonal().mean()
        rhs = torch.zeros(n + 1, dtype=torch.float64)
        rhs[n] = -1.0
        c = torch.linalg.lstsq(M, rhs, driver="gelsd").solution
        new = sum(float(c[i]) * hist[i][0] for i in range(n))
        t1, t2 = new[:t1.numel()].reshape(t1.shape), new[t1.numel():].reshape(t2.shape)
    tau = t2 + E("ia,jb->ijab", t1, t1)
    return t1, t2, float((tau * L).sum()), I, eo, ev


def _triples(t1, t2, I, eo, ev):
    """E[4]T and E[5]ST of the closed-shell (T) correction."""
    o, v = t1.shape
    G = I["ovvv"].permute(0, 3, 2, 1).contiguous()       # G[k,b,c,d] = (bd|ck) = <kd|cb>
    D3 = ev[:, None, None] + ev[None, :, None] + ev[None, None, :]
    perms = list(itertools.permutations(range(3)))
    e4 = e5 = 0.0
    for i in range(o):
        for j in range(i + 1):
            for k in range(j + 1):
                w, x = torch.zeros_like(D3), torch.zeros_like(D3)
                for p in perms:
                    a, b, c = ((i, j, k)[q] for q in p)
                    y = (t2[a, b] @ G[c].permute(2, 0, 1).reshape(v, v * v)).reshape(v, v, v)
                    y = y - torch.tensordot(t2[a].permute(1, 2, 0), I["ooov"][:, c, b, :],
                                            dims=([2], [0]))
                    inv = [p.index(q) for q in range(3)]
                    w = w + y.permute(inv)
                x = t1[i][:, None, None] * I["oovv"][j, k][None] \
                    + t1[j][None, :, None] * I["oovv"][i, k][:, None, :] \
                    + t1[k][None, None, :] * I["oovv"][i, j][:, :, None]
                D = eo[i] + eo[j] + eo[k] - D3
                mult = 6 if i == j == k else (2 if i == j or j == k else 1)
                for p in perms:
                    wp, xp = w.permute(p), x.permute(p)
                    z = (4 * wp + wp.permute(1, 2, 0) + wp.permute(2, 0, 1)) / D
                    e4 += float((z * (wp - wp.permute(2, 1, 0))).sum()) / (3 * mult)
                    e5 += float((z * (xp - xp.permute(2, 1, 0))).sum()) / (3 * mult)
    return e4, e5


def exact(case, seed):
    if case["kind"] == "xgemm":
        A, B, C0 = _xgemm_inputs(case, seed)
        a = A.T if case["ta"] == "N" else A
        b = B.T if case["tb"] == "N" else B
        out = (a @ b).T
        return (out + C0 if case["beta"] else out).contiguous()
    pop, vrt, eps, B = _system(case, seed)
    g, o = case["irreps"], case["o"]
    so, sv = _orbs(pop), _orbs(vrt)
    if case["kind"] == "lists":
        space = {"o": so, "v": sv}
        out = {}
        for lst, idx in ((13, "oooo"), (10, "ooov"), (16, "vvoo"), (25, "vovo"), (30, "vvvo"),
                         (233, "vvvv")):
            sp = [space[c] for c in idx]
            out["list%d" % lst] = _blocks(_eri(B, o, idx), sp[:2], sp[2:], g)
        return out
    t1, t2, e, I, eo, ev = _ccsd(eps, B, o)
    irr = [(h, a, i) for h in range(g) for i in so[h] for a in sv[h]]
    out = {"t1": [torch.stack([t1[i, a] for _, a, i in irr])[None]],
           "t2": _blocks(t2.permute(2, 3, 0, 1), (sv, sv), (so, so), g), "e": e}
    if case["triples"]:
        out["e_t4"], out["e_st5"] = _triples(t1, t2, I, eo, ev)
    if case["lam"]:   # no plain closed form here: held to the bound of their type
        out["l1"] = out["l2"] = out["density"] = None
    if case["eom"]:
        out["omega"] = None
    return out
