"""GPU test of products called from one host thread while another runs a CC
solve: the products grow from call to call (each needs larger planes and
partial sums than the one before) and so do those of the solve's first pass.
No call may be handed memory that the other one's kernels still use, so every
result equals the one computed alone bit for bit."""
import threading

import pytest
import torch

import acesb200 as ab
from oracle.hamiltonian import synthetic
from test_gpu_ccsd import setup_lists

pytestmark = pytest.mark.gpu

SHAPES = [(200, 150, 6000), (310, 140, 9000), (700, 300, 9001), (1300, 600, 8000),
          (1300, 2200, 4000), (2561, 1297, 4099)]


@pytest.mark.parametrize("prec", [ab.PREC_FP64, ab.PREC_BF16X3])
def test_products_beside_a_solve(prec):
    lib = ab.load()
    lib.init(0)
    setup_lists(lib, synthetic(8, 60, 100, seed=4, bscale=0.5))
    g = torch.Generator(device="cuda").manual_seed(7)
    jobs = []
    for m, n, k in SHAPES:
        A = torch.randn((m, k), generator=g, dtype=torch.float64, device="cuda")
        B = torch.randn((n, k), generator=g, dtype=torch.float64, device="cuda")
        jobs.append((m, n, k, A, B, torch.zeros((n, m), dtype=torch.float64, device="cuda")))

    def product(j):
        m, n, k, A, B, C = j
        lib.xgemm("T", "N", m, n, k, 1.0, A.data_ptr(), k, B.data_ptr(), k, 0.0, C.data_ptr(), m,
                  precision=prec)

    def solve():
        e = lib.xvcc(cc_conv=7, cc_maxcyc=60, cc_exporder=5, precision=prec).e_ccsd
        nr, nc = lib.list_dims(1, 46)
        return e, torch.from_numpy(lib.getlst(1, nc, 1, 46).copy())

    torch.cuda.synchronize()
    alone = []
    for j in jobs:
        product(j)
        alone.append(j[5].clone())
    e0, t0 = solve()
    torch.cuda.synchronize()
    bad, done = [], threading.Event()

    def products():
        while not done.is_set():
            for j, ref in zip(jobs, alone):
                product(j)
                if not torch.equal(j[5], ref):
                    bad.append(j[:3])

    t = threading.Thread(target=products)
    t.start()
    try:
        for _ in range(5):
            e, t2 = solve()
            if e != e0 or not torch.equal(t2, t0):
                bad.append("solve")
    finally:
        done.set()
        t.join()
    assert not bad
