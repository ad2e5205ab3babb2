"""GPU test of products called from several host threads at once: each call's
split-K partials are its own, so every product equals the one computed alone
bit for bit (FP64 with split K, and split precision with split K)."""
import threading

import pytest
import torch

import acesb200 as ab

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [ab.PREC_FP64, ab.PREC_BF16X3])
def test_concurrent_products(prec):
    lib = ab.load()
    lib.init(0)
    g = torch.Generator(device="cuda").manual_seed(5)
    jobs = []
    for m, n, k in ((200, 150, 6000), (96, 300, 9000), (310, 40, 12000), (150, 150, 20000)):
        A = torch.randn((m, k), generator=g, dtype=torch.float64, device="cuda")
        B = torch.randn((n, k), generator=g, dtype=torch.float64, device="cuda")
        C = torch.zeros((n, m), dtype=torch.float64, device="cuda")
        jobs.append((m, n, k, A, B, C))

    def run(j):
        m, n, k, A, B, C = j
        lib.xgemm("T", "N", m, n, k, 1.0, A.data_ptr(), k, B.data_ptr(), k, 0.0, C.data_ptr(), m,
                  precision=prec)

    torch.cuda.synchronize()
    alone = []
    for j in jobs:
        run(j)
        alone.append(j[5].clone())
    torch.cuda.synchronize()
    bad = []

    def worker(j, ref):
        for _ in range(20):
            run(j)
            if not torch.equal(j[5], ref):
                bad.append(j[:3])

    threads = [threading.Thread(target=worker, args=(j, r)) for j, r in zip(jobs, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
