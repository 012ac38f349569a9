"""Threads that run plans of different sizes at once: the same kernels are launched with different amounts
of shared memory (sort histograms of 4 (Nx - 1) words, the contraction's node flags, FFT grids, rotation
rows), and none may take another's limit.  Each thread's alm equal those it gets alone, to
1e-12 x max|alm| (the FP64 level's bound)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_plans_of_different_sizes_at_once():
    import torch
    from directsht_b200 import DirectSHT
    rng = np.random.default_rng(0)
    N = 3000
    pts = [torch.from_numpy(a).cuda() for a in (np.arccos(rng.uniform(-1, 1, N)), rng.uniform(0, 2 * np.pi, N),
                                                rng.normal(size=N))]
    plans = [DirectSHT(Nl, Nx) for Nl, Nx in ((20, 12000), (40, 20), (300, 4), (20, 6000), (64, 300), (120, 8))]
    for d, bins in zip(plans, ("fp64", "nufft", "nufft", "fp64", "nufft", "nufft")):
        d.tune(bin_sums=bins)
    alone = [d(*pts) for d in plans]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(150):
                    got = plans[i](*pts)
                    if not (got - alone[i]).abs().max() <= 1e-12 * alone[i].abs().max():
                        raise AssertionError("alm differ")
        except Exception as e:  # reported by the test
            wrong.append((i, repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(plans))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
