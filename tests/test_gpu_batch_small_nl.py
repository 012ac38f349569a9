"""Batches at the smallest Nl, where a transform just below the NUFFT sums' least number of points has
more (smaller) pieces than the largest one of the batch: every transform gives the alm of its own call
and of the oracle, to 1e-12 x max|alm| (the FP64 level's bound)."""
import numpy as np
import pytest

from oracle import dsht_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nl,Nx,N", [(1, 16, 84480), (1, 40, 219648), (2, 16, 42240)])
def test_sizes_on_both_sides_of_the_rule(Nl, Nx, N):
    from directsht_b200 import DirectSHT
    rng = np.random.default_rng(Nx)
    d, tab = DirectSHT(Nl, Nx), O.build_tables(Nl, Nx)
    sets = []
    for n in (N, N - 1, N // 2, 7):
        x = rng.uniform(-1, 1, n) ** 3  # uneven bins
        sets.append((np.arccos(x), rng.uniform(0, 2 * np.pi, n), rng.uniform(0.5, 1.5, n)))
    for got, s in zip(d.call_batch(sets), sets):
        for ref in (d(*s), O.direct_sht(tab, *s)):
            assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
