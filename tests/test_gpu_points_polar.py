"""The scatter pass queues each warp's polar points and does them 32 at a time: skies without polar points, with
nothing else, and with queue remainders of every kind, for records of cosines and sines (direct sums) and of turns
(NUFFT sums), against the oracle.  Tolerance 1e-12 x max|alm|, the FP64 level's bound."""
import numpy as np
import pytest

from oracle import dsht_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sums", ["fp64", "nufft"])
@pytest.mark.parametrize("npol,neq", [(0, 2048), (1, 0), (33, 0), (4097, 0), (31, 4000), (700, 700), (60000, 130000)])
def test_polar_queue(npol, neq, sums):
    from directsht_b200 import DirectSHT
    rng = np.random.default_rng(npol + neq)
    x = np.concatenate([rng.uniform(0.9, 0.999, npol) * rng.choice([-1, 1], npol), rng.uniform(-0.8, 0.8, neq)])
    th = rng.permutation(np.arccos(x))
    ph, w = rng.uniform(0, 2 * np.pi, x.size), rng.normal(size=x.size)
    Nl, Nx = 12, 40
    sht = DirectSHT(Nl, Nx)
    sht.tune(bin_sums=sums)
    ref = O.direct_sht(O.build_tables(Nl, Nx), th, ph, w)
    assert np.abs(sht(th, ph, w) - ref).max() <= 1e-12 * np.abs(ref).max()
