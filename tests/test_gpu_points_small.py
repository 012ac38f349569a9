"""The sort at the edges of its scatter tiles (512 points upwards) and key runs (1024 threads of the scan):
the FP64 level against the oracle.  Tolerance 1e-12 x max|alm|, the FP64 level's bound."""
import numpy as np
import pytest

from oracle import dsht_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nx,N", [(2, 511), (257, 512), (258, 513), (300, 1023), (1025, 2000), (700, 151551), (16, 151552),
                                  (16, 151553), (40, 300001)])
def test_scatter_tiles_and_key_runs(Nx, N):
    from directsht_b200 import DirectSHT
    rng = np.random.default_rng(N)
    th, ph, w = np.arccos(rng.uniform(-1, 1, N)), rng.uniform(0, 2 * np.pi, N), rng.normal(size=N)
    Nl = 12
    ref = O.direct_sht(O.build_tables(Nl, Nx), th, ph, w)
    got = DirectSHT(Nl, Nx)(th, ph, w)
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
