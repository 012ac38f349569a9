"""The FP64 level's NUFFT node sums against the direct FP64 sums and the oracle, where they can go
wrong: grid sizes of every FFT shape, runs that share nodes between CTAs, bins of several pieces,
single points, all points in one cell, azimuths at and beyond the ends of [0, 2 pi).

Tolerance 1e-12 x max|alm|, the FP64 level's bound: with at most 3e5 points of unit weights the
truncation (2.4e-15) and the rounding of the transforms (a few 2^-53 log2 n of the root sum
square) stay two decades below it."""
import numpy as np
import pytest

from oracle import dsht_oracle as O

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


def _pair(Nl, Nx, th, ph, w, **kw):
    from directsht_b200 import DirectSHT
    d = DirectSHT(Nl, Nx, **kw)
    d.tune(bin_sums="fp64")
    ref = d(th, ph, w)
    d.tune(bin_sums="nufft")
    return d, d(th, ph, w), ref


# n = 128 (radix 16, 8) .. 8192 (16, 8, 8, 8), one and two grids, both oversamplings
@pytest.mark.parametrize("Nl,Nx,N", [(1, 5, 40), (2, 3, 2000), (16, 40, 3000), (17, 9, 500), (33, 70, 9000),
                                     (64, 33, 20000), (65, 40, 4000), (128, 60, 5000), (250, 100, 30000),
                                     (257, 64, 20000), (512, 90, 30000), (513, 50, 20000), (1024, 40, 30000),
                                     (1025, 30, 20000), (2048, 12, 10000)])
def test_against_direct_sums(Nl, Nx, N):
    rng = np.random.default_rng(Nl)
    th, ph = np.arccos(rng.uniform(-1, 1, N)), rng.uniform(0, 2 * np.pi, N)
    _, got, ref = _pair(Nl, Nx, th, ph, rng.normal(size=N))
    assert _rel(got, ref) <= 1e-12


@pytest.mark.parametrize("case", ["one_point", "one_cell", "one_bin", "two_far_bins", "many_pieces", "edges"])
def test_point_layouts(case):
    rng = np.random.default_rng(3)
    Nl, Nx = 70, 30
    N = 1 if case == "one_point" else 60000 if case == "many_pieces" else 5000
    x, ph = rng.uniform(-0.7, 0.7, N), rng.uniform(0, 2 * np.pi, N)
    if case in ("one_cell", "one_bin", "many_pieces"):
        x = rng.uniform(0.301, 0.309, N)
    if case == "one_cell":
        ph = 1.0 + 1e-4 * rng.uniform(size=N)
    if case == "two_far_bins":
        x = np.where(rng.uniform(size=N) < 0.5, 0.301, -0.601)
    if case == "edges":
        ph = rng.choice([0.0, -0.0, 2 * np.pi, np.nextafter(2 * np.pi, 0), -np.pi, np.pi, -1e-300, 1e-17, 7.0, -40.0,
                         1e4, 3e7], N)
    th, w = np.arccos(x), rng.uniform(0.5, 1.5, N)
    d, got, ref = _pair(Nl, Nx, th, ph, w)
    assert _rel(got, ref) <= 1e-12
    assert _rel(got, O.direct_sht(O.build_tables(Nl, Nx), th, ph, w)) <= 1e-12


def test_maps_and_batch_share_the_route():
    from directsht_b200 import DirectSHT
    rng = np.random.default_rng(5)
    Nl, Nx, N = 60, 40, 30000  # 190 points per key: the automatic choice
    th, ph = np.arccos(rng.uniform(-1, 1, N)), rng.uniform(0, 2 * np.pi, N)
    w = rng.normal(size=(5, N))
    d = DirectSHT(Nl, Nx)
    maps = d.call_maps(th, ph, w)
    sets = d.call_batch([(th[:n], ph[:n], w[0, :n]) for n in (N, 200, 20000)])
    d.tune(bin_sums="fp64")
    for k in range(5):
        assert _rel(maps[k], d(th, ph, w[k])) <= 1e-12
    for got, n in zip(sets, (N, 200, 20000)):
        assert _rel(got, d(th[:n], ph[:n], w[0, :n])) <= 1e-12


def test_weights_that_are_not_finite_reach_every_coefficient():
    from directsht_b200 import DirectSHT
    rng = np.random.default_rng(6)
    th, ph = np.arccos(rng.uniform(-0.7, 0.7, 4000)), rng.uniform(0, 2 * np.pi, 4000)
    for bad in (np.nan, np.inf):
        w = np.ones(4000)
        w[17] = bad
        d = DirectSHT(20, 12)
        d.tune(bin_sums="nufft")
        assert not np.isfinite(d(th, ph, w)).any()


@pytest.mark.parametrize("scale", [2.0**1013, 2.0**-1000])
def test_weights_at_the_ends_of_the_range(scale):
    """Weights near the largest double (their sums still finite) and tiny ones: the alm are those of the
    unscaled weights times the power of two, as with the direct sums."""
    from directsht_b200 import DirectSHT
    rng = np.random.default_rng(8)
    th, ph, w = np.arccos(rng.uniform(-0.7, 0.7, 3000)), rng.uniform(0, 2 * np.pi, 3000), rng.normal(size=3000)
    w[5] = 1000.0
    d = DirectSHT(20, 12)
    for method in ("fp64", "nufft"):
        d.tune(bin_sums=method)
        ref, got = d(th, ph, w), d(th, ph, w * scale) / scale
        assert np.isfinite(ref).all() and np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max(), method
