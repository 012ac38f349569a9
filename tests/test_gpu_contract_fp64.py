"""The FP64 contraction at the edges of its tiles: blocks of 128 rows, stages of 32 nodes, groups
of eight nodes, one to four maps per pass, odd and tiny Nx.

Tolerance: the FP64 level's bound, 1e-12 x max|alm| (a product of K = 2 Nx rounded terms errs by
at most K 2^-53 of the sum of their magnitudes, below 1e-13 of it for these sizes)."""
import numpy as np
import pytest

from oracle import dsht_oracle as O

pytestmark = pytest.mark.gpu


def _sky(rng, N):
    return np.arccos(rng.uniform(-1, 1, N)), rng.uniform(0, 2 * np.pi, N)


@pytest.mark.parametrize("Nl,Nx", [(1, 2), (2, 3), (8, 7), (9, 8), (16, 9), (17, 31), (63, 32), (65, 33), (127, 64),
                                   (128, 65), (129, 17), (130, 130), (257, 40)])
def test_row_and_node_edges(Nl, Nx):
    from directsht_b200 import DirectSHT
    rng = np.random.default_rng(Nl * 1000 + Nx)
    th, ph = _sky(rng, 400)
    w = rng.normal(size=400)
    ref = O.direct_sht(O.build_tables(Nl, Nx), th, ph, w)
    got = DirectSHT(Nl, Nx)(th, ph, w)
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("nmaps", [1, 2, 3, 4, 5, 9])
@pytest.mark.parametrize("Nl,Nx", [(40, 77), (140, 50)])
def test_maps_per_pass(Nl, Nx, nmaps):
    from directsht_b200 import DirectSHT
    rng = np.random.default_rng(nmaps)
    th, ph = _sky(rng, 300)
    w = rng.normal(size=(nmaps, 300))
    tab = O.build_tables(Nl, Nx)
    d = DirectSHT(Nl, Nx)
    got = d.call_maps(th, ph, w)
    for k in range(nmaps):
        ref = O.direct_sht(tab, th, ph, w[k])
        assert np.abs(got[k] - ref).max() <= 1e-12 * np.abs(ref).max(), k


def test_point_sets_with_other_empty_nodes_share_a_pass():
    """Stages that are empty for one set of a batch and not for the other."""
    from directsht_b200 import DirectSHT
    rng = np.random.default_rng(7)
    Nl, Nx = 150, 300
    tab = O.build_tables(Nl, Nx)
    sets = []
    for lo, hi in ((0.1, 0.2), (-0.74, -0.6), (0.0, 0.74), (0.3, 0.31)):
        sets.append((np.arccos(rng.uniform(lo, hi, 200)), rng.uniform(0, 2 * np.pi, 200), rng.normal(size=200)))
    got = DirectSHT(Nl, Nx).call_batch(sets)
    for g, (t, p, w) in zip(got, sets):
        ref = O.direct_sht(tab, t, p, w)
        assert np.abs(g - ref).max() <= 1e-12 * np.abs(ref).max()


def test_no_points_in_range_gives_zeros():
    from directsht_b200 import DirectSHT
    got = DirectSHT(140, 40)(np.full(5, np.nan), np.zeros(5), np.ones(5))
    assert not got.any()


# grids whose padding nodes (beyond Nx, up to a whole group of eight) include x = 1
@pytest.mark.parametrize("precision", ["fp64", "mixed_f64_tables", "mixed"])
@pytest.mark.parametrize("Nl,Nx,xmax", [(20, 4, 0.75), (20, 10, 0.75), (20, 17, 0.8), (20, 19, 0.9), (40, 49, 0.96),
                                        (40, 100, 0.99)])
def test_padding_nodes_at_x_equal_to_one(Nl, Nx, xmax, precision):
    from directsht_b200 import DirectSHT
    dx = xmax / (Nx - 1)
    assert any(j * dx == 1.0 for j in range(Nx, (Nx + 7) // 8 * 8))
    rng = np.random.default_rng(Nx)
    th, ph = _sky(rng, 600)  # below the 1024 points from which the mixed levels leave the FP64 stages
    w = rng.normal(size=(2, 600))
    tab = O.build_tables(Nl, Nx, xmax)
    d = DirectSHT(Nl, Nx, xmax, precision=precision)
    maps = d.call_maps(th, ph, w)
    for k in range(2):
        ref = O.direct_sht(tab, th, ph, w[k])
        tol = 1e-12 * np.abs(ref).max()
        assert np.abs(d(th, ph, w[k]) - ref).max() <= tol
        assert np.abs(maps[k] - ref).max() <= tol
