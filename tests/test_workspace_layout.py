"""Workspaces hold every transform that runs on them (no device needed: the sizes are host arithmetic).

A transform of n points on K = min(keys, n) bins with points, in pieces of p points, has at most
K + (n - K) // p pieces: sum of ceil(c / p) over the bins, largest with c = 1 mod p in all bins but one."""
import ctypes as ct

import pytest

from directsht_b200 import _lib as L

LEVELS = [L.DSHT_PREC_FP64, L.DSHT_PREC_MIXED, L.DSHT_PREC_MIXED_F64_TABLES]


def layout(Nl, Nx, level, N, ntrans, n, bin_sums=0, piece_max=0):
    out = (ct.c_int64 * 6)()
    L.check(L.load().dsht_test_layout(Nl, Nx, level, bin_sums, piece_max, N, ntrans, n, out))
    return dict(zip(("bytes", "call", "pieces", "nufft", "piece", "grid"), out))


def nufft_from(Nl, Nx, level, **kw):
    """Fewest points that take the NUFFT sums."""
    lo, hi = 0, 1 << 31
    while hi - lo > 1:
        mid = (lo + hi) // 2
        if layout(Nl, Nx, level, mid, 0, mid, **kw)["nufft"] >= 0:
            hi = mid
        else:
            lo = mid
    return hi


@pytest.mark.parametrize("level", LEVELS)
@pytest.mark.parametrize("piece_max", [0, 256, 1024, 65536])
def test_batch_lists_hold_the_pieces_of_every_smaller_transform(level, piece_max):
    for Nl, Nx in ((1, 2), (1, 16), (1, 40), (2, 3), (2, 16), (3, 90), (8, 40), (33, 300), (257, 64), (513, 1000), (2048, 9)):
        kw = dict(piece_max=piece_max)
        start = nufft_from(Nl, Nx, level, **kw)
        keys = 4 * (Nx - 1)
        for N in (start, start + 1, start + 4097, 3 * start, 524289, 600001, 5000001):
            for n in (1, keys, start // 2, start - 2, start - 1, start, 524288, 524289, 4194304, N - 1, N):
                if not 1 <= n <= N:
                    continue
                got = layout(Nl, Nx, level, N, 2, n, **kw)
                K = min(keys, n)
                assert K + (n - K) // got["piece"] <= got["pieces"], (Nl, Nx, N, n, got)


@pytest.mark.parametrize("level", LEVELS)
def test_a_workspace_for_the_nufft_sums_serves_the_direct_sums_below(level):
    for Nl, Nx in ((1, 2), (1, 16), (2, 16), (3, 90), (33, 300), (47, 835), (257, 64), (513, 1000)):
        start = nufft_from(Nl, Nx, level)
        for ntrans in (0, 3):
            sizes = [layout(Nl, Nx, level, N, ntrans, 1)["bytes"] for N in (start // 2, start - 1, start, 2 * start)]
            assert sizes == sorted(sizes), (Nl, Nx, sizes)
