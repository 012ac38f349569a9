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


def test_a_size_asked_for_once_serves_every_precision_level():
    for Nl, Nx in ((1, 16), (16, 40), (47, 835), (257, 64), (513, 1000), (2048, 9), (100, 9000)):
        for ntrans in (0, 1, 5):
            for N in (1, 1000, 1023, 1024, 30_000, 400_000, 3_000_000):
                got = [layout(Nl, Nx, level, N, ntrans, 1) for level in LEVELS]
                assert len({g["bytes"] for g in got}) == 1
                assert all(g["call"] <= g["bytes"] for g in got)


def _per_piece_layout(Nl, Nx, N, level):
    """Bytes of a single transform with every list kept, sums per piece of the direct sums (at the mixed
    levels of pieces of 8192 points from 512 points per key) and both halves' alm beside the result: what
    fits the fixed scratch of dsht_execute_noalloc in this form is promised to fit it."""
    keys, nlm = 4 * (Nx - 1), Nl * (Nl + 1) // 2
    if level != L.DSHT_PREC_FP64 and N >= max(1024, 512 * keys):
        extra = max(-(-N // 8192), 2048, -(-512 * keys // 2048))
    else:
        extra = -(-N // min(2048, max(256, -(-N // 2048))))
    pieces = min(keys, N) + extra
    fold = max(128 * Nl * Nx, 32 * Nl * ((2 * Nx + 63) // 64 * 64))
    parts = ([4 * N, 32 * N] + 4 * [4 * (keys + 1)] + [4 * pieces, 8 * pieces, 4 * pieces, 4 * pieces, 8 * pieces, 4, 4]
             + [64 * Nl * pieces, fold, 4, 16, 4, 2 * -(-Nx // 128), 2 * -(-Nx // 256), 16 * nlm, 16 * nlm])
    return sum(-(-b // 256) * 256 for b in parts)


def test_what_fits_the_fixed_scratch_per_piece_fits_it():
    import math
    import random
    rng = random.Random(3)
    scratch = L.load().dsht_noalloc_scratch_bytes()
    sizes = [(47, 835), (16, 3275), (14, 3074), (56, 833), (54, 6065), (67, 7601), (53, 9537)]
    sizes += [(int(math.exp(rng.uniform(0, math.log(2048)))), int(math.exp(rng.uniform(math.log(2), math.log(12288)))))
              for _ in range(1500)]
    for Nl, Nx in sizes:
        for level in LEVELS:
            if _per_piece_layout(Nl, Nx, 1, level) > scratch:
                continue
            lo, hi = 1, 2_000_000  # the largest N that fits
            while hi - lo > 1:
                mid = (lo + hi) // 2
                lo, hi = (mid, hi) if _per_piece_layout(Nl, Nx, mid, level) <= scratch else (lo, mid)
            for N in {lo, max(1, lo - rng.randrange(300)), rng.randrange(1, lo + 1), min(lo, 1023), min(lo, 1024)}:
                if _per_piece_layout(Nl, Nx, N, level) <= scratch:
                    assert layout(Nl, Nx, level, N, 0, 1)["bytes"] <= scratch, (Nl, Nx, N, level)


def test_autotune_times_pieces_that_differ():
    from directsht_b200.batch import piece_candidates
    for level in LEVELS:
        cand = piece_candidates(level == L.DSHT_PREC_MIXED)
        for Nl, Nx, N in ((200, 100, 1_000_000), (1024, 300, 2_000_000), (2048, 4096, 9_000_000), (500, 1000, 100_000)):
            got = [layout(Nl, Nx, level, N, 1, N, piece_max=c)["piece"] for c in cand if c < 2048]
            assert len(set(got)) == len(got), (level, Nl, Nx, N, got)
