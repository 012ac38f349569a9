"""Transforms that fit the fixed 64 MiB scratch with the direct sums also fit it where the FP64 level takes the NUFFT
sums: accepted, and equal to the ordinary call to 1e-12 x max|alm| (both the FP64 level's bound)."""
import ctypes as ct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nl,Nx,N", [(64, 2, 1000), (300, 256, 100_000), (300, 256, 200_000), (400, 64, 100_000),
                                     (400, 64, 200_000), (400, 129, 30_000)])
def test_nufft_sums_fit_where_the_direct_sums_do(Nl, Nx, N):
    import torch
    from directsht_b200 import DirectSHT, _lib as L
    lib = L.load()
    g = torch.Generator(device="cuda").manual_seed(N)
    u = torch.rand(3, N, generator=g, device="cuda", dtype=torch.float64)
    th, ph, w = torch.arccos(1.6 * u[0] - 0.8).contiguous(), (2 * np.pi * u[1]).contiguous(), u[2].contiguous()
    sht = DirectSHT(Nl, Nx)
    auto, direct = ct.c_size_t(), ct.c_size_t()
    L.check(lib.dsht_workspace_size(sht._plan, N, ct.byref(auto)))
    ref = sht(th, ph, w)
    alm = torch.empty(sht.Nlm, dtype=torch.complex128, device="cuda")
    L.check(lib.dsht_execute_noalloc(sht._plan, L.ptr(th), L.ptr(ph), L.ptr(w), N, L.DSHT_MODE_CALL, L.ptr(alm), None))
    torch.cuda.synchronize()
    assert (alm - ref).abs().max() <= 1e-12 * ref.abs().max()
    sht.tune(bin_sums="fp64")
    L.check(lib.dsht_workspace_size(sht._plan, N, ct.byref(direct)))
    # beyond the direct sums' scratch: the node slots of at most two runs per SM, and list padding
    assert auto.value <= direct.value + 4 * 8 * Nl * (4 * (Nx - 1) + 4 + 4 * 148) + (1 << 16)


# sizes within 0.2 % of the scratch, whose lists of the NUFFT sums must not push them over it
@pytest.mark.parametrize("Nl,Nx,N,precision", [(47, 835, 1267619, "fp64"), (16, 3275, 1229312, "fp64"),
                                               (14, 3074, 1337432, "fp64"), (67, 7601, 310, "fp64"),
                                               (56, 833, 1156000, "mixed"), (54, 657, 1283368, "mixed_f64_tables")])
def test_sizes_at_the_limit(Nl, Nx, N, precision):
    import torch
    from directsht_b200 import DirectSHT, _lib as L
    lib = L.load()
    g = torch.Generator(device="cuda").manual_seed(N)
    u = torch.rand(3, N, generator=g, device="cuda", dtype=torch.float64)
    th, ph, w = torch.arccos(2 * u[0] - 1).contiguous(), (2 * np.pi * u[1]).contiguous(), u[2].contiguous()
    sht = DirectSHT(Nl, Nx, precision=precision)
    size = ct.c_size_t()
    L.check(lib.dsht_workspace_size(sht._plan, N, ct.byref(size)))
    assert size.value <= lib.dsht_noalloc_scratch_bytes()
    ref = sht(th, ph, w)
    alm = torch.empty(sht.Nlm, dtype=torch.complex128, device="cuda")
    L.check(lib.dsht_execute_noalloc(sht._plan, L.ptr(th), L.ptr(ph), L.ptr(w), N, L.DSHT_MODE_CALL, L.ptr(alm), None))
    torch.cuda.synchronize()
    assert (alm - ref).abs().max() <= (1e-12 if precision == "fp64" else 1e-7) * ref.abs().max()
