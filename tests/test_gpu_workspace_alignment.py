"""A workspace that is aligned to 16 bytes only serves every bin-sum method as one aligned to 256 does: the
tensor-core sums' stores of whole sectors need 32.  The same transform twice; differences come from the order of FP64
sums alone (1e-12 x max|alm|; the points of a key lie in one piece)."""
import ctypes as ct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level,sums", [("mixed", "tc"), ("mixed", "nufft"), ("mixed_f64_tables", "tc"), ("fp64", "fp64"),
                                        ("fp64", "nufft")])
@pytest.mark.parametrize("Nl", [64, 100, 33])
def test_sixteen_byte_workspace(Nl, level, sums):
    import torch
    from directsht_b200 import DirectSHT, _lib as L
    lib = L.load()
    N, Nx = 5000, 40
    g = torch.Generator(device="cuda").manual_seed(Nl)
    u = torch.rand(3, N, generator=g, device="cuda", dtype=torch.float64)
    th, ph, w = torch.arccos(2 * u[0] - 1).contiguous(), (2 * np.pi * u[1]).contiguous(), u[2].contiguous()
    sht = DirectSHT(Nl, Nx, precision=level)
    sht.tune(bin_sums=sums)
    nb = ct.c_size_t()
    L.check(lib.dsht_workspace_size(sht._plan, N, ct.byref(nb)))
    ws = torch.empty(nb.value + 256, dtype=torch.uint8, device="cuda")
    assert ws.data_ptr() % 256 == 0
    alms = []
    for off in (0, 16, 48):
        alm = torch.empty(sht.Nlm, dtype=torch.complex128, device="cuda")
        L.check(lib.dsht_execute(sht._plan, L.ptr(th), L.ptr(ph), L.ptr(w), N, L.DSHT_MODE_CALL, L.ptr(alm),
                                 ct.c_void_p(ws.data_ptr() + off), nb.value,
                                 ct.c_void_p(torch.cuda.current_stream().cuda_stream)))
        torch.cuda.synchronize()
        alms.append(alm)
    for a in alms[1:]:
        assert (a - alms[0]).abs().max() <= 1e-12 * alms[0].abs().max()
