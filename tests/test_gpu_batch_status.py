"""A contraction pass serves several transforms of a batch; when a bounded wait inside it runs out, the
alm of all of them are invalid, and the status word of each says so -- and of no other transform.  The
test hook makes the next contraction launch withhold one signal (a barrier that nothing completes): the
kernel gives up after about a second, the device stays usable and the next batch is right."""
import ctypes as ct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed_f64_tables", "mixed"])
def test_timeout_reaches_every_status_of_the_pass(precision):
    import torch
    from directsht_b200 import DirectSHT
    from directsht_b200 import _lib as L
    Nl, Nx, N, n = 64, 40, 2000, 5
    rng = np.random.default_rng(0)
    sets = [tuple(torch.from_numpy(a).cuda() for a in (np.arccos(rng.uniform(-1, 1, N)),
                                                       rng.uniform(0, 2 * np.pi, N), rng.normal(size=N)))
            for _ in range(n)]
    d = DirectSHT(Nl, Nx, precision=precision)
    d.tune(maps_per_pass=3)  # passes of transforms 0-2 and 3-4
    alms = [torch.empty(d.Nlm, dtype=torch.complex128, device="cuda") for _ in range(n)]
    status = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    nb = ct.c_size_t()
    L.check(d._lib.dsht_workspace_size_batch(d._plan, N, n, ct.byref(nb)))
    ws = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    arr = lambda k: (ct.c_void_p * n)(*[s[k].data_ptr() for s in sets])

    def run():
        out = (ct.c_void_p * n)(*[a.data_ptr() for a in alms])
        L.check(d._lib.dsht_enqueue_batch(d._plan, n, arr(0), arr(1), arr(2), (ct.c_int64 * n)(*[N] * n),
                                          L.DSHT_MODE_CALL, out, L.ptr(status), L.ptr(ws), ws.numel(),
                                          ct.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return [d._lib.dsht_status(int(f) & 0xffffffff, L.DSHT_MODE_CALL) for f in status.cpu().numpy()]

    assert run() == [L.DSHT_OK] * n
    good = [a.cpu().numpy() for a in alms]
    assert d._lib.dsht_test_stall_next_contraction() == L.DSHT_OK
    assert run() == [L.DSHT_ERR_CUDA] * 3 + [L.DSHT_OK] * 2
    assert run() == [L.DSHT_OK] * n
    for a, g in zip(alms, good):
        assert np.abs(a.cpu().numpy() - g).max() <= 1e-12 * np.abs(g).max()
