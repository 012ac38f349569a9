"""Host <-> device copies through pinned chunks: sizes around the direct-copy limit and the chunk
boundaries come back byte for byte, from several threads and streams at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sizes():
    from directsht_b200 import hostcopy as H
    c, m = H._CHUNK // 8, H._MIN_BYTES // 8
    return [0, 1, m - 1, m, m + 1, c - 1, c, c + 1, 3 * c, 3 * c + 5, 7 * c - 3]


def test_round_trip():
    from directsht_b200.hostcopy import to_device, to_host
    rng = np.random.default_rng(0)
    for n in _sizes():
        a = rng.normal(size=n)
        keep = a.copy()
        d = to_device(a, "cuda")
        a[:] = 0.0  # the source may change at once
        np.testing.assert_array_equal(to_host(d), keep)
    for a in (rng.normal(size=(3, 250001)).astype(np.float32), rng.normal(size=400001) + 1j * rng.normal(size=400001)):
        d = to_device(a, "cuda")
        assert tuple(d.shape) == a.shape
        np.testing.assert_array_equal(to_host(d), a)
    d = to_device(rng.normal(size=(1000, 600)), "cuda")
    np.testing.assert_array_equal(to_host(d.t()), d.t().cpu().numpy())  # not contiguous


def test_threads_and_streams():
    import torch
    from directsht_b200.hostcopy import to_device, to_host
    bad = []

    def work(seed):
        rng = np.random.default_rng(seed)
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(5):
                a = rng.normal(size=900000)
                if not np.array_equal(to_host(to_device(a, "cuda") * 2.0), a * 2.0):
                    bad.append(seed)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_pinned_views_are_copied_directly():
    """A numpy view of pinned memory keeps the link's rate: one copy, no staging, the same bytes."""
    import torch
    from directsht_b200.hostcopy import to_device
    p = torch.empty(3 << 20, dtype=torch.uint8).pin_memory()
    a = p.numpy()
    a[:] = np.arange(a.size, dtype=np.int64) % 251
    d = to_device(a, torch.device("cuda"))
    assert torch.equal(d.cpu(), p)


def test_other_default_device():
    """Programs that make CUDA the default device (or float32 the default type) get the same copies."""
    import torch
    from directsht_b200.hostcopy import to_device, to_host
    a = np.random.default_rng(1).normal(size=700001)
    with torch.device("cuda"):
        np.testing.assert_array_equal(to_host(to_device(a, "cuda")), a)


@pytest.mark.parametrize("threads", [1, 2, 4])
def test_any_number_of_host_threads(threads):
    """Few intra-op threads take the direct copies up to 32 MB and the staged ones above (out, or from two
    threads in): the same bytes either way."""
    import torch
    from directsht_b200 import hostcopy as H
    keep = torch.get_num_threads()
    try:
        torch.set_num_threads(threads)
        small, large = H._LARGE - 8, H._LARGE + 8
        assert [H._staged(small, 2), H._staged(large, 2), H._staged(small, 1), H._staged(large, 1)] == \
            [threads >= 4, threads >= 2, threads >= 4, True]
        for nbytes in (H._MIN_BYTES - 8, H._MIN_BYTES, small, large):
            a = np.random.default_rng(threads).normal(size=nbytes // 8)
            np.testing.assert_array_equal(H.to_host(H.to_device(a, "cuda")), a)
    finally:
        torch.set_num_threads(keep)
