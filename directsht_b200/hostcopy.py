"""Copies between pageable host arrays and the device through pinned chunks.

A copy from or to pageable memory runs at the driver's single-threaded staging rate (17 GB/s in,
13 GB/s out measured).  Here the host side of every chunk is copied by all intra-op threads into (out of)
one of three pinned buffers while the chunk before it is on the link: 30 GB/s in, 27 GB/s out (11 MB: 630
to 370 us in, 860 to 420 us out).  The buffers (6 MB per call) come from PyTorch's pinned-memory
allocator, which reuses them and keeps a freed one until the copies queued from it have run.  Below
_MIN_BYTES a direct copy is as fast.  All but the large arrays are copied directly where few intra-op
threads are set (launchers of several processes set one): there the host side is the slower one.
"""
from __future__ import annotations

import numpy as np
import torch

_CHUNK = 1 << 21      # bytes per pinned buffer
_BUFFERS = 3
_MIN_BYTES = 1 << 20
_LARGE = 32 << 20     # arrays that the host allocator maps afresh


def _staged(nbytes, threads_if_large):
    """Whether all intra-op threads together outrun the driver's copy: with four threads and more (16 MB
    in / out 900 / 941 us direct, 634 / 573 staged), not with fewer (one: 1368 / 1493, two: 1002 / 882);
    from _LARGE with threads_if_large: pages are first touched on the way (100 MB in with one thread 8.5
    ms direct, 10.1 staged, with two 6.7; out 48 direct, 39 with one).  A call with arrays of 500000 points
    took 1406 us staged with one thread, 1068 directly."""
    return torch.get_num_threads() >= (threads_if_large if nbytes >= _LARGE else 4)


def _chunks(nbytes):
    return [(o, min(_CHUNK, nbytes - o)) for o in range(0, nbytes, _CHUNK)]


def _buffers(count):
    n = min(_BUFFERS, count)
    return ([torch.empty(_CHUNK, dtype=torch.uint8, device="cpu", pin_memory=True) for _ in range(n)],
            [torch.cuda.Event() for _ in range(n)])


def to_device(a: np.ndarray, device) -> torch.Tensor:
    """A device copy of a contiguous host array, queued on the current stream; ``a`` may be changed as
    soon as this returns."""
    src = torch.from_numpy(a)
    # (pinned memory, of a tensor, say, needs no staging: 55 GB/s)
    if a.nbytes < _MIN_BYTES or not _staged(a.nbytes, 2) or src.is_pinned():
        return src.to(device=device, non_blocking=False)
    out = torch.empty(src.shape, dtype=src.dtype, device=device)
    s, d = src.reshape(-1).view(torch.uint8), out.reshape(-1).view(torch.uint8)
    parts = _chunks(a.nbytes)
    bufs, events = _buffers(len(parts))
    for i, (o, n) in enumerate(parts):
        b, e = bufs[i % len(bufs)], events[i % len(bufs)]
        if i >= len(bufs):
            e.synchronize()  # the buffer's last copy has left it
        b[:n].copy_(s[o:o + n])
        d[o:o + n].copy_(b[:n], non_blocking=True)
        e.record()
    return out


def to_host(t: torch.Tensor) -> np.ndarray:
    """A host copy of a device tensor (waits for the work queued on the current stream)."""
    nbytes = t.numel() * t.element_size()
    if nbytes < _MIN_BYTES or not _staged(nbytes, 1) or not t.is_contiguous():
        return t.cpu().numpy()
    out = torch.empty(t.shape, dtype=t.dtype, device="cpu")
    flat = (torch.view_as_real(t) if t.is_complex() else t).reshape(-1).view(torch.uint8)
    dst = (torch.view_as_real(out) if t.is_complex() else out).reshape(-1).view(torch.uint8)
    parts = _chunks(nbytes)
    bufs, events = _buffers(len(parts))

    def issue(i):
        o, n = parts[i]
        bufs[i % len(bufs)][:n].copy_(flat[o:o + n], non_blocking=True)
        events[i % len(bufs)].record()

    for i in range(len(bufs)):
        issue(i)
    for i, (o, n) in enumerate(parts):
        events[i % len(bufs)].synchronize()
        dst[o:o + n].copy_(bufs[i % len(bufs)][:n])
        if i + len(bufs) < len(parts):
            issue(i + len(bufs))
    return out.numpy()
