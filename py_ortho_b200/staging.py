"""Copies of large host arrays to and from the device.

A copy between the device and ordinary (pageable) host memory goes through the driver on one thread:
measured 11 GB/s up, and 2.7 GB/s down into freshly allocated arrays, whose pages it touches one
after another. Here large arrays move in pieces through two pinned buffers, copied between the buffers
and the array by torch's CPU threads while the other buffer is on the bus. The buffers are taken from
torch's pinned-memory cache for the call and go back at its end; small arrays take the plain copy.
"""
from __future__ import annotations

import numpy as np
import torch

PIECE = 8 << 20          # bytes per pinned buffer
LARGE = 4 << 20          # arrays from this size on are staged


class _Ring:
    """Two pinned buffers of one dtype, used in turn."""

    def __init__(self, dtype: torch.dtype):
        n = PIECE // torch.empty((), dtype=dtype).element_size()
        self.n = n
        self.buf = [torch.empty(n, dtype=dtype, pin_memory=True) for _ in range(2)]
        self.done = [torch.cuda.Event() for _ in range(2)]


def _ring(dtype: torch.dtype):
    """A _Ring, or None where no memory can be pinned (a limit on locked pages): then the plain copy."""
    try:
        return _Ring(dtype)
    except RuntimeError:
        return None


def _plain() -> bool:
    """Staging waits for its own copies: not possible while the stream is being captured."""
    return torch.cuda.is_current_stream_capturing()


class _Readable:
    """An array's memory as torch.from_numpy takes it without a warning when the array is read-only."""

    def __init__(self, a: np.ndarray):
        self.array = a
        self.__array_interface__ = {**a.__array_interface__, "data": (a.__array_interface__["data"][0], False)}


def to_device(a: np.ndarray, device) -> torch.Tensor:
    """torch.from_numpy(a).to(device) for a C-contiguous array, which is only read (a decoded image or a
    mapped file may be read-only)."""
    src = torch.from_numpy(a if a.flags.writeable else np.asarray(_Readable(a)))
    if a.nbytes < LARGE or _plain():
        return src.to(device)
    ring = _ring(src.dtype)
    if ring is None:
        return src.to(device)
    out = torch.empty(src.shape, dtype=src.dtype, device=device)
    with torch.cuda.device(out.device):
        flat, dst = src.reshape(-1), out.view(-1)
        for k, o in enumerate(range(0, flat.numel(), ring.n)):
            m, b = min(ring.n, flat.numel() - o), k & 1
            if k >= 2:
                ring.done[b].synchronize()
            ring.buf[b][:m].copy_(flat[o:o + m])
            dst[o:o + m].copy_(ring.buf[b][:m], non_blocking=True)
            ring.done[b].record()
        for e in ring.done:
            e.synchronize()
    return out


def to_host(t: torch.Tensor) -> np.ndarray:
    """t.cpu().numpy(): waits for the work before it on the current stream, as .cpu() does."""
    if t.device.type != "cuda" or not t.is_contiguous() or t.numel() * t.element_size() < LARGE:
        return t.cpu().numpy()
    ring = _ring(t.dtype)
    if ring is None:
        return t.cpu().numpy()
    out = torch.empty(t.shape, dtype=t.dtype)
    with torch.cuda.device(t.device):
        src, dst = t.view(-1), out.view(-1)
        pieces = [(o, min(ring.n, src.numel() - o)) for o in range(0, src.numel(), ring.n)]

        def fetch(k):
            o, m = pieces[k]
            ring.buf[k & 1][:m].copy_(src[o:o + m], non_blocking=True)
            ring.done[k & 1].record()

        for k in range(min(2, len(pieces))):
            fetch(k)
        for k, (o, m) in enumerate(pieces):
            ring.done[k & 1].synchronize()
            dst[o:o + m].copy_(ring.buf[k & 1][:m])
            if k + 2 < len(pieces):
                fetch(k + 2)
    return out.numpy()
