"""Small host arrays to the device without stalling the host.

A copy from ordinary host memory makes the caller wait until the stream has drained; a copy
from pinned memory does not, but reads the pinned bytes when the stream gets to it, by which
time the host may have written the next step's values.  So every array is first copied into
the next buffer of a ring of pinned buffers and sent from there; a buffer is reused only after
the copy that read it has run (an event per buffer says so).  The ring is native code
(``csrc/upload.cu``): a step sends two or three such arrays before its first kernel.
"""
from __future__ import annotations

import ctypes
import threading
import weakref
from typing import Optional

import numpy as np
import torch


def _close(native, ring: int, slab: torch.Tensor) -> None:
    """Waits for the copies that still read the pinned memory, which goes back to torch's allocator with its last reference."""
    native.qnn_upload_ring_free(ring)


class PinnedUploader:
    def __init__(self, device, entries: int = 8, nbytes: int = 1 << 16):
        self.device = torch.device(device)
        self.on_gpu = self.device.type == "cuda"
        self.entries = entries
        self._nbytes = nbytes
        self._ring: Optional[int] = None
        self._lib = None
        self._opening = threading.Lock()
        self.bytes_sent = 0

    def _open(self) -> None:
        from ..kernels import lib
        with self._opening:
            if self._ring is not None:
                return
            ring, native = ctypes.c_void_p(), lib.load()
            slab = torch.empty(self.entries * self._nbytes, dtype=torch.uint8, pin_memory=True)
            lib.check(native.qnn_upload_ring(self.entries, self._nbytes, slab.data_ptr(), ctypes.byref(ring)), "upload_ring", 0)
            self._lib = lib
            self._ring = ring.value
            weakref.finalize(self, _close, native, ring.value, slab)

    def send(self, dst: torch.Tensor, src: np.ndarray) -> None:
        """dst (contiguous) = src, ordered on the current stream of dst's device; a dst in host memory gets the bytes at once."""
        src = np.ascontiguousarray(src)
        n = src.nbytes
        if dst.numel() * dst.element_size() != n or not dst.is_contiguous():
            raise ValueError(f"upload of {n} bytes into a tensor of {dst.numel() * dst.element_size()} bytes")
        self.bytes_sent += n
        if n == 0:
            return
        if not self.on_gpu or not dst.is_cuda:
            dst.view(torch.uint8).reshape(-1).copy_(torch.from_numpy(src.view(np.uint8).reshape(-1)))
            return
        if self._ring is None:
            self._open()
        stream = torch._C._cuda_getCurrentRawStream(dst.device.index)
        self._lib.check(self._lib.load().qnn_upload(self._ring, dst.data_ptr(), src.__array_interface__["data"][0], n, dst.device.index, stream),
                        "upload", 0)
