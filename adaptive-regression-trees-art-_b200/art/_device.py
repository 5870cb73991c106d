"""Device plumbing: PyTorch owns device memory and streams; kernels run through the C ABI."""

from __future__ import annotations

import threading

import numpy as np


def torch():
    import torch as _torch

    return _torch


def require_cuda():
    """Return the current CUDA device, raising if the B200 path cannot run."""

    t = torch()
    if not t.cuda.is_available():
        raise RuntimeError(
            "art_b200 requires a CUDA device (sm_100); no CPU fallback exists for this path."
        )
    return t.device("cuda", t.cuda.current_device())


def stream_handle(stream=None) -> int:
    t = torch()
    s = t.cuda.current_stream() if stream is None else stream
    return int(s.cuda_stream)


def ptr(tensor) -> int | None:
    if tensor is None:
        return None
    return int(tensor.data_ptr())


def to_device(array, dtype=None, device=None):
    """numpy / torch -> contiguous CUDA tensor (no copy if already suitable)."""

    t = torch()
    device = require_cuda() if device is None else device
    if isinstance(array, t.Tensor):
        out = array.to(device=device, dtype=dtype if dtype is not None else array.dtype)
        return out.contiguous()
    arr = np.ascontiguousarray(array, dtype=None if dtype is None else _np_dtype(dtype))
    if not arr.flags.writeable:  # read-only views (broadcasts, loaded buffers): torch wants a writable array
        arr = arr.copy()
    return t.from_numpy(arr).to(device=device, non_blocking=False).contiguous()


# Staging through pinned memory: a pageable copy moves 17 GB/s here, threads
# fill pinned chunks at 190 GB/s and those move at 53 GB/s.  A call holds at
# most _CHUNKS chunks, which torch's allocator of pinned memory keeps for the
# next call of any thread; nothing is shared between calls.
_CHUNK = 2 << 20
_CHUNKS = 3


def _pinned(nbytes):
    t = torch()
    return t.empty(nbytes, dtype=t.uint8, pin_memory=True)


def upload_rows(array, dtype=None, device=None):
    """to_device for large host arrays, by pinned chunks: complete on the current
    stream, not on others; the host array is free when it returns."""

    t = torch()
    device = require_cuda() if device is None else device
    if isinstance(array, t.Tensor):
        return to_device(array, dtype, device)
    arr = np.ascontiguousarray(array, dtype=None if dtype is None else _np_dtype(dtype))
    if arr.nbytes < _CHUNK or not arr.flags.writeable or t.get_num_threads() == 1:
        return to_device(arr, dtype, device)
    src = t.from_numpy(arr)
    out = t.empty(src.shape, dtype=src.dtype, device=device)
    flat, to = src.view(-1).view(t.uint8), out.view(-1).view(t.uint8)
    slots = []
    for k, at in enumerate(range(0, arr.nbytes, _CHUNK)):
        n = min(_CHUNK, arr.nbytes - at)
        if k < _CHUNKS:
            slots.append([_pinned(_CHUNK), None])
        buf, done = slot = slots[k % _CHUNKS]
        if done is not None:
            done.synchronize()
        buf[:n].copy_(flat[at:at + n])
        to[at:at + n].copy_(buf[:n], non_blocking=True)
        if at + _CHUNKS * _CHUNK < arr.nbytes:
            slot[1] = t.cuda.Event()
            slot[1].record()
    return out


def pack(arrays, device=None):
    """Host arrays as views of one device buffer, each at a 256-byte boundary, by
    one copy on the current stream."""

    t = torch()
    device = require_cuda() if device is None else device
    places, total = [], 0
    for a in arrays:
        places.append(total)
        total += -(-a.nbytes // 256) * 256
    host = _pinned(total)
    for a, at in zip(arrays, places):
        host[at:at + a.nbytes].numpy().view(a.dtype).reshape(a.shape)[...] = a
    dev = t.empty(total, dtype=t.uint8, device=device)
    dev.copy_(host, non_blocking=True)
    return [dev[at:at + a.nbytes].view(t.from_numpy(a[:0]).dtype).view(a.shape) for a, at in zip(arrays, places)]


def download(*tensors):
    """numpy arrays of device tensors, with one wait for all of them."""

    t = torch()
    total = sum(x.numel() * x.element_size() for x in tensors)
    if not 0 < total <= _CHUNKS * _CHUNK:
        return [x.cpu().numpy() for x in tensors]
    host, at, views = _pinned(total), 0, []
    for x in tensors:  # widest elements first: every view is aligned
        n = x.numel() * x.element_size()
        views.append(host[at:at + n].view(x.dtype).view(x.shape))
        views[-1].copy_(x, non_blocking=True)
        at += n
    t.cuda.current_stream().synchronize()
    return [t.empty(v.shape, dtype=v.dtype).copy_(v).numpy() for v in views]


def _np_dtype(torch_dtype):
    t = torch()
    return {
        t.float64: np.float64,
        t.float32: np.float32,
        t.int64: np.int64,
        t.int32: np.int32,
        t.int8: np.int8,
        t.uint8: np.uint8,
    }[torch_dtype]


class _WorkspaceCache:
    """One growing byte buffer per (device, stream): workspaces must not be shared
    by calls that may overlap on the GPU."""

    def __init__(self):
        self._buffers = {}
        self._lock = threading.Lock()

    def get(self, nbytes: int, stream=None):
        t = torch()
        device = require_cuda()
        key = (device.index, stream_handle(stream))
        with self._lock:
            buf = self._buffers.get(key)
            if buf is None or buf.numel() < nbytes:
                size = max(int(nbytes), 1 << 16)
                if buf is not None:
                    size = max(size, 2 * buf.numel())
                buf = t.empty(size, dtype=t.uint8, device=device)
                self._buffers[key] = buf
            return buf


WORKSPACES = _WorkspaceCache()
