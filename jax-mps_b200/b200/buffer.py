"""The device array of the Python face. A module of its own because its class derives from a type of the extension module
(csrc/hot.c), which `import b200` alone does not load."""
from __future__ import annotations

import ctypes as C

import numpy as np

from . import _DT_NAMES, _DT_TO_NP, _P, BF16, Event, _check, _hot, load_library


class Buffer(_hot.Handle):
    """A device array (PJRT_Buffer), made from its client and its handle (`_h`), which it owns."""

    @property
    def dtype_code(self) -> int:
        return load_library().b200_buffer_dtype(self._h)

    @property
    def dtype(self) -> str:
        return _DT_NAMES[self.dtype_code]

    @property
    def shape(self) -> tuple:
        lib = load_library()
        n = lib.b200_buffer_num_dims(self._h)
        d = lib.b200_buffer_dims(self._h)
        return tuple(int(d[i]) for i in range(n))

    @property
    def nbytes(self) -> int:
        return load_library().b200_buffer_on_device_size(self._h)

    def device_pointer(self) -> int:
        return load_library().b200_buffer_device_pointer(self._h) or 0

    def is_deleted(self) -> bool:
        return bool(load_library().b200_buffer_is_deleted(self._h))

    def delete(self):
        _check(load_library().b200_buffer_delete(self._h))

    def copy(self) -> "Buffer":
        out = _P()
        _check(load_library().b200_buffer_copy(self._h, C.byref(out)))
        return Buffer(self.client, out.value)

    def block_until_ready(self) -> "Buffer":
        ev = _P()
        _check(load_library().b200_buffer_ready_event(self._h, C.byref(ev)))
        Event(ev.value).wait()
        return self

    def to_host_async(self, out: np.ndarray) -> Event:
        """Start a device-to-host copy into `out` (same shape/dtype; pinned memory makes it truly asynchronous)."""
        size = C.c_size_t(out.nbytes)
        ev = _P()
        _check(load_library().b200_buffer_to_host(self._h, out.ctypes.data_as(_P), C.byref(size), C.byref(ev)))
        return Event(ev.value)

    def to_numpy(self) -> np.ndarray:
        """bf16 buffers come back as float32 (exactly representable)."""
        code = self.dtype_code
        nbytes = self.nbytes
        if 65536 <= nbytes <= 1 << 24:
            block = _hot.to_block(self, nbytes)              # page-locked memory, given back with the array
            if block is not None:
                out = np.frombuffer(block, dtype=_DT_TO_NP[code]).reshape(self.shape)
                return (out.astype(np.uint32) << 16).view(np.float32) if code == BF16 else out
        out = np.empty(self.shape, dtype=_DT_TO_NP[code])
        size = C.c_size_t(out.nbytes)
        _check(load_library().b200_buffer_to_host(self._h, out.ctypes.data_as(_P), C.byref(size), None))
        if code == BF16:
            return (out.astype(np.uint32) << 16).view(np.float32)
        return out

    def __array__(self, dtype=None, copy=None):
        a = self.to_numpy()
        return a.astype(dtype) if dtype is not None else a
