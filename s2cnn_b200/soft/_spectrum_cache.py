"""Per-module caches around the transform of the kernel.

``S2Convolution`` / ``SO3Convolution`` transform ``kernel * scaling`` to the spectral domain in
every forward pass (s2cnn/soft/s2_conv.py:41, so3_conv.py:47).

* ``KernelSpectrumCache``: the result depends on the weights alone, so in inference it is the same
  tensor pass after pass; the cache keeps it while the parameter has not been written to (its version
  counter, storage and device are unchanged) and no gradient with respect to it is being recorded.
  During training the transform runs every time, as autograd needs it in the graph.
* ``FourierMatrices``: the Fourier matrices of the layer's grid; the products scale the kernel while
  they read it and its gradient while they write it, so neither ``kernel * scaling`` nor its gradient is
  a pass, or a matrix, of its own.

Each keeps one entry as a single tuple: replaced in one assignment, so a reader in another thread
never sees half of one entry and half of another.  Copies and pickles of a module start empty.

Passes may run on any stream: a spectrum is read elsewhere only after the event that follows its
making, and the allocator learns which streams read a kept tensor (``s2_ft.read_on_current_stream``).
A pass under capture reads what was there before (``torch.cuda.graph`` synchronizes the device before
it captures) and leaves nothing: what it makes itself is filled by the replays only.
"""
import torch

from ..s2_ft import _raw_stream, made_on_current_stream, read_on_current_stream


class _OneEntry:
    def __init__(self):
        self._entry = None

    def __deepcopy__(self, memo):
        return type(self)()

    def __reduce__(self):
        return (type(self), ())

    def clear(self):
        self._entry = None


class KernelSpectrumCache(_OneEntry):
    def get(self, kernel, transform):
        if torch.is_grad_enabled() and kernel.requires_grad:
            return transform(kernel)
        key = (kernel._version, kernel.data_ptr(), kernel.device, kernel.shape)
        entry = self._entry
        if entry is not None and entry[0] == key:
            _, value, event, index, stream = entry
            if event is not None and stream != _raw_stream(index):
                read_on_current_stream(value, event=event)
            return value
        with torch.no_grad():
            value = transform(kernel)
        event = index = stream = None
        if value.is_cuda:
            if torch.cuda.is_current_stream_capturing():
                return value
            event = torch.cuda.current_stream(value.device).record_event()
            made_on_current_stream(value)
            index = value.device.index
            stream = _raw_stream(index)
        self._entry = (key, value, event, index, stream)
        return value


class FourierMatrices(_OneEntry):
    def get(self, setup, b, grid, scaling, device):
        """``setup(b, grid, device_type, device_index)`` -> (F, Ft); returns (F, Ft, scaling), the
        arguments of ``ag_rft``.  The grid (a tuple of hundreds of angles, costly to hash) is
        compared by identity first."""
        entry = self._entry
        key = (b, scaling, device)
        if entry is None or entry[0] is not grid or entry[1] != key:
            F, Ft = setup(b, grid, device_type=device.type, device_index=device.index)
            entry = (grid, key, (F, Ft, scaling))
            self._entry = entry
        read_on_current_stream(entry[2][0], entry[2][1])
        return entry[2]
