"""s2_rft: transform of a kernel sampled on a few sphere points to its S2 spectrum.

Mirrors s2cnn/s2_ft.py:8-24.  The Fourier matrix F[i, (l,m)] = 2b conj(D^l_m0(alpha_i, beta_i, 0))
is generated in float64 by the library's host code (no lie_learn), cached per (b, grid, device)
like the reference's lru_cache (s2_ft.py:53-60); the product with the kernel and its transpose
(for autograd) run as CUDA kernels.
"""
from functools import lru_cache

import torch

from .ops import cuda_ops


def _raw_stream(index):
    """The current stream of a CUDA device, as a number (a stream object costs a microsecond)."""
    return torch._C._cuda_getCurrentRawStream(index)


def made_on_current_stream(*tensors):
    """Notes, on tensors that will be kept between calls, the stream they were allocated on."""
    for t in tensors:
        if t is not None and t.is_cuda:
            t._made_on = _raw_stream(t.get_device())


def read_on_current_stream(first, *others, event=None):
    """Kept tensors, made together, are about to be read on the current stream: where that is not their
    own it waits for ``event`` (recorded after they were written; None: they were complete before they
    were kept), and the allocator does not hand their memory on before the reader is done, whoever drops
    them."""
    if not first.is_cuda or first._made_on == _raw_stream(first.get_device()):
        return
    if torch.cuda.is_current_stream_capturing():   # the graph keeps them (GraphedForward)
        return
    stream = torch.cuda.current_stream(first.device)
    if event is not None:
        stream.wait_event(event)
    for t in (first,) + others:
        if t is not None:
            t.record_stream(stream)


def fourier_matrices(F_host, device):
    """(F, Ft) on the device, complete for every stream: Ft only for a CUDA device and an even number
    of grid points (the tensor-core product works on pairs along the contraction)."""
    F = torch.from_numpy(F_host).to(device)
    Ft = None
    if F.is_cuda:
        if F.size(0) % 2 == 0:
            Ft = F.permute(1, 2, 0).contiguous()
            torch.cuda.current_stream(device).synchronize()   # once per grid; the copy above has waited too
        made_on_current_stream(F, Ft)
    return F, Ft


@lru_cache(maxsize=32)
def _setup_s2_ft(b, grid, device_type, device_index):
    F = cuda_ops().s2_ft_matrix(b, grid)  # [n_grid, b^2, 2] float32, host
    return fourier_matrices(F, torch.device(device_type, device_index))


def s2_rft(x, b, grid):
    """
    Real Fourier Transform
    :param x: [..., beta_alpha]
    :param b: output bandwidth signal
    :param grid: tuple of (beta, alpha) tuples
    :return: [l * m, ..., complex]
    """
    F, Ft = _setup_s2_ft(b, grid, device_type=x.device.type, device_index=x.device.index)
    assert x.size(-1) == F.size(0)
    read_on_current_stream(F, Ft)
    return cuda_ops().ag_rft(x, F, Ft)
