"""so3_rft: transform of a kernel sampled on a few rotations to its SO(3) spectrum.

Mirrors s2cnn/so3_ft.py:8-24 with F[i, (l,m,n)] = conj(D^l_mn(alpha_i, beta_i, gamma_i)),
generated by the library's float64 host code and cached per (b, grid, device) as in
so3_ft.py:55-62.
"""
from functools import lru_cache

import torch

from .ops import cuda_ops
from .s2_ft import fourier_matrices, read_on_current_stream


@lru_cache(maxsize=32)
def _setup_so3_ft(b, grid, device_type, device_index):
    F = cuda_ops().so3_ft_matrix(b, grid)  # [n_grid, nspec, 2] float32, host
    return fourier_matrices(F, torch.device(device_type, device_index))


def so3_rft(x, b, grid):
    """
    Real Fourier Transform
    :param x: [..., beta_alpha_gamma]
    :param b: output bandwidth signal
    :param grid: tuple of (beta, alpha, gamma) tuples
    :return: [l * m * n, ..., complex]
    """
    F, Ft = _setup_so3_ft(b, grid, device_type=x.device.type, device_index=x.device.index)
    assert x.size(-1) == F.size(0)
    read_on_current_stream(F, Ft)
    return cuda_ops().ag_rft(x, F, Ft)
