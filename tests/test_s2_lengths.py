"""The S2 kernels at the lengths where they can go wrong: one-stage, two-stage and prime second steps, the two
power-of-two lengths with their own FFT, more than one block of rows, rows of N mod 4 = 2 in the tiled
contraction, the last size of the single-kernel analysis and the first beyond it, batch tiles of every size."""
import pytest
import torch

import backends
from oracle import s2cnn_oracle as O
from util import assert_close


@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.parametrize("b,b_spec,nb", [(1, 1, 1), (9, 9, 2), (16, 3, 70), (17, 11, 3), (29, 29, 1), (32, 32, 5), (33, 33, 9),
                                         (35, 34, 2), (40, 17, 1), (62, 40, 1), (63, 33, 2), (64, 64, 1), (64, 7, 3)])
def test_s2_transforms_at_edge_lengths(backend, b, b_spec, nb):
    ops, dev = backends.get(backend)
    gen = torch.Generator().manual_seed(100 * b + b_spec)
    x = torch.randn(nb, 2 * b, 2 * b, 2, generator=gen)
    s = torch.randn(b_spec * b_spec, nb, 2, generator=gen)
    xr = torch.stack((x[..., 0], torch.zeros_like(x[..., 0])), -1)
    for fg in (False, True):
        assert_close(ops.s2_fft(x.to(dev), fg, b_spec), O.s2_fft(x, for_grad=fg, b_out=b_spec), "complex")
        assert_close(ops.s2_fft(x[..., 0].to(dev), fg, b_spec, x_is_real=True), O.s2_fft(xr, for_grad=fg, b_out=b_spec), "real")
        want = O.s2_ifft(s, for_grad=fg, b_out=b)
        assert_close(ops.s2_ifft(s.to(dev), fg, b), want, "inverse complex")
        assert_close(ops.s2_ifft(s.to(dev), fg, b, out_is_real=True), want[..., 0], "inverse real")
