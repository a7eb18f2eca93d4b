"""The plane kernels of 32 < 2b < 64 against the three separate passes they replace (same arithmetic:
the results agree to the last bit up to the sign of zeros) and, for one size, the oracle: lengths with one
or several stages per step, prime blocks, ragged beta groups (N mod 4 = 2 with four planes per block),
dropped degrees, both weightings, a bias, and complex signals (strided access)."""
import pytest
import torch

import backends
from oracle import s2cnn_oracle as O
from util import assert_close

n3 = O.so3_nspec


@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.parametrize("b,b_spec,nb", [(17, 17, 2), (18, 5, 3), (21, 12, 1), (25, 13, 2), (27, 9, 1), (28, 20, 1),
                                         (29, 3, 2), (30, 30, 2), (31, 7, 1)])
def test_mid_planes_match_three_passes(backend, b, b_spec, nb):
    ops, dev = backends.get(backend)
    if backend == "cuda":
        nb = nb * 33
    gen = torch.Generator().manual_seed(b)
    x = torch.randn(nb, 2 * b, 2 * b, 2 * b, generator=gen).to(dev)
    s = torch.randn(n3(b_spec), nb, 2, generator=gen).to(dev)
    bias = torch.randn(nb, generator=gen).to(dev)

    def all_four():
        return [ops.so3_rfft(x, b_out=b_spec), ops.so3_rfft(x, b_out=b_spec, for_grad=True),
                ops.so3_rifft(s, b_out=b, bias=bias), ops.so3_rifft(s, b_out=b, for_grad=True)]

    got = all_four()
    ops.lib.s2c_debug_force_general_path(2)
    try:
        want = all_four()
    finally:
        ops.lib.s2c_debug_force_general_path(0)
    for g, w in zip(got, want):
        if backend == "cuda":
            assert torch.equal(g, w)
        else:   # the host compiler rounds the generic FFT's products differently
            assert_close(g, w, "planes vs passes")


@pytest.mark.parametrize("backend", backends.BACKENDS)
def test_mid_planes_complex_signal_matches_oracle(backend):
    ops, dev = backends.get(backend)
    gen = torch.Generator().manual_seed(3)
    b = 18
    x = torch.randn(2, 2 * b, 2 * b, 2 * b, 2, generator=gen)
    s = ops.so3_fft(x.to(dev), b_out=7)
    assert_close(s, O.so3_fft(x, b_out=7), "so3_fft")
    assert_close(ops.so3_ifft(s, b_out=b), O.so3_ifft(s.cpu(), b_out=b), "so3_ifft")


@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.parametrize("b,b_spec,nb", [(17, 17, 2), (20, 11, 3), (30, 4, 1)])
def test_mid_planes_fused_relu_sums_and_product(backend, b, b_spec, nb):
    """ReLU on load, its gradient's mask on store, per-signal sums and the S2 product evaluated while the spectrum
    is staged, against the separate operations."""
    ops, dev = backends.get(backend)
    gen = torch.Generator().manual_seed(7 * b)
    x = torch.randn(nb, 2 * b, 2 * b, 2 * b, generator=gen).to(dev)
    s = torch.randn(n3(b_spec), nb, 2, generator=gen).to(dev)
    assert_close(ops.so3_rfft(x, b_out=b_spec, relu=True), ops.so3_rfft(torch.relu(x), b_out=b_spec), "relu")
    assert_close(ops.so3_rifft_relu_grad(s, x), ops.so3_rifft(s, b_out=b, for_grad=True) * (x > 0), "mask")
    spec, sums = ops.so3_rfft_with_sums(x, for_grad=True, b_out=b_spec)
    assert_close(spec, ops.so3_rfft(x, b_out=b_spec, for_grad=True), "spectrum")
    assert (sums.double() - x.double().sum(dim=(-3, -2, -1))).abs().max().item() < 1e-3 * (2 * b) ** 1.5
    if b <= 20:
        xs = torch.randn(b * b, nb, 2, 2, generator=gen).to(dev)
        ys = torch.randn(b * b, 2, 3, 2, generator=gen).to(dev)
        bias = torch.randn(3, generator=gen).to(dev)
        got = ops.s2_conv_synthesis(xs, ys, bias)
        assert_close(got, ops.so3_rifft(ops.s2_mm(xs, ys), bias=bias), "product")
