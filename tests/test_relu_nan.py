"""The fused ReLUs treat NaN as torch.relu and its backward do: max(NaN, 0) is NaN, and a gradient
passes where the activation is NaN.  Every place that applies one, on each path: the analysis while it
reads, the synthesis' mask, both integrals, both relays; the signals beside the one with the NaN are
not touched."""
import pytest
import torch

import backends
from oracle import s2cnn_oracle as O

n3 = O.so3_nspec


def same_nan(got, want, what):
    assert torch.equal(torch.isnan(got), torch.isnan(want)), what
    ok = ~torch.isnan(want)
    assert torch.allclose(got[ok], want[ok], rtol=1e-4, atol=1e-4 * want[ok].abs().max().item()), what


@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.parametrize("b,mode", [(5, 1), (5, 2), (10, 1), (10, 2), (10, 3), (11, 1), (11, 3), (17, 0), (18, 0)])
def test_fused_relu_passes_nan(backend, b, mode):
    ops, dev = backends.get(backend)
    gen = torch.Generator().manual_seed(b)
    nb, n, nan = 3, 2 * b, float("nan")
    x = torch.randn(nb, n, n, n, generator=gen)
    x[1, 3, 2, 1] = nan
    x = x.to(dev)
    s = torch.randn(n3(b), nb, 2, generator=gen)
    clean = s.to(dev)
    s[2, 1, 0] = nan
    s = s.to(dev)
    xs = torch.randn(b * b, nb, 2, 2, generator=gen)
    xs[3, 1, 0, 1] = nan
    xs = xs.to(dev)
    ys = torch.randn(b * b, 2, 2, 2, generator=gen).to(dev)
    bias = torch.randn(nb, generator=gen).to(dev)
    ops.lib.s2c_debug_cluster(mode)
    try:
        same_nan(ops.so3_rfft(x, b_out=b, relu=True), ops.so3_rfft(torch.relu(x), b_out=b), "analysis")
        plain = ops.so3_rifft(clean, for_grad=True)
        same_nan(ops.so3_rifft_relu_grad(clean, x), torch.where(x <= 0, torch.zeros_like(plain), plain), "mask")
        if b <= 16:
            signal = torch.relu(ops.so3_rifft(s, bias=bias))
            assert bool(torch.isnan(signal[1]).any()) and not bool(torch.isnan(signal[0]).any())
            same_nan(ops.so3_rifft_relu_integrate(s, bias=bias), ops.so3_integrate(signal), "synthesis + integral")
            if mode != 2 or b <= 10:
                same_nan(ops.so3_rifft_relu_rfft(s, bias, b, b), ops.so3_rfft(signal), "relay")
                product = torch.relu(ops.s2_conv_synthesis(xs, ys, None))
                same_nan(ops.s2_conv_relu_so3_rfft(xs, ys, None, b), ops.so3_rfft(product), "product relay")
    finally:
        ops.lib.s2c_debug_cluster(0)


@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.parametrize("b", [3, 4])
def test_integral_of_relu_passes_nan(backend, b):
    ops, dev = backends.get(backend)
    gen = torch.Generator().manual_seed(b)
    x = torch.randn(3, 2 * b, 2 * b, 2 * b, generator=gen)
    x[2, 1, 1, 1] = float("nan")
    x = x.to(dev)
    same_nan(ops.so3_integrate(x, relu=True), ops.so3_integrate(torch.relu(x)), "integral")
    g = torch.randn(3, generator=gen).to(dev)
    plain = ops.so3_integrate_backward(g, b)
    same_nan(ops.so3_integrate_backward(g, b, x=x, relu=True), torch.where(x <= 0, torch.zeros_like(plain), plain), "backward")
