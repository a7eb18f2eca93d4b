"""S2 transforms of real signals compute the frequencies m >= 0 alone (analysis: from 33 degrees on): against the transforms
of complex signals, which compute all, at lengths with and without a remainder modulo 4 and numbers of signals that fill
tiles or do not.  The synthesis returns the real part of any spectrum's signal."""
import pytest
import torch

import backends
from oracle import s2cnn_oracle as O

CASES = [(33, 33, 1), (34, 33, 9), (40, 34, 3), (12, 7, 5), (45, 45, 2)]
GPU = [(64, 64, 192), (64, 33, 7), (64, 32, 70), (60, 50, 17), (63, 40, 65), (50, 34, 3)]


@pytest.mark.parametrize("backend,b,k,nb", [pytest.param("emul", *c) for c in CASES] +
                         [pytest.param("cuda", *c, marks=pytest.mark.gpu) for c in CASES + GPU])
def test_real_transforms_equal_the_complex_ones(backend, b, k, nb):
    ops, dev = backends.get(backend)
    gen = torch.Generator().manual_seed(b + nb)
    x = torch.randn(nb, 2 * b, 2 * b, generator=gen).to(dev)
    s = torch.randn(k * k, nb, 2, generator=gen).to(dev)            # not the spectrum of a real signal
    for grad in (False, True):
        a, w = ops.s2_fft(x, grad, k, True), ops.s2_fft(torch.stack([x, torch.zeros_like(x)], -1), grad, k)
        # float32 sums of at most 2 b terms: 2b * 2^-24 < 1e-5
        assert ((a - w).norm() / w.norm()).item() < 2e-6
        a, w = ops.s2_ifft(s, grad, b, True), ops.s2_ifft(s, grad, b)[..., 0]
        assert ((a - w).norm() / w.norm()).item() < 2e-6


@pytest.mark.parametrize("backend,b,k,nb", [pytest.param("emul", *c) for c in ((34, 34, 3), (64, 20, 2), (40, 35, 3))] +
                         [pytest.param("cuda", *c, marks=pytest.mark.gpu) for c in
                          ((34, 34, 8), (40, 35, 8), (48, 48, 8), (64, 64, 24), (64, 40, 24), (64, 20, 24), (30, 30, 8))])
def test_real_transforms_are_no_less_precise(backend, b, k, nb):
    """Against float64, beside the transforms of complex signals, whose two signs of a frequency are two sums with independent
    roundings: the signal of any spectrum, and from 33 degrees on, where the analysis takes half, the spectrum's symmetric
    part (what a transform behind it reads) and the way there and back."""
    ops, dev = backends.get(backend)
    gen = torch.Generator().manual_seed(b + k)
    x, s = torch.randn(nb, 2 * b, 2 * b, generator=gen), torch.randn(k * k, nb, 2, generator=gen)
    half, whole = ops.s2_fft(x.to(dev), False, k, True), ops.s2_fft(torch.stack([x, torch.zeros_like(x)], -1).to(dev), False, k)

    def off(a, w):
        return ((a.cpu().double() - w).norm() / w.norm()).item()

    def off_symmetric(a, w):
        d = torch.view_as_complex(a.cpu().double() - w)
        for l in range(k):
            r = slice(l * l, (l + 1) ** 2)
            sign = (1.0 - 2.0 * (torch.arange(-l, l + 1).abs() % 2)).view(-1, 1)
            d[r] = (d[r] + sign * d[r].flip(0).conj()) / 2
        return (d.abs().norm() / w.norm()).item()
    with O.float64():
        want = O.s2_fft(torch.stack([x.double(), torch.zeros_like(x).double()], -1), False, k)
        trip, signal = O.s2_ifft(want, False, b)[..., 0], O.s2_ifft(s.double(), False, b)[..., 0]
    s = s.to(dev)
    assert off(ops.s2_ifft(s, False, b, True), signal) <= off(ops.s2_ifft(s, False, b)[..., 0], signal)
    if k > 32:
        assert off_symmetric(half, want) <= off_symmetric(whole, want)
        assert off(ops.s2_ifft(half, False, b, True), trip) <= off(ops.s2_ifft(whole, False, b)[..., 0], trip)
