"""S2 transforms of real signals compute the frequencies m >= 0 alone (analysis: from 33 degrees on): against the transforms
of complex signals, which compute all, at lengths with and without a remainder modulo 4 and numbers of signals that fill
tiles or do not.  The synthesis returns the real part of any spectrum's signal."""
import pytest
import torch

import backends

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
