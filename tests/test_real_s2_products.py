"""The S2 product inside a synthesis, for spectra of real signals (``real=True``): half of the products, the other half
mirrored.  For factors with x[l,-m] = (-1)^m conj x[l,m] to the last bit the result equals the full product's to the last
bit, in every kernel that evaluates it: cluster, walking, plane (several signals per row or not) and tiled ones."""
import pytest
import torch

import backends
from oracle import s2cnn_oracle as O
from util import assert_close


def real_s2_spectrum(b, *shape, gen):
    rows = []
    for l in range(b):
        x = torch.view_as_complex(torch.randn(l + 1, *shape, 2, generator=gen))     # m = 0 .. l
        x[0] = x[0].real.to(x.dtype)
        sign = torch.tensor([(-1.0) ** m for m in range(l, 0, -1)]).view(-1, *[1] * len(shape))
        rows.append(torch.view_as_real(torch.cat([sign * x[1:].flip(0).conj().resolve_conj(), x])))
    return torch.cat(rows).contiguous()


CASES = [(3, 2, 3, 2, 5), (5, 4, 2, 3, 8), (10, 6, 3, 1, 4), (16, 10, 2, 2, 3), (18, 9, 2, 2, 3)]
GPU = [(10, 6, 40, 1, 20), (9, 5, 70, 2, 9), (16, 10, 20, 6, 100), (14, 8, 30, 3, 60), (12, 8, 16, 2, 100), (16, 9, 3, 8, 101),
       (30, 15, 5, 1, 7), (34, 16, 1, 2, 3)]


@pytest.mark.parametrize("backend,b,b_next,nb,fi,fo",
                         [pytest.param("emul", *c) for c in CASES] +
                         [pytest.param("cuda", *c, marks=pytest.mark.gpu) for c in CASES + GPU])
def test_real_products_equal_the_full_ones(backend, b, b_next, nb, fi, fo):
    ops, dev = backends.get(backend)
    gen = torch.Generator().manual_seed(b * 10 + nb)
    xs, ys = real_s2_spectrum(b, nb, fi, gen=gen).to(dev), real_s2_spectrum(b, fi, fo, gen=gen).to(dev)
    bias = torch.randn(fo, generator=gen).to(dev)
    want = ops.s2_conv_synthesis(xs, ys, bias)
    if b <= 16 and nb * fo <= 60:
        assert_close(want, O.so3_rifft(O.s2_mm(xs.cpu(), ys.cpu())) + bias.cpu().view(1, -1, 1, 1, 1), "full product")
    try:
        for mode in (0, 1, 2, 3) if b <= 16 else (0,):      # by size, cluster, walking, planes
            ops.lib.s2c_debug_cluster(mode)
            assert torch.equal(ops.s2_conv_synthesis(xs, ys, bias, real=True), want), mode
            if b <= 10 or (b <= 16 and mode in (0, 1, 3)):
                assert torch.equal(ops.s2_conv_relu_so3_rfft(xs, ys, bias, b_next, real=True),
                                   ops.s2_conv_relu_so3_rfft(xs, ys, bias, b_next)), ("relay", mode)
    finally:
        ops.lib.s2c_debug_cluster(0)
