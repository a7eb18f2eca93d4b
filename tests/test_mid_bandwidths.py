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
