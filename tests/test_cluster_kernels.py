"""The cluster kernels and the plane kernels of 2b <= 32 against the kernels whose blocks walk beta: same sums in the same order, so
equal to the last bit on the GPU.  One block per cluster, two, four and eight, betas that do not divide evenly
(2b = 12, 18, 22, 26, 30: a short last block; 28: an empty one), batches that end inside a group of four, more degrees
than the grid holds, a fused product with a feature count that is no multiple of four, masks, sums, the integral, a tile of 128 signals and a rest."""
import pytest
import torch

import backends
from oracle import s2cnn_oracle as O
from util import assert_close

n3 = O.so3_nspec


@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.parametrize("b,b_spec,nb", [(1, 1, 1), (3, 3, 5), (5, 2, 4), (6, 8, 3), (9, 9, 2), (10, 6, 9), (11, 11, 4),
                                         (9, 4, 131), (12, 5, 3), (13, 4, 1), (14, 14, 8), (15, 9, 6), (16, 16, 4)])
def test_cluster_kernels_match_walking_kernels(backend, b, b_spec, nb):
    ops, dev = backends.get(backend)
    gen = torch.Generator().manual_seed(31 * b + b_spec)
    low = min(b, b_spec)
    x = torch.randn(nb, 2 * b, 2 * b, 2 * b, generator=gen).to(dev)
    s = torch.randn(n3(b_spec), nb, 2, generator=gen).to(dev)
    bias = torch.randn(nb, generator=gen).to(dev)
    xs = torch.randn(b * b, 2, 3, 2, generator=gen).to(dev)
    ys = torch.randn(b * b, 3, nb, 2, generator=gen).to(dev)

    def all_ops():
        out = {"rfft": ops.so3_rfft(x, b_out=b_spec), "relu": ops.so3_rfft(x, b_out=b_spec, relu=True),
               "rifft": ops.so3_rifft(s, b_out=b, bias=bias), "grad": ops.so3_rifft(s, b_out=b, for_grad=True),
               "ifft": ops.so3_ifft(s, b_out=b), "mask": ops.so3_rifft_relu_grad(s, x),
               "fft": ops.so3_fft(torch.stack((x, x.flip(0)), -1), b_out=b_spec),
               "product": ops.s2_conv_synthesis(xs, ys, bias)}
        out["sums spectrum"], out["sums"] = ops.so3_rfft_with_sums(x, for_grad=True, b_out=b_spec)
        out["integral"] = ops.so3_rifft_relu_integrate(s, bias=bias, b_out=b)
        if b <= 10 and b_spec <= b:
            out["relay"] = ops.so3_rifft_relu_rfft(s, bias, b, low)
            out["product relay"] = ops.s2_conv_relu_so3_rfft(xs, ys, bias, low)
        return out

    res = []
    for mode in (2, 1, 3):
        ops.lib.s2c_debug_cluster(mode)
        try:
            res.append(all_ops())
        finally:
            ops.lib.s2c_debug_cluster(0)
    for k in res[0]:
        for other, mode in zip(res[1:], (1, 3)):
            if k in ("sums", "integral") or backend != "cuda":    # summed over threads in another order
                assert_close(other[k], res[0][k], "%s, mode %d" % (k, mode))
            else:
                assert torch.equal(other[k], res[0][k]), (k, mode)
