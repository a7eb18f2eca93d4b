"""Paths that the size-by-size tests do not reach by themselves: the relays of 22 <= 2b <= 32 (cluster and plane
kernels) against the separate operations, a spectrum with more degrees than the grid holds in the column Wigner
kernel, and every plane path with a workspace that holds part of the batch only (bias, mask, sums and S2-product
indices of a later chunk)."""
import pytest
import torch

import backends
from oracle import s2cnn_oracle as O
from util import assert_close

n3 = O.so3_nspec


@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.parametrize("b,b_in,b_next,nb", [(11, 11, 11, 3), (12, 5, 7, 2), (13, 13, 6, 4), (14, 9, 14, 1), (15, 15, 15, 2),
                                              (16, 16, 10, 5), (10, 10, 4, 6), (9, 7, 9, 5)])
def test_relays_match_separate_operations(backend, b, b_in, b_next, nb):
    ops, dev = backends.get(backend)
    gen = torch.Generator().manual_seed(b)
    fo = 3
    s = torch.randn(n3(b_in), nb, fo, 2, generator=gen).to(dev)
    xs = torch.randn(b * b, nb, 5, 2, generator=gen).to(dev)
    ys = torch.randn(b * b, 5, fo, 2, generator=gen).to(dev)
    bias = torch.randn(fo, generator=gen).to(dev)
    want = ops.so3_rfft(torch.relu(ops.so3_rifft(s, b_out=b, bias=bias)), b_out=b_next)
    want_p = ops.so3_rfft(torch.relu(ops.s2_conv_synthesis(xs, ys, bias)), b_out=b_next)
    got = {}
    for mode in (1, 3):
        ops.lib.s2c_debug_cluster(mode)
        try:
            got[mode] = (ops.so3_rifft_relu_rfft(s, bias, b, b_next), ops.s2_conv_relu_so3_rfft(xs, ys, bias, b_next))
        finally:
            ops.lib.s2c_debug_cluster(0)
        assert_close(got[mode][0], want.cpu(), "relay, mode %d" % mode)
        assert_close(got[mode][1], want_p.cpu(), "product relay, mode %d" % mode)
    if backend == "cuda":   # same sums in the same order
        assert all(torch.equal(a, c) for a, c in zip(got[1], got[3]))


@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.parametrize("b,b_spec,nb", [(9, 16, 5), (13, 15, 2), (15, 16, 3)])
def test_column_kernel_with_degrees_beyond_the_grid(backend, b, b_spec, nb):
    ops, dev = backends.get(backend)
    x = torch.randn(nb, 2 * b, 2 * b, 2 * b, generator=torch.Generator().manual_seed(b))
    ops.lib.s2c_debug_cluster(3)
    try:
        for grad in (False, True):
            assert_close(ops.so3_rfft(x.to(dev), grad, b_spec), O.so3_rfft(x, grad, b_spec), "rfft")
        assert_close(ops.so3_rfft(x.to(dev), b_out=b_spec, relu=True), O.so3_rfft(torch.relu(x), b_out=b_spec), "relu")
    finally:
        ops.lib.s2c_debug_cluster(0)


def v_bytes(b, k):
    """One signal of the plane kernels' scratch array: k x (2k - 1) frequency pairs of 2b betas."""
    return k * (2 * k - 1) * 2 * b * 8


# 2b <= 32: the least workspace the plane kernels take is a tile of 64 signals; 2b > 32: one signal
@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.parametrize("b,b_spec,per,nb", [(9, 9, 64, 130), (10, 4, 64, 129), (17, 17, 1, 3), (18, 7, 2, 5)])
def test_later_chunks(backend, b, b_spec, per, nb):
    ops, dev = backends.get(backend)
    lib = ops.lib
    stream = torch.cuda.current_stream().cuda_stream if dev.type == "cuda" else None
    gen = torch.Generator().manual_seed(b)
    n, k = 2 * b, min(b, b_spec)
    x = torch.randn(nb, n, n, n, generator=gen).to(dev)
    s = torch.randn(n3(b_spec), nb, 2, generator=gen).to(dev)
    bias = torch.randn(5, generator=gen).to(dev)
    fo = 5 if nb % 5 == 0 else 3 if nb % 3 == 0 else 1
    xs = torch.randn(b * b, nb // fo, 2, 2, generator=gen).to(dev)
    ys = torch.randn(b * b, 2, fo, 2, generator=gen).to(dev)
    bias_p = torch.randn(fo, generator=gen).to(dev)

    def run(limit):
        """Every call with room for `limit` signals."""
        def ws(signal_bytes):
            t = torch.empty(signal_bytes * limit, dtype=torch.uint8, device=dev)
            keep.append(t)
            return t.data_ptr(), t.numel()
        keep, out = [], {}

        def call(name, shape, args, signal_bytes):
            o = torch.full(shape, float("nan"), device=dev)
            p, size = ws(signal_bytes)
            lib.call(name, *args(o), p, size, stream)
            out[name] = o
        spec, vb = (n3(b_spec), nb, 2), v_bytes(b, k)
        sums = torch.full((nb,), float("nan"), device=dev)
        call("s2c_so3_rfft", spec, lambda o: (x.data_ptr(), o.data_ptr(), nb, b, b_spec, 0), vb)
        call("s2c_so3_rfft_relu", spec, lambda o: (x.data_ptr(), o.data_ptr(), nb, b, b_spec), vb)
        call("s2c_so3_rfft_sums_ws", spec, lambda o: (x.data_ptr(), o.data_ptr(), sums.data_ptr(), nb, b, b_spec, 1), vb)
        out["sums"] = sums
        call("s2c_so3_rifft", x.shape, lambda o: (s.data_ptr(), o.data_ptr(), nb, b_spec, b, 0, bias.data_ptr(), 5), vb)
        call("s2c_so3_rifft_relu_grad_ws", x.shape, lambda o: (s.data_ptr(), x.data_ptr(), o.data_ptr(), nb, b_spec, b), vb)
        call("s2c_s2_conv_synthesis", x.shape, lambda o: (xs.data_ptr(), ys.data_ptr(), o.data_ptr(), nb // fo, 2, fo, b,
                                                          bias_p.data_ptr()), v_bytes(b, b))
        if b <= 16:
            both = v_bytes(b, b_spec) + v_bytes(b, 5)
            call("s2c_so3_rifft_relu_rfft_ws", (n3(5), nb, 2), lambda o: (s.data_ptr(), o.data_ptr(), nb, b_spec, b, 5,
                                                                          bias.data_ptr(), 5), both)
            call("s2c_s2_conv_relu_so3_rfft_ws", (n3(5), nb, 2), lambda o: (
                xs.data_ptr(), ys.data_ptr(), o.data_ptr(), nb // fo, 2, fo, b, 5, bias_p.data_ptr()), v_bytes(b, b) + v_bytes(b, 5))
        if dev.type == "cuda":
            torch.cuda.synchronize()
        return out

    lib.s2c_debug_cluster(3)
    try:
        whole, parts = run(nb), run(per)
    finally:
        lib.s2c_debug_cluster(0)
    for name in whole:
        assert not torch.isnan(whole[name]).any(), name
        assert torch.equal(whole[name], parts[name]), name
    z = nb - 1     # the last signal against the oracle
    assert_close(parts["s2c_so3_rfft"][:, z], O.so3_rfft(x[z:].cpu(), b_out=b_spec)[:, 0], "rfft")
    assert_close(parts["s2c_so3_rifft"][z], O.so3_rifft(s[:, z:].cpu(), b_out=b)[0] + bias[z % 5].item(), "rifft")
    assert_close(parts["s2c_s2_conv_synthesis"][z], O.so3_rifft(O.s2_mm(xs[:, -1:].cpu(), ys.cpu()))[0, -1] + bias_p[-1].item(), "product")
