"""Kernels are launched before the ones ahead of them in the stream have finished (``stream_order_wait`` in backend.h): a
chain of calls that read and overwrite the same few buffers gives what it gives with a wait after every call."""
import os
import re

import pytest
import torch

import s2cnn_b200 as S


def _chain(sync):
    torch.manual_seed(0)
    dev = torch.device("cuda:0")
    grid = S.so3_near_identity_grid(n_alpha=4, n_beta=2, n_gamma=3)
    convs = [S.SO3Convolution(3, 5, 6, 6, grid).to(dev), S.SO3Convolution(5, 3, 6, 6, grid).to(dev)]
    x = torch.randn(4, 3, 12, 12, 12, device=dev)
    y = torch.randn(9, 64, 64, device=dev)
    z = torch.randn(2, 64, 64, 64, device=dev)
    done = torch.cuda.synchronize if sync else (lambda: None)
    from s2cnn_b200.soft.s2_fft import S2_fft_real, S2_ifft_real
    from s2cnn_b200.soft.so3_fft import so3_rfft, so3_rifft
    with torch.no_grad():
        for k in range(12):
            h = torch.relu(convs[0](x)); done()
            g = convs[1](h); done()
            x = g / g.std(); done()                                   # (freed buffers go round)
            x = S.so3_rotation(x, 0.3 * k, 0.2, 0.1); done()
            y = S2_ifft_real.apply(S2_fft_real.apply(y, 20), 32); done()
            y = y / y.abs().max(); done()
            z = so3_rifft(so3_rfft(z, b_out=21), b_out=32); done()
    torch.cuda.synchronize()
    return x, y, z


@pytest.mark.gpu
def test_chains_without_waits_equal_chains_with_them():
    want = _chain(True)
    for _ in range(3):
        for a, b in zip(_chain(False), want):
            assert torch.equal(a, b)


@pytest.mark.gpu
def test_two_streams_with_chains_of_their_own():
    want = _chain(True)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = []
    for s in streams:
        with torch.cuda.stream(s):
            got.append(_chain(False))
    torch.cuda.synchronize()
    for res in got:
        for a, b in zip(res, want):
            assert torch.equal(a, b)


def test_kernels_wait_before_they_touch_what_others_do():
    """Every kernel waits, and the tensor-core one takes tensor memory behind the wait, not while a kernel ahead may
    still want its own."""
    csrc = os.path.join(os.path.dirname(S.__file__), "csrc")
    kernels = 0
    for name in sorted(os.listdir(csrc)):
        text = open(os.path.join(csrc, name)).read()
        text = re.sub(r"//.*", "", text)
        for part in re.split(r"__global__\s+void", text)[1:]:
            kernels += 1
            head, wait = part.find("run("), part.find("stream_order_wait()")
            alloc = part.find("tcgen05.alloc")
            first = min(p for p in (head, alloc) if p >= 0)
            assert 0 <= wait < first, (name, part[:60])
    assert kernels >= 15
