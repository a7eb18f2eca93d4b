"""Kernels are launched before the ones ahead of them in the stream have finished (``stream_order_wait`` in backend.h): a
chain of calls that read and overwrite the same few buffers gives what it gives with a wait after every call."""
import os
import re

import pytest
import torch

import s2cnn_b200 as S


def _steps(sync, result):
    """A chain of calls, one per step of the generator; `result` gets its outputs."""
    torch.manual_seed(0)
    dev = torch.device("cuda:0")
    grid = S.so3_near_identity_grid(n_alpha=4, n_beta=2, n_gamma=3)
    convs = [S.SO3Convolution(3, 5, 6, 6, grid).to(dev), S.SO3Convolution(5, 3, 6, 6, grid).to(dev)]
    x = torch.randn(4, 3, 12, 12, 12, device=dev)
    y = torch.randn(9, 64, 64, device=dev)
    z = torch.randn(2, 64, 64, 64, device=dev)
    from s2cnn_b200.soft.s2_fft import S2_fft_real, S2_ifft_real
    from s2cnn_b200.soft.so3_fft import so3_rfft, so3_rifft
    for k in range(12):
        for step in range(7):
            with torch.no_grad():
                if step == 0:
                    h = torch.relu(convs[0](x))
                elif step == 1:
                    g = convs[1](h)
                elif step == 2:
                    x = g / g.std()                                   # (freed buffers go round)
                elif step == 3:
                    x = S.so3_rotation(x, 0.3 * k, 0.2, 0.1)
                elif step == 4:
                    y = S2_ifft_real.apply(S2_fft_real.apply(y, 20), 32)
                elif step == 5:
                    y = y / y.abs().max()
                else:
                    z = so3_rifft(so3_rfft(z, b_out=21), b_out=32)
            if sync:
                torch.cuda.synchronize()
            yield
    result.extend((x, y, z))


def _chain(sync):
    result = []
    for _ in _steps(sync, result):
        pass
    torch.cuda.synchronize()
    return result


@pytest.mark.gpu
def test_chains_without_waits_equal_chains_with_them():
    want = _chain(True)
    for _ in range(3):
        for a, b in zip(_chain(False), want):
            assert torch.equal(a, b)


@pytest.mark.gpu
def test_two_streams_with_chains_of_their_own():
    """Both in flight: the host issues a step of one and a step of the other in turn and waits at the end."""
    want = _chain(True)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = [[], []]
    torch.cuda.synchronize()
    chains = [_steps(False, g) for g in got]
    for _ in range(12 * 7 + 1):
        for s, c in zip(streams, chains):
            with torch.cuda.stream(s):
                next(c, None)
    torch.cuda.synchronize()
    for res in got:
        assert len(res) == 3
        for a, b in zip(res, want):
            assert torch.equal(a, b)


def _gradients(sync):
    """Kernel and input gradients whose tiles several clusters share (a memset of their counters in front)."""
    from s2cnn_b200.ops import cuda_ops
    ops = cuda_ops()
    nspec = 4495                                                      # 15 degrees
    assert ops.lib.s2c_rft_backward_workspace(128, 36, nspec) > 0
    gen = torch.Generator().manual_seed(3)
    F = torch.randn(36, nspec, 2, generator=gen).cuda()
    x, y = torch.randn(nspec, 2, 8, 2, generator=gen).cuda(), torch.randn(nspec, 8, 16, 2, generator=gen).cuda()
    done = torch.cuda.synchronize if sync else (lambda: None)
    out = []
    for k in range(6):
        z = ops.so3_mm_real(x, y); done()
        gx = ops.so3_mm_real_gradx(z, y, 2, 8); done()
        gy = ops.so3_mm_real_grady(z, x, 16); done()
        gk = ops.rft_backward(gy, F, 0.5); done()
        out += [gx, gk]
        x = gx / gx.std(); done()
        del z, gx, gy                                                 # (freed buffers go round)
    torch.cuda.synchronize()
    return out


@pytest.mark.gpu
def test_gradients_without_waits_equal_gradients_with_them():
    want = _gradients(True)
    for _ in range(3):
        for a, b in zip(_gradients(False), want):
            assert torch.equal(a, b)


@pytest.mark.gpu
def test_training_steps_without_waits():
    """Forward and backward of two layers, several steps in flight, against a wait after every pass."""
    grid = S.so3_near_identity_grid(n_alpha=6, n_beta=2, n_gamma=3)

    def steps(sync):
        torch.manual_seed(1)
        convs = torch.nn.ModuleList([S.SO3Convolution(8, 16, 15, 15, grid), S.SO3Convolution(16, 6, 15, 7, grid)]).cuda()
        x = torch.randn(2, 8, 30, 30, 30, device="cuda")
        grads = []
        for _ in range(4):
            convs.zero_grad(set_to_none=True)
            h = torch.relu(convs[0](x))
            if sync:
                torch.cuda.synchronize()
            convs[1](h).square().sum().backward()
            if sync:
                torch.cuda.synchronize()
            grads += [p.grad for p in convs.parameters()]
        torch.cuda.synchronize()
        return grads
    want = steps(True)
    for a, b in zip(steps(False), want):
        assert torch.equal(a, b)


@pytest.mark.gpu
def test_captured_graph_that_forks_and_joins():
    """Two branches of a captured graph, each a chain of kernels, on their own streams between a fork and a join."""
    from s2cnn_b200.soft.so3_fft import so3_rfft, so3_rifft
    grid = S.so3_near_identity_grid(n_alpha=4, n_beta=2, n_gamma=3)
    torch.manual_seed(2)
    convs = [S.SO3Convolution(3, 5, 9, 9, grid).cuda() for _ in range(2)]
    after = S.SO3Convolution(5, 4, 9, 5, grid).cuda()
    x = torch.randn(6, 3, 18, 18, 18, device="cuda")
    side = torch.cuda.Stream()

    def branch(k, h):
        return torch.relu(convs[k](S.so3_rotation(h, 0.3 + k, 0.2, 0.1)))

    def run():
        with torch.no_grad():
            h = so3_rifft(so3_rfft(x, b_out=9), b_out=9)
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                b = branch(1, h)
            a = branch(0, h)
            torch.cuda.current_stream().wait_stream(side)
            return after(a + b)
    main = torch.cuda.Stream()
    with torch.cuda.stream(main):
        want = run().clone()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=main):
            out = run()
        for _ in range(5):
            out.zero_()
            graph.replay()
        torch.cuda.synchronize()
    assert torch.equal(out, want)


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
