"""What layers keep between calls (kernel spectra, Fourier matrices) and passes on several streams: a spectrum made
behind a long kernel on one stream and read on another, a pass under capture that finds no spectrum, a graph whose
weights change after the capture; and that a layer keeps no second copy of its Fourier matrix."""
import pytest
import torch

import backends
from util import assert_close


def layer(S, dev, fi=3, fo=4):
    torch.manual_seed(5)
    return S.SO3Convolution(fi, fo, 4, 3, S.so3_near_identity_grid(n_alpha=4, n_beta=1)).to(dev)


@pytest.mark.parametrize("backend", backends.BACKENDS)
def test_no_scaled_copy_of_the_fourier_matrix_is_kept(backend):
    import s2cnn_b200 as S
    from s2cnn_b200.so3_ft import _setup_so3_ft
    with backends.active(backend) as (ops, dev):
        conv = layer(S, dev)
        x = torch.randn(2, 3, 8, 8, 8, device=dev)
        conv(x).square().sum().backward()
        F, Ft = _setup_so3_ft(conv.b_out, conv.grid, device_type=dev.type, device_index=conv.kernel.device.index)
        kept = [t for t in conv._fourier._entry[2] if isinstance(t, torch.Tensor)]
        assert all(t is F or t is Ft for t in kept)
        # the gradient carries the scaling all the same
        k = conv.kernel.detach().clone().requires_grad_(True)
        y = ops.ag_rft(k * conv.scaling, F, Ft)
        g = torch.randn_like(y)
        y.backward(g)
        k2 = conv.kernel.detach().clone().requires_grad_(True)
        ops.ag_rft(k2, F, Ft, conv.scaling).backward(g)
        assert_close(k2.grad, k.grad, "kernel gradient")


@pytest.mark.gpu
def test_spectrum_made_on_another_stream():
    import s2cnn_b200 as S
    conv = layer(S, "cuda")
    x = torch.randn(2, 3, 8, 8, 8, device="cuda")
    with torch.no_grad():
        want = conv(x)
        for _ in range(3):
            conv._spectrum_cache.clear()
            conv._fourier.clear()
            _setup_clear()
            torch.cuda.synchronize()
            a, b = torch.cuda.Stream(), torch.cuda.Stream()
            with torch.cuda.stream(a):
                torch.cuda._sleep(20_000_000)      # about 10 ms in front of the kernel transform
                first = conv(x)
            with torch.cuda.stream(b):
                second = conv(x)
                conv._spectrum_cache.clear()       # dropped while b still reads it
            with torch.cuda.stream(a):
                for _ in range(8):
                    torch.full((1 << 14,), float("nan"), device="cuda")
            torch.cuda.synchronize()
            assert torch.equal(first, want) and torch.equal(second, want)


@pytest.mark.gpu
def test_spectrum_made_under_capture_is_not_kept():
    import s2cnn_b200 as S
    conv = layer(S, "cuda")
    x = torch.randn(2, 3, 8, 8, 8, device="cuda")
    with torch.no_grad():
        want = conv(x)
        conv._spectrum_cache.clear()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = conv(x)
        assert conv._spectrum_cache._entry is None
        assert torch.equal(conv(x), want)          # before any replay
        graph.replay()
        assert torch.equal(out, want)


@pytest.mark.gpu
def test_graph_reads_its_spectrum_after_the_weights_have_changed():
    import s2cnn_b200 as S
    from s2cnn_b200.graph import GraphedForward
    conv = layer(S, "cuda")
    x = torch.randn(2, 3, 8, 8, 8, device="cuda")
    with torch.no_grad():
        want = conv(x)
        fwd = GraphedForward(conv, x)
        conv.kernel.mul_(2)
        conv(x)                                    # replaces the module's own entry
        torch.cuda.synchronize()
        junk = [torch.full_like(conv._spectrum_cache._entry[1], float("nan")) for _ in range(4)]
        assert torch.equal(fwd(x), want)
        del junk


def _setup_clear():
    from s2cnn_b200.so3_ft import _setup_so3_ft
    _setup_so3_ft.cache_clear()
