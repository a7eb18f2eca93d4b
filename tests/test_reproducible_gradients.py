"""Gradients are the same to the last bit from run to run, also where a tile's contraction is shared by several
thread blocks: both gradient products and the transposed kernel transform, shared by one cluster of two to eight
blocks (some without a K block of their own) and by up to fifteen clusters, with even and odd channel counts, and
with another stream's work on the same SMs, which changes the order in which the blocks finish.  Without a
workspace at most one cluster shares a tile: the same values up to rounding."""
import pytest
import torch

from oracle import s2cnn_oracle as O
from util import assert_close

n3 = O.so3_nspec


@pytest.mark.gpu
@pytest.mark.parametrize("nl,nb,fi,fo", [(6, 32, 20, 40), (7, 5, 13, 9), (5, 32, 100, 255), (15, 4, 16, 24), (20, 1, 2, 2)])
def test_gradient_products_repeat(nl, nb, fi, fo):
    from s2cnn_b200.ops import cuda_ops
    ops = cuda_ops()
    gen = torch.Generator(device="cuda").manual_seed(nl)
    x = torch.randn(n3(nl), nb, fi, 2, generator=gen, device="cuda")
    y = torch.randn(n3(nl), fi, fo, 2, generator=gen, device="cuda")
    gz = torch.randn(n3(nl), nb, fo, 2, generator=gen, device="cuda")
    run = lambda: (ops.so3_mm_gradx(gz, y, nb, fi), ops.so3_mm_grady(gz, x, fo))  # noqa: E731
    _repeat(run)
    gx, gy = run()
    stream = torch.cuda.current_stream().cuda_stream
    for name, a, want in (("gradx", y, gx), ("grady", x, gy)):
        got = torch.empty_like(want)
        ops.lib.call("s2c_so3_mm_" + name, gz.data_ptr(), a.data_ptr(), got.data_ptr(), nl, nb, fi, fo, stream)
        assert_close(got, want.cpu(), name + " without a workspace")


@pytest.mark.gpu
@pytest.mark.parametrize("nf,ng,ns", [(800, 192, 286), (117, 192, 455), (128, 36, 4495), (7, 24, 100), (1, 2, 40000)])
def test_kernel_gradient_repeats(nf, ng, ns):
    from s2cnn_b200.ops import cuda_ops
    ops = cuda_ops()
    gen = torch.Generator(device="cuda").manual_seed(nf)
    F = torch.randn(ng, ns, 2, generator=gen, device="cuda")
    g = torch.randn(ns, nf, 2, generator=gen, device="cuda")
    _repeat(lambda: (ops.rft_backward(g, F, scale=0.37),))
    want = 0.37 * torch.einsum("sfc,asc->fa", g.double(), F.double())
    assert_close(ops.rft_backward(g, F, scale=0.37), want.float().cpu(), "kernel gradient")
    got = torch.empty(nf, ng, device="cuda")
    ops.lib.call("s2c_rft_backward", g.data_ptr(), F.data_ptr(), got.data_ptr(), nf, ng, ns, torch.cuda.current_stream().cuda_stream)
    assert_close(0.37 * got, want.float().cpu(), "without a workspace")


def _repeat(run):
    first = run()
    other, noise = torch.cuda.Stream(), torch.randn(1 << 22, device="cuda")
    other.wait_stream(torch.cuda.current_stream())
    for k in range(30):
        if k % 3:
            with torch.cuda.stream(other):
                for _ in range(k % 5):
                    noise.mul_(1.0000001)
        for a, b in zip(run(), first):
            assert torch.equal(a, b), k
    torch.cuda.synchronize()
