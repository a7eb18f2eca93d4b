"""Spectral products of real signals (``so3_mm_real`` and its gradients): half of the result is computed, the
other half is its mirror.  Checked against the full product in float64 on spectra with the symmetry
X[l,-m,-n] = (-1)^(m-n) conj X[l,m,n], at row counts around the 128-row tiles, odd sizes, one degree, and tiles
shared by several thread blocks.  A spectrum that a caller hands to a layer keeps the full product unless the
caller vouches for the symmetry."""
import numpy as np
import pytest
import torch

import s2cnn_b200 as S
import backends
from oracle import s2cnn_oracle as O
from util import assert_close

n3 = O.so3_nspec


def mirrored(x, nl):
    """(-1)^(m-n) conj X[l,-m,-n]; within a degree the mirror reverses the order and the sign alternates."""
    out = torch.empty_like(x)
    for l in range(nl):
        s = slice(n3(l), n3(l + 1))
        q = torch.arange((2 * l + 1) ** 2)
        sign = (1.0 - 2.0 * (q % 2)).view(-1, 1, 1, 1).to(x.dtype)
        out[s] = x[s].flip(0) * sign * torch.tensor([1.0, -1.0], dtype=x.dtype)
    return out


def real_spectrum(nl, *shape, gen):
    x = torch.randn(n3(nl), *shape, 2, generator=gen)
    return (x + mirrored(x, nl)) / 2


def products64(x, y, gz, nl):
    xc, yc, gc = (torch.view_as_complex(t.double()) for t in (x, y, gz))
    z, gx, gy = torch.zeros_like(gc), torch.zeros_like(xc), torch.zeros_like(yc)
    for l in range(nl):
        L, s = 2 * l + 1, slice(n3(l), n3(l + 1))
        xl, yl, gl = (t[s].reshape(L, L, *t.shape[1:]) for t in (xc, yc, gc))
        z[s] = torch.einsum("mpik,npkj->mnij", xl, yl.conj()).reshape(L * L, *z.shape[1:])
        gx[s] = torch.einsum("mnij,npkj->mpik", gl, yl).reshape(L * L, *gx.shape[1:])
        gy[s] = torch.einsum("mnij,mpik->npkj", gl.conj(), xl).reshape(L * L, *gy.shape[1:])
    return [torch.view_as_real(t) for t in (z, gx, gy)]


@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.parametrize("nl,nb,fi,fo", [(1, 1, 2, 2), (4, 32, 4, 6), (4, 33, 3, 5), (2, 64, 8, 12), (2, 65, 2, 3),
                                         (7, 1, 20, 8), (9, 2, 1, 1), (3, 128, 26, 10), (6, 3, 24, 16)])
def test_half_products_match_the_full_ones(backend, nl, nb, fi, fo):
    ops, dev = backends.get(backend)
    gen = torch.Generator().manual_seed(nl * 31 + nb)
    x, y, gz = (real_spectrum(nl, *s, gen=gen) for s in ((nb, fi), (fi, fo), (nb, fo)))
    want = products64(x, y, gz, nl)
    xd, yd, gd = x.to(dev), y.to(dev), gz.to(dev)
    got = [ops.so3_mm_real(xd, yd), ops.so3_mm_real_gradx(gd, yd, nb, fi), ops.so3_mm_real_grady(gd, xd, fo)]
    full = [ops.so3_mm(xd, yd), ops.so3_mm_gradx(gd, yd, nb, fi), ops.so3_mm_grady(gd, xd, fo)]
    for name, g, f, w in zip(("z", "gx", "gy"), got, full, want):
        g, f = g.cpu(), f.cpu()
        # 3xTF32: 2^-22 for the split and at most 2^-23 per truncated addition of a chain of 66: below 1e-5
        err = [((t.double() - w).norm() / w.norm()).item() for t in (g, f)]
        assert err[0] < 1e-5, (name, err)
        assert_close(g, f, name)
        if backend == "cuda":     # the halves mirror each other exactly (index 0 is its own half: computed as a whole)
            m0 = torch.cat([(torch.arange((2 * l + 1) ** 2) // (2 * l + 1) == l) if name == "gx" else
                            (torch.arange((2 * l + 1) ** 2) % (2 * l + 1) == l) for l in range(nl)])
            assert torch.equal(g[~m0], mirrored(g, nl)[~m0]), name
    if backend == "cuda":
        from s2cnn_b200 import _lib
        assert _lib.cuda_lib().s2c_so3_mm_tc_status() == 0


# layers whose forward products are not segmented: contractions too long for eight segments (partial sums every seven
# blocks), or too many tiles for clusters (one chain, the products with a lo part in an accumulator of their own)
WIDE = [(10, 2, 100, 100), (5, 3, 100, 255), (15, 2, 16, 16), (15, 2, 8, 16)]
# ... too short for segments; pairs of CTAs per tile, with segments and without; one CTA per tile where pairs do not fit
PAIRS = [(2, 16, 32, 64), (7, 32, 16, 24), (15, 7, 8, 16), (6, 64, 8, 46), (8, 32, 24, 46), (5, 20, 9, 7)]


@pytest.mark.gpu
@pytest.mark.parametrize("nl,nb,fi,fo", WIDE + PAIRS)
def test_wide_half_products_match_the_full_ones(nl, nb, fi, fo):
    test_half_products_match_the_full_ones("cuda", nl, nb, fi, fo)


@pytest.mark.gpu
@pytest.mark.parametrize("nl,fi,fo", [(6, 20, 40), (3, 32, 64), (7, 13, 9), (2, 4, 4), (7, 16, 24), (12, 24, 3)] +
                         [(nl, fi, fo) for nl, _, fi, fo in WIDE + PAIRS])
def test_forward_does_not_depend_on_the_batch(nl, fi, fo):
    """A tile's segments, one to a block of a cluster (few signals) or one after the other, give the same bits."""
    ops, dev = backends.get("cuda")
    gen = torch.Generator().manual_seed(fo)
    x, y = real_spectrum(nl, 300, fi, gen=gen).to(dev), real_spectrum(nl, fi, fo, gen=gen).to(dev)
    z = ops.so3_mm_real(x, y)
    for n in (1, 3, 17, 32, 129):
        assert torch.equal(ops.so3_mm_real(x[:, :n].contiguous(), y), z[:, :n]), n


def real_s2_spectrum(b, *shape, gen):
    out = real_spectrum(b, *shape, gen=gen)
    return torch.cat([out[n3(l) + l * (2 * l + 1):n3(l) + (l + 1) * (2 * l + 1)] for l in range(b)]).contiguous()  # m = 0


@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.parametrize("nl,nb,fi,fo", [(1, 1, 1, 1), (4, 65, 1, 3), (7, 3, 8, 5), (5, 2, 9, 4), (12, 20, 6, 33)])
def test_half_s2_gradients_match_the_full_ones(backend, nl, nb, fi, fo):
    """f_in above 8 takes the general product."""
    ops, dev = backends.get(backend)
    gen = torch.Generator().manual_seed(nl + fo)
    gz = real_spectrum(nl, nb, fo, gen=gen).to(dev)
    x, y = real_s2_spectrum(nl, nb, fi, gen=gen).to(dev), real_s2_spectrum(nl, fi, fo, gen=gen).to(dev)
    for name, a, b in (("gx", ops.s2_mm_gradx(gz, y, nb, fi, real=True), ops.s2_mm_gradx(gz, y, nb, fi)),
                       ("gy", ops.s2_mm_grady(gz, x, fo, real=True), ops.s2_mm_grady(gz, x, fo))):
        # both are sums of at most (2 nl - 1) * max(nb, fo) terms in float32, in other orders
        assert ((a - b).norm() / b.norm()).item() < 5e-6, name


# Relative error of the symmetric part, which is what the transforms behind a gradient read, of gx and gy when every row was
# computed (float32 against float64, mean of four draws): mirrored rows have no two independent roundings to average and
# must not be further off
WHOLE_ERROR = [((6, 16, 1, 10), 0.98e-7, 1.53e-7), ((10, 4, 1, 32), 2.02e-7, 0.87e-7), ((12, 5, 3, 60), 3.05e-7, 0.72e-7)]
WHOLE_ERROR_GPU = [((10, 32, 1, 20), 1.62e-7, 1.10e-7), ((30, 32, 1, 8), 1.77e-7, 1.74e-7), ((30, 7, 1, 8), 1.79e-7, 1.55e-7),
                   ((16, 32, 6, 100), 4.49e-7, 1.66e-7), ((16, 30, 3, 40), 2.87e-7, 1.19e-7), ((14, 64, 1, 16), 1.72e-7, 1.49e-7)]


@pytest.mark.parametrize("backend,sizes,gx,gy", [pytest.param("emul", *c) for c in WHOLE_ERROR] +
                         [pytest.param("cuda", *c, marks=pytest.mark.gpu) for c in WHOLE_ERROR + WHOLE_ERROR_GPU])
def test_half_s2_gradients_are_no_less_precise(backend, sizes, gx, gy):
    ops, dev = backends.get(backend)
    nl, nb, fi, fo = sizes
    off = {"gx": [], "gy": []}
    for seed in range(4):
        gen = torch.Generator().manual_seed(seed)
        gz = real_spectrum(nl, nb, fo, gen=gen)
        x, y = real_s2_spectrum(nl, nb, fi, gen=gen), real_s2_spectrum(nl, fi, fo, gen=gen)
        gc, xc, yc = (torch.view_as_complex(t.double()) for t in (gz, x, y))
        want = {"gx": torch.zeros_like(xc), "gy": torch.zeros_like(yc)}
        for l in range(nl):
            L, s = 2 * l + 1, slice(l * l, (l + 1) ** 2)
            gl = gc[n3(l):n3(l + 1)].reshape(L, L, nb, fo)
            want["gx"][s] = torch.einsum("mnij,nkj->mik", gl, yc[s])
            want["gy"][s] = torch.einsum("mnij,mik->nkj", gl.conj(), xc[s])
        gd, xd, yd = gz.to(dev), x.to(dev), y.to(dev)
        for name, got in (("gx", ops.s2_mm_gradx(gd, yd, nb, fi, real=True)), ("gy", ops.s2_mm_grady(gd, xd, fo, real=True))):
            w = torch.view_as_real(want[name])     # (mirrored itself, as got is: the difference is the symmetric part's)
            off[name].append(((got.cpu().double() - w).norm() / w.norm()).item())
    assert sum(off["gx"]) / 4 <= gx and sum(off["gy"]) / 4 <= gy, off


@pytest.mark.gpu
def test_a_given_spectrum_keeps_the_full_product():
    torch.manual_seed(3)
    conv = S.SO3Convolution(3, 4, 5, 4, S.so3_near_identity_grid()).cuda()
    x = torch.randn(n3(4), 2, 3, 2)                      # no symmetry
    y = O.so3_rft(conv.kernel.detach().cpu() * conv.scaling, 4, conv.grid)
    want = O.so3_rifft(O.so3_mm(x, y))                  # the synthesis takes the symmetric part of the product
    with torch.no_grad():
        assert_close(conv(x.cuda(), input_spectrum=True), want, "given spectrum")
        xs = real_spectrum(4, 2, 3, gen=torch.Generator().manual_seed(1))
        a = conv(xs.cuda(), input_spectrum=True)
        b = conv(xs.cuda(), input_spectrum=True, real_spectrum=True)
    assert_close(b, a, "real spectrum")


@pytest.mark.gpu
def test_wide_layer_without_gradients():
    """40 -> 60 channels at ten degrees, the half product with partial sums, through the module (no gradient recorded)."""
    torch.manual_seed(5)
    grid = S.so3_near_identity_grid(n_alpha=4, n_beta=2, n_gamma=3)
    conv = S.SO3Convolution(40, 60, 10, 10, grid)
    x = torch.randn(2, 40, 20, 20, 20)
    want = O.so3_convolution(x, conv.kernel.detach(), conv.bias.detach(), 10, 10, grid)
    with torch.no_grad():
        assert_close(conv.cuda()(x.cuda()), want, "y")


@pytest.mark.gpu
def test_layer_gradients_with_half_products():
    """SO3Convolution forward and backward against the oracle in float64 (odd channel counts, b_out < b_in)."""
    torch.manual_seed(4)
    grid = S.so3_near_identity_grid(max_beta=np.pi / 8, n_alpha=4, n_beta=2, n_gamma=3)
    conv = S.SO3Convolution(5, 3, 6, 4, grid)
    x, gy = torch.randn(3, 5, 12, 12, 12), torch.randn(3, 3, 8, 8, 8)
    xo, ko = x.clone().requires_grad_(True), conv.kernel.detach().clone().requires_grad_(True)
    O.so3_convolution(xo, ko, conv.bias.detach(), 6, 4, grid).backward(gy)
    conv = conv.cuda()
    xd = x.cuda().requires_grad_(True)
    conv(xd).backward(gy.cuda())
    assert_close(xd.grad, xo.grad, "gx")
    assert_close(conv.kernel.grad, ko.grad, "gkernel")
