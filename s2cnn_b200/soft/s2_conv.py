"""S2Convolution (s2cnn/soft/s2_conv.py:13-47): same constructor, parameters, init and scaling."""
import math

import torch
from torch.nn.modules import Module
from torch.nn.parameter import Parameter

from ..ops import cuda_ops
from ..s2_ft import _setup_s2_ft
from .s2_fft import S2_fft_real
from .so3_fft import SO3_fft_real, SO3_fft_real_relu
from ._spectrum_cache import FourierMatrices, KernelSpectrumCache
from ._recompute import fused_or_recompute


def _product_synthesis(x, y, bias):
    """``SO3_ifft_real(s2_mm(x, y)) + bias`` (s2_conv.py:42-45) as one differentiable op: for small
    bandwidths the product is evaluated inside the synthesis kernel and the SO(3) spectrum never
    reaches memory.  ``x`` and ``y`` are spectra of real signals (half products
    where no gradient is recorded)."""
    return cuda_ops().ag_s2_product_synthesis(x, y, bias)


class S2Convolution(Module):
    def __init__(self, nfeature_in, nfeature_out, b_in, b_out, grid):
        """Correlation of a signal on the sphere with a learned kernel supported on a few points of
        the sphere; the result is a signal on SO(3).

        nfeature_in, nfeature_out: channel counts of the input and output signals.
        b_in, b_out: bandwidths; the input lives on the 2 b_in x 2 b_in sphere grid, the output on
            the (2 b_out)^3 SOFT grid.
        grid: the points (beta, alpha) on which the kernel has a weight, a tuple of 2-tuples;
            ``kernel`` holds one weight per (input channel, output channel, point).
        """
        super().__init__()
        self.nfeature_in = nfeature_in
        self.nfeature_out = nfeature_out
        self.b_in = b_in
        self.b_out = b_out
        self.grid = grid
        # one uniform_(-1, 1) draw on the default generator, as s2_conv.py:28
        self.kernel = Parameter(torch.empty(nfeature_in, nfeature_out, len(grid)).uniform_(-1, 1))
        self.scaling = 1. / math.sqrt(len(self.grid) * self.nfeature_in * (self.b_out ** 4.) / (self.b_in ** 2.))
        self.bias = Parameter(torch.zeros(1, nfeature_out, 1, 1, 1))
        self._spectrum_cache = KernelSpectrumCache()
        self._fourier = FourierMatrices()

    def _kernel_spectrum(self, kernel):
        """s2_rft(kernel * scaling, b_out, grid)"""
        return cuda_ops().ag_rft(kernel, *self._fourier.get(_setup_s2_ft, self.b_out, self.grid, self.scaling,
                                                            kernel.device))

    def forward(self, x, relu_so3_fft=None, channel_scale=None, bias=None):
        '''
        :x:      [batch, feature_in,  beta, alpha]
        :relu_so3_fft: (extension) bandwidth b_next of the SO3Convolution that follows: return
                 SO3_fft_real(relu(conv(x)), b_next) - that layer's input spectrum
                 [l * m * n, batch, feature_out, complex] (pass it on with ``input_spectrum=True,
                 real_spectrum=True``; without the latter the layer computes whole products).
                 Without autograd and for 2 b_out <= 32 the signal between the layers is never written.
        :channel_scale, bias: (extension, used by ``s2cnn_b200.fuse`` to fold an eval-mode BatchNorm3d
                 into the layer) multiply output channel j by channel_scale[j] - applied to the
                 kernel's spectrum - and add ``bias`` ([1, f_out, 1, 1, 1]) instead of the layer's own
        :return: [batch, feature_out, beta, alpha, gamma]
        '''
        assert x.size(1) == self.nfeature_in
        assert x.size(2) == 2 * self.b_in
        assert x.size(3) == 2 * self.b_in
        x = S2_fft_real.apply(x, self.b_out)  # [l * m, batch, feature_in, complex]
        # [l * m, feature_in, feature_out, complex]; kept between calls while the weights stand still
        y = self._spectrum_cache.get(self.kernel, self._kernel_spectrum)
        if channel_scale is not None:
            y = y * channel_scale.view(1, 1, -1, 1)
        own_bias = self.bias if bias is None else bias
        if relu_so3_fft is not None:
            b_next = int(relu_so3_fft)
            if 2 * self.b_out <= 32:   # ReLU applied while the next layer's analysis reads the signal
                plain = lambda xx, yy, bb: SO3_fft_real_relu.apply(_product_synthesis(xx, yy, bb), b_next)  # noqa: E731
            else:
                plain = lambda xx, yy, bb: SO3_fft_real.apply(torch.relu(_product_synthesis(xx, yy, bb)), b_next)  # noqa: E731
            if 2 * self.b_out <= 32 and b_next <= self.b_out:
                grad = torch.is_grad_enabled() and (x.requires_grad or y.requires_grad or own_bias.requires_grad)
                # a recorded pass computes whole products: its backward recomputes them through the unfused chain
                fused = lambda xx, yy, bb: cuda_ops().s2_conv_relu_so3_rfft(xx, yy, bb, b_next, real=not grad)  # noqa: E731
                return fused_or_recompute(fused, plain, (x, y, own_bias), grad,
                                          getattr(self, "fused_training", False))
            return plain(x, y, own_bias)
        # s2_mm -> SO3_ifft_real -> + bias, fused: [batch, feature_out, beta, alpha, gamma]
        return _product_synthesis(x, y, own_bias)
