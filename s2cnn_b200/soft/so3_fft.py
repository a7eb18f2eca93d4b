"""SO(3) generalised FFTs and their autograd wrappers.

Same names, arguments and shapes as s2cnn/soft/so3_fft.py (so3_fft :12, so3_rfft :64, so3_ifft
:115, so3_rifft :158, SO3_fft_real :446, SO3_ifft_real :459).  The work is done by the CUDA
library; tensors must be float32 CUDA tensors.

Two deliberate differences, both invisible at the reference's own tolerances:

* ``so3_rifft`` returns the real part of the complex synthesis for any spectrum (the reference's
  CPU semantics); the reference's CUDA kernel assumed a Hermitian spectrum.
* ``SO3_fft_real.backward`` therefore uses the real-output synthesis directly instead of the
  complex one followed by ``[..., 0]`` (so3_fft.py:453-456) - same values, half the work.
"""
from ..ops import cuda_ops


def so3_fft(x, for_grad=False, b_out=None):
    '''
    :param x: [..., beta, alpha, gamma, complex]
    :return: [l * m * n, ..., complex]
    '''
    return cuda_ops().so3_fft(x, for_grad=for_grad, b_out=b_out)


def so3_rfft(x, for_grad=False, b_out=None):
    '''
    :param x: [..., beta, alpha, gamma]
    :return: [l * m * n, ..., complex]
    '''
    return cuda_ops().so3_rfft(x, for_grad=for_grad, b_out=b_out)


def so3_ifft(x, for_grad=False, b_out=None):
    '''
    :param x: [l * m * n, ..., complex]
    :return: [..., beta, alpha, gamma, complex]
    '''
    return cuda_ops().so3_ifft(x, for_grad=for_grad, b_out=b_out)


def so3_rifft(x, for_grad=False, b_out=None):
    '''
    :param x: [l * m * n, ..., complex]
    :return: [..., beta, alpha, gamma]
    '''
    return cuda_ops().so3_rifft(x, for_grad=for_grad, b_out=b_out)


class SO3_fft_real:
    """``so3_rfft``, differentiable: ``SO3_fft_real.apply(x, b_out)``."""

    @staticmethod
    def apply(x, b_out=None):
        return cuda_ops().ag_so3_fft_real(x, b_out)


class SO3_fft_real_relu:
    """``SO3_fft_real`` of ``relu(x)`` with the activation applied while the signal is read (the
    ReLU between two convolutions of the reference's models, e.g. examples/mnist/run.py:88-93,
    folded into the consumer); its backward writes 0 where x <= 0 inside the synthesis kernel, without
    a separate pass over the gradient signal.  Needs 2 b_in < 64."""

    @staticmethod
    def apply(x, b_out=None):
        return cuda_ops().ag_so3_fft_real(x, b_out, True)


class SO3_ifft_real:
    """``so3_rifft``, differentiable: ``SO3_ifft_real.apply(x, b_out)``."""

    @staticmethod
    def apply(x, b_out=None):
        return cuda_ops().ag_so3_ifft_real(x, b_out)


class SO3_ifft_real_bias:
    """``SO3_ifft_real`` followed by ``+ bias`` ([1, f_out, 1, 1, 1]) in one pass: the addition
    of s2cnn/soft/s2_conv.py:45 and so3_conv.py:56 is fused into the last synthesis kernel."""

    @staticmethod
    def apply(x, bias):
        return cuda_ops().ag_so3_ifft_real_bias(x, bias)
