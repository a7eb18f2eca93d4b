"""S2 generalised FFTs and their autograd wrappers.

Same names, arguments and shapes as s2cnn/soft/s2_fft.py (s2_fft :13, s2_ifft :61, S2_fft_real
:226, S2_ifft_real :239).  ``S2_fft_real`` feeds the real signal straight to the kernel instead of
first materialising a complex copy (the reference's as_complex at :232).
"""
from ..ops import cuda_ops


def s2_fft(x, for_grad=False, b_out=None):
    '''
    :param x: [..., beta, alpha, complex]
    :return:  [l * m, ..., complex]
    '''
    return cuda_ops().s2_fft(x, for_grad=for_grad, b_out=b_out)


def s2_ifft(x, for_grad=False, b_out=None):
    '''
    :param x: [l * m, ..., complex]
    :return: [..., beta, alpha, complex]
    '''
    return cuda_ops().s2_ifft(x, for_grad=for_grad, b_out=b_out)


class S2_fft_real:
    """Spectrum of a real signal, differentiable: ``S2_fft_real.apply(x, b_out)``, x [..., beta, alpha]
    -> [l * m, ..., complex]."""

    @staticmethod
    def apply(x, b_out=None):
        return cuda_ops().ag_s2_fft_real(x, b_out)


class S2_ifft_real:
    """Real signal of a spectrum, differentiable: ``S2_ifft_real.apply(x, b_out)``."""

    @staticmethod
    def apply(x, b_out=None):
        return cuda_ops().ag_s2_ifft_real(x, b_out)
