"""so3_mm: per-degree block product of an SO(3) signal spectrum with a kernel spectrum.

Mirrors s2cnn/so3_mm.py:8-122 (function and autograd rule).
"""
from .ops import bandwidth_from_so3_nspec, cuda_ops


def so3_mm(x, y):
    '''
    :param x: [l * m * n,   batch,    feature_in,  complex]
    :param y: [l * m * n, feature_in, feature_out, complex]
    :return:  [l * m * n,   batch,    feature_out, complex]
    '''
    assert y.size(3) == 2
    assert x.size(3) == 2
    assert y.size(1) == x.size(2)
    assert y.size(0) == x.size(0)
    bandwidth_from_so3_nspec(x.size(0))  # asserts a valid spectrum length
    return cuda_ops().ag_so3_mm(x, y)
