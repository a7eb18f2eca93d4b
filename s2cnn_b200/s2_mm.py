"""s2_mm: per-degree product of an S2 signal spectrum with an S2 kernel spectrum.

Mirrors s2cnn/s2_mm.py:10-101 (function and autograd rule); all three products run in the
grouped complex GEMM kernel of the library.
"""
from .ops import cuda_ops


def s2_mm(x, y):
    '''
    :param x: [l * m,     batch,      feature_in,  complex]
    :param y: [l * m,     feature_in, feature_out, complex]
    :return:  [l * m * n, batch,      feature_out, complex]
    '''
    assert y.size(3) == 2
    assert x.size(3) == 2
    assert y.size(1) == x.size(2)
    assert y.size(0) == x.size(0)
    return cuda_ops().ag_s2_mm(x, y)
