"""so3_integrate: Haar integral of a signal on SO(3) (s2cnn/soft/so3_integrate.py:7-29)."""
from ..ops import cuda_ops


def so3_integrate(x):
    """
    Integrate a signal on SO(3) using the Haar measure

    :param x: [..., beta, alpha, gamma] (..., 2b, 2b, 2b)
    :return y: [...] (...)
    """
    assert x.size(-1) == x.size(-2)
    assert x.size(-2) == x.size(-3)
    return cuda_ops().ag_so3_integrate(x, False)


def so3_relu_integrate(x):
    """``so3_integrate(relu(x))`` in one pass over x (the activation is applied while reading)."""
    assert x.size(-1) == x.size(-2)
    assert x.size(-2) == x.size(-3)
    return cuda_ops().ag_so3_integrate(x, True)
