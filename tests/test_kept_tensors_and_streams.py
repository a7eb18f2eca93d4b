"""What layers keep between calls: no second copy of the Fourier matrix."""
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
