"""The native host path writes through raw pointers, which torch.jit.trace and forward-mode differentiation do not
see.  The differentiable ops are recorded by a tracer as one node each (values and gradients of the traced function
on new inputs are the eager ones); the plain ops refuse to be traced, and every op refuses dual tensors - nothing is
recorded as an uninitialised buffer and no tangent is dropped."""
import pytest
import torch
import torch.autograd.forward_ad as fwd

import backends
from oracle import s2cnn_oracle as O

n3 = O.so3_nspec


def ops_and_inputs(S, b=3):
    from s2cnn_b200.soft.s2_fft import S2_fft_real, S2_ifft_real
    from s2cnn_b200.soft.so3_fft import SO3_fft_real, SO3_fft_real_relu, SO3_ifft_real
    grid = S.s2_near_identity_grid()
    return {
        "s2 analysis": (lambda a: S2_fft_real.apply(a, 2), (2, 1, 2 * b, 2 * b)),
        "s2 synthesis": (lambda a: S2_ifft_real.apply(a), (b * b, 2, 2)),
        "so3 analysis": (lambda a: SO3_fft_real.apply(a, 2), (2, 2 * b, 2 * b, 2 * b)),
        "so3 analysis of relu": (lambda a: SO3_fft_real_relu.apply(a, 2), (2, 2 * b, 2 * b, 2 * b)),
        "so3 synthesis": (lambda a: SO3_ifft_real.apply(a), (n3(b), 2, 2)),
        "integral": (S.so3_integrate, (2, 2 * b, 2 * b, 2 * b)),
        "s2 kernel transform": (lambda a: S.s2_rft(a, b, grid), (2, len(grid))),
    }


@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.filterwarnings("ignore")
def test_traced_ops_give_the_eager_values_and_gradients(backend):
    import s2cnn_b200 as S
    with backends.active(backend) as (ops, dev):
        gen = torch.Generator().manual_seed(1)
        for name, (f, shape) in ops_and_inputs(S).items():
            x, x2 = (torch.randn(*shape, generator=gen).to(dev) for _ in range(2))
            for grad in (False, True):
                traced = torch.jit.trace(f, x.clone().requires_grad_(grad), check_trace=False)
                assert torch.equal(traced(x2), f(x2)), name
            a, b = (x2.clone().requires_grad_(True) for _ in range(2))
            traced(a).square().sum().backward()
            f(b).square().sum().backward()
            assert torch.equal(a.grad, b.grad), name


@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.filterwarnings("ignore")
def test_plain_ops_refuse_to_be_traced(backend):
    ops, dev = backends.get(backend)
    x = torch.randn(2, 4, 4, 4, device=dev)
    with pytest.raises(RuntimeError, match="torch.jit.trace"):
        torch.jit.trace(lambda a: ops.so3_rfft(a), x, check_trace=False)


@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.parametrize("grad", [False, True])
def test_forward_mode_is_refused(backend, grad):
    import s2cnn_b200 as S
    with backends.active(backend) as (ops, dev):
        for name, (f, shape) in ops_and_inputs(S).items():
            x = torch.randn(*shape, device=dev).requires_grad_(grad)
            with fwd.dual_level():
                with pytest.raises(NotImplementedError, match="jvp"):
                    f(fwd.make_dual(x, torch.ones_like(x)))
