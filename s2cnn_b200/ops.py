"""The op table: torch tensors in, torch tensors out, one method per entry point of the C ABI
(include/s2cnn_b200.h).

``Ops(lib)`` binds one build of the library to the native host path (host/host_ops.cpp), which checks
dtype and shape, allocates the output and the scratch space with torch (device memory management is
all torch is used for here) and passes raw pointers plus the current CUDA stream.  The public,
reference-named API in the sibling modules is built on ``cuda_ops()``, which is bound to the CUDA
build and refuses CPU tensors.

Methods: the ops themselves (``so3_rfft``, ``so3_rifft``, ``s2_fft``, ``so3_mm``, ... with the argument
names of their definitions in host_ops.cpp) and, under ``ag_...``, the differentiable ones with the
reference's autograd rules.
"""
import logging
import os

import torch

from . import _lib


def so3_nspec(b):
    return b * (4 * b * b - 1) // 3


def bandwidth_from_so3_nspec(nspec):
    b = round((3.0 / 4.0 * nspec) ** (1.0 / 3.0))  # as s2cnn/soft/so3_fft.py:121-122
    assert nspec == so3_nspec(b), "not an SO(3) spectrum length: %d" % nspec
    return b


def _log_new_tables(what, n):
    """The reference logs "Compute Wigner ..." on the "trainer" logger whenever a table is built
    (s2cnn/soft/so3_fft.py:223, s2_fft.py:127); the native path calls this when the library's count
    has grown."""
    logging.getLogger("trainer").info("Compute Wigner tables (%s): %d computed by this process", what, n)


def _flag(name):
    return os.environ.get(name, "0") not in ("", "0")


class _Traced(torch.autograd.Function):
    """One differentiable op inside ``torch.jit.trace``, recorded as a single Python call.  Its backward
    runs the op again and differentiates that with the op's own rule."""

    @staticmethod
    def forward(ctx, op, *args):
        ctx.op, ctx.others = op, [None if isinstance(a, torch.Tensor) else a for a in args]
        ctx.save_for_backward(*[a if isinstance(a, torch.Tensor) else None for a in args])
        with _lib.host_module().InsideTracedOp():
            return op(*args)

    @staticmethod
    def backward(ctx, grad):
        args = [o if t is None else t.detach().requires_grad_(need) for t, o, need in
                zip(ctx.saved_tensors, ctx.others, ctx.needs_input_grad[1:])]
        with torch.enable_grad():
            out = ctx.op(*args)
        wanted = [a for a, need in zip(args, ctx.needs_input_grad[1:]) if need]
        grads = iter(torch.autograd.grad(out, wanted, grad, allow_unused=True))
        return (None,) + tuple(next(grads) if need else None for need in ctx.needs_input_grad[1:])


def _traced(native, name, *args):
    return _Traced.apply(getattr(native, name), *args)


class Ops:
    def __init__(self, lib):
        self.lib = lib
        # S2CNN_B200_NVTX: every library call in an NVTX range of its name; S2CNN_B200_CHECK_TC: wait
        # for the device after every spectral product and raise if a tensor-core product gave up on one
        # of its bounded barrier waits (check_tensor_core_status - a training loop can call that once
        # per step instead)
        native = _lib.host_module().Ops(lib.path, _log_new_tables, _flag("S2CNN_B200_NVTX"),
                                        bool(os.environ.get("S2CNN_B200_CHECK_TC")))
        for name in dir(native):
            if not name.startswith("_"):
                setattr(self, name, getattr(native, name))

    # -- host generators -----------------------------------------------------------------------
    def so3_rotation_matrices(self, b, alpha, beta, gamma):
        """Host: concatenated Wigner-D matrices [b(4b^2-1)/3, 2] of one rotation."""
        import numpy as np
        U = np.empty((so3_nspec(b), 2), dtype=np.float32)
        self.lib.call("s2c_so3_rotation_matrices", b, float(alpha), float(beta), float(gamma),
                      U.ctypes.data)
        return U

    def so3_ft_matrix(self, b, grid):
        import numpy as np
        g = np.ascontiguousarray(np.asarray(grid, dtype=np.float64).reshape(len(grid), 3))
        F = np.empty((len(grid), so3_nspec(b), 2), dtype=np.float32)
        self.lib.call("s2c_so3_ft_matrix", b, g.ctypes.data, len(grid), F.ctypes.data)
        return F

    def s2_ft_matrix(self, b, grid):
        import numpy as np
        g = np.ascontiguousarray(np.asarray(grid, dtype=np.float64).reshape(len(grid), 2))
        F = np.empty((len(grid), b * b, 2), dtype=np.float32)
        self.lib.call("s2c_s2_ft_matrix", b, g.ctypes.data, len(grid), F.ctypes.data)
        return F


_cuda_ops = None


def cuda_ops():
    global _cuda_ops
    if _cuda_ops is None:
        _cuda_ops = Ops(_lib.cuda_lib())
    return _cuda_ops
