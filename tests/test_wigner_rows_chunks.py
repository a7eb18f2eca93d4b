"""2b = 64 and 128: chunks of 3, 5, 6 and 7 signals (the analysis takes them in fours, the synthesis in eights, so the last
four or eight are ragged), degrees that are no multiple of the four rows or sixteen frequencies a kernel takes at a time,
and a workspace aligned to 16 bytes only, against the separate passes (``s2c_debug_force_general_path(2)``)."""
import ctypes

import pytest
import torch

import backends
from oracle import s2cnn_oracle as O
from util import assert_close


@pytest.mark.parametrize("backend,width,b_out", [pytest.param("emul", 5, 6)] +
                         [pytest.param("cuda", w, k, marks=pytest.mark.gpu) for w, k in
                          ((3, 32), (5, 31), (6, 17), (7, 18), (5, 2))])
def test_ragged_chunks(backend, width, b_out):
    ops, dev = backends.get(backend)
    gen = torch.Generator().manual_seed(width)
    x = torch.randn(width, 64, 64, 64, generator=gen).to(dev)
    s = torch.randn(O.so3_nspec(b_out), width, 2, generator=gen).to(dev)
    xc = torch.randn(width, 64, 64, 64, 2, generator=gen).to(dev) if backend == "cuda" else None
    res = []
    try:
        for level in (2, 0):
            ops.lib.s2c_debug_force_general_path(level)
            res.append([ops.so3_rfft(x, b_out=b_out), ops.so3_rifft(s, b_out=32)])
            if xc is not None:
                res[-1] += [ops.so3_fft(xc, b_out=b_out), ops.so3_ifft(s, b_out=32)]
    finally:
        ops.lib.s2c_debug_force_general_path(0)
    for a, b in zip(res[1], res[0]):
        assert_close(a, b.cpu())


@pytest.mark.gpu
def test_workspace_aligned_to_16_bytes():
    ops, dev = backends.get("cuda")
    lib, p = ops.lib, ctypes.c_void_p
    s = torch.randn(O.so3_nspec(32), 6, 2, device=dev)
    want = ops.so3_rifft(s)
    n = lib.s2c_so3_synthesis_workspace(6, 32, 32)
    ws = torch.empty(n + 64, dtype=torch.uint8, device=dev)
    out, spec = torch.empty_like(want), torch.empty_like(s)
    at = ws.data_ptr() // 32 * 32 + 48
    stream = p(torch.cuda.current_stream().cuda_stream)
    lib.call("s2c_so3_rifft", p(s.data_ptr()), p(out.data_ptr()), 6, 32, 32, 0, None, 1, p(at), n, stream)
    lib.call("s2c_so3_rfft", p(want.data_ptr()), p(spec.data_ptr()), 6, 32, 32, 0, p(at), n, stream)
    torch.cuda.synchronize()
    assert torch.equal(out, want) and torch.equal(spec, ops.so3_rfft(want))


@pytest.mark.gpu
@pytest.mark.parametrize("b,width,k", [(32, 300, 13), (64, 35, 9)])
def test_long_chunks_equal_short_ones(b, width, k):
    """300 signals at b = 32: two chunks of 152 and 148, 35 at b = 64: of 24 and 11, against chunks of 8; equal to the last bit."""
    ops, dev = backends.get("cuda")
    gen = torch.Generator(device=dev).manual_seed(4)
    x = torch.randn(width, 2 * b, 2 * b, 2 * b, generator=gen, device=dev)
    res = []
    try:
        for width in (0, 8):
            ops.lib.s2c_debug_plane_chunk(width)
            spec = ops.so3_rfft(x, b_out=k)
            res.append((spec, ops.so3_rifft(spec, b_out=b)))
    finally:
        ops.lib.s2c_debug_plane_chunk(0)
    assert torch.equal(res[0][0], res[1][0]) and torch.equal(res[0][1], res[1][1])
