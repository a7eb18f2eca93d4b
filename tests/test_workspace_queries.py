"""The workspace queries answer for the kernels that the call will take: nothing for the single-kernel paths (which
then run with a null pointer), and otherwise a size with which the call gives what it gives with any larger one.
The host path allocates no more than that."""
import pytest
import torch

import backends
from oracle import s2cnn_oracle as O

n3 = O.so3_nspec
MB = 1 << 20


def stream(dev):
    return torch.cuda.current_stream().cuda_stream if dev.type == "cuda" else None


@pytest.mark.parametrize("backend", backends.BACKENDS)
def test_single_kernel_paths_need_no_workspace(backend):
    lib = backends.get(backend)[0].lib
    for b, b_spec, nb in ((1, 1, 1), (5, 4, 7), (8, 8, 5000), (10, 6, 64), (16, 16, 40), (16, 5, 200)):
        assert lib.s2c_so3_analysis_workspace(nb, b, b_spec) == 0
        assert lib.s2c_so3_synthesis_workspace(nb, b_spec, b) == 0
    assert lib.s2c_s2_conv_synthesis_workspace(5, 8, 16) == 0
    assert lib.s2c_so3_relay_workspace(20, 16, 16, 10) == 0 and lib.s2c_so3_relay_workspace(40, 16, 16, 10) > 0
    assert lib.s2c_s2_conv_relu_so3_rfft_workspace(5, 8, 16, 10) == 0      # 40 signals: a product takes planes later
    assert lib.s2c_s2_conv_relu_so3_rfft_workspace(64, 20, 10, 6) > 0
    for nb in (300, 4000, 100000):                                         # bounded, whatever the batch
        assert 0 < lib.s2c_so3_analysis_workspace(nb, 16, 16) <= 192 * MB
        assert 0 < lib.s2c_so3_synthesis_workspace(nb, 30, 30) <= 192 * MB
    # 34 <= 2b <= 62: the product is evaluated inside the contraction, its spectrum needs no room
    assert lib.s2c_s2_conv_synthesis_workspace(3, 5, 20) == lib.s2c_so3_synthesis_workspace(15, 20, 20)


@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.parametrize("b_in,b_out", [(32, 32), (64, 64), (32, 64), (64, 32)])
def test_query_for_both_directions_takes_the_larger_one(backend, b_in, b_out):
    lib = backends.get(backend)[0].lib
    for nb in (1, 8, 31, 64, 256, 300):
        both = max(lib.s2c_so3_analysis_workspace(nb, b_in, b_out), lib.s2c_so3_synthesis_workspace(nb, b_in, b_out))
        assert lib.s2c_so3_fft_workspace(nb, b_in, b_out) == max(both, lib.s2c_so3_fft_workspace_min(b_in, b_out)) <= 256 * MB, nb


@pytest.mark.parametrize("backend", backends.BACKENDS)
def test_queries_answer_nonsense_with_nothing(backend):
    lib = backends.get(backend)[0].lib
    for name in ("so3_fft", "so3_analysis", "so3_synthesis", "s2_fft"):
        for bad in ((4, 0, 3), (4, 3, 0), (4, -2, 3), (4, 3, -1)):
            assert getattr(lib, "s2c_%s_workspace" % name)(*bad) == 0, (name, bad)
    assert lib.s2c_so3_relay_workspace(0, 3, 3, 3) == 0 and lib.s2c_so3_relay_workspace(5, 3, 0, 3) == 0
    assert lib.s2c_s2_conv_synthesis_workspace(2, 3, 0) == 0 and lib.s2c_s2_conv_synthesis_workspace(0, 3, 3) == 0
    assert lib.s2c_so3_mm_gradx_workspace(0, 1, 1, 1) == 0 and lib.s2c_rft_backward_workspace(3, 0, 5) == 0


@pytest.mark.parametrize("backend", backends.BACKENDS)
@pytest.mark.parametrize("b,b_spec,nb", [(4, 6, 3), (9, 9, 2), (13, 13, 130), (17, 5, 3), (18, 18, 2), (33, 7, 1)])
def test_calls_run_with_what_the_query_says(backend, b, b_spec, nb):
    ops, dev = backends.get(backend)
    gen = torch.Generator().manual_seed(b)
    x = torch.randn(nb, 2 * b, 2 * b, 2 * b, generator=gen).to(dev)
    s = torch.randn(n3(b_spec), nb, 2, generator=gen).to(dev)
    calls = {
        "rfft": ("s2c_so3_rfft", x, (n3(b_spec), nb, 2), (b, b_spec, 0), ops.lib.s2c_so3_analysis_workspace(nb, b, b_spec)),
        "rifft": ("s2c_so3_rifft", s, tuple(x.shape), (b_spec, b, 0, None, 0), ops.lib.s2c_so3_synthesis_workspace(nb, b_spec, b)),
    }
    for name, src, shape, args, size in calls.values():
        got = []
        for n in (size, size + 64 * MB if size else 0):
            ws = torch.empty(n, dtype=torch.uint8, device=dev) if n else None
            out = torch.full(shape, float("nan"), device=dev)
            ops.lib.call(name, src.data_ptr(), out.data_ptr(), nb, *args, ws.data_ptr() if n else None, n, stream(dev))
            got.append(out)
        assert torch.equal(*got) and not torch.isnan(got[0]).any(), name


@pytest.mark.gpu
@pytest.mark.parametrize("b,nb,fo", [(16, 2, 12), (10, 4, 20), (12, 8, 6)])
def test_fused_calls_of_small_batches_take_their_results_only(b, nb, fo):
    from s2cnn_b200.ops import cuda_ops
    ops = cuda_ops()
    xs, ys = torch.randn(b * b, nb, 3, 2, device="cuda"), torch.randn(b * b, 3, fo, 2, device="cuda")
    spec, sig = torch.randn(n3(b), nb, fo, 2, device="cuda"), torch.randn(nb, fo, 2 * b, 2 * b, 2 * b, device="cuda")
    for call in (lambda: ops.s2_conv_relu_so3_rfft(xs, ys, None, b), lambda: ops.so3_rifft_relu_rfft(spec, None, b, b),
                 lambda: ops.s2_conv_synthesis(xs, ys, None), lambda: ops.so3_rfft_with_sums(sig, for_grad=True),
                 lambda: ops.so3_rifft_relu_grad(spec, sig), lambda: ops.so3_rfft(sig), lambda: ops.so3_rifft(spec)):
        call()
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        out = call()
        own = sum(t.numel() * 4 for t in (out if isinstance(out, tuple) else (out,)))
        assert torch.cuda.max_memory_allocated() - before <= own + 4096
