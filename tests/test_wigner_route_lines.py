"""2b >= 66 with 2b mod 4 = 2: the untiled Wigner kernels serve few signals and the tiled ones more.  Both add the
same terms in the same order, so the signals of a batch just above the line are, to the last bit, those of a batch
just below it; one of them against the oracle."""
import pytest
import torch

from oracle import s2cnn_oracle as O
from util import assert_close

n3 = O.so3_nspec


@pytest.mark.gpu
@pytest.mark.parametrize("b,b_spec,few_analysis,few_synthesis", [(33, 33, 33, 12), (35, 20, 32, 11), (45, 45, 24, 8)])
def test_both_sides_of_the_line_agree(b, b_spec, few_analysis, few_synthesis):
    from s2cnn_b200.ops import cuda_ops
    ops = cuda_ops()
    gen = torch.Generator(device="cuda").manual_seed(b)
    x = torch.randn(few_analysis + 1, 2 * b, 2 * b, 2 * b, generator=gen, device="cuda")
    more, few = ops.so3_rfft(x, b_out=b_spec), ops.so3_rfft(x[:-1], b_out=b_spec)
    assert torch.equal(more[:, :-1], few)
    s = torch.randn(n3(b_spec), few_synthesis + 1, 2, generator=gen, device="cuda")
    more_s, few_s = ops.so3_rifft(s, b_out=b), ops.so3_rifft(s[:, :-1].contiguous(), b_out=b)
    assert torch.equal(more_s[:-1], few_s)
    assert_close(few[:, :1], O.so3_rfft(x[:1].cpu(), b_out=b_spec), "analysis")
    assert_close(few_s[:1], O.so3_rifft(s[:, :1].cpu(), b_out=b), "synthesis")
