"""A bulk copy that does not land within the bound of its wait: the kernel reads the data from global memory, starts no
further copy while the barrier's phase is not over, and gives the late one a second wait before the block ends.  On the CPU,
where the emulation holds one copy back and counts copies into an unfinished phase and copies that outlive their block."""
import pytest
import torch

import backends
from oracle import s2cnn_oracle as O

CALLS = {
    # analysis at 2b = 64: a block walks items, two copies each; 3 blocks
    "rows": lambda ops, x, s: ops.so3_rfft(x, b_out=18),
    # single-kernel synthesis (walking blocks) and relay: a copy per group of betas
    "fused": lambda ops, x, s: ops.so3_rifft(s, b_out=7),
    "integral": lambda ops, x, s: ops.so3_rifft_relu_integrate(s),
    "relay": lambda ops, x, s: ops.so3_rifft_relu_rfft(s, None, 7, 5),
}


@pytest.mark.parametrize("name", CALLS)
@pytest.mark.parametrize("never", [0, 1])
@pytest.mark.parametrize("nth", [1, 2, 3, 4, 7])
def test_late_copy(name, nth, never):
    ops, _ = backends.get("emul")
    gen = torch.Generator().manual_seed(1)
    x = torch.randn(2, 64, 64, 64, generator=gen) if name == "rows" else None
    s = torch.randn(O.so3_nspec(7), 5, 2, generator=gen)
    ops.lib.s2c_debug_cluster(2)
    try:
        want = CALLS[name](ops, x, s)
        hold = ops.lib.s2c_emul_hold_copy
        hold(nth, never)
        got = CALLS[name](ops, x, s)
        faults = hold(0, 0)
    finally:
        ops.lib.s2c_debug_cluster(0)
    assert faults == 0
    if never and name != "rows":     # not a number wherever a copy is missing, and nothing wrong elsewhere
        assert torch.equal(torch.where(torch.isnan(got), want, got), want)
    else:
        assert torch.equal(got, want)
