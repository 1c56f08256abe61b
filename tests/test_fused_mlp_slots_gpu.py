r"""The fused MLP backward at the edges of its plan: one to four row tiles in flight per CTA, ragged rows and tiles, rows that
cannot be fetched in 16-byte chunks, every activation, with and without biases; against the storage-rounded oracle."""
import pytest
import torch

from test_fused_mlp_gpu import NAMES, make_params, nerr, rows_outside, run_both

from triton_helpers_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(
    "rows,d_in,d_hid,d_out,depth,bias,activation,dtype",
    [
        (1, 32, 64, 16, 2, False, "relu", torch.float16),  # four slots, one row
        (129, 32, 64, 16, 1, True, "relu", torch.float16),
        (128 * 148 * 5 + 3, 32, 32, 16, 1, False, "none", torch.float16),  # more than one tile per slot
        (1000, 27, 64, 3, 2, True, "relu", torch.float16),  # three slots, rows of odd width
        (4099, 48, 64, 48, 2, False, "relu", torch.bfloat16),  # the output gradient in a tile of its own
        (20011, 32, 64, 3, 3, True, "silu", torch.float16),  # two slots
        (300, 64, 64, 64, 3, True, "relu2", torch.float16),
        (300, 16, 64, 8, 6, False, "none", torch.float16),  # one slot
        (777, 32, 16, 16, 9, True, "none", torch.bfloat16),  # the most layers that fit
    ],
)
def test_backward_at_the_edges_of_the_slot_plan(rows, d_in, d_hid, d_out, depth, bias, activation, dtype):
    p = make_params(d_in, d_hid, d_out, depth, dtype, bias=bias, seed=rows)
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(1, rows, d_in, generator=g).to(dtype)
    go = (torch.randn(1, rows, d_out, generator=g) * 0.1).to(dtype)
    want, got = run_both(x, p, go, activation, rounded=True)
    tight = 2e-3 if dtype == torch.float16 else 1.6e-2
    for name, w, gg in zip(NAMES, want, got):
        assert (w is None) == (gg is None), name
        if w is None:
            continue
        if name == "dx":
            assert rows_outside(gg, w, tight) <= 1e-2, f"dx rows outside: {rows_outside(gg, w, tight)}"
        else:
            assert nerr(gg, w) <= (tight if name == "y" else 5 * tight), f"{name}: {nerr(gg, w)}"
    assert _lib.lib().th_mlp_tc_status() == 0
