r"""The fused MLP backward's ring of row buffers: more tiles per CTA than buffers, rows by TMA, by threads and mixed, against the
storage-rounded oracle."""
import pytest
import torch

from test_fused_mlp_gpu import NAMES, make_params, nerr, rows_outside, run_both

from triton_helpers_b200 import _lib

pytestmark = pytest.mark.gpu

WRAPS = 148 * 128 * 6 + 77  # six to seven tiles per CTA, at most five buffers


@pytest.mark.parametrize(
    "rows,d_in,d_out,depth,bias",
    [
        (WRAPS, 32, 16, 2, False),  # four slots, five buffers; both by TMA
        (WRAPS, 27, 3, 2, True),  # both by threads
        (WRAPS, 32, 1, 3, False),  # mixed
        (WRAPS, 27, 16, 1, False),
        (WRAPS, 64, 64, 2, False),  # as many buffers as slots
        (WRAPS, 16, 32, 4, True),  # two slots; 32- and 64-byte rows
        (128 * 148 * 2 + 1, 48, 24, 2, True),
    ],
)
def test_backward_through_the_ring_of_rows(rows, d_in, d_out, depth, bias):
    dtype = torch.float16
    p = make_params(d_in, 64, d_out, depth, dtype, bias=bias, seed=d_in)
    g = torch.Generator().manual_seed(d_out)
    x = torch.randn(1, rows, d_in, generator=g).to(dtype)
    go = (torch.randn(1, rows, d_out, generator=g) * 0.1).to(dtype)
    want, got = run_both(x, p, go, "relu", rounded=True)
    for name, w, gg in zip(NAMES, want, got):
        if w is None:
            continue
        if name == "dx":
            assert rows_outside(gg, w, 2e-3) <= 1e-2, f"dx rows outside: {rows_outside(gg, w, 2e-3)}"
        else:  # as for the other shapes: one rounding of y, sums in another order for the parameters
            assert nerr(gg, w) <= (2e-3 if name == "y" else 1e-2), f"{name}: {nerr(gg, w)}"
    assert _lib.lib().th_mlp_tc_status() == 0
