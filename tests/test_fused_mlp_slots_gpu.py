r"""The fused MLP backward at the edges of its plan: one to four row tiles in flight per CTA, ragged rows and tiles, rows that
cannot be fetched in 16-byte chunks, every activation, with and without biases; against the storage-rounded oracle."""
import pytest
import torch

from test_fused_mlp_gpu import NAMES, make_params, nerr, rows_outside, run_both

from triton_helpers_b200 import _lib
from triton_helpers_b200.layers.fully_fused_mlp import fully_fused_mlp

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


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_silu_of_every_16_bit_value(dtype):
    # identity weights: hidden = silu(z), and the input's gradient is silu'(z).  Half a unit of the last place for the rounding to
    # 16 bits, and what __expf is off by in float32: 2 + 1.17 |z| units, |z| <= 104 before the result is 0 -> 1.5e-5, 0.03 units in float16.
    z = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(dtype)
    z = z[torch.isfinite(z.float())].cuda()
    x = torch.zeros(1, z.numel(), 16, device="cuda", dtype=dtype)
    x[0, :, 0] = z
    x.requires_grad_(True)
    eye = torch.eye(16, device="cuda", dtype=dtype)
    y = fully_fused_mlp(x, eye, None, eye, None, None, None, "silu")
    go = torch.zeros_like(x)
    go[..., 0] = 1
    (dx,) = torch.autograd.grad(y, x, go)
    zd = z.double()
    s = torch.sigmoid(zd)
    info = torch.finfo(dtype)
    for got, want in ((y[0, :, 0], zd * s), (dx[0, :, 0], s * (1 + zd * (1 - s)))):
        unit = info.eps * 2.0 ** torch.floor(torch.log2(want.abs().clamp_min(info.tiny)))
        assert float(((got.detach().double() - want).abs() / unit).max()) <= 0.53
