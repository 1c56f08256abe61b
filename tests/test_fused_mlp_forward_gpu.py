r"""The multi-slot MLP forward where its output and its biases take paths of their own, against the float32 oracle."""
import pytest
import torch

from oracle import fused_mlp as oracle
from triton_helpers_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize(
    "rows,d_out,depth",
    # 16 layers before the last: the most whose biases fit as operand tiles, without room for the staging; 17: they no longer do
    [(r, d, 6) for r in (1, 33, 128, 19001) for d in (24, 40, 64)] + [(r, d, n) for r in (33, 148 * 128 * 4 + 9) for d in (16, 64) for n in (16, 17)],
)
def test_wide_outputs_and_biases_of_the_multi_slot_forward(rows, d_out, depth, dtype):
    # outputs of more than 16 columns leave through shared memory (edges: a part of a warp's 32 rows, of a 32-column box; padding
    # between rows stays as it was); biases are a K step of each layer's GEMM (seven layers: two operand tiles of them)
    g = torch.Generator().manual_seed(rows + d_out)
    d_in, hidden = 32, 64
    lin = lambda o, i: ((torch.rand(o, i, generator=g) * 2 - 1) * (3 / i) ** 0.5).to(dtype).cuda()  # noqa: E731
    x = torch.randn(1, rows, d_in, generator=g).to(dtype).cuda()
    w_in, w_hid, w_out = lin(hidden, d_in), torch.cat([lin(hidden, hidden) for _ in range(depth - 1)]), lin(d_out, hidden)
    b_in, b_hid, b_out = (torch.randn(n, generator=g).to(dtype).cuda() for n in (hidden, (depth - 1) * hidden, d_out))
    b_hid = b_hid.view(depth - 1, hidden)
    b_hid[1, 5] = float("-inf")  # a unit that is switched off: the other layers' biases must not meet it
    want = oracle.forward(x.cpu(), *(t.cpu() for t in (w_in, b_in, w_out, b_out, w_hid, b_hid)))
    lib = _lib.lib()
    wide = torch.full((rows, d_out + 8), 7.0, dtype=dtype, device="cuda")
    rc = lib.th_mlp_fwd(x.data_ptr(), d_in, w_in.data_ptr(), b_in.data_ptr(), w_hid.data_ptr(), b_hid.data_ptr(), w_out.data_ptr(), b_out.data_ptr(),
                        wide.data_ptr(), d_out + 8, rows, d_in, hidden, d_out, depth, 1, _lib.DTYPE_CODE[dtype], 0, _lib.stream_ptr(x.device))  # fmt: skip
    assert rc == 0
    got = wide[:, :d_out].float().cpu()
    assert torch.isfinite(got).all() and (wide[:, d_out:] == 7).all()
    # depth + 1 layers rounded to 11 (8) bits, in the largest output: as many units of 2^-11 (2^-8), and as much again for the sums behind them
    assert (got - want[0]).abs().max() <= 2 * (depth + 1) * (2**-11 if dtype == torch.float16 else 2**-8) * want.abs().max()
