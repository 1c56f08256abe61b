r"""The multi-slot MLP forward where its output and its biases take paths of their own, against the float32 oracle."""
import pytest
import torch

from oracle import fused_mlp as oracle
from triton_helpers_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d_out", [24, 40, 64])
@pytest.mark.parametrize("rows", [1, 33, 128, 19001])
def test_wide_outputs_and_biases_of_the_multi_slot_forward(d_out, rows):
    # outputs of more than 16 columns leave through shared memory (edges: a part of a warp's 32 rows, of a 32-column box; padding
    # between rows stays as it was); biases are a K step of each layer's GEMM (seven layers: two operand tiles of them)
    g = torch.Generator().manual_seed(rows + d_out)
    depth, d_in, hidden = 6, 32, 64
    lin = lambda o, i: ((torch.rand(o, i, generator=g) * 2 - 1) * (3 / i) ** 0.5).half().cuda()  # noqa: E731
    x = torch.randn(1, rows, d_in, generator=g).half().cuda()
    w_in, w_hid, w_out = lin(hidden, d_in), torch.cat([lin(hidden, hidden) for _ in range(depth - 1)]), lin(d_out, hidden)
    b_in, b_hid, b_out = (torch.randn(n, generator=g).half().cuda() for n in (hidden, (depth - 1) * hidden, d_out))
    b_hid = b_hid.view(depth - 1, hidden)
    b_hid[1, 5] = float("-inf")  # a unit that is switched off: the other layers' biases must not meet it
    want = oracle.forward(x.cpu(), *(t.cpu() for t in (w_in, b_in, w_out, b_out, w_hid, b_hid)))
    lib = _lib.lib()
    wide = torch.full((rows, d_out + 8), 7.0, dtype=torch.half, device="cuda")
    rc = lib.th_mlp_fwd(x.data_ptr(), d_in, w_in.data_ptr(), b_in.data_ptr(), w_hid.data_ptr(), b_hid.data_ptr(), w_out.data_ptr(), b_out.data_ptr(),
                        wide.data_ptr(), d_out + 8, rows, d_in, hidden, d_out, depth, 1, _lib.DTYPE_CODE[torch.half], 0, _lib.stream_ptr(x.device))  # fmt: skip
    assert rc == 0
    got = wide[:, :d_out].float().cpu()
    assert torch.isfinite(got).all() and (wide[:, d_out:] == 7).all()
    # seven layers rounded to 11 bits, in the largest output: 7 * 2^-11, and as much again for the sums behind them
    assert (got - want[0]).abs().max() <= 14 * 2**-11 * want.abs().max()
