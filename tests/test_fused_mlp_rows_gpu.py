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
@pytest.mark.parametrize("activation", ["relu", "none"])
def test_backward_through_the_ring_of_rows(rows, d_in, d_out, depth, bias, activation):
    dtype = torch.float16
    p = make_params(d_in, 64, d_out, depth, dtype, bias=bias, seed=d_in)
    g = torch.Generator().manual_seed(d_out)
    x = torch.randn(1, rows, d_in, generator=g).to(dtype)
    go = (torch.randn(1, rows, d_out, generator=g) * 0.1).to(dtype)
    want, got = run_both(x, p, go, activation, rounded=True)
    for name, w, gg in zip(NAMES, want, got):
        if w is None:
            continue
        if name == "dx" and activation == "none":
            # no ReLU that could switch: every row, the ragged tile's included, within one unit in the last place (2^-11 of the largest)
            # for each of the 2 depth + 1 stored roundings behind it; a row of another tile, or of none, is off by the size of a row
            assert nerr(gg, w) <= (2 * depth + 1) * 2**-11, f"dx: {nerr(gg, w)}"
        elif name == "dx":
            assert rows_outside(gg, w, 2e-3) <= 1e-2, f"dx rows outside: {rows_outside(gg, w, 2e-3)}"
            assert nerr(gg, w) <= 0.5
        else:  # as for the other shapes: one rounding of y, sums in another order for the parameters
            assert nerr(gg, w) <= (2e-3 if name == "y" else 1e-2), f"{name}: {nerr(gg, w)}"
    assert _lib.lib().th_mlp_tc_status() == 0


@pytest.mark.parametrize("rows", [1, 33, 129, 148 * 128 * 3 + 50])
@pytest.mark.parametrize("d_in,d_out", [(64, 64), (61, 33), (32, 17), (16, 9), (8, 64), (9, 8), (48, 1), (3, 48)])
def test_rows_off_their_alignment_give_the_gradients_of_aligned_ones(rows, d_in, d_out):
    # One element off and with gaps between rows: the copies by threads, whole rows of a thread and lanes along a row.  Rows do not
    # depend on one another, so the input gradient is the same bits as that of aligned rows.
    hidden, depth, dtype = 64, 2, torch.float16
    p = {k: None if v is None else v.cuda() for k, v in make_params(d_in, hidden, d_out, depth, dtype, bias=False, seed=rows).items()}
    g = torch.Generator().manual_seed(rows + d_in)
    lib = _lib.lib()

    def backward(off, pad_in, pad_out):
        torch.manual_seed(1)
        wide = lambda cols, pad: torch.full((rows * (cols + pad) + 2,), 7.0, dtype=dtype, device="cuda")  # noqa: E731
        view = lambda t, cols, pad: t[off : off + rows * (cols + pad)].view(rows, cols + pad)  # noqa: E731
        xs, gos, dxs = wide(d_in, pad_in), wide(d_out, pad_out), wide(d_in, pad_in)
        view(xs, d_in, pad_in)[:, :d_in] = x.cuda()
        view(gos, d_out, pad_out)[:, :d_out] = go.cuda()
        dw = [torch.empty_like(p[k]) for k in ("w_in", "w_hid", "w_out")]
        size = lib.th_mlp_workspace_bytes(d_in, hidden, d_out, depth)
        ws = torch.empty(size, dtype=torch.uint8, device="cuda")
        rc = lib.th_mlp_bwd(
            xs.data_ptr() + 2 * off, d_in + pad_in, p["w_in"].data_ptr(), None, p["w_hid"].data_ptr(), None, p["w_out"].data_ptr(), None,
            gos.data_ptr() + 2 * off, d_out + pad_out, dxs.data_ptr() + 2 * off, d_in + pad_in,
            dw[0].data_ptr(), None, dw[1].data_ptr(), None, dw[2].data_ptr(), None, ws.data_ptr(), size,
            rows, d_in, hidden, d_out, depth, _lib.ACTIVATION_CODE["relu"], _lib.DTYPE_CODE[dtype], 0, _lib.stream_ptr(xs.device),
        )  # fmt: skip
        assert rc == 0
        got = view(dxs, d_in, pad_in)
        assert (got[:, d_in:] == 7).all() and (dxs[:off] == 7).all() and (dxs[off + rows * (d_in + pad_in) :] == 7).all()
        return got[:, :d_in].clone(), dw

    x = torch.randn(rows, d_in, generator=g).to(dtype)
    go = (torch.randn(rows, d_out, generator=g) * 0.1).to(dtype)
    want, dw_want = backward(0, -d_in % 8, -d_out % 8)  # rows of whole 16-byte chunks
    for off, pad_in, pad_out in ((1, 0, 0), (0, 1, 3), (1, 7, 8)):
        got, dw = backward(off, pad_in, pad_out)
        assert torch.equal(got, want)
        for a, b in zip(dw, dw_want):
            assert nerr(a, b) <= 2e-3  # float32 sums in another order, rounded once: one unit in the last place of the largest
    assert _lib.lib().th_mlp_tc_status() == 0
