r"""Reversible backward with biases and with activations that need the pre-activation, at the sizes where its tensor-core path can
go wrong: the first full tile, a ragged last one, several tiles per CTA, narrow widths; against the storage-rounded oracle."""
import pytest
import torch

from oracle import reversible_mlp as oracle
from test_reversible_mlp_gpu import TIGHT, make_params, nerr, rows_outside, to_cuda

from triton_helpers_b200 import _lib
from triton_helpers_b200.layers.reversible_mlp import reversible_mlp_backward, reversible_mlp_forward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(
    "rows,d_model,hidden,blocks,bias,activation,dtype",
    [
        (128, 128, 64, 2, True, "silu", torch.float16),
        (129, 64, 16, 3, True, "none", torch.bfloat16),
        (1000, 96, 48, 2, True, "relu", torch.float16),
        (300, 128, 64, 2, False, "silu", torch.bfloat16),
        (300, 32, 32, 1, False, "relu2", torch.float16),
        (128 * 300 + 5, 64, 32, 2, True, "silu", torch.float16),
    ],
)
def test_biased_and_preactivation_backward(rows, d_model, hidden, blocks, bias, activation, dtype):
    weights, biases = make_params(blocks, d_model // 2, hidden, bias, dtype, seed=rows)
    g = torch.Generator().manual_seed(rows)
    x = torch.randn(rows, d_model, generator=g).to(dtype)
    go = torch.randn(rows, d_model, generator=g).to(dtype)
    wc, bc = to_cuda(weights), to_cuda(biases)
    y = reversible_mlp_forward(x.cuda(), wc, bc, activation)
    got = reversible_mlp_backward(y, go.cuda(), wc, bc, activation, reconstruct=True)
    _, dx_r, grads_r, xrec_r = oracle.forward_backward_storage_rounded(x, weights, biases, go, activation, y_saved=y.cpu())
    assert rows_outside(got.dx, dx_r, 2 * TIGHT[dtype]) <= 5e-2
    assert rows_outside(got.x_reconstructed, xrec_r, 2 * TIGHT[dtype]) <= 5e-2
    for name, want, have in zip(("dw_f1", "dw_f2", "dw_g1", "dw_g2", "db_f1", "db_f2", "db_g1", "db_g2"), grads_r, got[1:9]):
        assert (want is None) == (have is None), name
        if want is not None:
            assert nerr(have, want) <= 5 * TIGHT[dtype], f"{name}: {nerr(have, want)}"
    assert _lib.lib().th_rev_tc_status() == 0


@pytest.mark.parametrize("half", [16, 32, 48, 64])
@pytest.mark.parametrize("hidden", [16, 32, 48, 64])
@pytest.mark.parametrize("activation,dtype", [("relu", torch.float16), ("none", torch.bfloat16)])
def test_every_width(half, hidden, activation, dtype):
    # the kernels know the half at compile time; a full tile and a ragged one, two blocks
    rows, blocks = 200, 2
    weights, biases = make_params(blocks, half, hidden, False, dtype, seed=half + hidden)
    g = torch.Generator().manual_seed(hidden)
    x = torch.randn(rows, 2 * half, generator=g).to(dtype)
    go = torch.randn(rows, 2 * half, generator=g).to(dtype)
    wc = to_cuda(weights)
    y = reversible_mlp_forward(x.cuda(), wc, biases, activation)
    got = reversible_mlp_backward(y, go.cuda(), wc, biases, activation, reconstruct=True)
    y_r, _, _, _ = oracle.forward_backward_storage_rounded(x, weights, biases, go, activation)
    _, dx_r, grads_r, xrec_r = oracle.forward_backward_storage_rounded(x, weights, biases, go, activation, y_saved=y.cpu())
    assert rows_outside(y, y_r, TIGHT[dtype]) <= 1e-2
    assert rows_outside(got.dx, dx_r, 2 * TIGHT[dtype]) <= 5e-2
    assert rows_outside(got.x_reconstructed, xrec_r, 2 * TIGHT[dtype]) <= 5e-2
    for name, want, have in zip(("dw_f1", "dw_f2", "dw_g1", "dw_g2"), grads_r, got[1:5]):
        assert nerr(have, want) <= 5 * TIGHT[dtype], f"{name}: {nerr(have, want)}"
