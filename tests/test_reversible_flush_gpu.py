r"""The reversible backward's weight gradients on their way out: several row tiles per CTA, every
pair of widths (the two accumulators of a branch share tensor-memory columns), with and without biases."""
import pytest
import torch

from test_reversible_mlp_gpu import TIGHT, make_params, nerr, to_cuda

from oracle import reversible_mlp as oracle
from triton_helpers_b200 import _lib
from triton_helpers_b200.layers.reversible_mlp import reversible_mlp_backward, reversible_mlp_forward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize(
    "rows,half,hidden",
    [
        (128 * 148 * 2 + 5, 64, 64),  # two to three tiles per CTA, more CTAs than accumulators
        (128 * 17 + 1, 64, 64),  # eighteen CTAs
        (129, 64, 64),
        (128 * 40, 64, 32),
        (128 * 40 - 1, 32, 64),
        (128 * 40 + 64, 48, 48),
        (2000, 16, 48),
        (2000, 48, 16),
    ],
)
def test_weight_gradients_of_every_width_and_batch(rows, half, hidden, bias):
    # no ReLU that could switch: every block's gradients are tight
    dtype, blocks = torch.float16, 3
    weights, biases = make_params(blocks, half, hidden, bias, dtype, seed=half + hidden)
    weights = tuple((w.float() * 0.5).to(dtype) for w in weights)
    g = torch.Generator().manual_seed(rows)
    x, go = torch.randn(rows, 2 * half, generator=g).to(dtype), torch.randn(rows, 2 * half, generator=g).to(dtype)
    wc, bc = to_cuda(weights), to_cuda(biases)
    y = reversible_mlp_forward(x.cuda(), wc, bc, "none")
    got = reversible_mlp_backward(y, go.cuda(), wc, bc, "none", reconstruct=True)
    _, dx, grads, xrec = oracle.forward_backward_storage_rounded(x, weights, biases, go, "none", y_saved=y.cpu())
    assert nerr(got.dx, dx) <= 5 * TIGHT[dtype] and nerr(got.x_reconstructed, xrec) <= 5 * TIGHT[dtype]
    for want, have in zip(grads, got[1:]):
        if want is None:
            continue
        per_block = want.shape[0] // blocks
        for b in range(blocks):
            s = slice(b * per_block, (b + 1) * per_block)
            assert nerr(have[s], want[s]) <= 5 * TIGHT[dtype], (b, nerr(have[s], want[s]))
    assert _lib.lib().th_rev_tc_status() == 0


@pytest.mark.parametrize("rows,blocks", [(128 * 148 * 3 + 5, 2), (128 * 148 * 4, 1), (128 * 40, 8)])
def test_weight_gradients_repeat_bit_for_bit(rows, blocks):
    # an accumulator has one owner that adds to it in order, and the copies are summed in order: no call differs from another
    dtype, half = torch.float16, 64
    weights, _ = make_params(blocks, half, half, False, dtype, seed=3)
    g = torch.Generator().manual_seed(rows)
    x, go = torch.randn(rows, 2 * half, generator=g).to(dtype).cuda(), torch.randn(rows, 2 * half, generator=g).to(dtype).cuda()
    wc, bc = to_cuda(weights), to_cuda((None,) * 4)
    y = reversible_mlp_forward(x, wc, bc, "relu")
    first = reversible_mlp_backward(y, go, wc, bc, "relu")
    for _ in range(8):
        for want, have in zip(first, reversible_mlp_backward(y, go, wc, bc, "relu")):
            assert want is None or torch.equal(want, have)
