r"""Reversible backward with biases and with activations that need the pre-activation, at the sizes where its tensor-core path can
go wrong: the first full tile, a ragged last one, several tiles per CTA, narrow widths; against the storage-rounded oracle."""
import pytest
import torch

from oracle import reversible_mlp as oracle
from test_reversible_mlp_gpu import TIGHT, make_params, nerr, rows_outside, to_cuda

from triton_helpers_b200 import _lib
from triton_helpers_b200.layers.reversible_mlp import ReversibleMLP, reversible_mlp_backward, reversible_mlp_forward

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


def float64_gradients(x, params, go, half, hidden, blocks):
    r"""Gradients of the biased ReLU stack by autograd in float64: ``[dx, dw_f1, dw_f2, dw_g1, dw_g2, db_f1, db_f2, db_g1, db_g2]``."""
    x, *params = (t.detach().double().requires_grad_(True) for t in (x, *params))
    w_f1, w_f2, w_g1, w_g2, b_f1, b_f2, b_g1, b_g2 = params

    def branch(u, w1, b1, w2, b2, k):
        h = torch.relu(u @ w1[k * hidden : (k + 1) * hidden].t() + b1[k])
        return h @ w2[k * half : (k + 1) * half].t() + b2[k]

    x1, x2 = x[:, :half], x[:, half:]
    for k in range(blocks):
        x1 = x1 + branch(x2, w_f1, b_f1, w_f2, b_f2, k)
        x2 = x2 + branch(x1, w_g1, b_g1, w_g2, b_g2, k)
    return torch.autograd.grad(torch.cat([x1, x2], -1), [x, *params], go.double())


@pytest.mark.parametrize(
    "dtype,rows,blocks,dx,dw,db",
    [
        # relative errors against float64 of the mma.sync backward, which took biased stacks before: mean of four seeds
        (torch.float16, 128, 8, 0.00920, 0.01042, 0.01029),
        (torch.float16, 1000, 10, 0.01274, 0.01361, 0.01398),
        (torch.float16, 4099, 8, 0.01046, 0.01218, 0.01242),
        (torch.bfloat16, 128, 10, 0.03707, 0.04045, 0.04113),
        (torch.bfloat16, 1000, 8, 0.03007, 0.03535, 0.03714),
        (torch.bfloat16, 4099, 10, 0.03517, 0.03881, 0.04028),
    ],
)
def test_deep_biased_stacks_are_as_exact_as_on_mma_sync(dtype, rows, blocks, dx, dw, db):
    # what remains is where ReLUs within a rounding of zero switch, which depends on the last bits: over 24 such combinations the ratio
    # of the two kernels' errors is 0.995 +- 0.006 (float16) and 1.0004 +- 0.002
    errors = torch.zeros(3, dtype=torch.float64)
    for seed in range(4):
        torch.manual_seed(seed)
        layer = ReversibleMLP(128, blocks, 64, "relu", bias=True).cuda().to(dtype)
        x = torch.randn(rows, 128, device="cuda").to(dtype).requires_grad_(True)
        go = torch.randn(rows, 128, device="cuda").to(dtype)
        params = [getattr(layer, n) for n in ("w_f1", "w_f2", "w_g1", "w_g2", "b_f1", "b_f2", "b_g1", "b_g2")]
        got = torch.autograd.grad(layer(x), [x, *params], go)
        want = float64_gradients(x, params, go, 64, 64, blocks)
        e = torch.tensor([float((g.double() - w).norm() / w.norm()) for g, w in zip(got, want)], dtype=torch.float64)
        errors += torch.stack([e[0], e[1:5].mean(), e[5:].mean()]) / 4
    assert (errors <= 1.05 * torch.tensor([dx, dw, db], dtype=torch.float64)).all(), errors
