r"""A biased network's backward recomputes what its forward computed: the same ReLUs are open in both, also where a
pre-activation is a sum that cancels to within its rounding."""
import pytest
import torch

from triton_helpers_b200 import _lib
from triton_helpers_b200.layers.fully_fused_mlp import fully_fused_mlp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows", [300, 100_003])
@pytest.mark.parametrize("d_in,hidden", [(32, 64), (64, 64), (27, 64), (48, 32), (19, 16)])  # 27 and 19: rows TMA cannot describe
def test_backward_opens_the_relus_the_forward_opened(d_in, hidden, rows, dtype):
    g = torch.Generator().manual_seed(d_in + rows)
    w = torch.randn(hidden, d_in, generator=g).to(dtype)
    centre = torch.rand(d_in, generator=g) * 8 + 8
    step = 2.0**-7 if dtype == torch.float16 else 2.0**-4  # the spacing of the storage type there
    x = (centre.to(dtype).float() + step * torch.randint(-2, 3, (rows, d_in), generator=g)).to(dtype)
    b = -(w.double() @ centre.to(dtype).double()).to(dtype)  # x . w is some tens, x . w + b within a few hundredths of zero
    eye, zero = torch.eye(hidden).to(dtype), torch.zeros(hidden).to(dtype)
    xc = x[None].cuda().requires_grad_(True)
    y = fully_fused_mlp(xc, w.cuda(), b.cuda(), eye.cuda(), zero.cuda(), None, None, activation="relu")
    (dx,) = torch.autograd.grad(y, xc, torch.ones_like(y))
    open_ = (y > 0).double()[0].cpu()
    assert 0.2 < open_.mean() < 0.8
    want = open_ @ w.double()
    # one rounding of the largest sum; a ReLU that differs moves its row by a row of w, whose largest entry is above one
    limit = (2.0**-10 if dtype == torch.float16 else 2.0**-7) * want.abs().max()
    assert limit < w.double().abs().amax(-1).min()
    assert (dx[0].cpu().double() - want).abs().max() <= limit
    assert _lib.lib().th_mlp_tc_status() == 0
