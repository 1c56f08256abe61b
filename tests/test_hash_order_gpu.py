r"""The encoding over a spatially ordered batch: the order itself, and forward / backward against the unordered kernels."""
import pytest
import torch

from triton_helpers_b200 import _lib
from triton_helpers_b200.layers.hash_encoding.helpers import level_geometry
from triton_helpers_b200.layers.hash_encoding.kernel import PI_1, PI_2, PI_3

pytestmark = pytest.mark.gpu


def ordered_and_unordered(n, d, feats, dtype, cap, max_res, points, keep_order, levels=16):
    g = torch.Generator(device="cuda").manual_seed(n + d)
    x = torch.rand(n, d, device="cuda", generator=g)
    if points == "one cell":
        x = x * 0.01 + 0.3
    elif points == "clustered":
        x = (torch.rand(4, d, device="cuda", generator=g)[torch.randint(0, 4, (n,), device="cuda", generator=g)] * 0.8 + 0.1
             + 0.01 * torch.randn(n, d, device="cuda", generator=g)).clamp_(0, 1)  # fmt: skip
    elif points != "uniform":  # a cube of this width above the unit range, next to points inside it
        x = torch.where(torch.rand(n, 1, device="cuda", generator=g) < 0.8, 1.2 + points * x, x)
    geo = level_geometry(levels, cap, d, 16, max_res)
    table = torch.randn(geo.total_rows, feats, device="cuda", generator=g).to(dtype)
    go = torch.randn(n, levels * feats, device="cuda", generator=g).to(dtype)
    lib, code, stream = _lib.lib(), _lib.DTYPE_CODE[dtype], _lib.stream_ptr(x.device)
    args = (n, d, feats, levels, _lib.i32_array(geo.resolutions), _lib.i64_array(geo.rows), _lib.i64_array(geo.offsets),
            _lib.i64_array([PI_1, PI_2, PI_3][:d]))  # fmt: skip
    out, out_o = torch.empty_like(go), torch.empty_like(go)
    de, de_o = torch.zeros_like(table), torch.zeros_like(table)
    _lib.check(lib.th_hash_fwd(x.data_ptr(), d, 1, 0, table.data_ptr(), code, out.data_ptr(), levels * feats, *args, 1.0, 0, levels, stream), "fwd")
    _lib.check(lib.th_hash_bwd(x.data_ptr(), d, 1, 0, go.data_ptr(), levels * feats, de.data_ptr(), code, *args, 1.0, 0, levels, stream), "bwd")
    order = torch.empty(n, 4, device="cuda")
    scratch = torch.empty(lib.th_hash_order_scratch_bytes(n, d), dtype=torch.uint8, device="cuda")
    _lib.check(lib.th_hash_order(x.data_ptr(), d, 1, 0, n, d, 1.0, order.data_ptr(), scratch.data_ptr(), scratch.numel(), stream), "order")
    rows = order[:, 3].view(torch.int32).long()
    assert torch.equal(rows.sort().values, torch.arange(n, device="cuda")), "every point once"
    assert torch.equal(order[:, :d], x[rows])
    if keep_order:
        go = go[rows].contiguous()
    _lib.check(lib.th_hash_fwd_ordered(order.data_ptr(), keep_order, table.data_ptr(), code, out_o.data_ptr(), levels * feats, *args, 0, levels, stream), "fwd")
    _lib.check(lib.th_hash_bwd_ordered(order.data_ptr(), keep_order, go.data_ptr(), levels * feats, de_o.data_ptr(), code, *args, 0, levels, stream), "bwd")
    assert torch.equal(out_o, out[rows] if keep_order else out), "forward: the same arithmetic per point"
    return de, de_o


def same_rows(de, de_o):
    r"""Entries that are zero on one side only are sums that cancel to a rounding error in another order."""
    apart = (de != 0) != (de_o != 0)
    return not apart.any() or float((de - de_o)[apart].abs().max()) <= 1e-6 * float(de.abs().max())


@pytest.mark.parametrize("points", ["uniform", "clustered", "one cell"])
@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 20001])
def test_ordered_matches_unordered(n, points):
    # one point, the edges of a tile of 1024, several tiles; cells of one point and cells of a whole tile
    de, de_o = ordered_and_unordered(n, 3, 2, torch.float32, 2**14, 512, points, keep_order=0)
    assert float((de - de_o).abs().max() / de.abs().max()) <= 2e-5
    assert same_rows(de, de_o)


@pytest.mark.parametrize("d,feats,dtype", [(1, 1, torch.float32), (2, 2, torch.float16), (2, 8, torch.float32), (3, 4, torch.float32),
                                           (3, 1, torch.float16), (3, 8, torch.bfloat16), (3, 2, torch.bfloat16)])  # fmt: skip
@pytest.mark.parametrize("keep_order", [0, 1])
def test_ordered_shapes(d, feats, dtype, keep_order):
    de, de_o = ordered_and_unordered(5000, d, feats, dtype, 2**12, 2048, "uniform", keep_order, levels=8)
    tol = {torch.float32: 2e-5, torch.float16: 2e-2, torch.bfloat16: 1e-1}[dtype]
    assert float((de.float() - de_o.float()).abs().max() / de.float().abs().max()) <= tol


def test_several_passes_over_a_large_table():
    # 16 levels of up to 16 MB: more than one pass of levels, each of them sorting some tiles
    de, de_o = ordered_and_unordered(2**17 + 77, 3, 4, torch.float32, 2**20, 4096, "clustered", keep_order=0)
    assert float((de - de_o).abs().max() / de.abs().max()) <= 2e-5
    assert same_rows(de, de_o)


@pytest.mark.parametrize("d,max_res,width", [(3, 1000, 0.005), (2, 60000, 2.5e-4)])
def test_cells_above_the_unit_range_keep_their_rows(d, max_res, width):
    # many points per cell, on grids whose cells fit the packed key only inside the unit range
    de, de_o = ordered_and_unordered(6000, d, 2, torch.float32, 2**14, max_res, width, keep_order=0)
    assert float((de - de_o).abs().max() / de.abs().max()) <= 2e-5
    assert same_rows(de, de_o)
