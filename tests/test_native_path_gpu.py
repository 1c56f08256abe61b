r"""The operators' native host path (``_native``) against their Python autograd functions: same outputs, same
gradients, same errors, and the calls it leaves to Python."""
import warnings

import pytest
import torch
import torch.autograd.forward_ad as forward_ad

from triton_helpers_b200 import _lib
from triton_helpers_b200.layers.fully_fused_mlp import FullyFusedMLP, fully_fused_mlp
from triton_helpers_b200.layers.hash_encoding import HashEncoding, hash_encoding
from triton_helpers_b200.layers.hash_encoding.helpers import level_geometry
from triton_helpers_b200.layers.neural_field import hash_encoded_mlp
from triton_helpers_b200.layers.neural_field.kernel import FieldUnsupported
from triton_helpers_b200.layers.reversible_mlp import ReversibleMLP
from triton_helpers_b200.training import NeuralFieldTrainer

pytestmark = pytest.mark.gpu


def both(call, leaves):
    r"""``call``'s output and the gradients of ``leaves``: native, then Python."""
    results = []
    for deferred in (False, True):
        _lib.native().defer(deferred)
        try:
            y = call()
            assert "Backward" in y.grad_fn.name() and isinstance(y.grad_fn, torch.autograd.function.BackwardCFunction) == deferred
            g = torch.Generator(device="cuda").manual_seed(5)
            go = torch.randn(y.shape, device="cuda", generator=g).to(y.dtype)
            results.append((y.detach(), *torch.autograd.grad(y, leaves, go)))
        finally:
            _lib.native().defer(False)
    return results


def close(native, python, rel):
    for a, b in zip(native, python):
        assert a.shape == b.shape and a.dtype == b.dtype
        assert float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30)) <= rel


@pytest.mark.parametrize("shape,dtype", [((1, 3), torch.float32), ((257, 2), torch.float16), ((5, 40, 3), torch.float32)])
@pytest.mark.parametrize("own_primes", [False, True])
def test_hash_encoding(shape, dtype, own_primes):
    layer = HashEncoding(2**12, 8, shape[-1], 2, 16, 128).cuda().to(dtype)
    layer.pi = layer.pi.long()
    x = torch.rand(*shape, device="cuda")
    pi = torch.tensor([1, 7919, 104729], device="cuda") if own_primes else None
    call = lambda: hash_encoding(x, layer.embeddings, None, pi, 2**12, 16, 128, 8)  # noqa: E731
    native, python = both(call, [layer.embeddings])
    assert torch.equal(native[0], python[0])
    close(native, python, 1e-5 if dtype == torch.float32 else 5e-3)


@pytest.mark.parametrize("rows,bias,depth,activation,dtype", [(1, True, 1, "relu", torch.float16), (300, True, 3, "silu", torch.bfloat16),
                                                              (129, False, 2, "none", torch.float16), (1, True, 1, "relu", torch.float32),
                                                              (300, True, 3, "silu", torch.float32)])  # fmt: skip
def test_fused_mlp(rows, bias, depth, activation, dtype):
    layer = FullyFusedMLP(16, 32, 8, depth, activation, bias=bias).cuda().to(dtype)
    x = torch.randn(1, rows, 16, device="cuda").to(dtype).requires_grad_(True)
    native, python = both(lambda: layer(x), [x, *layer.parameters()])
    assert torch.equal(native[0], python[0])
    close(native, python, 2e-3 if dtype == torch.float16 else 1e-2)


@pytest.mark.parametrize("rows,bias", [(1, False), (333, True)])
def test_reversible_mlp(rows, bias):
    layer = ReversibleMLP(64, 3, 32, bias=bias).cuda().half()
    x = torch.randn(rows, 64, device="cuda").half().requires_grad_(True)
    native, python = both(lambda: layer(x), [x, *layer.parameters()])
    assert torch.equal(native[0], python[0])
    close(native, python, 2e-3)


@pytest.mark.parametrize("rows,depth", [(1, 1), (1000, 2)])
def test_hash_encoded_mlp(rows, depth):
    table = (torch.randn(level_geometry(16, 2**12, 3, 16, 128).total_rows, 2, device="cuda") * 0.1).half().requires_grad_(True)
    mlp = FullyFusedMLP(32, 64, 16, depth, bias=False).cuda().half()
    x = torch.rand(rows, 3, device="cuda")
    leaves = [table, mlp.w_in, mlp.w_out] + ([mlp.w_hid] if depth > 1 else [])
    native, python = both(lambda: hash_encoded_mlp(x, table, mlp.w_in, mlp.w_out, mlp.w_hid, None, 2**12, 16, 128, 16), leaves)
    assert torch.equal(native[0], python[0])
    close(native, python, 1e-2)


def test_what_the_native_path_leaves_to_python():
    layer = FullyFusedMLP(16, 32, 8, 2).cuda().half()
    x = torch.randn(1, 64, 16, device="cuda").half()
    args = (layer.w_in, layer.b_in, layer.w_out, layer.b_out, layer.w_hid, layer.b_hid, "relu")
    fast = _lib.native().fully_fused_mlp
    assert fast(x, *args) is not NotImplemented
    with torch.autocast("cuda"):
        assert fast(x, *args) is NotImplemented
    with _lib.KernelTimer() as timer:
        assert fast(x, *args) is NotImplemented
        layer(x)
    assert timer.summary()["th_mlp_fwd"][0] == 1 and fast(x, *args) is not NotImplemented
    assert fast(x.cpu(), *args) is NotImplemented and fast(x[..., ::2], *args) is NotImplemented
    with pytest.raises(AssertionError, match="Input dimension mismatch"):
        layer(x[..., :8])
    # a graph is gone after one backward pass, and a parameter changed in between is noticed
    y = layer(x)
    y.sum().backward()
    with pytest.raises(RuntimeError, match="second time"):
        y.sum().backward()
    y = layer(x)
    with torch.no_grad():
        layer.w_in.add_(1)
    with pytest.raises(RuntimeError, match="inplace operation"):
        y.sum().backward()
    # frozen input, one live parameter: only its gradient arrives
    for p in layer.parameters():
        p.requires_grad_(False)
        p.grad = None
    layer.w_out.requires_grad_(True)
    y = fully_fused_mlp(x, *args)
    y.sum().backward()
    assert layer.w_out.grad is not None and all(p.grad is None for p in layer.parameters() if p is not layer.w_out)


def operator(name):
    r"""A call of one tensor, that tensor, and a parameter the call differentiates."""
    torch.manual_seed(0)
    if name == "encoding":
        layer = HashEncoding(2**12, 8, 3, 2, 16, 128).cuda()
        return layer, torch.rand(40, 3, device="cuda"), layer.embeddings
    if name in ("mlp", "mlp float32"):
        layer = FullyFusedMLP(16, 32, 8, 2).cuda()
        layer = layer if name == "mlp float32" else layer.half()
        return layer, torch.randn(1, 40, 16, device="cuda").to(layer.w_in.dtype), layer.w_in
    if name == "reversible":
        layer = ReversibleMLP(64, 2, 32).cuda().half()
        return layer, torch.randn(40, 64, device="cuda").half(), layer.w_f1
    table = (torch.randn(level_geometry(16, 2**12, 3, 16, 128).total_rows, 2, device="cuda") * 0.1).half()
    mlp = FullyFusedMLP(32, 64, 16, 2, bias=False).cuda().half()
    call = lambda x: hash_encoded_mlp(x, table, mlp.w_in, mlp.w_out, mlp.w_hid, None, 2**12, 16, 128, 16)  # noqa: E731
    return call, torch.rand(40, 3, device="cuda"), mlp.w_in


OPERATORS = ["encoding", "mlp", "mlp float32", "reversible", "field"]


@pytest.mark.parametrize("name", OPERATORS)
def test_forward_mode_is_refused(name):
    call, x, _ = operator(name)
    with forward_ad.dual_level(), pytest.raises(NotImplementedError, match="jvp"):
        call(forward_ad.make_dual(x, torch.ones_like(x)))


@pytest.mark.parametrize("name", OPERATORS[:4])  # the fifth closes over its tensors, which a trace cannot hold
def test_a_trace_follows_its_input(name):
    layer, x, _ = operator(name)
    with torch.no_grad():
        traced = torch.jit.trace(layer, x, check_trace=False)
        assert torch.equal(traced(x * 0.5), layer(x * 0.5))


def test_a_saved_tensor_hook_may_change_the_layout():
    # rows of a wider array come back from the host packed
    layer, _, leaf = operator("mlp")
    x = torch.randn(1, 40, 32, device="cuda").half()[..., :16]
    assert _lib.native().fully_fused_mlp(x, *(getattr(layer, n) for n in ("w_in", "b_in", "w_out", "b_out", "w_hid", "b_hid")), "relu") is not NotImplemented
    go = torch.randn(1, 40, 8, device="cuda").half()
    (want,) = torch.autograd.grad(layer(x), leaf, go)
    with torch.autograd.graph.save_on_cpu():
        y = layer(x)
    (got,) = torch.autograd.grad(y, leaf, go)
    assert torch.equal(got, want)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t[..., :8]):
        y = layer(x)
    with pytest.raises(RuntimeError, match="saved-tensor hook"):
        torch.autograd.grad(y, leaf, go)


@pytest.mark.parametrize("name,kept", zip(OPERATORS, [40 * 3 * 4, 40 * 16 * 2, None, 40 * 64 * 2, 40 * 32 * 2]))
def test_saved_tensors_go_through_their_hooks(name, kept):
    # the bytes of the rows an operator keeps (a float32 network: one buffer of all its 16-bit operands) reach the hook
    call, x, leaf = operator(name)
    kept = kept or sum((t.numel() + 15) // 16 * 16 * 2 for t in (x, *call.parameters()))
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.numel() * t.element_size()) or t.cpu(), lambda t: t.cuda()):
        y = call(x)
    assert kept in packed, packed
    go = torch.randn_like(y)
    (got,) = torch.autograd.grad(y, leaf, go)
    (want,) = torch.autograd.grad(call(x), leaf, go)
    assert float((got - want).norm() / want.norm()) <= 1e-2  # float16 sums in no fixed order


@pytest.mark.parametrize("deferred", [False, True])
def test_a_saved_order_goes_through_its_hooks(deferred):
    layer, x, packed = HashEncoding(2**12, 16, 3, 2, 16, 128).cuda(), torch.rand(2**21, 3, device="cuda"), []
    _lib.native().defer(deferred)
    try:
        with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.numel() * t.element_size()) or t, lambda t: t):
            layer(x)
    finally:
        _lib.native().defer(False)
    assert 16 * 2**21 in packed


def test_a_network_too_deep_for_the_fused_backward_says_so():
    table = (torch.randn(level_geometry(16, 2**12, 3, 16, 128).total_rows, 2, device="cuda") * 0.1).half().requires_grad_(True)
    mlp = FullyFusedMLP(32, 64, 16, 8, bias=False).cuda().half()
    y = hash_encoded_mlp(torch.rand(40, 3, device="cuda"), table, mlp.w_in, mlp.w_out, mlp.w_hid, None, 2**12, 16, 128, 16)
    with pytest.raises(FieldUnsupported):
        y.sum().backward()


def test_a_tensor_subclass_keeps_its_type():
    class Rows(torch.Tensor):
        pass

    layer, x, _ = operator("mlp")
    y = layer(x.as_subclass(Rows))
    assert type(y) is Rows and torch.equal(y.as_subclass(torch.Tensor), layer(x))


@pytest.mark.parametrize("n,dtype,bias,depth", [(1, torch.float16, False, 1), (1000, torch.bfloat16, True, 3), (2**20 + 3, torch.float16, False, 2),
                                                (1, torch.float32, True, 1), (5003, torch.float32, False, 3)])  # fmt: skip
def test_training_step(n, dtype, bias, depth, monkeypatch):
    # the last 16-bit case runs over spatially ordered points
    def train(deferred):
        torch.manual_seed(0)
        encoding, mlp = HashEncoding(2**12, 8, 3, 2, 16, 256), FullyFusedMLP(16, 32, 8, depth, bias=bias)
        with torch.no_grad():
            encoding.embeddings.mul_(0.1)
        trainer = NeuralFieldTrainer(encoding.cuda().to(dtype), mlp.cuda().to(dtype), lr=1e-3, fused=False)
        g = torch.Generator(device="cuda").manual_seed(3)
        x, t = torch.rand(n, 3, device="cuda", generator=g), torch.rand(n, 8, device="cuda", generator=g).to(dtype)
        answers, ask = [], _lib.native().train_gradients
        monkeypatch.setattr(_lib.native(), "train_gradients", lambda *args: answers.append(ask(*args)) or answers[-1])
        _lib.native().defer(deferred)
        try:
            losses = [float(trainer.step(x, t)) for _ in range(3)]
        finally:
            _lib.native().defer(False)
            monkeypatch.undo()
        assert len(answers) == 3 and all((a is NotImplemented) == deferred for a in answers), "the native step is taken, or not"
        assert trainer.skipped_elements() == 0
        return losses, [p.detach().double() for p in trainer.parameters()]

    (loss_n, params_n), (loss_p, params_p) = train(False), train(True)
    for a, b in zip(loss_n, loss_p):
        assert abs(a - b) <= 2e-3 * abs(b)
    for a, b in zip(params_n, params_p):  # Adam's first steps are lr * sign: entries whose gradient nearly cancels may differ
        assert float((a - b).norm() / b.norm()) <= 2e-3


def float32_trainer(d_out=8, feats=2, levels=8, d=3, depth=2, bias=True):
    torch.manual_seed(0)
    encoding, mlp = HashEncoding(2**12, levels, d, feats, 16, 256), FullyFusedMLP(levels * feats, 32, d_out, depth, bias=bias)
    with torch.no_grad():
        encoding.embeddings.mul_(0.1)
    return NeuralFieldTrainer(encoding.cuda(), mlp.cuda(), lr=1e-3)


def batch(n=1000, d=3, d_out=8):
    g = torch.Generator(device="cuda").manual_seed(1)
    return torch.rand(n, d, device="cuda", generator=g), torch.rand(n, d_out, device="cuda", generator=g)


@pytest.mark.parametrize("hook", ["post accumulate", "parameter", "module", "every module", "before the optimizer", "after the optimizer"])
def test_hooks_run_in_a_float32_step(hook):
    trainer, seen = float32_trainer(), []
    call = lambda *args, **kwargs: seen.append(1)  # noqa: E731
    register = {
        "post accumulate": trainer.mlp.w_in.register_post_accumulate_grad_hook,
        "parameter": trainer.mlp.w_in.register_hook,
        "module": trainer.mlp.register_forward_hook,
        "every module": torch.nn.modules.module.register_module_forward_hook,
        "before the optimizer": trainer.optimizer.register_step_pre_hook,
        "after the optimizer": trainer.optimizer.register_step_post_hook,
    }[hook]
    handle = register(call)
    try:
        trainer.step(*batch())
    finally:
        handle.remove()
    assert seen


def test_a_scheduler_sees_the_float32_steps():
    trainer = float32_trainer()
    scheduler = torch.optim.lr_scheduler.StepLR(trainer.optimizer, 1)
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        trainer.step(*batch())
        scheduler.step()


def test_a_gradient_replaced_by_a_hook_leaves_nothing_behind():
    # the table's gradient is dropped before one step: the next one starts from zero
    def run(drop):
        trainer = float32_trainer()
        table = trainer.encoding.embeddings
        handle = trainer.optimizer.register_step_pre_hook(lambda *args, **kwargs: setattr(table, "grad", None)) if drop else None
        before = table.detach().clone()
        trainer.step(*batch())
        if drop:
            handle.remove()
            assert torch.equal(table, before)
            return float(trainer._state.table_grad.abs().max())
        return float((table - before).abs().max())

    assert run(drop=True) == 0 and run(drop=False) > 0


def test_anomaly_detection_sees_a_float32_step():
    x, target = batch()
    target[0] = float("nan")
    with pytest.raises(RuntimeError, match="nan"), torch.autograd.detect_anomaly(check_nan=True):
        float32_trainer().step(x, target)


@pytest.mark.parametrize("kw", [dict(d=1), dict(feats=1, levels=16), dict(d_out=3)])
def test_a_float32_step_keeps_buffers_only_where_it_uses_them(kw):
    trainer = float32_trainer(**kw)
    trainer.step(*batch(d=kw.get("d", 3), d_out=kw.get("d_out", 8)))
    assert trainer._state is None


def test_a_replaced_network_is_not_trained_by_the_old_optimizer():
    # as through the graph: the optimizer holds the first network's parameters
    trainer, other = float32_trainer(depth=1, bias=False), FullyFusedMLP(16, 32, 8, 1).cuda()
    trainer.step(*batch())
    before = [p.detach().clone() for p in other.parameters()]
    trainer.mlp = other
    trainer.step(*batch())
    assert all(torch.equal(a, b) for a, b in zip(before, other.parameters()))
    # a network of another layout under a new optimizer gets buffers of its own
    trainer.optimizer = type(trainer.optimizer)(trainer.parameters(), lr=1e-3)
    trainer.step(*batch())
    assert not any(torch.equal(a, b) for a, b in zip(before, other.parameters()))


@pytest.mark.parametrize("n,d,hidden,depth,fused", [(2**19 + 3, 2, 32, 1, True), (2**18 + 3, 3, 16, 2, True), (2**19 - 1, 2, 32, 1, False), (2**18 + 3, 3, 32, 2, False)])
def test_sixty_four_features_and_a_small_network(n, d, hidden, depth, fused):
    # forward + backward in the fused kernels from this size on; same gradients as the two layers
    table = (torch.randn(level_geometry(16, 2**12, d, 16, 128).total_rows, 4, device="cuda") * 0.1).half().requires_grad_(True)
    mlp = FullyFusedMLP(64, hidden, 8, depth, bias=False).cuda().half()
    x, go = torch.rand(n, d, device="cuda"), torch.randn(n, 8, device="cuda").half() * 1e-3
    leaves = [table, mlp.w_in, mlp.w_out]
    y = hash_encoded_mlp(x, table, mlp.w_in, mlp.w_out, mlp.w_hid, None, 2**12, 16, 128, 16)
    assert isinstance(y.grad_fn, torch.autograd.function.BackwardCFunction) == fused
    got = [y.detach(), *torch.autograd.grad(y, leaves, go)]
    z = mlp(hash_encoding(x, table, None, None, 2**12, 16, 128, 16).unsqueeze(0)).squeeze(0)
    close(got, [z.detach(), *torch.autograd.grad(z, leaves, go)], 1e-2)
