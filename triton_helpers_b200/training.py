r"""Neural-field training step: hash encoding -> fused MLP -> MSE -> backward -> gradient sum -> Adam.

The step benchmark configuration 3 describes, built only from this package's operators.  It
has no counterpart in triton_helpers (which stops at the two layers); the layers it drives are
the drop-in ``HashEncoding`` and ``FullyFusedMLP`` modules.

Two ways through the step:

* **direct** (table and MLP share one 16-bit dtype): the trainer calls the C ABI itself on buffers it
  keeps from step to step - ``th_hash_fwd``, ``th_mlp_fwd_mse``, ``th_mlp_bwd``, ``th_hash_bwd`` (their ordered forms for
  large batches) from one native call, or on request the fused pair ``th_field_fwd`` (encoding + MLP + loss) and
  ``th_field_bwd`` (MLP backward + encoding backward); then ``th_scale_cast`` and ``th_adam_steps``.  All gradients live in ONE flat 16-bit
  buffer ``[table gradient | MLP gradients]`` so that a step costs one all-reduce:

  - the table part holds ``grad_out_scale * sum over the local batch`` (the encoding backward adds
    into it with 16-bit reductions; Adam clears it in the pass that consumes it);
  - the MLP part holds the MEAN over the local batch of the unscaled gradient: the float32 sums
    ``th_mlp_bwd`` leaves in its workspace are divided by ``rows * grad_out_scale`` before they are
    rounded.  A sum over 2^21 rows reaches 1e4..1e5 and four ranks of that exceed float16's 65504;
    means stay below one at any batch size and world size.

* **float32 parameters**: on one rank the same sequence in one native call, the MLP on 16-bit copies of its
  parameters; otherwise forward and backward through the layers' autograd functions and
  ``parallel.allreduce_gradients`` on the float32 gradients.

With more than one process the point batch is split across ranks (every rank passes the same
number of points), parameters are replicated and their gradients summed once per step.
"""
import math
from typing import List, Optional, Tuple, Union

import torch
import torch.distributed as dist
import torch.nn as nn
from torch import Tensor

from . import _lib
from .layers.fully_fused_mlp import FullyFusedMLP
from .layers.fully_fused_mlp.kernel import _f32_operand_dtype
from .layers.hash_encoding import HashEncoding
from .layers.hash_encoding.helpers import level_geometry
from .layers.hash_encoding.kernel import _Launch
from .layers.neural_field.kernel import FieldUnsupported, field_backward, field_forward
from .optim import FusedAdam, adam_updates
from .parallel import PendingReduce, allreduce_gradients, gradient_scales, level_passes


@torch.no_grad()
def mse_grad(pred: Tensor, target: Tensor, grad_scale: float) -> Tuple[Tensor, Tensor]:
    r"""``(grad, loss_sum)``: ``grad = (pred - target) * grad_scale`` in ``pred``'s dtype and the
    float32 sum of squared differences (a one-element device tensor), in one kernel."""
    assert pred.shape == target.shape and pred.dtype == target.dtype, "Prediction / target mismatch"
    device = _lib.require_cuda(pred, target)
    pred, target = pred.contiguous(), target.contiguous()
    grad = torch.empty_like(pred)
    loss_sum = torch.zeros(1, dtype=torch.float32, device=device)
    with torch.cuda.device(device):
        _lib.check(
            _lib.lib().th_mse_grad(
                pred.data_ptr(), target.data_ptr(), grad.data_ptr(), loss_sum.data_ptr(), pred.numel(), grad_scale,
                _lib.dtype_code(pred), _lib.stream_ptr(device),
            ),
            "th_mse_grad",
        )  # fmt: skip
    return grad, loss_sum


def default_grad_out_scale(global_points: int) -> float:
    r"""Loss scale for 16-bit table gradients: the power of two nearest below ``2^18 / global_points``,
    kept within ``[2^-8, 1]``.  A row of the coarsest level collects a share of EVERY point of every
    rank, so its 16-bit sum grows with the global batch (measured on the float32 CPU port of
    configuration 3: max |row sum| = 260 per 2^19 points at unit scale); dividing the scale by the
    batch keeps that sum near 130 whatever the number of ranks, two orders of magnitude inside
    float16's range, while single contributions on the fine levels (1e-4 .. 1 at unit scale) stay
    representable."""
    scale = 2.0 ** math.floor(math.log2(max(2.0**18 / max(global_points, 1), 2.0**-8)))
    return min(scale, 1.0)


class NeuralFieldTrainer(nn.Module):
    r"""Hash-encoded MLP regressed on targets with MSE and Adam.

    Args:
        encoding, mlp: the two layers (moved to the device and dtype the caller wants; float16
            tables and weights for benchmark configuration 3).  In direct mode the MLP's parameters
            are re-pointed into one flat buffer (their values, names and shapes are unchanged).
        lr, betas, eps: Adam hyper-parameters.
        grad_out_scale: the MLP receives ``(pred - target) * grad_out_scale`` as its output
            gradient, i.e. the loss is scaled so 16-bit table gradients neither underflow nor
            overflow; Adam undoes the scale exactly.  ``None``: ``default_grad_out_scale`` of the
            global batch of the first step.
        group: process group for data parallelism (``None``: the default group, if initialised).
        fused: direct mode only; which steps run in the kernels that fuse the encoding with the MLP.
            ``None`` (default) or ``False``: none, the separate operators, over spatially ordered points where
            that pays (benchmark configuration 3 on a B200: 1.48 ms per step; with the fused backward 1.73 ms);
            ``"backward"``: the backward pass, raise if it is not covered; ``True``: forward and backward, raise
            if not covered.
        backward_passes: ``None`` (default): one encoding backward, then one gradient sum over the
            ranks.  An integer n (direct mode): the encoding backward runs in n level ranges, finest
            first; the gradient rows of a finished range are summed over the ranks (NCCL,
            asynchronously) while the kernels of the next range run, and the MLP gradients travel
            with the first range.  Measured on 2 and 8 B200 with the cfg 3 step it gains nothing -
            the sum of 24 MB over NVLink takes about as long as the second pass over the points
            costs extra - so it is left to the caller to switch on (slower interconnects, larger tables).
    """

    def __init__(
        self,
        encoding: HashEncoding,
        mlp: FullyFusedMLP,
        lr: float = 1e-2,
        betas: Tuple[float, float] = (0.9, 0.99),
        eps: float = 1e-15,
        grad_out_scale: Optional[float] = None,
        group: Optional[dist.ProcessGroup] = None,
        backward_passes: Optional[int] = None,
        fused: Union[None, bool, str] = None,
    ):
        super().__init__()
        self.fused = fused
        self._no_fused_forward = self._no_fused_backward = self._no_ordered = False
        self.encoding = encoding
        self.mlp = mlp
        self.grad_out_scale = grad_out_scale
        self.group = group
        self.backward_passes = backward_passes
        self.lr, self.betas, self.eps = lr, betas, eps
        table_dtype, mlp_dtype = encoding.embeddings.dtype, mlp.w_in.dtype
        sixteen = (torch.float16, torch.bfloat16)
        if table_dtype == mlp_dtype and table_dtype in sixteen:
            self.direct = True
        elif table_dtype in sixteen or mlp_dtype in sixteen:
            raise ValueError(
                "NeuralFieldTrainer takes a table and an MLP of one 16-bit dtype, or float32 for both "
                f"(got {table_dtype} and {mlp_dtype}): unnormalised 16-bit MLP gradients cannot be summed over ranks"
            )
        else:
            self.direct = False
        self.optimizer = None if self.direct else FusedAdam(self.parameters(), lr=lr, betas=betas, eps=eps)
        self._state = None  # direct mode: buffers, created on the first step
        self._steps = 0

    def world_size(self) -> int:
        return dist.get_world_size(self.group) if dist.is_available() and dist.is_initialized() else 1

    def forward(self, coords: Tensor) -> Tensor:
        r"""Prediction ``(N, d_out)`` for coordinates ``(N, D)``."""
        return self.mlp(self.encoding(coords).unsqueeze(0)).squeeze(0)

    def skipped_elements(self) -> int:
        r"""Parameter elements Adam has passed over so far because their gradient was not finite
        (reads the device: synchronises).  Zero in a healthy run."""
        if self.direct:
            return 0 if self._state is None else int(self._state.skipped.item())
        return self.optimizer.skipped_elements()

    def step(self, coords: Tensor, targets: Tensor) -> Tensor:
        r"""One optimisation step on this rank's points; returns the local mean squared error
        (float32, on the device, not synchronised)."""
        if self.grad_out_scale is None:
            self.grad_out_scale = default_grad_out_scale(coords.shape[0] * self.world_size())
        self._steps += 1
        return self._step_direct(coords, targets) if self.direct else self._step_autograd(coords, targets)

    # ---- autograd mode (float32 parameters) --------------------------------------------------------

    def _step_autograd(self, coords: Tensor, targets: Tensor) -> Tensor:
        world = self.world_size()
        loss = self._step_float32(coords, targets) if world == 1 else None
        if loss is not None:
            return loss
        pred = self.mlp(self.encoding(coords).unsqueeze(0)).squeeze(0)
        grad_out, loss_sum = mse_grad(pred, targets.to(pred.dtype), self.grad_out_scale)
        pred.backward(grad_out)
        allreduce_gradients([p.grad for p in self.parameters() if p.grad is not None], self.group)
        # d(mean over the global batch)/d pred = 2 (pred - target) / (N_global * C)
        self.optimizer.step(grad_scale=2.0 / (pred.numel() * world * self.grad_out_scale))
        for p in self.parameters():
            p.grad = None
        return loss_sum / pred.numel()

    def _step_float32(self, coords: Tensor, targets: Tensor) -> Optional[Tensor]:
        r"""The same step without an autograd graph: forward and backward in one native call on kept buffers, then the
        optimizer's step.  ``None`` where the graph has to be built: hooks of modules or parameters, anomaly detection,
        frozen parameters, subclasses of the layers, or a call the native path does not take."""
        enc, mlp = self.encoding, self.mlp
        if type(enc) is not HashEncoding or type(mlp) is not FullyFusedMLP or len(self.optimizer.param_groups) != 1 or coords.ndim != 2:
            return None
        if _hooked(enc) or _hooked(mlp) or nn.modules.module._has_any_global_hook() or torch.is_anomaly_enabled():
            return None
        params = [p for p in (enc.embeddings, mlp.w_in, mlp.b_in, mlp.w_hid, mlp.b_hid, mlp.w_out, mlp.b_out) if p is not None]
        if not all(p.requires_grad and p.grad is None and not p._backward_hooks and not p._post_accumulate_grad_hooks for p in params):
            return None
        held = {id(p) for p in self.optimizer.param_groups[0]["params"]}
        if any(id(p) not in held for p in params) or not _float32_native(enc, mlp, coords):
            return None
        layout = _Float32State.layout(enc, mlp)
        st = self._state
        if st is None or st.key != layout:
            st = self._state = _Float32State(enc, mlp)
        st.resize(coords.shape[0])
        scale = float(self.grad_out_scale)
        loss = _lib.native().train_gradients(
            coords, targets, enc.embeddings, st.table_grad, (mlp.w_in, mlp.b_in, mlp.w_hid, mlp.b_hid, mlp.w_out, mlp.b_out),
            st.sums, st.feats, st.grad_pred, st.grad_feats, None, enc.pi, enc.max_entries_per_level, enc.min_res, enc.max_res,
            enc.num_levels, mlp.activation, scale, 1.0,
        )  # fmt: skip
        if loss is NotImplemented:
            self._state = None
            return None
        grads = [st.table_grad] + [g.view_as(p) for p, g in zip(params[1:], st.mlp_grads)]
        # d(mean over the batch)/d pred = 2 (pred - target) / (N * C); Adam clears the table gradient as it consumes it
        adam_scale = 2.0 / (coords.shape[0] * st.d_out * scale)
        try:
            if self.optimizer.watched():  # by step hooks or a scheduler: the public step, on the parameters' grad
                for p, g in zip(params, grads):
                    p.grad = g
                self.optimizer.step(grad_scale=adam_scale, zero_grad=True)
                if enc.embeddings.grad is not st.table_grad:
                    st.table_grad.zero_()  # a hook put another gradient in its place
                for p in params:
                    p.grad = None
            else:
                zero = [True] + [False] * (len(params) - 1)
                self.optimizer.update(self.optimizer.param_groups[0], params, grads, [adam_scale] * len(params), zero)
        except BaseException:
            self._state = None  # its table gradient may not be zero
            raise
        return loss

    # ---- direct mode (one 16-bit dtype) ------------------------------------------------------------

    def _step_direct(self, coords: Tensor, targets: Tensor) -> Tensor:
        loss = self._step_native(coords, targets)
        if loss is not None:
            return loss
        st = self._prepare(coords)
        enc, mlp, lib = self.encoding, self.mlp, _lib.lib()
        device, dtype = st.device, st.dtype
        n, world, scale = coords.shape[0], self.world_size(), float(self.grad_out_scale)
        targets = targets.to(dtype)
        if targets.stride(-1) != 1:
            targets = targets.contiguous()
        d_coord = coords.shape[1]
        launch = _Launch(coords, st.primes, d_coord, enc.max_entries_per_level, enc.num_levels, enc.min_res, enc.max_res, 1.0)
        cast_scale, table_adam_scale, mlp_adam_scale = gradient_scales(n, world, st.d_out, scale)
        code, act = _lib.dtype_code(st.flat_grad), _lib.ACTIVATION_CODE[mlp.activation]
        mlp_ptrs = (st.w_in.data_ptr(), _lib.ptr(st.b_in), _lib.ptr(st.w_hid), _lib.ptr(st.b_hid), st.w_out.data_ptr(), _lib.ptr(st.b_out))
        dims = (st.d_feat, st.d_hidden, st.d_out, st.depth)
        fuse_fwd, fuse_bwd = self._fusion_plan(st)
        with torch.cuda.device(device):
            stream = _lib.stream_ptr(device)
            st.loss_sum.zero_()
            geometry = (launch.n, d_coord, st.n_feats, enc.num_levels, launch.res, launch.rows, launch.offsets, launch.primes, launch.scale)
            weights = (st.w_in, st.w_out, st.w_hid)
            # ---- forward: encoding, MLP, loss ----
            if fuse_fwd:
                try:
                    field_forward(launch, enc.embeddings.data, *weights, mlp.activation, enc.num_levels, feats_out=st.feats,
                                  target=targets, grad_out=st.grad_pred, loss_sum=st.loss_sum, grad_scale=scale,
                                  biases=(st.b_in, st.b_hid, st.b_out))  # fmt: skip
                except FieldUnsupported:
                    if self.fused is True:
                        raise
                    self._no_fused_forward = True  # nothing was launched: the separate operators from now on
                    fuse_fwd = False
            # ---- or, for large batches, in spatial order from the features to the table gradient ----
            # (the loss epilogue takes whole 16-byte chunks of targets and gradients: decided before anything is ordered)
            order = None
            if not (fuse_fwd or fuse_bwd or self.backward_passes or self._no_ordered or st.d_out % 8):
                order = launch.order(st.n_feats, st.n_feats * st.flat_grad.element_size(), True)
            if order is not None and (targets.stride(0) % 8 or targets.data_ptr() % 16):
                targets = targets.clone(memory_format=torch.contiguous_format)
            if order is not None:
                _lib.check(
                    lib.th_hash_fwd_ordered(order.data_ptr(), 1, enc.embeddings.data_ptr(), code, st.feats.data_ptr(), st.d_feat, *geometry[:-1],
                                            0, enc.num_levels, stream),
                    "th_hash_fwd_ordered",
                )  # fmt: skip
                rc = lib.th_mlp_fwd_mse_ordered(
                    st.feats.data_ptr(), st.d_feat, *mlp_ptrs, targets.data_ptr(), targets.stride(0), code, order.data_ptr(),
                    st.grad_pred.data_ptr(), st.d_out, st.loss_sum.data_ptr(), 1.0, scale, n, *dims, act, code, stream,
                )  # fmt: skip
                if rc == _lib.TH_ERR_UNSUPPORTED:
                    order, self._no_ordered = None, True  # a switch turned its kernel off: the unordered operators from now on
                else:
                    _lib.check(rc, "th_mlp_fwd_mse_ordered")
            if not fuse_fwd and order is None:
                _lib.check(
                    lib.th_hash_fwd(*launch.coord_args, enc.embeddings.data_ptr(), code, st.feats.data_ptr(), st.d_feat,
                                    *geometry, 0, enc.num_levels, stream),
                    "th_hash_fwd",
                )  # fmt: skip
                rc = lib.th_mlp_fwd_mse(
                    st.feats.data_ptr(), st.d_feat, *mlp_ptrs, None, st.d_out, targets.data_ptr(), targets.stride(0),
                    st.grad_pred.data_ptr(), st.d_out, st.loss_sum.data_ptr(), scale, n, *dims, act, code, stream,
                )  # fmt: skip
                if rc == _lib.TH_ERR_UNSUPPORTED:  # shapes the fused forward + loss does not take: the two kernels it stands for
                    _lib.check(lib.th_mlp_fwd(st.feats.data_ptr(), st.d_feat, *mlp_ptrs, st.pred.data_ptr(), st.d_out, n, *dims, act, code, 0, stream), "th_mlp_fwd")
                    t = targets.contiguous()
                    _lib.check(lib.th_mse_grad(st.pred.data_ptr(), t.data_ptr(), st.grad_pred.data_ptr(), st.loss_sum.data_ptr(), n * st.d_out, scale, code, stream), "th_mse_grad")
                else:
                    _lib.check(rc, "th_mlp_fwd_mse")
            # ---- backward: MLP, then the encoding's table gradient into the flat buffer ----
            if fuse_bwd:
                try:
                    field_backward(launch, st.feats, st.grad_pred, *weights, mlp.activation, enc.num_levels, st.table_grad, st.workspace)
                except FieldUnsupported:
                    if self.fused in (True, "backward"):
                        raise
                    self._no_fused_backward = True
                    fuse_bwd = False
            if not fuse_bwd:
                _lib.check(
                    lib.th_mlp_bwd(st.feats.data_ptr(), st.d_feat, *mlp_ptrs, st.grad_pred.data_ptr(), st.d_out, st.grad_feats.data_ptr(),
                                   st.d_feat, None, None, None, None, None, None, st.workspace.data_ptr(), st.workspace.numel() * 4,
                                   n, *dims, act, code, 0, stream),
                    "th_mlp_bwd",
                )  # fmt: skip
            # float32 sums over this rank's rows -> mean of the unscaled gradient, rounded into the flat buffer's tail
            _lib.check(lib.th_scale_cast(st.workspace.data_ptr(), st.mlp_grad.data_ptr(), st.mlp_grad.numel(), cast_scale, code, stream), "th_scale_cast")
            pending = PendingReduce(self.group, bucket_bytes=0)
            if fuse_bwd:
                pending.start([st.flat_grad])
            elif order is not None:
                _lib.check(
                    lib.th_hash_bwd_ordered(order.data_ptr(), 1, st.grad_feats.data_ptr(), st.d_feat, st.table_grad.data_ptr(), code,
                                            *geometry[:-1], 0, enc.num_levels, stream),
                    "th_hash_bwd_ordered",
                )  # fmt: skip
                pending.start([st.flat_grad])
            else:
                passes = [(0, enc.num_levels)] if not self.backward_passes else level_passes(launch.geo.rows, self.backward_passes)
                for i, (begin, end) in enumerate(passes):  # finest first
                    _lib.check(
                        lib.th_hash_bwd(*launch.coord_args, st.grad_feats.data_ptr(), st.d_feat, st.table_grad.data_ptr(), code,
                                        *geometry, begin, end, stream),
                        "th_hash_bwd",
                    )  # fmt: skip
                    first = launch.geo.offsets[begin] * st.n_feats
                    last = st.flat_grad.numel() if i == 0 else (launch.geo.offsets[end - 1] + launch.geo.rows[end - 1]) * st.n_feats
                    pending.start([st.flat_grad[first:last]])  # one collective per range; the first carries the MLP gradients
            pending.finish()
        self._adam_direct(st, table_adam_scale, mlp_adam_scale)
        return st.loss_sum / (n * st.d_out)

    def _adam_direct(self, st: "_DirectState", table_scale: float, mlp_scale: float) -> None:
        adam_updates(
            (self.encoding.embeddings.data.view(-1), st.mlp_flat), (st.table_grad_flat, st.mlp_grad), (st.table_m, st.mlp_m), (st.table_v, st.mlp_v),
            (table_scale, mlp_scale), (True, False), self._steps, self.lr, self.betas, self.eps, st.skipped,
        )  # fmt: skip

    def _step_native(self, coords: Tensor, targets: Tensor) -> Optional[Tensor]:
        r"""The direct step with its forward and backward in one native call; ``None`` where the Python sequence has to run
        (fused kernels or level passes asked for, calls the native path does not take)."""
        if self.fused not in (None, False) or self.backward_passes:
            return None
        st = self._prepare(coords)
        enc = self.encoding
        world, scale = self.world_size(), float(self.grad_out_scale)
        cast_scale, table_adam_scale, mlp_adam_scale = gradient_scales(coords.shape[0], world, st.d_out, scale)
        loss = _lib.native().train_gradients(
            coords, targets, enc.embeddings.data, st.table_grad, (st.w_in, st.b_in, st.w_hid, st.b_hid, st.w_out, st.b_out),
            st.workspace, st.feats, st.grad_pred, st.grad_feats, st.mlp_grad, enc.pi, enc.max_entries_per_level, enc.min_res, enc.max_res,
            enc.num_levels, self.mlp.activation, scale, cast_scale,
        )  # fmt: skip
        if loss is NotImplemented:
            return None
        if world > 1:
            pending = PendingReduce(self.group, bucket_bytes=0)
            pending.start([st.flat_grad])
            pending.finish()
        self._adam_direct(st, table_adam_scale, mlp_adam_scale)
        return loss

    def _fusion_plan(self, st: "_DirectState") -> Tuple[bool, bool]:
        r"""(fused forward?, fused backward?) for this step; see ``fused`` in the class docstring."""
        mode = self.fused
        if not mode:
            return False, False
        want_fwd = mode is True
        want_bwd = mode in (True, "backward")
        if st.b_in is not None or self.backward_passes:
            # the fused backward is built for bias-free networks; level-range passes need the separate encoding backward
            if mode in (True, "backward"):
                raise FieldUnsupported("the fused backward takes bias-free networks and one pass over all levels")
            want_bwd = False
        return want_fwd and not self._no_fused_forward, want_bwd and not self._no_fused_backward

    def _prepare(self, coords: Tensor) -> "_DirectState":
        st = self._state
        if st is None:
            st = self._state = _DirectState(self.encoding, self.mlp)
        assert coords.ndim == 2 and 1 <= coords.shape[1] <= 3, "coordinates must be (N, D) with D in 1..3"
        st.resize(coords.shape[0])
        return st


def _hooked(module: nn.Module) -> bool:
    return bool(module._forward_hooks or module._forward_pre_hooks or module._backward_hooks or module._backward_pre_hooks)


def _float32_native(enc: HashEncoding, mlp: FullyFusedMLP, coords: Tensor) -> bool:
    r"""What the native float32 step declines for good, before buffers are made for it: shapes it has no kernels for, batches that
    are better ordered in space (the layers' own functions do that), modes in which the native path stands back."""
    n, d = coords.shape
    feats, hidden, d_out = enc.embeddings.shape[1], mlp.w_in.shape[0], mlp.w_out.shape[0]
    depth = 1 if mlp.w_hid is None else mlp.w_hid.shape[0] // hidden + 1
    if not coords.is_cuda or n < 1 or d not in (2, 3) or feats not in (2, 4) or hidden not in (16, 32, 64) or depth >= 4:
        return False
    if d_out > 64 or d_out % 8 or enc.num_levels * feats > 64 or torch.is_autocast_enabled("cuda") or _lib.timing():
        return False
    if n < 2**17:  # no batch below is ordered, whatever its form
        return True
    rows = level_geometry(enc.num_levels, enc.max_entries_per_level, d, enc.min_res, enc.max_res).total_rows
    return not _lib.lib().th_hash_order_pays(n, d, feats, enc.num_levels, 4 * feats, rows, 1)


class _Float32State:
    r"""Buffers the float32 step keeps: the table's gradient (zero between steps), the float32 sums of the MLP's gradients,
    16-bit rows."""

    @staticmethod
    def layout(enc: HashEncoding, mlp: FullyFusedMLP) -> tuple:
        r"""What the buffers depend on."""
        table, hidden = enc.embeddings, mlp.w_hid
        return table.device, table.dtype, table.shape, mlp.w_in.shape, None if hidden is None else hidden.shape, mlp.w_out.shape, mlp.b_in is None

    def __init__(self, enc: HashEncoding, mlp: FullyFusedMLP):
        self.key = self.layout(enc, mlp)
        table = enc.embeddings
        self.device = table.device
        self.d_hidden, self.d_feat = mlp.w_in.shape
        self.d_out = mlp.w_out.shape[0]
        depth = 1 if mlp.w_hid is None else mlp.w_hid.shape[0] // self.d_hidden + 1
        self.table_grad = torch.zeros_like(table)
        self.sums = torch.zeros(_lib.lib().th_mlp_workspace_bytes(self.d_feat, self.d_hidden, self.d_out, depth) // 4, device=self.device)
        # slices of the sums in the order w_in, b_in, w_hid, b_hid, w_out, b_out of the parameters that exist
        h, offset, place = self.d_hidden, 0, {}
        sizes = (("w_in", h * self.d_feat), ("w_hid", (depth - 1) * h * h), ("w_out", self.d_out * h), ("b_in", h), ("b_hid", (depth - 1) * h), ("b_out", self.d_out))
        for name, size in sizes:
            place[name] = self.sums[offset : offset + size]
            offset += size
        self.mlp_grads = [place[name] for name in ("w_in", "b_in", "w_hid", "b_hid", "w_out", "b_out") if getattr(mlp, name) is not None]
        self.rows = -1

    def resize(self, n: int) -> None:
        if n == self.rows:
            return
        kw = dict(dtype=_f32_operand_dtype(), device=self.device)
        self.feats = torch.empty(n, self.d_feat, **kw)
        self.grad_feats = torch.empty(n, self.d_feat, **kw)
        self.grad_pred = torch.empty(n, self.d_out, **kw)
        self.rows = n


class _DirectState:
    r"""Buffers the direct step keeps: the flat gradient, Adam moments, the MLP's flat parameter
    buffer, per-batch intermediates."""

    def __init__(self, enc: HashEncoding, mlp: FullyFusedMLP):
        table = enc.embeddings
        self.device, self.dtype = table.device, table.dtype
        _lib.require_cuda(table, mlp.w_in)
        assert table.is_contiguous(), "the embedding table must be contiguous"
        self.n_feats = table.shape[1]
        self.primes = enc.pi
        self.d_hidden, self.d_feat = mlp.w_in.shape
        self.d_out = mlp.w_out.shape[0]
        self.depth = 1 if mlp.w_hid is None else mlp.w_hid.shape[0] // self.d_hidden + 1
        assert self.d_feat == enc.num_levels * self.n_feats, "the MLP's input width must be levels * features"

        # MLP parameters in one flat buffer, in the order of th_mlp_bwd's workspace
        has_bias = mlp.b_in is not None
        ordered: List[Tuple[str, Optional[nn.Parameter]]] = [("w_in", mlp.w_in), ("w_hid", mlp.w_hid), ("w_out", mlp.w_out)]
        if has_bias:
            ordered += [("b_in", mlp.b_in), ("b_hid", mlp.b_hid), ("b_out", mlp.b_out)]
        total = _lib.lib().th_mlp_workspace_bytes(self.d_feat, self.d_hidden, self.d_out, self.depth) // 4
        self.mlp_flat = torch.zeros(total, dtype=self.dtype, device=self.device)
        table_elems = table.numel()
        tail = (table_elems + 15) // 16 * 16  # 32-byte aligned start of the MLP part
        self.flat_grad = torch.zeros(tail + total, dtype=self.dtype, device=self.device)
        self.table_grad_flat = self.flat_grad[:table_elems]
        self.table_grad = self.table_grad_flat.view_as(table)
        self.mlp_grad = self.flat_grad[tail:]
        offset = 0
        for name, p in ordered:
            setattr(self, name, None)
            if p is None:
                continue
            view = self.mlp_flat[offset : offset + p.numel()].view_as(p)
            view.copy_(p.data)
            p.data = view
            p.grad = self.mlp_grad[offset : offset + p.numel()].view_as(p)
            setattr(self, name, view)
            offset += p.numel()
        if not has_bias:
            self.b_in = self.b_hid = self.b_out = None
        table.grad = self.table_grad
        f32 = dict(dtype=torch.float32, device=self.device)
        self.table_m, self.table_v = torch.zeros(table_elems, **f32), torch.zeros(table_elems, **f32)
        self.mlp_m, self.mlp_v = torch.zeros(total, **f32), torch.zeros(total, **f32)
        self.workspace = torch.zeros(total, **f32)
        self.loss_sum = torch.zeros(1, **f32)
        self.skipped = torch.zeros(1, dtype=torch.int32, device=self.device)
        self.rows = -1

    def resize(self, n: int) -> None:
        if n == self.rows:
            return
        kw = dict(dtype=self.dtype, device=self.device)
        self.feats = torch.empty(n, self.d_feat, **kw)
        self.grad_feats = torch.empty(n, self.d_feat, **kw)
        self.grad_pred = torch.empty(n, self.d_out, **kw)
        self.pred = torch.empty(n, self.d_out, **kw)
        self.rows = n
