"""Tensor-core scoring for every model whose score is ``compose(h, r) · t`` (+ a per-query scalar), or a distance.

:mod:`fused_step` covers the models whose composition is one of the algebra products the lookup kernel knows.  The
rest of the bilinear zoo produces its query vector with ordinary PyTorch modules: the convolutional gates of ConEx /
AConEx / ConvQ / AConvQ / ConvO / AConvO, DualE's dual-quaternion product, and any covered model once input dropout
or a normaliser sits between the embedding and the product.  For those the step is split:

* **autograd side** (PyTorch): gather ``E[h]``, ``R[r]``, dropout / normalisers / gates / product → ``Q [B, d]``;
* **kernel side** (:class:`FusedScoring`, one ``autograd.Function``): ``Q`` is scored against the whole entity table
  by the two tcgen05 launches of :func:`~dice_embeddings_b200.ops.kernels.kvsall_fused` — loss and dense ``dE`` with
  the table stationary, ``dQ`` with the queries stationary — with labels from the resident CSR as bit masks; nothing of
  size ``B × |E|`` exists.  ``backward`` hands ``dQ`` to autograd, which carries it through the gates to every other
  parameter;
* the entity table itself never meets autograd: the gathered head rows are a leaf whose gradient is scatter-added into
  the dense ``dE`` the kernel produced, and the table is updated by the fused optimiser kernel (bf16 shadow refreshed
  in the same sweep).  All other parameters are stepped by the model's own optimiser.

Two epilogue variants of the scoring kernel widen the contract.  Models whose score adds a scalar that depends on the
query only — the general Clifford models Keci / CKeci (p, q) and DeCaL (p, q, r), whose σ_pp / σ_qq / σ_pq / … terms
are summed into one number per (h, r) (``dicee/models/clifford.py:258-305``, ``:601-790``) — pass it as a per-query bias
(a column bias in the launch that keeps the table stationary, a row bias in the other, which also returns its
gradient).  TransE (``dicee/models/real.py:52-76``) uses the distance epilogue: ``margin − sqrt(‖q‖² + ‖e‖² − 2 q·e)``
from the same dot products, with the squared norms as per-row scalars; the kernel's second GEMM then yields
``Σ w e`` with ``w = dS / distance`` together with ``Σ w``, and the gradient is ``Σ w e − (Σ w) q``.

The reference runs these models as ``conv2d`` / ``Linear`` / four to eight ``torch.mm`` against the table plus
``BCEWithLogitsLoss`` on dense labels (``dicee/models/complex.py:33-62``, ``dicee/models/quaternion.py:242-319``,
``dicee/models/octonion.py:206-313``, ``dicee/models/dualE.py:102-127``, ``dicee/models/base_model.py:25-46``).
"""
from __future__ import annotations

import logging
import os
import types
from collections import OrderedDict
from typing import Optional

import torch

from . import kernels as K
from .fused_step import SUPPORTED_DIMS, SUPPORTED_SCORING, _EngineOptimizer, fused_model_code


#: attribute types of a module that its forward may read and a captured step therefore has fixed (momentum, eps, probabilities,
#: modes, replaced functions ...)
_PLAIN = frozenset((bool, int, float, str, tuple, type(None), torch.dtype, types.FunctionType, types.BuiltinFunctionType,
                    types.MethodType))


def hybrid_supported(model) -> bool:
    """Bilinear contract (with or without a per-query bias) or TransE's distance, a width the scoring kernel takes,
    ordinary index inputs."""
    if getattr(model, "byte_pair_encoding", False):
        return False
    if model.embedding_dim not in SUPPORTED_DIMS or model.optimizer_name not in K.OPT_CODE:
        return False
    if type(model).__name__ == "TransE":
        return True
    return bool(getattr(model, "bilinear", False)) and hasattr(model, "compose")


class FusedScoring(torch.autograd.Function):
    """``loss = mean BCE-with-logits(logits(Q, E), labels)`` with the gradient w.r.t. ``Q`` (and the per-query bias)
    computed in the same call.  ``mode`` 0: ``Q Eᵀ``; 1: ``Q Eᵀ + bias[:, None]``; 2: ``margin − cdist(Q, E)``."""

    @staticmethod
    def forward(ctx, q: torch.Tensor, bias: Optional[torch.Tensor], engine: "ExternalQueryEngine", dp: torch.Tensor,
                mode: int):
        n = q.shape[0]
        b = engine._buffers(n)
        scale = 1.0 / (float(n) * float(engine.NE))
        b.Q.copy_(q.detach())                                  # fp32 -> bf16 operand
        b.dQ.zero_()
        engine.loss_acc.zero_()
        b.mask_q.zero_()
        b.mask_e.zero_()
        K.build_label_masks(dp, engine.offsets, engine.values, n, 1, 0, b.mask_q, b.mask_e,
                            num_data_points=engine.num_data_points, num_local_rows=engine.NE, status=engine.status)
        common = dict(pos_delta=engine.pos_weight, score_mode=mode, margin=engine.margin)
        if mode == 0:
            e_kw, q_kw = {}, {}
        elif mode == 1:
            b.q_scalar[:n].copy_(bias.detach())
            b.q_sum.zero_()
            e_kw = dict(y_bias=b.q_scalar)
            q_kw = dict(x_bias=b.q_scalar, x_dsum=b.q_sum)
        else:
            # squared norms of the operands as the tensor cores see them (bf16-rounded)
            torch.sum(b.Q.float() ** 2, dim=1, out=b.q_scalar[:n])
            torch.sum(engine.E_bf16.float() ** 2, dim=1, out=engine.e_scalar[:engine.NE])
            b.q_sum.zero_()
            engine.e_sum.zero_()
            e_kw = dict(x_bias=engine.e_scalar, y_bias=b.q_scalar, x_dsum=engine.e_sum)
            q_kw = dict(x_bias=b.q_scalar, y_bias=engine.e_scalar, x_dsum=b.q_sum)
        K.kvsall_fused(engine.E_bf16, b.Q, engine.gE, engine.loss_acc, engine.status, engine.base, scale, True,
                       mask=b.mask_e, **common, **e_kw)
        K.kvsall_fused(b.Q, engine.E_bf16, b.dQ, None, engine.status, engine.base, scale, False,
                       mask=b.mask_q, **common, **q_kw)
        if mode == 2:
            # d logit / d x = (y − x) / distance: the kernels returned Σ w y and Σ w
            engine.gE.addcmul_(engine.e_sum[:, None], engine.E, value=-1.0)
            b.dQ.addcmul_(b.q_sum[:, None], q.detach(), value=-1.0)
        ctx.dq, ctx.dbias = b.dQ, (b.q_sum if mode == 1 else None)
        return (engine.loss_acc * scale).to(torch.float32).reshape(())

    @staticmethod
    def backward(ctx, grad_out):
        return grad_out * ctx.dq, (None if ctx.dbias is None else grad_out * ctx.dbias), None, None, None


class ExternalQueryEngine:
    #: captured steps kept (one per batch size as a rule); the least recently used one makes room for another
    MAX_GRAPHS = 4
    #: plain steps of a kind before it takes the place of another: a capture takes 2 to 13 ms, a replay saves 0.35 to 1.2 ms
    STEPS_BEFORE_REPLACING = 16
    #: kinds of steps whose number is remembered
    MAX_KINDS = 64

    def __init__(self, model, dataset, batch_size: int, lr: float, weight_decay: float = 0.0, device=None,
                 use_graph: bool = True):
        assert hybrid_supported(model)
        self.model = model
        self.device = dev = torch.device(device or model.device)
        self.D, self.NE = model.embedding_dim, model.num_entities
        self.lr, self.weight_decay = float(lr), float(weight_decay)
        self.opt_kind = K.OPT_CODE[model.optimizer_name]
        self.betas = (0.9, 0.9999) if self.opt_kind == 3 else (0.9, 0.999)
        self.eps = 1e-6 if self.opt_kind == 3 else 1e-8
        self.E = model.entity_embeddings.weight.data
        assert self.E.is_cuda and self.E.is_contiguous() and self.E.dtype == torch.float32
        self.E_bf16 = torch.empty(self.NE, self.D, dtype=torch.bfloat16, device=dev)
        K.cast_bf16(self.E, self.E_bf16)
        self.gE = torch.zeros_like(self.E)
        self.mE, self.vE = torch.zeros_like(self.E), torch.zeros_like(self.E)
        self.step_count = torch.zeros(1, dtype=torch.int64, device=dev)
        self.loss_acc = torch.zeros(1, dtype=torch.float64, device=dev)
        self.status = torch.zeros(1, dtype=torch.int32, device=dev)
        # every parameter but the entity table belongs to the model's own optimiser
        model.entity_embeddings.weight.requires_grad_(False)
        rest = [p for p in model.parameters() if p.requires_grad]
        self.rest_optimizer = model.configure_optimizers(rest) if rest else None
        if self.rest_optimizer is not None:
            for g in self.rest_optimizer.param_groups:
                g["lr"] = self.lr
        # The step is about a hundred small launches: as plain launches the host needs twice as long as the GPU (ConEx,
        # batch 1024, d = 256: 1685 us against 890), so it is replayed from a CUDA graph.  Adam and AdamW keep their step
        # counters on the device for that.
        self.use_graph = use_graph and os.environ.get("DICE_B200_NO_GRAPH") != "1"
        if type(self.rest_optimizer) in (torch.optim.Adam, torch.optim.AdamW):
            for g in self.rest_optimizer.param_groups:
                g["capturable"], g["fused"], g["foreach"] = True, True, False
        elif self.rest_optimizer is not None and type(self.rest_optimizer) is not torch.optim.SGD:
            self.use_graph = False
        self._graphs = OrderedDict()
        self._seen = OrderedDict()      # kind of step: plain launches so far
        self.dataset = dataset
        dataset.sparse_labels = True
        if hasattr(dataset, "offsets"):
            self.offsets, self.values = dataset.offsets.to(dev).contiguous(), dataset.values.to(dev).contiguous()
            pos, base = dataset.label_constants()
        else:  # 1vsAll: one positive per data point
            pairs = dataset.train_data.to(dev)
            self.offsets = torch.arange(pairs.shape[0] + 1, dtype=torch.int64, device=dev)
            self.values = pairs[:, 2].contiguous()
            pos, base = 1.0, 0.0
        self.pos_weight, self.base = float(pos - base), float(base)
        self.distance = type(model).__name__ == "TransE"
        self.margin = float(getattr(model, "margin", 0.0)) if self.distance else 0.0
        if self.distance:
            self.e_scalar = torch.zeros(K.padded_rows(self.NE), device=dev)
            self.e_sum = torch.zeros(self.NE, device=dev)
        self.num_data_points = int(self.offsets.numel() - 1)
        self.label_mode = "mask"
        self._bufs = {}

    def _buffers(self, n: int):
        if n not in self._bufs:
            from types import SimpleNamespace
            dev = self.device
            b = SimpleNamespace()
            b.Q = torch.zeros(n, self.D, dtype=torch.bfloat16, device=dev)
            b.dQ = torch.zeros(n, self.D, dtype=torch.float32, device=dev)
            b.mask_q = torch.zeros(n, K.mask_stride(self.NE), dtype=torch.int32, device=dev)
            b.mask_e = torch.zeros(self.NE, K.mask_stride(n), dtype=torch.int32, device=dev)
            b.q_scalar = torch.zeros(K.padded_rows(n), device=dev)     # per-query bias or squared norm
            b.q_sum = torch.zeros(n, device=dev)
            b.x_in = torch.zeros(n, 2, dtype=torch.int64, device=dev)
            b.dp = torch.zeros(n, dtype=torch.int64, device=dev)
            self._bufs[n] = b
        return self._bufs[n]

    def step(self, batch) -> torch.Tensor:
        """``batch = (x [n, 2] int64, data-point ids [n] int64)`` on the device; returns the loss (device scalar)."""
        x, dp = batch[0], batch[1]
        key = self._graph_key(x)
        if key is None:
            return self._step(x, dp)
        entry = self._graphs.get(key)
        if entry is None:
            if self._seen.get(key, 0) < (1 if len(self._graphs) < self.MAX_GRAPHS else self.STEPS_BEFORE_REPLACING):
                loss = self._step(x, dp)   # the first step of a kind sets up libraries and the optimiser's state
                self._count(self._graph_key(x))
                return loss
            entry = self._capture(x.shape[0], key)
            if entry is None:
                return self._step(x, dp)
        self._graphs.move_to_end(key)
        graph, loss, grads = entry
        b = self._buffers(x.shape[0])
        K.stage((b.x_in, x[:, :2]), (b.dp, dp))
        graph.replay()
        for p, g in grads:
            p.grad = g
        return loss.clone()

    def _count(self, key) -> None:
        self._seen[key] = self._seen.pop(key, 0) + 1
        if len(self._seen) > self.MAX_KINDS:
            self._seen.popitem(last=False)

    def _graph_key(self, x):
        """Everything a captured step has fixed, or ``None`` where the step has to run as plain launches: hooks, autocast,
        anomaly mode and saved-tensor hooks act on the Python side of a step, which a replay does not run."""
        if not self.use_graph or not x.is_cuda or x.dim() != 2 or x.shape[1] < 2:
            return None
        if torch.cuda.is_current_stream_capturing() or torch.is_autocast_enabled("cuda") or torch.is_anomaly_enabled() \
                or not torch.is_grad_enabled() or torch.is_inference_mode_enabled() or torch._C._len_torch_dispatch_stack() \
                or torch._C._len_torch_function_stack() or torch._C._autograd._top_saved_tensors_default_hooks(True) is not None:
            return None
        from torch.nn.modules import module as nn_module
        if nn_module._global_forward_hooks or nn_module._global_forward_pre_hooks or nn_module._global_backward_hooks \
                or nn_module._global_backward_pre_hooks:
            return None
        # one walk over the modules (38 us for ConEx, against 59 for modules(), parameters() and buffers() one after the other)
        kinds, tensors, todo = [], [], [self.model]
        while todo:
            m = todo.pop()
            if m is None:
                continue
            if m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks:
                return None
            kinds.append(type(m))
            kinds += [kv for kv in m.__dict__.items() if type(kv[1]) in _PLAIN]
            for p in m._parameters.values():
                if p is not None:
                    if p._backward_hooks or p._post_accumulate_grad_hooks:
                        return None
                    tensors += (p.data_ptr(), p.requires_grad)
            tensors += [t.data_ptr() for t in m._buffers.values() if t is not None]
            todo += m._modules.values()
        opt = []
        if self.rest_optimizer is not None:
            o = self.rest_optimizer
            if o._optimizer_step_pre_hooks or o._optimizer_step_post_hooks:
                return None
            for g in o.param_groups:
                opt.append(tuple((k, repr(v)) for k, v in sorted(g.items()) if k != "params"))
                if any(isinstance(v, torch.Tensor) for k, v in g.items() if k != "params"):
                    return None
                opt += [t.data_ptr() for p in g["params"] for t in o.state.get(p, {}).values() if isinstance(t, torch.Tensor)]
        mm, cudnn = torch.backends.cuda.matmul, torch.backends.cudnn
        flags = (mm.allow_tf32, mm.allow_fp16_reduced_precision_reduction, mm.allow_bf16_reduced_precision_reduction, cudnn.enabled,
                 cudnn.benchmark, cudnn.allow_tf32, cudnn.deterministic, torch.are_deterministic_algorithms_enabled(),
                 torch.get_default_dtype())
        mine = (self.lr, self.weight_decay, self.betas, self.eps, self.opt_kind, self.margin, self.pos_weight, self.base)
        key = (x.shape[0], mine, tuple(kinds), tuple(tensors), tuple(opt), flags)
        try:
            hash(key)
        except TypeError:       # a tuple of lists or the like: nothing to recognise a step by
            return None
        return key

    def _capture(self, n: int, key):
        b = self._buffers(n)
        if len(self._graphs) >= self.MAX_GRAPHS:
            torch.cuda.synchronize(self.device)      # no replay is under way when its memory is given back
            self._graphs.popitem(last=False)
        graph, pool, stream = torch.cuda.CUDAGraph(), torch.cuda.graph_pool_handle(), torch.cuda.current_stream(self.device)
        try:
            with torch.cuda.graph(graph, pool=pool, capture_error_mode="thread_local"):
                loss = self._step(b.x_in, b.dp)
        except RuntimeError as err:
            # the step cannot be captured, or there is no memory for a graph's own pool (nothing has run): plain launches from
            # here on, which raise what is wrong with the step itself
            self._leave_failed_capture(pool, stream)
            # the text alone: the exception holds the frames of the step, and they its tensors
            logging.getLogger(__name__).warning("training step runs as plain launches, its capture failed: %s",
                                                (str(err) or type(err).__name__).splitlines()[0])
            self.use_graph = False
            self._graphs.clear()
            return None
        grads = [(p, p.grad) for p in self.model.parameters() if p.grad is not None]
        self._graphs[key] = (graph, loss, grads)
        return self._graphs[key]

    def _leave_failed_capture(self, pool, stream) -> None:
        """What the end of a capture does and an invalidated one leaves undone: the caller's stream is current again, the
        allocator no longer waits for the capture's end, and the random generator (whose mark only the end of a whole capture
        takes off) gives numbers outside of captures."""
        torch.cuda.set_stream(stream)
        try:
            torch._C._cuda_endAllocateToPool(self.E.device.index, pool)
        except RuntimeError:
            pass        # it was ended
        with torch.cuda.graph(torch.cuda.CUDAGraph(), capture_error_mode="thread_local"):
            self.loss_acc.add_(0.0)     # recorded, never run

    def _step(self, x: torch.Tensor, dp: torch.Tensor) -> torch.Tensor:
        m = self.model
        if self.rest_optimizer is not None:
            self.rest_optimizer.zero_grad(set_to_none=True)
        h_idx = x[:, 0].contiguous()
        head_rows = self.E[h_idx].requires_grad_(True)          # leaf: the table itself stays outside autograd
        h = m.normalize_head_entity_embeddings(m.input_dp_ent_real(head_rows))
        r = m.normalize_relation_embeddings(m.input_dp_rel_real(m.relation_embeddings(x[:, 1])))
        if self.distance:
            q, bias, mode = h + r + m._eps, None, 2
        else:
            q, bias = m.compose(h, r)
            mode = 0 if bias is None else 1
            if bias is not None:
                bias = bias.float().reshape(-1).contiguous()
        loss = FusedScoring.apply(q.float().contiguous(), bias, self, dp.contiguous(), mode)
        loss.backward()
        self.gE.index_add_(0, h_idx, head_rows.grad)           # row gradients of the lookups join the dense dE
        if self.rest_optimizer is not None:
            self.rest_optimizer.step()
        b1, b2 = self.betas
        K.optimizer_step(self.opt_kind, self.E, self.gE, self.mE, self.vE, self.E_bf16, self.step_count, self.lr, b1,
                         b2, self.eps, self.weight_decay)
        self.step_count += 1
        return loss.detach()

    def launches_per_step(self) -> int:
        return 5

    def sync_to_model(self) -> None:
        K.check_status(self.status, "in the external-query training step")

    def optimizer_view(self):
        return _HybridOptimizer(self)


class _HybridOptimizer(_EngineOptimizer):
    """LR-scheduling callbacks steer both halves: the kernel-side table update and the model's own optimiser."""

    def __init__(self, engine: ExternalQueryEngine):
        super().__init__(engine)
        self.param_groups = [_BothLr(engine)]


class _BothLr(dict):
    def __init__(self, engine):
        super().__init__(lr=engine.lr)
        self._e = engine

    def __setitem__(self, k, v):
        super().__setitem__(k, v)
        if k == "lr":
            self._e.lr = float(v)
            if self._e.rest_optimizer is not None:
                for g in self._e.rest_optimizer.param_groups:
                    g["lr"] = float(v)


def build_hybrid_engine(model, dataset, args, device) -> Optional[ExternalQueryEngine]:
    """An :class:`ExternalQueryEngine` when the fully fused engine does not cover the model but the bilinear contract
    holds; ``None`` otherwise."""
    if fused_model_code(model) is not None or not hybrid_supported(model):
        return None
    if getattr(args, "scoring_technique", None) not in SUPPORTED_SCORING:
        return None
    if dataset is None or not hasattr(dataset, "train_data") or torch.cuda.get_device_capability(device)[0] != 10:
        return None
    mask_bytes = 2 * int(args.batch_size) * model.num_entities / 8
    if mask_bytes > (1 << 30):
        return None
    return ExternalQueryEngine(model, dataset, batch_size=args.batch_size, lr=args.lr,
                               weight_decay=getattr(args, "weight_decay", 0.0) or 0.0, device=device)
