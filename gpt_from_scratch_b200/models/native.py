"""The GPT model's forward and backward as a handful of native calls.

Module by module, a transformer block costs the host about 0.3 ms forward and 0.5 ms backward (eight
autograd functions, about twenty launches through ctypes), which is more than its kernels take at small
and ordinary sizes. ``GPTModel.forward`` therefore hands the whole model to this file when nothing needs
the module-by-module path: the stack of blocks with the final norm is ONE call into the library per
direction (csrc/model.cu), and autograd sees one function for the model. Same kernels, same order, same
results.

The modules stay the owners of the parameters and every condition is looked up again in each pass
(``_Plan.refresh``), so replacing a module or a parameter, registering a hook, freezing a weight or
switching a module to another implementation sends the next pass down the module path.
"""
from __future__ import annotations

import ctypes
import weakref
from ctypes import byref, c_float, c_int, c_size_t, c_ulonglong, c_void_p

import torch

from ..ops import _lib
from ..ops import gemm as gemm_ops
from ..ops.embedding import embedding_bwd_native, embedding_fwd_native, sort_ids_async
from ..ops.grad_sink import GradSink
from ..parallel import parallel_state as ps
from ..parallel.layers import ColumnParallelLinear, RowParallelLinear, VocabParallelEmbedding
from .mlp import ParallelMLP
from .normalization import RMSNorm
from .position_embeddings import RotaryEmbedding


class _Dims(ctypes.Structure):
    """GfsBlockDims in csrc/model.cu."""
    _fields_ = [("S", c_int), ("B", c_int), ("H", c_int), ("nh", c_int), ("D", c_int), ("I", c_int),
                ("n_layers", c_int), ("pair_min_tiles", c_int), ("grouped_wgrad", c_int),
                ("dropout_p", c_float), ("eps_final", c_float), ("cos_table", c_void_p), ("sin_table", c_void_p)]


class _BlockParams(ctypes.Structure):
    """GfsBlockParams in csrc/model.cu."""
    _fields_ = [("w", c_void_p * 6), ("g", c_void_p * 6), ("accumulate", c_int * 6), ("eps", c_float * 2),
                ("seed", c_ulonglong * 2)]


class _Top(ctypes.Structure):
    """GfsModelTop in csrc/model.cu."""
    _fields_ = [("w", c_void_p * 3), ("g", c_void_p * 3), ("accumulate", c_int * 3), ("V", c_int)]


def _hook_dicts(module: torch.nn.Module):
    return (module._forward_hooks, module._forward_pre_hooks, module._backward_hooks, module._backward_pre_hooks)


def _native_weight(w) -> bool:
    return w.is_cuda and w.dtype == torch.bfloat16 and w.is_contiguous() and w.data_ptr() % 16 == 0


def _consume(p: torch.nn.Parameter) -> int:
    """1 if the gradient slice already holds this step's gradient (see GradSink.consume_accumulate)."""
    fresh = getattr(p, "_grad_fresh", False)
    p._grad_fresh = False
    return 0 if fresh else 1


class _Plan:
    """What a pass of one model needs, kept between passes; ``refresh`` brings it up to date."""

    def __init__(self, layer_type, attention_type):
        self.layer_type, self.attention_type = layer_type, attention_type
        self.layers: list = []          # the blocks the arrays below were built for
        self.shape = None               # (S, B) the workspace sizes were computed for
        self.dims = _Dims()
        self.params = None              # ctypes array of _BlockParams
        self.weights: list = []         # per block: its six parameters
        self.hooks: list = []
        self.ptrs: list = []
        self.step_shape = None          # (S, B, dropout) step_bytes was computed for
        self.top_args = _Top()

    def _bind(self, model) -> bool:
        """Structural checks and everything that depends on the modules only."""
        self.ptrs = []
        layers = list(model.layers)
        head, emb, fin = model.output, model.embedding, model.final_norm
        if (type(head) is not ColumnParallelLinear or head.bias is not None or
                type(emb) is not VocabParallelEmbedding or type(fin) is not RMSNorm):
            return False
        modules = [emb, fin, head]
        for layer in layers:
            a, m = layer.attention, layer.mlp
            if (type(layer) is not self.layer_type or type(a) is not self.attention_type or
                    type(m) is not ParallelMLP or type(layer.input_norm) is not RMSNorm or
                    type(layer.post_attention_norm) is not RMSNorm or
                    type(a.qkv_proj) is not ColumnParallelLinear or type(a.out_proj) is not RowParallelLinear or
                    type(m.gate_up_proj) is not ColumnParallelLinear or type(m.down_proj) is not RowParallelLinear or
                    type(a.rotary_emb) is not RotaryEmbedding):
                return False
            if any(x.bias is not None for x in (a.qkv_proj, a.out_proj, m.gate_up_proj, m.down_proj)):
                return False
            modules += [layer, a, m, layer.input_norm, layer.post_attention_norm, a.qkv_proj, a.out_proj,
                        m.gate_up_proj, m.down_proj, a.rotary_emb]
        H = fin.weight.shape[0]
        for layer in layers:
            a, m = layer.attention, layer.mlp
            if (a.hidden_size != H or a.head_dim not in (64, 128) or a.num_heads_per_partition * a.head_dim != H or
                    a.head_dim != layers[0].attention.head_dim or a.qkv_proj.weight.shape != (3 * H, H) or
                    a.out_proj.weight.shape != (H, H) or m.down_proj.weight.shape != (H, m.intermediate_size) or
                    m.gate_up_proj.weight.shape != (2 * m.intermediate_size, H) or
                    m.intermediate_size != layers[0].mlp.intermediate_size or m.intermediate_size % 8):
                return False
            r, r0 = a.rotary_emb, layers[0].attention.rotary_emb
            if (layer.dropout_prob != layers[0].dropout_prob or
                    (r.base, r.head_dim, r.round_to_activation_dtype) !=
                    (r0.base, r0.head_dim, r0.round_to_activation_dtype)):
                return False
        if not layers or H % 8 or head.weight.shape[1] != H or emb.weight.shape[1] != H or head.weight.shape[0] % 8:
            return False
        if any(not _native_weight(p) for p in model.parameters()):
            return False
        self.layers = layers
        self.hooks = [d for x in modules for d in _hook_dicts(x)]
        self.params = (_BlockParams * len(layers))()
        self.weights = [self._weights_of(layer) for layer in layers]
        for bp, layer, ws in zip(self.params, layers, self.weights):
            for k, w in enumerate(ws):
                bp.w[k] = w.data_ptr()
            bp.eps[0], bp.eps[1] = layer.input_norm.eps, layer.post_attention_norm.eps
        self.top = (emb.weight, fin.weight, head.weight)
        for k, w in enumerate(self.top):
            self.top_args.w[k] = w.data_ptr()
        self.top_args.V = head.weight.shape[0]
        self.all_params = [w for ws in self.weights for w in ws] + list(self.top)
        # A shared parameter (a tied head, a block that occurs twice) needs its overwrite-or-add flag taken where
        # each kernel runs, and its uses in one launch kept apart: the modules do both.
        if len({id(w) for w in self.all_params}) != len(self.all_params):
            return False
        d = self.dims
        d.H, d.nh, d.D = H, layers[0].attention.num_attention_heads, layers[0].attention.head_dim
        d.I, d.n_layers, d.eps_final = layers[0].mlp.intermediate_size, len(layers), fin.eps
        self.shape = self.step_shape = None
        self.ptrs = self._live_ptrs(model)
        return True

    @staticmethod
    def _weights_of(layer) -> tuple:
        m = layer._modules
        a, f = m["attention"]._modules, m["mlp"]._modules
        return (m["input_norm"]._parameters["weight"], a["qkv_proj"]._parameters["weight"],
                a["out_proj"]._parameters["weight"], m["post_attention_norm"]._parameters["weight"],
                f["gate_up_proj"]._parameters["weight"], f["down_proj"]._parameters["weight"])

    def _live_ptrs(self, model) -> list:
        """Identity of every parameter and address of its data as the modules hold them now."""
        top = model._modules
        ws = [w for layer in top["layers"]._modules.values() for w in self._weights_of(layer)]
        ws += [top["embedding"]._parameters["weight"], top["final_norm"]._parameters["weight"],
               top["output"]._parameters["weight"]]
        return [(id(w), w.data_ptr()) for w in ws]

    def refresh(self, model) -> bool:
        """True if this pass can run natively."""
        try:
            current = self._live_ptrs(model)
        except (KeyError, AttributeError):     # modules replaced by others
            return False
        if current != self.ptrs and not self._bind(model):
            return False
        if any(self.hooks) or torch.nn.modules.module._has_any_global_hook():
            return False
        training = self.layers[0].training
        for layer in self.layers:
            if layer.training != training or layer._modules["attention"].attention_impl != "fused":
                return False
        self.dropout = self.layers[0].dropout_prob if training else 0.0
        return True

    def set_shape(self, S: int, B: int) -> None:
        d = self.dims
        rot = self.layers[0].attention.rotary_emb
        cos, sin = rot(self.top[0], S)
        d.cos_table, d.sin_table = cos.data_ptr(), sin.data_ptr()
        d.pair_min_tiles = gemm_ops.pair_threshold()
        d.grouped_wgrad = 1 if gemm_ops._WGRAD_GROUPING else 0
        key = (S, B, self.dropout)
        if key != self.shape:
            d.S, d.B, d.dropout_p = S, B, self.dropout
            out_off = c_size_t()
            lib = _lib.lib()
            self.act_bytes = lib.gfs_blocks_act_bytes(byref(d), byref(out_off))
            self.bwd_bytes = lib.gfs_blocks_bwd_bytes(byref(d))
            self.shape = key

    def draw_seeds(self) -> list:
        """Two dropout seeds per block, in the order the modules would draw them."""
        seeds = torch.randint(0, 2 ** 62, (2 * len(self.layers),)).tolist()   # host generator: no device sync
        self.put_seeds(seeds)
        return seeds

    def put_gradients(self) -> None:
        """Where the blocks' weight gradients go, and whether they are added to what is there."""
        for bp, ws in zip(self.params, self.weights):
            g, acc = bp.g, bp.accumulate
            for k, w in enumerate(ws):
                g[k] = w.grad.data_ptr()
                acc[k] = _consume(w)

    def put_seeds(self, seeds: list) -> None:
        for bp, s0, s1 in zip(self.params, seeds[0::2], seeds[1::2]):
            bp.seed[0], bp.seed[1] = s0, s1


# beside the modules, not in them: a plan holds raw addresses, which must not travel with a model that
# is copied or pickled
_plans: "weakref.WeakKeyDictionary" = weakref.WeakKeyDictionary()


def plan_for(model, inputs: torch.Tensor):
    """The model's plan if this pass can run natively, else ``None``."""
    w = model.embedding.weight
    if not (_native_weight(w) and inputs.dim() == 2 and inputs.device == w.device and inputs.numel() > 0):
        return None
    if ps.get_tensor_model_parallel_world_size() != 1:
        return None
    plan = _plans.get(model)
    if plan is None:
        from .transformer_layer import ParallelAttention, TransformerLayer
        plan = _plans[model] = _Plan(TransformerLayer, ParallelAttention)
    if not plan.refresh(model):
        return None
    if torch.is_grad_enabled():
        slices = set()
        for p in plan.all_params:
            # every gradient goes to a slice of its own in the optimizer's buffer and nobody waits for single ones
            if not p.requires_grad or GradSink.of(p) is None or getattr(p, "_grad_ready_cb", None) is not None:
                return None
            slices.add(p.grad.data_ptr())
        if len(slices) != len(plan.all_params):
            return None
    return plan


def _stack_forward(plan: _Plan, x: torch.Tensor, keep: bool):
    """Blocks + final norm on ``x [S, B, H]`` -> (y [S*B, H], what the backward needs)."""
    S, B, H = x.shape
    dev = x.device
    n = len(plan.layers)
    seeds = plan.draw_seeds() if plan.dropout > 0.0 else None
    acts = [torch.empty(plan.act_bytes, dtype=torch.uint8, device=dev) for _ in range(n if keep else 1)]
    addr = (c_ulonglong * n)(*[(acts[i] if keep else acts[0]).data_ptr() for i in range(n)])
    y = torch.empty((S * B, H), dtype=torch.bfloat16, device=dev)
    rstd = torch.empty(S * B, dtype=torch.float32, device=dev)
    tmp = torch.empty_like(y) if seeds is not None else None
    launches = c_int(0)
    with _lib.nvtx("fused:blocks_fwd"):
        rc = _lib.lib().gfs_blocks_forward(byref(plan.dims), plan.params, plan.top[1].data_ptr(), x.data_ptr(), addr,
                                           _lib.ptr(tmp), y.data_ptr(), rstd.data_ptr(), byref(launches),
                                           _lib.stream_ptr())
    _lib.check(rc, "gfs_blocks_forward")
    _lib.add_launches(launches.value - 1)
    return y, (x, rstd, acts, seeds)


def _stack_backward(plan: _Plan, x, rstd, acts, seeds, dy: torch.Tensor) -> torch.Tensor:
    n = len(plan.layers)
    plan.put_gradients()
    if seeds is not None:
        plan.put_seeds(seeds)
    w_fin = plan.top[1]
    addr = (c_ulonglong * n)(*[t.data_ptr() for t in acts])
    scratch = torch.empty(plan.bwd_bytes, dtype=torch.uint8, device=x.device)
    dx = torch.empty_like(x)
    launches = c_int(0)
    with _lib.nvtx("fused:blocks_bwd"):
        rc = _lib.lib().gfs_blocks_backward(byref(plan.dims), plan.params, w_fin.data_ptr(), w_fin.grad.data_ptr(),
                                            _consume(w_fin), x.data_ptr(), addr, rstd.data_ptr(), dy.data_ptr(),
                                            scratch.data_ptr(), dx.data_ptr(), byref(launches), _lib.stream_ptr())
    _lib.check(rc, "gfs_blocks_backward")
    _lib.add_launches(launches.value - 1)
    return dx


class _ModelFn(torch.autograd.Function):
    """logits ``[S, B, V]`` (and, for the loss, the LM head's softmax statistics) from token ids. The
    embedding weight is an input so that the result requires a gradient; all weight gradients go
    to their sinks."""

    @staticmethod
    def forward(ctx, ids, w_emb, plan, ce_stats):
        B, S = ids.shape
        x = embedding_fwd_native(ids, w_emb, 0, w_emb.shape[0])
        ctx.sorted_ids = sort_ids_async(ids, 0, w_emb.shape[0])   # needed by the backward; side stream
        y, (x, rstd, acts, seeds) = _stack_forward(plan, x, keep=True)
        w_out = plan.top[2]
        logits, partials = gemm_ops.linear_fwd_ce(y, w_out) if ce_stats else (gemm_ops.linear_fwd(y, w_out), None)
        ctx.save_for_backward(ids, x, y, rstd, *acts)
        ctx.plan, ctx.seeds, ctx.key = plan, seeds, (S, B, plan.dropout)
        logits = logits.view(S, B, -1)
        if not ce_stats:
            return logits
        if partials is None:
            partials = x.new_empty(0, dtype=torch.float32)
        ctx.mark_non_differentiable(partials)
        return logits, partials

    @staticmethod
    def backward(ctx, dlogits, _dpartials=None):
        plan = ctx.plan
        ids, x, y, rstd, *acts = ctx.saved_tensors
        S, B, dropout = ctx.key
        if ctx.key != plan.shape:       # another pass of the model ran in between
            plan.dropout = dropout
            plan.set_shape(S, B)
        w_emb, _, w_out = plan.top
        d2 = dlogits.reshape(S * B, w_out.shape[0])
        if not d2.is_contiguous():
            d2 = d2.contiguous()
        dy = gemm_ops.linear_dgrad(d2, w_out)
        gemm_ops.linear_wgrad_to_sink(d2, y, GradSink(w_out))
        dx = _stack_backward(plan, x, rstd, acts, ctx.seeds, dy)
        embedding_bwd_native(ids, dx, w_emb.grad, 0, w_emb.shape[0], accumulate=bool(_consume(w_emb)),
                             sorted_ids=ctx.sorted_ids)
        return None, None, None, None


def forward(plan: _Plan, inputs: torch.Tensor, ce_stats: bool):
    """The model's forward on the native path: ``logits`` or ``(logits, partials or None)``."""
    ids = inputs.contiguous()
    if ids.dtype != torch.int64:
        ids = ids.long()
    B, S = ids.shape
    w_emb, _, w_out = plan.top
    plan.set_shape(S, B)
    if torch.is_grad_enabled():
        out = _ModelFn.apply(ids, w_emb, plan, ce_stats)
        if not ce_stats:
            return out
        logits, partials = out
        return logits, (partials if partials.numel() else None)
    x = embedding_fwd_native(ids, w_emb, 0, w_emb.shape[0])
    y, _ = _stack_forward(plan, x, keep=False)
    if not ce_stats:
        return gemm_ops.linear_fwd(y, w_out).view(S, B, -1)
    logits, partials = gemm_ops.linear_fwd_ce(y, w_out)
    return logits.view(S, B, -1), partials


def train_pass(model, inputs: torch.Tensor, labels: torch.Tensor):
    """Forward, mean loss and backward of one micro-batch (``[B, S]`` ids and labels) without autograd:
    returns the loss (0-dim fp32) with every weight gradient in its sink, or ``None`` if the model has to
    go through its modules. One call into the library; all intermediates lie in one buffer."""
    if (not torch.is_grad_enabled() or labels.shape != inputs.shape or not labels.is_cuda or
            model._forward_hooks or model._forward_pre_hooks or model._backward_hooks or model._backward_pre_hooks):
        return None
    plan = plan_for(model, inputs)
    if plan is None:
        return None
    B, S = inputs.shape
    if B * S > 32768:       # the embedding backward then sorts its ids with the library's sort
        return None
    ids, labels = inputs.contiguous(), labels.contiguous()
    if ids.dtype != torch.int64:
        ids = ids.long()
    if labels.dtype != torch.int64:
        labels = labels.long()
    dev = plan.top[0].device
    plan.set_shape(S, B)
    if plan.dropout > 0.0:
        plan.draw_seeds()
    lib, dims, top = _lib.lib(), byref(plan.dims), plan.top_args
    if plan.step_shape != plan.shape:
        plan.step_bytes = lib.gfs_model_step_bytes(dims, byref(top))
        plan.step_shape = plan.shape
    fresh = [getattr(p, "_grad_fresh", False) for p in plan.all_params]
    plan.put_gradients()
    for k, w in enumerate(plan.top):
        top.g[k] = w.grad.data_ptr()
        top.accumulate[k] = _consume(w)
    arena = torch.empty(plan.step_bytes, dtype=torch.uint8, device=dev)
    loss = torch.empty((), dtype=torch.float32, device=dev)
    launches = c_int(0)
    with _lib.nvtx("fused:model_step"):
        rc = lib.gfs_model_step(dims, plan.params, byref(top), ids.data_ptr(), labels.data_ptr(), arena.data_ptr(),
                                loss.data_ptr(), byref(launches), _lib.stream_ptr())
    if rc == -20:           # ids times tokens do not fit the sort's 32-bit keys: nothing was launched
        for p, f in zip(plan.all_params, fresh):
            p._grad_fresh = f
        return None
    _lib.check(rc, "gfs_model_step")
    _lib.add_launches(launches.value - 1)
    return loss
