"""The GPT model's forward and backward as a handful of native calls.

Module by module, a transformer block costs the host about 0.3 ms forward and 0.5 ms backward (eight
autograd functions, about twenty launches through ctypes), which is more than its kernels take at small
and ordinary sizes. ``GPTModel.forward`` therefore hands the whole model to this file when nothing needs
the module-by-module path: the stack of blocks with the final norm is ONE call into the library per
direction (csrc/model.cu), and autograd sees one function for the model. Same kernels and same logits; gradients
differ by roundings, because the weight gradients are grouped differently (csrc/model.cu says where).

The modules stay the owners of the parameters, and each pass compares what it is about to use with what they
hold: modules and their types, weights, biases, rotary tables, norm constants, dropout, hooks, ``forward`` methods
replaced on an instance or a class (``_Plan.current``, ``_Plan.plain_modules``). A change within what the native
passes compute is followed; any other one, a frozen weight included, sends the pass down the module path.
"""
from __future__ import annotations

import ctypes
import weakref
from ctypes import byref, c_float, c_int, c_ulonglong, c_void_p
from itertools import repeat
from operator import contains, getitem, is_

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
from .transformer_layer import ParallelAttention, TransformerLayer


class _Dims(ctypes.Structure):
    """GfsBlockDims in csrc/model.cu."""
    _fields_ = [("S", c_int), ("B", c_int), ("H", c_int), ("nh", c_int), ("D", c_int), ("I", c_int),
                ("n_layers", c_int), ("pair_min_tiles", c_int), ("grouped_wgrad", c_int),
                ("dropout_p", c_float), ("eps_final", c_float)]


class _BlockParams(ctypes.Structure):
    """GfsBlockParams in csrc/model.cu."""
    _fields_ = [("w", c_void_p * 6), ("g", c_void_p * 6), ("accumulate", c_int * 6), ("eps", c_float * 2),
                ("cos_table", c_void_p), ("sin_table", c_void_p), ("seed", c_ulonglong * 2)]


class _Top(ctypes.Structure):
    """GfsModelTop in csrc/model.cu."""
    _fields_ = [("w", c_void_p * 3), ("g", c_void_p * 3), ("accumulate", c_int * 3), ("V", c_int)]


def _native_tensor(t: torch.Tensor, dtype: torch.dtype) -> bool:
    return t.is_cuda and t.dtype == dtype and t.is_contiguous() and t.data_ptr() % 16 == 0


def _consume(p: torch.nn.Parameter) -> int:
    """1 if the gradient slice already holds this step's gradient (see GradSink.consume_accumulate)."""
    fresh = getattr(p, "_grad_fresh", False)
    p._grad_fresh = False
    return 0 if fresh else 1


# The methods whose work the native passes do: a class that has been given another one is asked.
_FORWARDS = tuple((c, c.forward) for c in (
    VocabParallelEmbedding, TransformerLayer, RMSNorm, ParallelAttention, RotaryEmbedding, ParallelMLP,
    ColumnParallelLinear, RowParallelLinear))


_model_class = _model_forward = None


def serve(model_class) -> None:
    """``model_class`` is the model that :func:`train_pass` restates (called where the class is defined)."""
    global _model_class, _model_forward
    _model_class, _model_forward = model_class, model_class.forward


class _Unsupported(Exception):
    """The modules compute something that the native passes do not."""


def _require(ok: bool) -> None:
    if not ok:
        raise _Unsupported


class _Plan:
    """What the passes of one model need, and everything it was derived from: the modules in their places, their
    weights, tables and settings (``dicts[i][keys[i]] is values[i]``) and what each tensor looked like. Built anew
    when any of it has changed (:meth:`current`)."""

    def __init__(self, model):
        self.dicts, self.keys, self.values = [], [], []
        self.modules, self.tensors, self.tables = [], [], []

        def read(place: dict, key: str):
            value = place[key]
            self.dicts.append(place)
            self.keys.append(key)
            self.values.append(value)
            return value

        def child(parent, name: str, cls):
            m = read(parent._modules, name)
            _require(type(m) is cls)
            self.modules.append(m)
            return m

        def weight(m, *shape):
            w = read(m._parameters, "weight")
            _require(_native_tensor(w, torch.bfloat16) and (not shape or tuple(w.shape) == shape))
            self.tensors.append(w)
            return w

        def linear(parent, name: str, cls, *shape):
            m = child(parent, name, cls)
            _require(read(m._parameters, "bias") is None)
            return weight(m, *shape)

        def norm(parent, name: str):
            m = child(parent, name, RMSNorm)
            eps = read(m.__dict__, "eps")
            _require(type(eps) in (int, float))
            return weight(m, H), eps

        emb = child(model, "embedding", VocabParallelEmbedding)
        w_emb = weight(emb)
        V, H = w_emb.shape
        _require(read(emb.__dict__, "vocab_start_index") == 0 and read(emb.__dict__, "vocab_end_index") == V)
        w_fin, eps_final = norm(model, "final_norm")
        w_out = linear(model, "output", ColumnParallelLinear)
        _require(w_out.shape[1] == H and w_out.shape[0] % 8 == 0 and H % 8 == 0)
        self.stack = read(model._modules, "layers")
        _require(type(self.stack) is torch.nn.ModuleList and len(self.stack) > 0)
        self.layers = list(self.stack)
        self.rotaries, self.weights, self.settings = [], [], set()
        self.table_rows = None
        self.params = (_BlockParams * len(self.layers))()
        for name, bp in zip(self.stack._modules, self.params):
            layer = child(self.stack, name, TransformerLayer)
            w1, eps1 = norm(layer, "input_norm")
            w2, eps2 = norm(layer, "post_attention_norm")
            a, m = child(layer, "attention", ParallelAttention), child(layer, "mlp", ParallelMLP)
            nh, D = read(a.__dict__, "num_heads_per_partition"), read(a.__dict__, "head_dim")
            _require(read(a.__dict__, "attention_impl") == "fused" and D in (64, 128) and nh * D == H)
            ws = (w1, linear(a, "qkv_proj", ColumnParallelLinear, 3 * H, H),
                  linear(a, "out_proj", RowParallelLinear, H, H), w2,
                  linear(m, "gate_up_proj", ColumnParallelLinear), linear(m, "down_proj", RowParallelLinear))
            I = ws[5].shape[1]
            _require(ws[4].shape == (2 * I, H) and ws[5].shape == (H, I) and I % 8 == 0)
            rot = child(a, "rotary_emb", RotaryEmbedding)
            cos, sin = read(rot._buffers, "cos_cached"), read(rot._buffers, "sin_cached")
            _require(_native_tensor(cos, torch.float32) and _native_tensor(sin, torch.float32))
            _require(cos.shape == sin.shape and cos.dim() == 2 and cos.shape[1] == D // 2)
            self.tables += (cos, sin)
            self.table_rows = min(self.table_rows or cos.shape[0], cos.shape[0])
            self.settings.add((nh, D, I, read(layer.__dict__, "dropout_prob")))
            self.rotaries.append(rot)
            self.weights.append(ws)
            for k, w in enumerate(ws):
                bp.w[k] = w.data_ptr()
            bp.eps[0], bp.eps[1] = eps1, eps2
            bp.cos_table, bp.sin_table = cos.data_ptr(), sin.data_ptr()
        _require(len(self.settings) == 1)
        nh, D, I, self.dropout_prob = self.settings.pop()
        _require(0.0 <= self.dropout_prob < 1.0)
        self.top = (w_emb, w_fin, w_out)
        self.all_params = [w for ws in self.weights for w in ws] + list(self.top)
        # A shared parameter (a tied head, a block that occurs twice) needs its overwrite-or-add flag taken where
        # each kernel runs, and its uses in one launch kept apart: the modules do both.
        _require(len({id(w) for w in self.all_params}) == len(self.all_params))
        self.types = [type(m) for m in self.modules]
        self.module_dicts = [m.__dict__ for m in self.modules]
        self.layer_dicts = [layer.__dict__ for layer in self.layers]
        self.hooks = [d for m in self.modules for d in (m._forward_hooks, m._forward_pre_hooks, m._backward_hooks,
                                                        m._backward_pre_hooks)]
        self.looks = self._looks()
        self.dims = _Dims(H=H, nh=nh, D=D, I=I, n_layers=len(self.layers), eps_final=eps_final)
        self.top_args = _Top(V=w_out.shape[0])
        for k, w in enumerate(self.top):
            self.top_args.w[k] = w.data_ptr()

    @classmethod
    def of(cls, model) -> "_Plan | None":
        try:
            return cls(model)
        except (_Unsupported, KeyError, AttributeError, TypeError, ValueError):   # others in our modules' places
            return None

    def _looks(self) -> tuple:
        ts = self.tensors
        return ([t.data_ptr() for t in ts], [t.shape for t in ts], [t.dtype for t in ts],
                [t.is_contiguous() for t in ts], [t.data_ptr() for t in self.tables])

    def current(self) -> bool:
        """True if nothing that the plan was built from has changed. (Loops in C: 60 us for 12 blocks.)"""
        try:
            if not all(map(is_, map(getitem, self.dicts, self.keys), self.values)):
                return False
        except KeyError:
            return False
        return (all(map(is_, map(type, self.modules), self.types)) and list(self.stack._modules.values()) == self.layers
                and self._looks() == self.looks)

    def plain_modules(self) -> bool:
        """No hook, no replaced method: calling a module is calling its class's ``forward``."""
        return not (any(self.hooks) or torch.nn.modules.module._has_any_global_hook() or
                    any(map(contains, self.module_dicts, repeat("forward"))) or
                    any(c.forward is not f for c, f in _FORWARDS))

    def grow_tables(self, S: int) -> bool:
        """Have the rotary modules make their tables for S positions, as they do when called."""
        grown = False
        for r in self.rotaries:
            if S > r.max_seq_len_cached or (r.round_to_activation_dtype and r._rounded_for is not torch.bfloat16):
                r(self.top[0], S)
                grown = True
        return grown

    def dropout_now(self) -> float | None:
        """The dropout probability of a pass that starts now; ``None`` if the blocks differ in it."""
        training = self.layer_dicts[0]["training"]
        if self.dropout_prob != 0.0 and any(d["training"] != training for d in self.layer_dicts):
            return None
        return self.dropout_prob if training else 0.0


class _Pass:
    """The arguments of one pass: copies of its own, because the library reads them without the interpreter lock
    while other threads start passes of the same model, and because a backward may come long after its forward."""
    __slots__ = ("plan", "S", "B", "dropout", "dims", "params", "gradients")

    def __init__(self, plan: _Plan, S: int, B: int, dropout: float):
        self.plan, self.S, self.B, self.dropout = plan, S, B, dropout     # the plan also keeps the tables alive
        self.gradients = None           # addresses of the gradients of plan.all_params when the pass began
        d = self.dims = _Dims.from_buffer_copy(plan.dims)
        d.S, d.B, d.dropout_p = S, B, dropout
        d.pair_min_tiles = gemm_ops.pair_threshold()
        d.grouped_wgrad = 1 if gemm_ops._WGRAD_GROUPING else 0
        self.params = type(plan.params).from_buffer_copy(plan.params)

    def act_bytes(self) -> int:
        return _lib.lib().gfs_blocks_act_bytes(byref(self.dims))

    def bwd_bytes(self) -> int:
        return _lib.lib().gfs_blocks_bwd_bytes(byref(self.dims))

    def draw_seeds(self) -> None:
        """Two dropout seeds per block, in the order the modules would draw them."""
        seeds = torch.randint(0, 2 ** 62, (2 * len(self.params),)).tolist()   # host generator: no device sync
        for bp, s0, s1 in zip(self.params, seeds[0::2], seeds[1::2]):
            bp.seed[0], bp.seed[1] = s0, s1

    def put_gradients(self, params, addresses, add) -> None:
        """Where the blocks' weight gradients go, and whether they are added to what is there (as :func:`_consume`
        says; both in the order of ``plan.all_params``)."""
        for i, bp in enumerate(params):
            bp.g[:] = addresses[6 * i:6 * i + 6]
            bp.accumulate[:] = add[6 * i:6 * i + 6]

    def for_backward(self, weights):
        """The blocks' arguments with ``weights`` (as autograd returns them) and their gradients."""
        params = type(self.params).from_buffer_copy(self.params)
        it = iter(weights)
        for bp, ws in zip(params, self.plan.weights):
            for k, w in enumerate(ws):
                t = next(it)
                assert t.shape == w.shape and _native_tensor(t, torch.bfloat16), "a weight changed since the forward"
                bp.w[k] = t.data_ptr()
        blocks = self.plan.all_params[:-3]
        self.put_gradients(params, [w.grad.data_ptr() for w in blocks], [_consume(w) for w in blocks])
        return params


# beside the modules, not in them: a plan holds raw addresses, which must not travel with a model that
# is copied or pickled
_plans: "weakref.WeakKeyDictionary" = weakref.WeakKeyDictionary()


def _renew(model) -> _Plan | None:
    plan = _Plan.of(model)
    if plan is None:
        _plans.pop(model, None)
    else:
        _plans[model] = plan
    return plan


def _sinks(params) -> list | None:
    """Addresses of the gradients if every one goes to a slice of its own in the optimizer's buffer (what
    GradSink.of asks for) and nobody waits for single ones or looks at them, else ``None``."""
    addresses = []
    for p in params:
        attrs, g = p.__dict__, p.grad
        if (g is None or not p.requires_grad or not attrs.get("_grad_sink_ok") or
                attrs.get("_grad_ready_cb") is not None or p._post_accumulate_grad_hooks or not g.is_contiguous()):
            return None
        for hook in p._backward_hooks.values() if p._backward_hooks else ():
            if not getattr(hook, "clears_slice", False):    # not the optimizer's own
                return None
        addresses.append(g.data_ptr())
    if len(set(addresses)) != len(addresses) or any(a % 16 for a in addresses):
        return None
    return addresses


def _autograd_is_watched() -> bool:
    """Somebody wants to see what autograd saves (hooks, as for offloading) or every gradient (anomaly mode)."""
    return torch.is_anomaly_enabled() or torch._C._autograd._top_saved_tensors_default_hooks(False) is not None


def plan_for(model, inputs: torch.Tensor) -> _Pass | None:
    """The arguments of a pass over ``inputs`` if it can run natively, else ``None``."""
    if not (inputs.dim() == 2 and inputs.numel() > 0) or ps.get_tensor_model_parallel_world_size() != 1:
        return None
    S = inputs.shape[1]
    plan = _plans.get(model)
    if plan is None or not plan.current():
        plan = _renew(model)
    if plan is None or not plan.plain_modules():
        return None
    if plan.grow_tables(S):
        plan = _renew(model)
        if plan is None:
            return None
    if torch.autograd.forward_ad._current_level >= 0:      # the modules refuse tangents, they must not get lost
        return None
    dropout = plan.dropout_now()
    if inputs.device != plan.top[0].device or S > plan.table_rows or dropout is None:
        return None
    run = _Pass(plan, S, inputs.shape[0], dropout)
    if torch.is_grad_enabled():
        if _autograd_is_watched():
            return None
        run.gradients = _sinks(plan.all_params)
        if run.gradients is None:
            return None
    return run


def _stack_forward(run: _Pass, x: torch.Tensor, keep: bool):
    """Blocks + final norm on ``x [S, B, H]`` -> (y [S*B, H], what the backward needs)."""
    S, B, H = x.shape
    dev = x.device
    n = len(run.params)
    drop = run.dropout > 0.0
    act_bytes = run.act_bytes()
    acts = [torch.empty(act_bytes, dtype=torch.uint8, device=dev) for _ in range(n if keep else 1)]
    addr = (c_ulonglong * n)(*[(acts[i] if keep else acts[0]).data_ptr() for i in range(n)])
    y = torch.empty((S * B, H), dtype=torch.bfloat16, device=dev)
    rstd = torch.empty(S * B, dtype=torch.float32, device=dev)
    tmp = torch.empty_like(y) if drop else None
    if drop:
        run.draw_seeds()
    launches = c_int(0)
    with _lib.nvtx("fused:blocks_fwd"):
        rc = _lib.lib().gfs_blocks_forward(byref(run.dims), run.params, run.plan.top[1].data_ptr(), x.data_ptr(), addr,
                                           _lib.ptr(tmp), y.data_ptr(), rstd.data_ptr(), byref(launches),
                                           _lib.stream_ptr())
    _lib.check(rc, "gfs_blocks_forward")
    _lib.add_launches(launches.value - 1)
    return y, rstd, acts


def _stack_backward(run: _Pass, weights, w_fin, x, rstd, acts, dy: torch.Tensor) -> torch.Tensor:
    n = len(run.params)
    addr = (c_ulonglong * n)(*[t.data_ptr() for t in acts])
    scratch = torch.empty(run.bwd_bytes(), dtype=torch.uint8, device=x.device)
    dx = torch.empty_like(x)
    p_fin = run.plan.top[1]
    params = run.for_backward(weights)
    launches = c_int(0)
    with _lib.nvtx("fused:blocks_bwd"):
        rc = _lib.lib().gfs_blocks_backward(byref(run.dims), params, w_fin.data_ptr(), p_fin.grad.data_ptr(),
                                            _consume(p_fin), x.data_ptr(), addr, rstd.data_ptr(), dy.data_ptr(),
                                            scratch.data_ptr(), dx.data_ptr(), byref(launches), _lib.stream_ptr())
    _lib.check(rc, "gfs_blocks_backward")
    _lib.add_launches(launches.value - 1)
    return dx


class _ModelFn(torch.autograd.Function):
    """logits ``[S, B, V]`` (and, for the loss, the LM head's softmax statistics) from token ids. The
    embedding weight is an input so that the result requires a gradient; all weight gradients go
    to their sinks. The other weights are saved like the modules save theirs: autograd notices one that is
    written to before the backward."""

    @staticmethod
    def forward(ctx, ids, w_emb, run, ce_stats):
        B, S = ids.shape
        x = embedding_fwd_native(ids, w_emb, 0, w_emb.shape[0])
        ctx.sorted_ids = sort_ids_async(ids, 0, w_emb.shape[0])   # needed by the backward; side stream
        y, rstd, acts = _stack_forward(run, x, keep=True)
        w_out = run.plan.top[2]
        logits, partials = gemm_ops.linear_fwd_ce(y, w_out) if ce_stats else (gemm_ops.linear_fwd(y, w_out), None)
        ctx.save_for_backward(ids, x, y, rstd, *acts, *run.plan.all_params[:-3], *run.plan.top[1:])
        ctx.run = run
        logits = logits.view(S, B, -1)
        if not ce_stats:
            return logits
        if partials is None:
            partials = x.new_empty(0, dtype=torch.float32)
        ctx.mark_non_differentiable(partials)
        return logits, partials

    @staticmethod
    def backward(ctx, dlogits, _dpartials=None):
        run = ctx.run
        n = len(run.params)
        ids, x, y, rstd, *saved = ctx.saved_tensors
        acts, weights, (w_fin, w_out) = saved[:n], saved[n:-2], saved[-2:]
        p_emb, _, p_out = run.plan.top
        d2 = dlogits.reshape(run.S * run.B, w_out.shape[0])
        if not d2.is_contiguous():
            d2 = d2.contiguous()
        dy = gemm_ops.linear_dgrad(d2, w_out)
        gemm_ops.linear_wgrad_to_sink(d2, y, GradSink(p_out))
        dx = _stack_backward(run, weights, w_fin, x, rstd, acts, dy)
        embedding_bwd_native(ids, dx, p_emb.grad, 0, p_emb.shape[0], accumulate=bool(_consume(p_emb)),
                             sorted_ids=ctx.sorted_ids)
        return None, None, None, None


def forward(run: _Pass, inputs: torch.Tensor, ce_stats: bool):
    """The model's forward on the native path: ``logits`` or ``(logits, partials or None)``."""
    ids = inputs.contiguous()
    if ids.dtype != torch.int64:
        ids = ids.long()
    w_emb, _, w_out = run.plan.top
    if torch.is_grad_enabled():
        out = _ModelFn.apply(ids, w_emb, run, ce_stats)
        if not ce_stats:
            return out
        logits, partials = out
        return logits, (partials if partials.numel() else None)
    x = embedding_fwd_native(ids, w_emb, 0, w_emb.shape[0])
    y, _, _ = _stack_forward(run, x, keep=False)
    if not ce_stats:
        return gemm_ops.linear_fwd(y, w_out).view(run.S, run.B, -1)
    logits, partials = gemm_ops.linear_fwd_ce(y, w_out)
    return logits.view(run.S, run.B, -1), partials


def train_pass(model, inputs: torch.Tensor, labels: torch.Tensor):
    """Forward, mean loss and backward of one micro-batch (``[B, S]`` ids and labels) without autograd:
    returns the loss (0-dim fp32) with every weight gradient in its sink, or ``None`` if the model has to
    go through its modules. One call into the library; all intermediates lie in one buffer."""
    if (type(model) is not _model_class or _model_class.forward is not _model_forward or "forward" in model.__dict__ or
            model._forward_hooks or model._forward_pre_hooks or model._backward_hooks or model._backward_pre_hooks):
        return None             # the model computes something of its own
    if not torch.is_grad_enabled() or not gemm_ops._CE_EPILOGUE:
        return None
    if labels.shape != inputs.shape or labels.device != inputs.device:
        return None
    run = plan_for(model, inputs)
    if run is None:
        return None
    plan = run.plan
    if plan.top[0].shape != plan.top[2].shape:      # a vocabulary for both
        return None
    lib, dims, top = _lib.lib(), byref(run.dims), _Top.from_buffer_copy(plan.top_args)
    step_bytes = lib.gfs_model_step_bytes(dims, byref(top))
    if step_bytes == 0:             # the embedding backward then sorts its ids with torch.sort
        return None
    ids, labels = inputs.contiguous(), labels.contiguous()
    if ids.dtype != torch.int64:
        ids = ids.long()
    if labels.dtype != torch.int64:
        labels = labels.long()
    dev = plan.top[0].device
    try:
        arena = torch.empty(step_bytes, dtype=torch.uint8, device=dev)
    except torch.OutOfMemoryError:  # no room in one piece: the modules' smaller tensors may still fit
        return None
    loss = torch.empty((), dtype=torch.float32, device=dev)
    if run.dropout > 0.0:
        run.draw_seeds()
    fresh = [p.__dict__.get("_grad_fresh", False) for p in plan.all_params]
    add = [_consume(p) for p in plan.all_params]
    run.put_gradients(run.params, run.gradients, add)
    top.g[:], top.accumulate[:] = run.gradients[-3:], add[-3:]
    launches = c_int(0)
    with _lib.nvtx("fused:model_step"):
        rc = lib.gfs_model_step(dims, run.params, byref(top), ids.data_ptr(), labels.data_ptr(), arena.data_ptr(),
                                loss.data_ptr(), byref(launches), _lib.stream_ptr())
    if rc != 0:             # the gradients hold nothing of this step
        for p, f in zip(plan.all_params, fresh):
            p._grad_fresh = f
    _lib.check(rc, "gfs_model_step")
    _lib.add_launches(launches.value - 1)
    return loss
