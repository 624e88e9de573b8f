"""When the whole-model native passes may serve a model, on the CPU: the device checks are stubbed out, nothing
is launched. A pass that the native path cannot serve has to go through the modules, also when an earlier pass of the
same model ran natively."""
import threading
import types
from contextlib import contextmanager

import pytest
import torch

from gpt_from_scratch_b200.config import GPTConfig
from gpt_from_scratch_b200.models import native
from gpt_from_scratch_b200.models.gpt import GPTModel
from gpt_from_scratch_b200.parallel import parallel_state as ps

IDS = torch.zeros(2, 8, dtype=torch.int64)


@pytest.fixture(autouse=True)
def _cpu_state():
    ps.destroy_model_parallel()
    ps.set_device("cpu")
    ps.initialize_parallel_state(1)
    yield
    ps.destroy_model_parallel()


@pytest.fixture
def model(monkeypatch):
    monkeypatch.setattr(native, "_native_tensor", lambda t, dtype: t.is_contiguous())
    m = GPTModel(GPTConfig(vocab_size=64, hidden_size=128, num_layers=3, num_attention_heads=2,
                           max_position_embeddings=16, intermediate_size=64))
    for p in m.parameters():
        p.grad = torch.zeros_like(p)
        p._grad_sink_ok = True
    assert native.plan_for(m, IDS) is not None
    return m


def _tie_head(m):
    m.output.weight = m.embedding.weight


def _repeat_block(m):
    m.layers[1] = m.layers[0]


def _share_norm(m):
    m.layers[2].input_norm.weight = m.layers[1].input_norm.weight


def _share_gradient(m):
    m.layers[2].mlp.down_proj.weight.grad = m.layers[1].mlp.down_proj.weight.grad


@pytest.mark.parametrize("share", [_tie_head, _repeat_block, _share_norm, _share_gradient])
def test_shared_parameters_take_the_module_path(model, share):
    share(model)
    assert native.plan_for(model, IDS) is None


class _OtherLinear(torch.nn.Module):
    bias = None

    def __init__(self, weight):
        super().__init__()
        self.weight = weight


def _subclass_linear(m):
    a = m.layers[1].attention
    new = type("Scaled", (type(a.out_proj),), {})(128, 128, bias=False)
    new.weight = a.out_proj.weight
    a.out_proj = new


def _other_linear(m):
    m.layers[1].mlp.down_proj = _OtherLinear(m.layers[1].mlp.down_proj.weight)


def _retype(m):
    m.layers[2].__class__ = type("Block", (type(m.layers[2]),), {})


def _own_forward(m):
    m.layers[0].mlp.forward = types.MethodType(lambda self, x, residual=None: x, m.layers[0].mlp)


def _attach_bias(m):
    m.layers[2].attention.qkv_proj.bias = torch.nn.Parameter(torch.zeros(384))


def _head_bias(m):
    m.output.bias = torch.nn.Parameter(torch.zeros(64))


def _other_impl(m):
    m.layers[1].attention.attention_impl = "reference"


def _hook(m):
    m.layers[1].attention.rotary_emb.register_forward_hook(lambda *a: None)


def _uneven_dropout(m):
    m.layers[1].dropout_prob = 0.25


def _vocabulary_slice(m):
    m.embedding.vocab_start_index = 8


def _other_stack(m):
    m.layers = torch.nn.Sequential(*m.layers)


def _view_of_weight(m):
    w = m.layers[1].attention.out_proj.weight        # same parameter, same address, other strides
    w.data = w.data.t()


def _shorter_table(m):
    r = m.layers[1].attention.rotary_emb
    r.cos_cached, r.sin_cached = r.cos_cached[:4], r.sin_cached[:4]


def _wrapped_embedding(m):
    m.embedding = torch.nn.Sequential(m.embedding)


def _freeze(m):
    m.layers[0].mlp.gate_up_proj.weight.requires_grad_(False)


@pytest.mark.parametrize("change", [
    _subclass_linear, _other_linear, _retype, _own_forward, _attach_bias, _head_bias, _other_impl, _hook, _uneven_dropout,
    _vocabulary_slice, _other_stack, _view_of_weight, _shorter_table, _wrapped_embedding, _freeze])
def test_changes_after_a_native_pass_take_the_module_path(model, change):
    change(model)
    assert native.plan_for(model, IDS) is None


@pytest.mark.parametrize("cls", ["RMSNorm", "TransformerLayer", "RotaryEmbedding"])
def test_replaced_class_method_takes_the_module_path(model, monkeypatch, cls):
    monkeypatch.setattr(getattr(native, cls), "forward", lambda self, *a, **k: None)
    assert native.plan_for(model, IDS) is None


def test_changed_settings_are_followed(model):
    """Values that the modules read in each pass, tables and weights that are exchanged for others."""
    model.layers[1].post_attention_norm.eps = 0.5
    model.final_norm.eps = 0.25
    for layer in model.layers:
        layer.dropout_prob = 0.125
    table = model.layers[2].attention.rotary_emb
    table.cos_cached = table.cos_cached * 0.5
    old = model.layers[0].mlp.down_proj.weight
    model.layers[0].mlp.down_proj.weight = new = torch.nn.Parameter(old.detach().clone())
    new.grad, new._grad_sink_ok = torch.zeros_like(new), True
    plan = native.plan_for(model, IDS)
    assert plan.params[1].eps[1] == 0.5 and plan.dims.eps_final == 0.25 and plan.dropout == 0.125
    assert plan.params[2].cos_table == table.cos_cached.data_ptr() != plan.params[1].cos_table
    assert plan.params[0].w[5] == new.data_ptr()
    model.eval()
    assert native.plan_for(model, IDS).dropout == 0.0


def test_tables_grow_with_the_sequence(model):
    """Positions past max_position_embeddings, as through the modules: every block's own table grows."""
    plan = native.plan_for(model, torch.zeros(1, 40, dtype=torch.int64))
    for bp, layer in zip(plan.params, model.layers):
        cos = layer.attention.rotary_emb.cos_cached
        assert cos.shape[0] == 40 and bp.cos_table == cos.data_ptr()


@pytest.fixture
def step(model, monkeypatch):
    """``step(model)``: whether the training step in one native call takes the model."""
    with _fake_library(monkeypatch, gfs_model_step=lambda *a: 0, gfs_model_step_bytes=lambda *a: 1):
        yield lambda m=model: native.train_pass(m, IDS, IDS) is not None


def test_training_step_takes_plain_models_only(model, step, monkeypatch):
    """A model with a forward of its own (a wrapper, a subclass, a method set on the instance or the class) is called."""
    assert step()

    class Wrapper(torch.nn.Module):
        def __init__(self, inner):
            super().__init__()
            self.inner = inner

    assert not step(Wrapper(model))
    model.forward = lambda *a, **k: None
    assert not step()
    del model.forward
    assert step()
    model.__class__ = type("Sub", (GPTModel,), {})
    assert not step()
    model.__class__ = GPTModel
    monkeypatch.setattr(GPTModel, "forward", lambda *a, **k: None)
    assert not step()


def test_engine_calls_its_own_forward_loss(monkeypatch):
    """``forward_loss`` replaced in a subclass, on the instance or on the class is what a step runs."""
    from gpt_from_scratch_b200 import engine as engine_mod
    cfg = GPTConfig(vocab_size=64, hidden_size=128, num_layers=1, num_attention_heads=2, max_position_embeddings=16,
                    intermediate_size=64)
    monkeypatch.setattr(native, "train_pass", lambda *a: torch.tensor(-1.0))
    base = engine_mod.TrainEngine.forward_loss

    def own(self, x, y):
        return base(self, x, y) * 0.0 + 7.0

    eng = engine_mod.TrainEngine(cfg, dtype=torch.float32)
    assert float(eng.train_step(IDS, IDS)) == -1.0
    eng.forward_loss = types.MethodType(own, eng)
    assert float(eng.train_step(IDS, IDS)) == 7.0
    del eng.forward_loss
    sub = type("Sub", (engine_mod.TrainEngine,), {"forward_loss": own})(cfg, dtype=torch.float32)
    assert float(sub.train_step(IDS, IDS)) == 7.0
    monkeypatch.setattr(engine_mod.TrainEngine, "forward_loss", own)
    assert float(eng.train_step(IDS, IDS)) == 7.0


def test_observers_of_gradients_are_served(model, step):
    """Who asks to see single gradients or what autograd saves gets a pass under autograd; tangents are refused by
    the modules, so they must reach them."""
    w = model.layers[1].mlp.down_proj.weight
    w.register_hook(lambda g: None).remove()
    assert step()
    for register in (w.register_hook, w.register_post_accumulate_grad_hook):
        handle = register(lambda g: None)
        assert native.plan_for(model, IDS) is None and not step()
        handle.remove()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t):
        assert native.plan_for(model, IDS) is None and not step()
    with torch.autograd.set_detect_anomaly(True):
        assert native.plan_for(model, IDS) is None and not step()
    with torch.autograd.forward_ad.dual_level(), torch.no_grad():
        assert native.plan_for(model, IDS) is None
    w.grad = torch.zeros_like(w.T.contiguous()).T            # of the weight's shape, but strided
    assert not step()
    w.grad = torch.zeros_like(w)
    assert step()


@contextmanager
def _fake_library(monkeypatch, **calls):
    """The native library with some entry points replaced; what runs around them does so on the CPU."""
    from gpt_from_scratch_b200.ops import _lib

    class Fake:
        def __getattr__(self, name):
            return calls.get(name) or getattr(real, name)
    real, fake = _lib.lib(), Fake()
    with monkeypatch.context() as m:
        m.setattr(_lib, "lib", lambda: fake)
        m.setattr(_lib, "stream_ptr", lambda: 0)
        m.setattr(native, "embedding_fwd_native", lambda ids, w, v0, v1: torch.zeros(*ids.T.shape, w.shape[1]))
        m.setattr(native.gemm_ops, "linear_fwd", lambda x, w: torch.zeros(x.shape[0], w.shape[0]))
        yield


def test_passes_of_two_threads_have_their_own_arguments(model, monkeypatch):
    """The library reads a pass's arguments without the interpreter lock, while another thread starts a pass of
    another shape (and another dropout mode) on the same model."""
    for layer in model.layers:
        layer.dropout_prob = 0.5
    inside, go_on, seen = threading.Event(), threading.Event(), []

    def blocks_forward(dims, params, *rest):
        first = not inside.is_set()
        before = (dims._obj.S, dims._obj.B, dims._obj.dropout_p, [tuple(p.seed) for p in params])
        if first:
            inside.set()
            assert go_on.wait(20)
        seen.append((before, (dims._obj.S, dims._obj.B, dims._obj.dropout_p, [tuple(p.seed) for p in params])))
        return 0

    def run(ids, train):
        with torch.no_grad():
            model.train(train)
            model(ids)

    with _fake_library(monkeypatch, gfs_blocks_forward=blocks_forward, gfs_blocks_bwd_bytes=lambda dims: 0):
        first = threading.Thread(target=run, args=(IDS, True))
        first.start()
        assert inside.wait(20)
        run(torch.zeros(3, 5, dtype=torch.int64), True)
        go_on.set()
        first.join()
    assert [before[:2] for before, _ in seen] == [(5, 3), (8, 2)]
    assert all(before == after for before, after in seen)


def test_step_refuses_before_it_starts(model):
    """Batches that the id sort cannot take are refused before anything is launched (on the CPU: before the
    first CUDA call fails)."""
    from ctypes import byref, c_int
    from gpt_from_scratch_b200.ops import _lib
    lib = _lib.lib()
    run = native.plan_for(model, IDS)
    top = native._Top.from_buffer_copy(run.plan.top_args)
    for S, B, V in ((32769, 1, 64), (256, 129, 64), (16384, 2, 1 << 17)):
        run.dims.S, run.dims.B, top.V = S, B, V
        assert lib.gfs_embedding_sort_shift(S * B, V) == -20
        assert lib.gfs_model_step_bytes(byref(run.dims), byref(top)) == 0
        launches = c_int(0)
        assert lib.gfs_model_step(byref(run.dims), run.params, byref(top), 0, 0, 0, 0, byref(launches), 0) == -1
        assert launches.value == 0
    assert [lib.gfs_embedding_sort_shift(n, 64) for n in (1, 2, 3, 4, 5, 32768)] == [1, 1, 2, 2, 3, 15]


def test_failed_or_refused_step_leaves_no_trace(model, monkeypatch):
    """Whether gradients are overwritten or added to, and the dropout generator, are as before the call."""
    for layer in model.layers:
        layer.dropout_prob = 0.5
    for i, p in enumerate(model.parameters()):
        p._grad_fresh = i % 2 == 0
    before = [p._grad_fresh for p in model.parameters()]
    rng = torch.get_rng_state()
    with _fake_library(monkeypatch, gfs_model_step=lambda *a: -13, gfs_model_step_bytes=lambda *a: 8):
        with pytest.raises(RuntimeError, match="gfs_model_step"):
            native.train_pass(model, IDS, IDS)
        assert [p._grad_fresh for p in model.parameters()] == before

        def no_room(*a, **k):
            raise torch.OutOfMemoryError("no room")
        with monkeypatch.context() as m:
            torch.set_rng_state(rng)
            m.setattr(torch, "empty", no_room)
            assert native.train_pass(model, IDS, IDS) is None
    with _fake_library(monkeypatch, gfs_model_step=lambda *a: 0, gfs_model_step_bytes=lambda *a: 0):
        assert native.train_pass(model, IDS, IDS) is None
    assert [p._grad_fresh for p in model.parameters()] == before and torch.equal(torch.get_rng_state(), rng)


def test_step_wants_one_vocabulary(model, step):
    head = model.output.weight = torch.nn.Parameter(torch.zeros(72, 128))
    head.grad, head._grad_sink_ok = torch.zeros_like(head), True
    assert native.plan_for(model, IDS) is not None and not step()
