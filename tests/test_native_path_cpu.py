"""When the whole-model native passes may serve a model, on the CPU: the device checks are stubbed out, nothing
is launched. A pass that the native path cannot serve has to go through the modules, also when an earlier pass of the
same model ran natively."""
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
    monkeypatch.setattr(native, "_native_weight", lambda w: True)
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
