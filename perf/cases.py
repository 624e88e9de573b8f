"""The work a user of this framework has it do, as cases that can be timed and compared.

Three kinds, each through the public entry points:

* ``step``: one optimisation step, ``TrainEngine.train_step(inputs, labels)`` (what train.py and
  bench.py loop over), replayed from a CUDA graph or launched kernel by kernel (train.py's default);
* ``forward``: a pass of ``TrainEngine.model`` without gradients, either for the loss of every token
  of held-out text (``vocab_parallel_cross_entropy``) or for the logits of a prompt;
* ``attention``: ``apply_flash_attn`` on ``[B, nh, S, D]`` tensors and its backward.

A case is a dict of plain values; see ``listed`` for the fields and what each case stands for.
"""
import gc
import math

import torch

from gpt_from_scratch_b200.config import GPTConfig
from gpt_from_scratch_b200.engine import TrainEngine
from gpt_from_scratch_b200.ops.attention import apply_flash_attn
from gpt_from_scratch_b200.parallel.loss import vocab_parallel_cross_entropy

GPT_TINY = dict(layers=2, hidden=256, heads=4, ffn=512, vocab=1024)
GPT_124M = dict(layers=12, hidden=768, heads=12, ffn=3072, vocab=50304)
GPT_1P3B = dict(layers=24, hidden=2048, heads=16, ffn=5632, vocab=50304)


def _step(name, model, batch, seq, graph, dropout=0.0, text="zipf"):
    return dict(name=name, kind="step", **model, batch=batch, seq=seq, graph=graph, dropout=dropout, text=text)


def _forward(name, model, batch, seq, want, text="zipf"):
    return dict(name=name, kind="forward", **model, batch=batch, seq=seq, want=want, text=text)


def _attention(name, batch, heads, seq, head_dim, causal=True, dtype="bf16"):
    return dict(name=name, kind="attention", batch=batch, heads=heads, seq=seq, head_dim=head_dim, causal=causal,
                dtype=dtype)


def listed():
    return [
        # A first run of somebody who tries the framework out, and the loop of its tests and of
        # bench.py's "tiny" configuration: all launches and host work.
        _step("tiny-step", GPT_TINY, 2, 256, graph=False),
        # The same model with the step in a CUDA graph: what is left is the latency of the kernels.
        _step("tiny-step-graph", GPT_TINY, 2, 256, graph=True),
        # `python train.py --data-path text.bin`: every default of the command line.
        _step("124m-step-default", GPT_124M, 8, 1024, graph=False),
        # The headline benchmark: bench.py's default workload with its uniform random tokens.
        _step("124m-step-bench", GPT_124M, 16, 1024, graph=True, text="uniform"),
        # A micro-batch that no tile divides: documents cut at an odd length, an odd number of them.
        _step("124m-step-ragged", GPT_124M, 3, 777, graph=True),
        # Fine-tuning with --dropout-prob 0.1 on short sequences (dropout keeps the eager loop).
        _step("124m-step-dropout", GPT_124M, 4, 512, graph=False, dropout=0.1),
        # The larger model of bench.py (head_dim 128), whole on one GPU: the largest step.
        _step("1.3b-step", GPT_1P3B, 4, 2048, graph=True),
        # Held-out text during training of the default model: the loss of every token.
        _forward("124m-eval-loss", GPT_124M, 8, 1024, want="loss"),
        # Logits of one prompt: the smallest forward call.
        _forward("124m-prompt-logits", GPT_124M, 1, 130, want="logits"),
        # The attention operator by itself in the shape of the headline benchmark.
        _attention("attention-124m", 16, 12, 1024, 64),
        # Long sequences and wide heads: one layer of the 7B configuration.
        _attention("attention-7b", 1, 32, 4096, 128),
        # The operator's other options: fp16 tensors, no mask, a length that no block divides.
        _attention("attention-fp16-full", 3, 5, 333, 64, causal=False, dtype="fp16"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_model(rng):
    head_dim = rng.choice([64, 64, 128])
    heads = max(1, _log_uniform(rng, 128, 2048) // head_dim)
    hidden = heads * head_dim
    ffn = max(64, int(hidden * rng.uniform(2.0, 4.0)) // 8 * 8)
    vocab = rng.choice([_log_uniform(rng, 256, 50304) // 8 * 8, 50304])
    return dict(layers=_log_uniform(rng, 1, 24), hidden=hidden, heads=heads, ffn=ffn, vocab=vocab)


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        kind = rng.choice(["step"] * 7 + ["forward"] * 2 + ["attention"] * 3)
        if kind == "attention":
            case = _attention("", _log_uniform(rng, 1, 32), _log_uniform(rng, 1, 32), _log_uniform(rng, 32, 8192),
                              rng.choice([64, 128]), causal=rng.random() < 0.75,
                              dtype="fp16" if rng.random() < 0.25 else "bf16")
            # at most a quarter GiB per tensor and the work of a few milliseconds
            fits = case["batch"] * case["heads"] * case["seq"] * case["head_dim"] <= 1 << 27
            fits = fits and work(case)["flops"] <= 4e12
        else:
            batch, seq = _log_uniform(rng, 1, 16), _log_uniform(rng, 64, 2048)
            text = rng.choice(["zipf", "zipf", "uniform"])
            if kind == "step":
                dropout = 0.1 if rng.random() < 0.2 else 0.0
                case = _step("", _draw_model(rng), batch, seq, graph=dropout == 0.0 and rng.random() < 0.5,
                             dropout=dropout, text=text)
            else:
                case = _forward("", _draw_model(rng), batch, seq, rng.choice(["loss", "logits"]), text=text)
            fits = batch * seq <= 16384 and work(case)["flops"] <= most
            # the logits of a forward case stay within half a GiB
            fits = fits and (kind == "step" or batch * seq * case["vocab"] <= 1 << 29)
        if fits:
            del case["name"]
            return case


# ---------------------------------------------------------------------------- inputs
def _tokens(case, gen, shape):
    """Token ids. ``zipf``: the frequencies of words in text, p(n) ~ 1 / (n + 2.7) for the n-th most
    frequent one (the first is some 3 % of all); ``uniform``: as in bench.py."""
    V = min(case["vocab"], 50257)
    if case["text"] == "uniform":
        return torch.randint(0, V, shape, generator=gen, device="cuda")
    u = torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64)
    rank = (2.7 * (torch.exp(u * math.log((V + 2.7) / 2.7)) - 1.0)).long()
    # the frequent words have no ids in a row: a fixed shuffle of the vocabulary
    order = torch.randperm(V, generator=torch.Generator().manual_seed(1)).cuda()
    return order[rank.clamp_(0, V - 1)]


def _engine(case, seed):
    gc.collect()        # a program that builds a new engine has let go of its old one
    cfg = GPTConfig(vocab_size=case["vocab"], hidden_size=case["hidden"], num_layers=case["layers"],
                    num_attention_heads=case["heads"], max_position_embeddings=case["seq"],
                    intermediate_size=case["ffn"], dropout_prob=case.get("dropout", 0.0))
    # the first steps of a linear warm-up to 3e-4 over a thousand steps: two right implementations,
    # whose gradients differ by roundings, still have the same weights after a few of them
    return TrainEngine(cfg, lr=3e-7, seed=seed, cuda_graph=case.get("graph", False), graph_warmup=2)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "attention":
        dtype = torch.float16 if case["dtype"] == "fp16" else torch.bfloat16
        shape = (case["batch"], case["heads"], case["seq"], case["head_dim"])
        q, k, v, dout = (torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32).to(dtype)
                         for _ in range(4))
        return dict(kind="attention", q=q.requires_grad_(), k=k.requires_grad_(), v=v.requires_grad_(), dout=dout,
                    causal=case["causal"])
    torch.manual_seed(seed)          # dropout masks
    engine = _engine(case, seed)
    text = _tokens(case, gen, (case["batch"], case["seq"] + 1))
    state = dict(kind=case["kind"], engine=engine, inputs=text[:, :-1].contiguous(), labels=text[:, 1:].contiguous())
    if case["kind"] == "forward":
        state["want"] = case["want"]
        return state
    if case["graph"]:
        # a training program is past its first steps: the graph exists
        for _ in range(3):
            engine.train_step(state["inputs"], state["labels"])
    opt = engine.optimizer
    moments = opt._adam_state()      # made on first use
    state["updated"] = dict(grads=opt.grad_buffer, params=opt.param_buffer, master=opt.fp32_master_shard.detach(),
                            exp_avg=moments["exp_avg"], exp_avg_sq=moments["exp_avg_sq"])
    return state


# ---------------------------------------------------------------------------- one pass
def run(state):
    if state["kind"] == "attention":
        q, k, v = state["q"], state["k"], state["v"]
        out = apply_flash_attn(q, k, v, state["causal"])
        dq, dk, dv = torch.autograd.grad(out, (q, k, v), state["dout"])
        return dict(out=out.detach(), dq=dq, dk=dk, dv=dv)
    engine = state["engine"]
    if state["kind"] == "forward":
        with torch.no_grad():
            if state["want"] == "loss":
                logits, stats = engine.model(state["inputs"], return_ce_stats=True)
                return vocab_parallel_cross_entropy(logits, state["labels"].transpose(0, 1).contiguous(), stats)
            return engine.model(state["inputs"])
    loss = engine.train_step(state["inputs"], state["labels"])
    return dict(state["updated"], loss=loss)


# ---------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    B, S = case["batch"], case["seq"]
    if case["kind"] == "attention":
        n = B * case["heads"] * S * case["head_dim"]
        # two products forward, five backward; half of each under the causal mask
        flops = 14.0 * n * S * (0.5 if case["causal"] else 1.0)
        return dict(bytes=8 * 2.0 * n, flops=flops)      # q, k, v, dout read; out, dq, dk, dv written
    H, I, L, V = case["hidden"], case["ffn"], case["layers"], case["vocab"]
    cfg = GPTConfig(vocab_size=V, hidden_size=H, num_layers=L, intermediate_size=I)
    n, tokens = cfg.num_parameters(), B * S
    flops = cfg.flops_per_token(S) * tokens
    if case["kind"] == "step":
        # per parameter: weight read, gradient written, fp32 master and both moments read and written,
        # new weight written; both token arrays
        return dict(bytes=30.0 * n + 16.0 * tokens, flops=flops)
    weights = 2.0 * (n - V * H) + 2.0 * H * min(tokens, V)
    out = 2.0 * tokens * V if case["want"] == "logits" else 4.0 * tokens
    return dict(bytes=weights + out + (16.0 if case["want"] == "loss" else 8.0) * tokens, flops=flops / 3.0)


def tolerance(case):
    if case["kind"] == "attention":
        return {"rel": 1e-2}
    if case["kind"] == "forward" and case["want"] == "loss":
        return {"rel": 1e-3}         # fp32 sums over bf16 logits near zero
    # bf16 activations through all layers. Gradients of uniform random tokens cancel to a few times
    # their rounding noise (two compositions of the same bf16 step differ by 8e-3), and the table rows of
    # the most frequent tokens hold gradients a hundred times the buffer's rms: their rounding alone is of
    # the order of that rms.
    return {"rel": 1.5e-2, "max": 0.99}
