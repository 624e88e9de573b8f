"""Steps of several models, forwards and attention passes; saves all results. Run by test_overlap_gpu.py with programmatic
launches on and off (GFS_PDL)."""
import sys

import torch

from gpt_from_scratch_b200.config import GPTConfig
from gpt_from_scratch_b200.engine import TrainEngine
from gpt_from_scratch_b200.models import native
from gpt_from_scratch_b200.ops import _lib
from gpt_from_scratch_b200.ops.attention import apply_flash_attn
from gpt_from_scratch_b200.parallel import parallel_state as ps

# layers, hidden, heads, ffn, vocab, batch, seq, dropout
MODELS = {
    "one-tile products, grouped weight gradients": (2, 256, 4, 512, 1024, 2, 256, 0.0),
    "few rows, ragged": (2, 192, 3, 520, 504, 3, 77, 0.0),
    "pairs, lone and grouped weight gradients": (2, 768, 12, 3072, 8192, 4, 512, 0.0),
    "pairs with K above 1024, head_dim 128": (2, 1152, 9, 3072, 4096, 8, 512, 0.0),
    "dropout, few rows": (2, 256, 4, 512, 1024, 2, 128, 0.1),
    "dropout, many rows": (2, 768, 12, 2048, 1024, 4, 512, 0.1),
}


def main(path):
    torch.cuda.set_device(0)
    ps.set_device(torch.device("cuda", 0))
    ps.initialize_parallel_state(1)
    out = {}
    for name, (L, H, nh, I, V, B, S, p) in MODELS.items():
        cfg = GPTConfig(vocab_size=V, hidden_size=H, num_layers=L, num_attention_heads=nh, max_position_embeddings=S,
                        intermediate_size=I, dropout_prob=p)
        g = torch.Generator().manual_seed(3)
        tokens = [torch.randint(0, V, (B, S + 1), generator=g).cuda() for _ in range(2)]
        for path_name in ("native", "modules"):
            torch.manual_seed(4)
            eng = TrainEngine(cfg, seed=5, lr=1e-3)
            if path_name == "modules":
                eng.model.layers[0].register_forward_hook(lambda *a: None)
            res = []
            for step in range(4):
                t = tokens[step % 2]
                res.append(eng.train_step(t[:, :-1].contiguous(), t[:, 1:].contiguous()).clone())
                res.append(eng.optimizer.grad_buffer.clone())
            res.append(eng.optimizer.param_buffer.clone())
            if path_name == "native":
                # two micro-batches: the second one's gradients are added
                eng.optimizer.overlap_grad_reduce = False
                eng.optimizer.zero_grad()
                for t in tokens:
                    res.append(native.train_pass(eng.model, t[:, :-1].contiguous(), t[:, 1:].contiguous()).clone())
                res.append(eng.optimizer.grad_buffer.clone())
                eng.model.eval()
                with torch.no_grad():
                    res.append(eng.model(tokens[0][:, :-1].contiguous()).clone())
            out[f"{name}, {path_name}"] = [r.cpu() for r in res]
    g = torch.Generator(device="cuda").manual_seed(6)
    for D, B, nh, S, causal in ((64, 1, 3, 130, True), (64, 3, 12, 777, False), (128, 2, 5, 300, True)):
        q, k, v, do = (torch.randn(B, nh, S, D, device="cuda", generator=g).bfloat16() for _ in range(4))
        for t in (q, k, v):
            t.requires_grad_()
        res = []
        for _ in range(10):
            o = apply_flash_attn(q, k, v, causal)
            res += [o.detach(), *torch.autograd.grad(o, (q, k, v), do)]
        out[f"attention {D} {S}"] = [r.cpu() for r in res]
    torch.cuda.synchronize()
    _lib.raise_on_status()
    torch.save(out, path)


if __name__ == "__main__":
    main(sys.argv[1])
