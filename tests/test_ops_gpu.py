"""Numerics of the single-GPU kernels against fp32 PyTorch references."""
import math
import pathlib
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(a, b, atol, rtol=0.0, what=""):
    a, b = a.float(), b.float()
    err = (a - b).abs()
    tol = atol + rtol * b.abs()
    bad = (err > tol)
    assert not bad.any(), f"{what}: max err {err.max().item():.4g} (tol {atol}), {int(bad.sum())} bad of {a.numel()}"


@pytest.mark.parametrize("B,nh,S,D", [(2, 2, 128, 64), (1, 3, 256, 64), (2, 2, 512, 128), (1, 2, 384, 128),
                                      (4, 12, 1024, 64), (1, 2, 2048, 64)])
def test_flash_attention_fwd_bwd(cuda_device, B, nh, S, D):
    from gpt_from_scratch_b200.ops.attention import apply_flash_attn, attention_reference
    g = torch.Generator(device="cuda").manual_seed(S + D)
    q, k, v = (torch.randn(B, nh, S, D, device=cuda_device, generator=g).bfloat16().requires_grad_() for _ in range(3))
    do = torch.randn(B, nh, S, D, device=cuda_device, generator=g).bfloat16()
    o = apply_flash_attn(q, k, v, True)
    o.backward(do)
    dq, dk, dv = q.grad.clone(), k.grad.clone(), v.grad.clone()
    qf, kf, vf = (t.detach().float().requires_grad_() for t in (q, k, v))
    of = attention_reference(qf, kf, vf, True)
    of.backward(do.float())
    # the reference repository's own tolerances: 1e-2 forward, 5e-2 gradients
    _close(o, of, 1e-2, what="O")
    _close(dq, qf.grad, 5e-2, what="dQ")
    _close(dk, kf.grad, 5e-2, what="dK")
    _close(dv, vf.grad, 5e-2, what="dV")
    # and a tighter relative check on the aggregate error
    for name, a, b in (("O", o, of), ("dQ", dq, qf.grad), ("dK", dk, kf.grad), ("dV", dv, vf.grad)):
        rel = (a.float() - b).norm() / (b.norm() + 1e-12)
        assert rel < 2e-2, f"{name}: relative error {rel:.4g}"


def test_flash_attention_fp16_inputs_run_the_native_kernels(cuda_device):
    """fp16 in, fp16 out (the reference's self-test dtype): served by the bf16 kernels, never by the
    eager fallback; compared against the fp32 oracle with the reference's tolerances."""
    from gpt_from_scratch_b200.ops import _lib
    from gpt_from_scratch_b200.ops.attention import apply_flash_attn, attention_reference
    g = torch.Generator(device="cuda").manual_seed(77)
    B, nh, S, D = 2, 3, 256, 64
    q, k, v = (torch.randn(B, nh, S, D, device=cuda_device, generator=g).half().requires_grad_() for _ in range(3))
    do = torch.randn(B, nh, S, D, device=cuda_device, generator=g).half()
    before = _lib.launch_count()
    o = apply_flash_attn(q, k, v, True)
    o.backward(do)
    assert _lib.launch_count() - before >= 2 and o.dtype == torch.float16 and q.grad.dtype == torch.float16
    qf, kf, vf = (t.detach().float().requires_grad_() for t in (q, k, v))
    of = attention_reference(qf, kf, vf, True)
    of.backward(do.float())
    _close(o, of, 2e-2, what="O")
    for name, a, b in (("O", o, of), ("dQ", q.grad, qf.grad), ("dK", k.grad, kf.grad), ("dV", v.grad, vf.grad)):
        _close(a, b, 5e-2, what=name)
        rel = (a.float() - b).norm() / (b.norm() + 1e-12)
        assert rel < 2e-2, f"{name}: relative error {rel:.4g}"
    with pytest.raises(ValueError):
        apply_flash_attn(q[..., :32], k[..., :32], v[..., :32], True)


@pytest.mark.parametrize("causal,D", [(True, 64), (False, 64), (True, 128)])
def test_flash_attention_growing_scores(cuda_device, causal, D):
    """Keys whose magnitude grows along the sequence: the row maximum rises by far more than 2^8
    from one key block to the next, so the head_dim-64 forward has to rescale the output it
    accumulates in tensor memory (with random-normal inputs the maximum settles in the first
    block and that path never runs). Some rows get a negative query, so their maximum stays."""
    from gpt_from_scratch_b200.ops.attention import apply_flash_attn, attention_reference
    g = torch.Generator(device="cuda").manual_seed(11)
    B, nh, S = 2, 3, 640
    q = torch.randn(B, nh, S, D, device=cuda_device, generator=g)
    k = torch.randn(B, nh, S, D, device=cuda_device, generator=g)
    v = torch.randn(B, nh, S, D, device=cuda_device, generator=g)
    ramp = torch.linspace(0.25, 6.0, S, device=cuda_device).view(1, 1, S, 1)
    k = k * ramp + 0.5 * ramp * torch.sign(q.mean(dim=2, keepdim=True))
    q[:, :, ::3] *= -1.0
    q, k, v = (t.bfloat16().requires_grad_() for t in (q, k, v))
    do = torch.randn(B, nh, S, D, device=cuda_device, generator=g).bfloat16()
    o = apply_flash_attn(q, k, v, causal)
    o.backward(do)
    qf, kf, vf = (t.detach().float().requires_grad_() for t in (q, k, v))
    of = attention_reference(qf, kf, vf, causal)
    of.backward(do.float())
    _close(o, of, 2e-2, what="O")
    for name, a, b in (("O", o, of), ("dQ", q.grad, qf.grad), ("dK", k.grad, kf.grad), ("dV", v.grad, vf.grad)):
        rel = (a.float() - b).norm() / (b.norm() + 1e-12)
        assert rel < 3e-2, f"{name}: relative error {rel:.4g}"


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,nh,S", [(1, 1, 1), (2, 1, 33), (1, 2, 63), (1, 1, 65), (2, 3, 127), (1, 2, 129), (3, 1, 193),
                                    (1, 3, 385), (3, 51, 257)])
def test_flash_attention_tile_edges(cuda_device, B, nh, S, D, causal):
    """Lengths around the tiles' edges (64 streamed rows, 32-row warp slices, 128-row items), and more items
    than pipelines. Tolerance: P and dS are rounded to bf16 (2^-9 relative), like the results."""
    from gpt_from_scratch_b200.ops.attention import apply_flash_attn, attention_reference
    g = torch.Generator(device="cuda").manual_seed(S * 2 + D)
    q, k, v = (torch.randn(B, nh, S, D, device=cuda_device, generator=g).bfloat16().requires_grad_() for _ in range(3))
    do = torch.randn(B, nh, S, D, device=cuda_device, generator=g).bfloat16()
    o = apply_flash_attn(q, k, v, causal)
    o.backward(do)
    qf, kf, vf = (t.detach().double().requires_grad_() for t in (q, k, v))
    of = attention_reference(qf, kf, vf, causal)
    of.backward(do.double())
    for name, a, b in (("O", o, of), ("dQ", q.grad, qf.grad), ("dK", k.grad, kf.grad), ("dV", v.grad, vf.grad)):
        if S == 1 and name in ("dQ", "dK"):     # a single key: zero up to fp32 sums in two orders
            assert a.float().abs().max() < 1e-3
            continue
        rel = (a.double() - b).norm() / b.norm()
        assert rel < 1e-2, f"{name}: relative error {rel:.4g}"


def test_flash_attention_noncausal_and_ragged(cuda_device):
    from gpt_from_scratch_b200.ops.attention import apply_flash_attn, attention_reference
    g = torch.Generator(device="cuda").manual_seed(3)
    for S, causal in ((192, True), (320, False), (64, True)):
        q, k, v = (torch.randn(1, 2, S, 64, device=cuda_device, generator=g).bfloat16().requires_grad_()
                   for _ in range(3))
        do = torch.randn(1, 2, S, 64, device=cuda_device, generator=g).bfloat16()
        o = apply_flash_attn(q, k, v, causal)
        o.backward(do)
        qf, kf, vf = (t.detach().float().requires_grad_() for t in (q, k, v))
        of = attention_reference(qf, kf, vf, causal)
        of.backward(do.float())
        _close(o, of, 1e-2, what=f"O S={S}")
        _close(q.grad, qf.grad, 5e-2, what=f"dQ S={S}")
        _close(k.grad, kf.grad, 5e-2, what=f"dK S={S}")
        _close(v.grad, vf.grad, 5e-2, what=f"dV S={S}")


@pytest.mark.parametrize("S,B,nh,D", [(256, 2, 4, 64), (128, 1, 2, 128)])
def test_fused_rope_attention_matches_composition(cuda_device, S, B, nh, D):
    from gpt_from_scratch_b200.ops.attention import attention_reference, fused_rope_attention
    from gpt_from_scratch_b200.ops.rope import rope_reference
    g = torch.Generator(device="cuda").manual_seed(9)
    qkv = torch.randn(S * B, 3 * nh * D, device=cuda_device, generator=g).bfloat16()
    pos = torch.arange(S, device=cuda_device, dtype=torch.float32)
    freqs = 10000.0 ** (-torch.arange(0, D, 2, device=cuda_device, dtype=torch.float32) / D)
    ang = pos[:, None] * freqs[None, :]
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    x = qkv.clone().requires_grad_()
    do = torch.randn(S * B, nh * D, device=cuda_device, generator=g).bfloat16()
    out = fused_rope_attention(x * 1, cos, sin, S, B, nh, D)
    out.backward(do)
    xf = qkv.float().requires_grad_()
    q, k, v = xf.view(S, B, 3, nh, D).unbind(2)
    qr, kr = rope_reference(q, cos, sin), rope_reference(k, cos, sin)
    of = attention_reference(qr.permute(1, 2, 0, 3), kr.permute(1, 2, 0, 3), v.permute(1, 2, 0, 3), True)
    of = of.permute(2, 0, 1, 3).reshape(S * B, nh * D)
    of.backward(do.float())
    _close(out, of, 1.5e-2, what="fused out")
    _close(x.grad, xf.grad, 6e-2, what="fused dqkv")
    rel = (x.grad.float() - xf.grad).norm() / xf.grad.norm()
    assert rel < 2e-2, rel


def test_rope_fwd_bwd(cuda_device):
    from gpt_from_scratch_b200.ops.rope import apply_rope, rope_reference
    S, B, nh, D = 96, 3, 5, 64
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn(S, B, nh, D, device=cuda_device, generator=g).bfloat16().requires_grad_()
    ang = torch.rand(S, D // 2, device=cuda_device, generator=g) * 6.28
    cos, sin = ang.cos(), ang.sin()
    y = apply_rope(x, cos, sin)
    gy = torch.randn_like(y)
    y.backward(gy)
    xf = x.detach().float().requires_grad_()
    yf = rope_reference(xf, cos, sin)
    yf.backward(gy.float())
    _close(y, yf, 2e-2, what="rope y")
    _close(x.grad, xf.grad, 2e-2, what="rope dx")
    # strided input (an unbind view of a packed buffer) must give the same answer
    packed = torch.randn(S, B, 3, nh, D, device=cuda_device, generator=g).bfloat16()
    q = packed[:, :, 0]
    _close(apply_rope(q, cos, sin), rope_reference(q.float(), cos, sin), 2e-2, what="rope strided")


@pytest.mark.parametrize("rows,H", [(64, 768), (1000, 2048), (33, 4096), (17, 8192), (4096, 768)])
def test_rmsnorm_fwd_bwd(cuda_device, rows, H):
    from gpt_from_scratch_b200.ops.rmsnorm import rmsnorm, rmsnorm_reference
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = (torch.randn(rows, H, device=cuda_device, generator=g) * 2).bfloat16().requires_grad_()
    w = (1 + 0.1 * torch.randn(H, device=cuda_device, generator=g)).bfloat16().requires_grad_()
    dy = torch.randn(rows, H, device=cuda_device, generator=g).bfloat16()
    y = rmsnorm(x, w, 1e-5)
    y.backward(dy)
    xf, wf = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    yf = rmsnorm_reference(xf, wf, 1e-5)
    yf.backward(dy.float())
    _close(y, yf, 3e-2, 1e-2, what="rmsnorm y")
    _close(x.grad, xf.grad, 3e-2, 2e-2, what="rmsnorm dx")
    rel = (w.grad.float() - wf.grad).norm() / wf.grad.norm()
    assert rel < 1e-2, f"rmsnorm dw rel {rel}"


def test_swiglu_fwd_bwd(cuda_device):
    from gpt_from_scratch_b200.ops.swiglu import swiglu, swiglu_reference
    g = torch.Generator(device="cuda").manual_seed(4)
    gu = torch.randn(300, 2 * 1408, device=cuda_device, generator=g).bfloat16().requires_grad_()
    da = torch.randn(300, 1408, device=cuda_device, generator=g).bfloat16()
    a = swiglu(gu)
    a.backward(da)
    gf = gu.detach().float().requires_grad_()
    af = swiglu_reference(gf)
    af.backward(da.float())
    _close(a, af, 2e-2, 1e-2, what="swiglu")
    _close(gu.grad, gf.grad, 2e-2, 1e-2, what="swiglu grad")


@pytest.mark.parametrize("M,H,I", [(256, 256, 384), (1000, 768, 704), (2048, 768, 3072)])
def test_fused_mlp_matches_unfused(cuda_device, M, H, I):
    """SwiGLU folded into the GEMM epilogues == separate GEMM / activation kernels."""
    from gpt_from_scratch_b200.ops.mlp_fused import _FusedMLP
    g = torch.Generator(device="cuda").manual_seed(M + I)
    x = torch.randn(M, H, device=cuda_device, generator=g).bfloat16()
    w_gu = (torch.randn(2 * I, H, device=cuda_device, generator=g) * 0.05).bfloat16()
    w_dn = (torch.randn(H, I, device=cuda_device, generator=g) * 0.05).bfloat16()
    res = torch.randn(M, H, device=cuda_device, generator=g).bfloat16()
    dout = torch.randn(M, H, device=cuda_device, generator=g).bfloat16()
    xa, wa, wb = x.clone().requires_grad_(), w_gu.clone().requires_grad_(), w_dn.clone().requires_grad_()
    ya = _FusedMLP.apply(xa, wa, wb, res, None, None)
    ya.backward(dout)
    xf, wf, wg = x.float().requires_grad_(), w_gu.float().requires_grad_(), w_dn.float().requires_grad_()
    gu = xf @ wf.t()
    act = torch.nn.functional.silu(gu[:, :I]) * gu[:, I:]
    yf = act @ wg.t() + res.float()
    yf.backward(dout.float())
    for name, a, b in (("y", ya, yf), ("dx", xa.grad, xf.grad), ("dW_gu", wa.grad, wf.grad), ("dW_down", wb.grad, wg.grad)):
        rel = (a.float() - b).norm() / (b.norm() + 1e-9)
        assert rel < 1.5e-2, f"{name}: relative error {rel:.4g}"


@pytest.mark.parametrize("M,H,I", [(512, 256, 384), (1000, 768, 704), (2048, 320, 1536)])
@pytest.mark.parametrize("pair", [False, True])
def test_swiglu_gemm_epilogues(cuda_device, M, H, I, pair):
    """SwiGLU forward / backward folded into the GEMM epilogue (single-CTA and CTA-pair kernels)
    against an fp32 reference of the same two steps."""
    from gpt_from_scratch_b200.ops import gemm as gemm_ops
    from gpt_from_scratch_b200.ops.mlp_fused import swiglu_gemm_bwd, swiglu_gemm_fwd
    g = torch.Generator(device="cuda").manual_seed(M + I + int(pair))
    x = torch.randn(M, H, device=cuda_device, generator=g).bfloat16()
    w_gu = (torch.randn(2 * I, H, device=cuda_device, generator=g) * 0.05).bfloat16()
    w_dn = (torch.randn(H, I, device=cuda_device, generator=g) * 0.05).bfloat16()
    dy = torch.randn(M, H, device=cuda_device, generator=g).bfloat16()
    with gemm_ops.pair_min_tiles(1 if pair else 10 ** 9):
        gu, act = swiglu_gemm_fwd(x, w_gu)
        dgu = swiglu_gemm_bwd(dy, w_dn, gu)
    gu_ref = x.float() @ w_gu.float().t()
    _close(gu, gu_ref, 2e-2, 2e-2, what="gate_up projection")
    guf = gu.float().requires_grad_()          # the kernels compute act and the gradient from the bf16 projection
    act_ref = torch.nn.functional.silu(guf[:, :I]) * guf[:, I:]
    _close(act, act_ref, 2e-2, 2e-2, what="act")
    dact = (dy.float() @ w_dn.float()).bfloat16().float()
    act_ref.backward(dact)
    _close(dgu, guf.grad, 3e-2, 3e-2, what="d_gate_up")


def test_dropout_residual_kernel(cuda_device):
    """Fused residual + dropout: keep rate, scaling, regenerated mask in the backward."""
    from gpt_from_scratch_b200.ops.dropout import dropout_add
    g = torch.Generator(device="cuda").manual_seed(11)
    x = (torch.rand(512, 768, device=cuda_device, generator=g) * 2 + 2).bfloat16().requires_grad_()   # in [2, 4]
    res = (torch.randn(512, 768, device=cuda_device, generator=g) * 0.25).bfloat16().requires_grad_()
    host_gen = torch.Generator().manual_seed(5)
    p = 0.25
    y = dropout_add(x, res, p, True, generator=host_gen)
    kept = (y.float() - res.float()).abs() > 0.5            # x is bounded away from zero
    rate = kept.float().mean().item()
    assert abs(rate - (1 - p)) < 0.01, rate
    expect = res.float() + torch.where(kept, x.float() / (1 - p), torch.zeros_like(x.float())).bfloat16().float()
    assert (y.float() - expect).abs().max() < 0.07
    dy = torch.randn_like(y)
    y.backward(dy)
    assert torch.equal(res.grad, dy)
    dx_expect = torch.where(kept, dy.float() / (1 - p), torch.zeros_like(dy.float()))
    assert (x.grad.float() - dx_expect).abs().max() < 0.05
    assert torch.equal(x.grad != 0, kept & (dy != 0))        # same mask in both directions
    # a different call draws a different mask; evaluation mode is the plain sum
    y2 = dropout_add(x.detach(), res.detach(), p, True, generator=host_gen)
    assert not torch.equal(y2, y.detach())
    assert torch.equal(dropout_add(x.detach(), res.detach(), p, False), res.detach() + x.detach())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,nh,S,D,causal", [(1, 1, 1, 64, True), (3, 5, 333, 64, False), (2, 3, 129, 128, True)])
def test_flash_attention_api_dtypes_and_layouts(cuda_device, dtype, B, nh, S, D, causal):
    """bf16 and fp16 tensors (the latter through the cast and fp16-storing variants), contiguous and as
    transposed views of a [B, S, nh, D] projection, at row counts around the pre-pass' 4-row groups. The
    bf16 roundings of P, dS and the inputs (2^-9 each) bound the relative error."""
    from gpt_from_scratch_b200.ops.attention import apply_flash_attn, attention_reference
    g = torch.Generator(device="cuda").manual_seed(S + D)
    for transposed in (False, True):
        shape = (B, S, nh, D) if transposed else (B, nh, S, D)
        q, k, v, do = (torch.randn(shape, device=cuda_device, generator=g).to(dtype) for _ in range(4))
        if transposed:
            q, k, v, do = (t.transpose(1, 2) for t in (q, k, v, do))
        q, k, v = (t.detach().requires_grad_() for t in (q, k, v))
        o = apply_flash_attn(q, k, v, causal)
        grads = torch.autograd.grad(o, (q, k, v), do)
        qf, kf, vf = (t.detach().float().requires_grad_() for t in (q, k, v))
        of = attention_reference(qf, kf, vf, causal)
        refs = torch.autograd.grad(of, (qf, kf, vf), do.float())
        assert o.dtype == dtype and all(t.dtype == dtype for t in grads)
        for name, a, b in zip(("O", "dQ", "dK", "dV"), (o, *grads), (of, *refs)):
            # one token: dQ and dK are exactly zero, what is left is the rounding of dO and V in dP - D
            err = (a.float() - b).norm()
            assert err <= 2e-2 * b.norm() + (2e-2 * D ** 0.5 if S == 1 else 0.0), (name, err.item(), b.norm().item())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("Sk,Sv", [(200, 130), (130, 200), (300, 300)])
def test_flash_attention_longer_keys(cuda_device, dtype, Sk, Sv):
    """k and v of more rows than q are read with their own strides: the first rows, one per query, also where all
    tensors are contiguous. The rows past them get no gradient. Shorter ones are refused. Tolerance as in
    test_flash_attention_api_dtypes_and_layouts."""
    from gpt_from_scratch_b200.ops.attention import apply_flash_attn, attention_reference
    B, nh, S, D = 2, 3, 130, 64
    g = torch.Generator(device="cuda").manual_seed(Sk)
    q, k, v, do = (torch.randn(B, nh, n, D, device=cuda_device, generator=g).to(dtype).requires_grad_()
                   for n in (S, Sk, Sv, S))
    for causal in (True, False):
        o = apply_flash_attn(q, k, v, causal)
        grads = torch.autograd.grad(o, (q, k, v), do.detach())
        qf, kf, vf = (t.detach().float().requires_grad_() for t in (q, k, v))
        of = attention_reference(qf, kf[:, :, :S], vf[:, :, :S], causal)
        refs = torch.autograd.grad(of, (qf, kf, vf), do.detach().float())
        for name, a, b in zip(("O", "dQ", "dK", "dV"), (o, *grads), (of, *refs)):
            assert a.shape == b.shape and (a.float() - b).norm() <= 2e-2 * b.norm(), name
    for wrong in (k[:, :, :S - 1], k[:, :1], k[:1], k[..., :32], k[0]):
        with pytest.raises(ValueError, match="cover q"):
            apply_flash_attn(q, wrong, v)
        with pytest.raises(ValueError, match="cover q"):
            apply_flash_attn(q, k, wrong)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_flash_attention_misaligned_tensors(cuda_device, dtype):
    """Contiguous q, k, v and gradient at odd addresses give what aligned copies of them give."""
    from gpt_from_scratch_b200.ops.attention import apply_flash_attn
    B, nh, S, D = 2, 3, 70, 64
    g = torch.Generator(device="cuda").manual_seed(1)
    flat = [torch.randn(1 + B * nh * S * D, device=cuda_device, generator=g).to(dtype) for _ in range(4)]
    results = []
    for copy in (True, False):
        q, k, v, do = (t[1:].view(B, nh, S, D) for t in flat)
        if copy:
            q, k, v, do = (t.clone() for t in (q, k, v, do))
        q, k, v = (t.detach().requires_grad_() for t in (q, k, v))
        o = apply_flash_attn(q, k, v)
        results.append((o, *torch.autograd.grad(o, (q, k, v), do)))
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("B,nh,S,D", [(2, 3, 129, 64), (1, 2, 300, 128)])
def test_flash_attention_fp16_output_may_be_written_to(cuda_device, B, nh, S, D):
    """The output of fp16 tensors belongs to the caller: written to in place, the gradients stay what they are. (A bf16
    output is saved itself, and autograd says so.)"""
    from gpt_from_scratch_b200.ops.attention import apply_flash_attn
    g = torch.Generator(device="cuda").manual_seed(1)
    t = [torch.randn(B, S, nh, D, device=cuda_device, generator=g).half().transpose(1, 2) for _ in range(4)]
    grads = []
    for write in (False, True):
        q, k, v = (x.detach().requires_grad_() for x in t[:3])
        o = apply_flash_attn(q, k, v)
        if write:
            o += 1.0
        grads.append(torch.autograd.grad(o, (q, k, v), t[3]))
    assert all(torch.equal(a, b) for a, b in zip(*grads))
    q, k, v = (x.detach().bfloat16().requires_grad_() for x in t[:3])
    o = apply_flash_attn(q, k, v)
    o += 1.0
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        o.sum().backward()


@pytest.mark.parametrize("B,nh,S,causal", [
    (1, 148, 100, True), (1, 149, 100, True),        # one item per SM, one more
    (1, 10, 2048, True), (1, 13, 2048, True),        # more items that find room behind short ones, and that do not
    (1, 19, 1024, True), (1, 20, 1024, True), (1, 9, 2048, False), (1, 10, 2048, False)])
def test_flash_forward_128_both_kernels(cuda_device, B, nh, S, causal):
    """head_dim 128, both sides of the line between its two forward kernels, in bf16 and fp16 (with and without the copy
    for the backward). Tolerance: one bf16 rounding of the output and of P (2^-9 each); fp16 inputs are rounded to bf16."""
    from gpt_from_scratch_b200.ops.attention import apply_flash_attn, attention_reference
    g = torch.Generator(device="cuda").manual_seed(S + nh)
    q, k, v = (torch.randn(B, nh, S, 128, device=cuda_device, generator=g).bfloat16() for _ in range(3))
    ref = attention_reference(q.double(), k.double(), v.double(), causal)
    assert (apply_flash_attn(q, k, v, causal).double() - ref).norm() < 4e-3 * ref.norm()
    q, k, v = (t.half() for t in (q, k, v))
    plain = apply_flash_attn(q, k, v, causal)
    assert (plain.double() - ref).norm() < 4e-3 * ref.norm()
    assert torch.equal(apply_flash_attn(q.requires_grad_(), k, v, causal).detach(), plain)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("nh", [4, 40])
def test_flash_forward_128_largest_probability_is_exact(cuda_device, nh, causal):
    """Scores of standard deviation 4: a row is mostly its largest probability, which is 1 before the division, exact in
    bf16, if the running maximum is the true one. What is left is the output's own rounding (1.66e-3 rms for bf16) and
    a part of P's: 1.74e-3 measured; 2.04e-3 and 2.16e-3 with a maximum that lags by up to 2^8."""
    from gpt_from_scratch_b200.ops.attention import apply_flash_attn, attention_reference
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k = (2 * torch.randn(1, nh, 1024, 128, device=cuda_device, generator=g) for _ in range(2))
    q, k, v = (t.bfloat16() for t in (q, k, torch.randn(1, nh, 1024, 128, device=cuda_device, generator=g)))
    ref = attention_reference(q.double(), k.double(), v.double(), causal)
    assert (apply_flash_attn(q, k, v, causal).double() - ref).norm() < 1.9e-3 * ref.norm()


@pytest.mark.parametrize("rows,H", [(1, 8), (9, 256), (1184, 264), (1185, 264), (2500, 8), (2500, 1024), (2500, 1032),
                                    (2500, 2048), (2500, 2056), (80000, 64)])
@pytest.mark.parametrize("residual", [False, True])
def test_rmsnorm_backward_ring(cuda_device, rows, H, residual):
    """Both sides of the lines at 1024 and 2048 columns and at a CTA per SM, a last vector that not every lane has, more
    than 32 rows per warp; against float64, weight gradients included. The normalised value is rounded to bf16
    (2^-9), as are the results."""
    from gpt_from_scratch_b200.ops import _lib
    lib = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(rows + H)
    rnd = lambda *s: torch.randn(*s, device=cuda_device, generator=g).bfloat16()  # noqa: E731
    x, dy, res, w = rnd(rows, H), rnd(rows, H), rnd(rows, H), (rnd(H).float() * 0.2 + 1).bfloat16()
    rstd = (x.float().pow(2).mean(1) + 1e-5).rsqrt().contiguous()
    dx = torch.full((rows + 1, H), 7.0, device=cuda_device, dtype=torch.bfloat16)
    dw = torch.empty(H, device=cuda_device, dtype=torch.bfloat16)
    partial = torch.empty(lib.gfs_rmsnorm_bwd_parts(rows) * H, device=cuda_device)
    assert lib.gfs_rmsnorm_bwd(dy.data_ptr(), x.data_ptr(), w.data_ptr(), rstd.data_ptr(), res.data_ptr() if residual else 0,
                               dx.data_ptr(), dw.data_ptr(), partial.data_ptr(), rows, H, 0, _lib.stream_ptr()) == 0
    xd, dyd, wd, r = x.double(), dy.double(), w.double(), rstd.double()[:, None]
    ref = r * dyd * wd - xd * r ** 3 * (dyd * wd * xd).mean(1, keepdim=True) + (res.double() if residual else 0)
    assert (dx[rows] == 7.0).all()
    assert (dx[:rows].double() - ref).norm() < 3e-3 * ref.norm()
    ref_w = (dyd * (xd * r)).sum(0)
    assert (dw.double() - ref_w).norm() < 6e-3 * (dyd * xd * r).pow(2).sum(0).sqrt().norm()


@pytest.mark.parametrize("rows,H", [(1, 8), (9, 1024), (77, 1032), (33, 2048), (5, 4104), (1184, 264), (1185, 264),
                                    (2500, 1024), (2500, 1032), (2500, 2048), (1300, 2056)])
@pytest.mark.parametrize("p", [0.0, 0.1, 0.999])
def test_rmsnorm_with_dropout(cuda_device, rows, H, p):
    """The norm that makes its input from a branch's dropped output, and the norm's backward that also writes that branch's
    gradient: the bits of the two kernels each, at the lines of both (columns kept in registers, rows per CTA)."""
    from gpt_from_scratch_b200.ops import _lib
    lib, st, seed = _lib.lib(), _lib.stream_ptr, 0x9876543210fedcba
    g = torch.Generator(device="cuda").manual_seed(rows + H)
    rnd = lambda *s: torch.randn(*s, device=cuda_device, generator=g).bfloat16()  # noqa: E731
    z, res, dy, w = rnd(rows, H), rnd(rows, H), rnd(rows, H), (rnd(H).float() * 0.2 + 1).bfloat16()
    out = [[torch.full((rows + 1, H), 7.0, device=cuda_device, dtype=torch.bfloat16) for _ in range(4)] for _ in range(2)]
    rstd = [torch.zeros(rows, device=cuda_device) for _ in range(2)]
    partial = [torch.zeros(lib.gfs_rmsnorm_bwd_parts(rows) * H, device=cuda_device) for _ in range(2)]
    P = lambda t: t.data_ptr()  # noqa: E731
    x, y, dx, dm = out[0]
    assert lib.gfs_dropout_residual(P(z), P(res), P(x), rows * H, p, seed, 0, st()) == 0
    assert lib.gfs_rmsnorm_fwd(P(x), P(w), P(y), P(rstd[0]), rows, H, 1e-5, st()) == 0
    assert lib.gfs_rmsnorm_bwd(P(dy), P(x), P(w), P(rstd[0]), P(res), P(dx), 0, P(partial[0]), rows, H, 0, st()) == 0
    assert lib.gfs_dropout_residual(P(dx), 0, P(dm), rows * H, p, seed, 1, st()) == 0
    x2, y2, dx2, dm2 = out[1]
    assert lib.gfs_dropout_residual_norm(P(z), P(res), P(x2), P(w), P(y2), P(rstd[1]), rows, H, 1e-5, p, seed, st()) == 0
    rc = lib.gfs_rmsnorm_bwd_dropout(P(dy), P(x2), P(w), P(rstd[1]), P(res), P(dx2), P(dm2), P(partial[1]), rows, H, p, seed,
                                     st())
    assert rc == (1 if rows <= 1184 or H > 2048 else 0)
    assert torch.equal(x, x2) and torch.equal(y, y2) and torch.equal(rstd[0], rstd[1])
    if rc == 0:
        assert torch.equal(dx, dx2) and torch.equal(dm, dm2) and torch.equal(partial[0], partial[1])


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,nh,S", [(7, 23, 333), (5, 30, 70), (2, 75, 257), (1, 160, 640)])
def test_flash_attention_many_items(cuda_device, B, nh, S, causal):
    """More work items than SMs at head_dim 64: pairs of query tiles with and without a second one, one to five key blocks;
    the output once more in fp16, which is stored twice."""
    from gpt_from_scratch_b200.ops.attention import apply_flash_attn, attention_reference
    g = torch.Generator(device="cuda").manual_seed(S)
    for dtype in (torch.bfloat16, torch.float16):
        q, k, v = (torch.randn(B, nh, S, 64, device=cuda_device, generator=g).to(dtype).requires_grad_() for _ in range(3))
        do = torch.randn(B, nh, S, 64, device=cuda_device, generator=g).to(dtype)
        o = apply_flash_attn(q, k, v, causal)
        got = (o, *torch.autograd.grad(o, (q, k, v), do))
        qf, kf, vf = (t.detach().bfloat16().float().requires_grad_() for t in (q, k, v))
        of = attention_reference(qf, kf, vf, causal)
        for name, a, b in zip(("O", "dQ", "dK", "dV"), got, (of, *torch.autograd.grad(of, (qf, kf, vf), do.float()))):
            rel = (a.float() - b).norm() / b.norm()
            assert rel < 1e-2, f"{name}: relative error {rel:.4g}"       # as in test_flash_attention_tile_edges


@pytest.mark.parametrize("op", ["rmsnorm", "linear"])
def test_first_call_may_be_captured(cuda_device, op):
    """A process whose first use of the library is inside a graph capture: what is set up on first use must not invalidate
    the capture. rmsnorm: more rows than two CTAs of eight warps per SM have warps, so that its backward is the kernel
    with bounded waits, which has status words."""
    code = f"""
import torch
from gpt_from_scratch_b200.ops import _lib
from gpt_from_scratch_b200.ops.gemm import gemm_bf16
from gpt_from_scratch_b200.ops.rmsnorm import rmsnorm, rmsnorm_reference
g = torch.Generator(device='cuda').manual_seed(1)
x, dy = (torch.randn(2500, 256, device='cuda', generator=g).bfloat16() for _ in range(2))
w = torch.ones(256, device='cuda', dtype=torch.bfloat16).requires_grad_()
x.requires_grad_()
graph = torch.cuda.CUDAGraph()
torch.cuda.synchronize()
with torch.cuda.graph(graph):
    if {op!r} == 'rmsnorm':
        got, = torch.autograd.grad(rmsnorm(x, w, 1e-5), (x,), dy)
    else:
        got = gemm_bf16(x.detach(), dy[:256])
graph.replay()
if {op!r} == 'rmsnorm':
    xd = x.detach().double().requires_grad_()
    ref, = torch.autograd.grad(rmsnorm_reference(xd, w.detach().double(), 1e-5), (xd,), dy.double())
else:
    ref = x.detach().double() @ dy[:256].double().t()
torch.cuda.synchronize()
_lib.raise_on_status()
assert (got.double() - ref).norm() < 3e-3 * ref.norm()      # results rounded to bf16, 2^-9
print('captured')
"""
    run = subprocess.run([sys.executable, "-c", code], cwd=pathlib.Path(__file__).resolve().parent.parent, text=True,
                         capture_output=True, timeout=300)
    assert run.returncode == 0 and "captured" in run.stdout, run.stderr[-2000:]


@pytest.mark.parametrize("repeat", [1, 12])
@pytest.mark.parametrize("H", [8, 264, 768, 4200])
def test_embedding_backward_runs_behind_one_load_of_keys(cuda_device, H, repeat):
    """Runs around the 31 keys that a warp's first load brings, and the 32 of each further one, between runs of one row, from
    the first position to the last; positions that several warps share and, with more of them, one each: bit for bit the fp32
    sum in the order of the positions, rounded once."""
    from gpt_from_scratch_b200.ops.embedding import embedding_bwd_native
    counts = [3, 1, 30, 1, 2, 62, 63, 1, 94, 95, 96, 1] * repeat
    g = torch.Generator(device="cuda").manual_seed(H)
    ids = torch.repeat_interleave(torch.arange(len(counts), device=cuda_device), torch.tensor(counts, device=cuda_device))
    ids = ids[torch.randperm(ids.numel(), generator=g, device=cuda_device)].view(1, -1)
    dout = torch.randn(ids.shape[1], 1, H, device=cuda_device, generator=g).bfloat16()
    dW = torch.randn(len(counts), H, device=cuda_device, generator=g).bfloat16()
    acc = dW.float()
    embedding_bwd_native(ids, dout, dW, 0, len(counts), accumulate=True)
    for s in range(ids.shape[1]):
        acc[ids[0, s]] += dout[s, 0].float()
    assert torch.equal(dW, acc.bfloat16())


@pytest.mark.parametrize("M,H,I,pair", [(130, 256, 384, False), (3000, 264, 1528, False), (512, 256, 384, True),
                                        (512, 1032, 384, True)])
def test_swiglu_fused_and_alone_agree(cuda_device, M, H, I, pair):
    """The activation of every product with a SwiGLU epilogue (tiles, persistent CTAs, pairs with sixteen and eight epilogue
    warps) has the bits of the kernel that makes it from the stored projection."""
    from gpt_from_scratch_b200.ops import gemm as gemm_ops
    from gpt_from_scratch_b200.ops.mlp_fused import swiglu_gemm_fwd
    from gpt_from_scratch_b200.ops.swiglu import swiglu
    g = torch.Generator(device="cuda").manual_seed(M + H)
    x = torch.randn(M, H, device=cuda_device, generator=g).bfloat16()
    w = (torch.randn(2 * I, H, device=cuda_device, generator=g) * 0.2).bfloat16()
    with gemm_ops.pair_min_tiles(1 if pair else 10 ** 9):
        gu, act = swiglu_gemm_fwd(x, w)
    assert torch.equal(act, swiglu(gu))
