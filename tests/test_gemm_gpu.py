"""Numerics of the tcgen05 GEMM against an fp32 PyTorch reference (all operand layouts)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(a, b, a_mn, b_mn, addend):
    A = a.float().t() if a_mn else a.float()
    B = b.float() if b_mn else b.float().t()
    y = A @ B
    if addend is not None:
        y = y + addend.float()
    return y


def _check(out, ref, K):
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item() + 1e-6
    # bf16 output rounding (2^-8 relative) plus accumulation-order noise
    assert err <= 1.5e-2 * scale + 1e-3, f"max err {err} vs scale {scale} (K={K})"


SHAPES = [
    (128, 256, 64), (128, 128, 128), (256, 512, 256), (384, 768, 768), (1000, 1384, 328),
    (130, 8, 72), (2048, 2304, 768), (96, 4096, 1024),
]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_gemm_layouts(cuda_device, M, N, K, a_mn, b_mn):
    from gpt_from_scratch_b200.ops.gemm import gemm_bf16
    if (a_mn and M % 8) or (b_mn and N % 8) or K % 8:
        pytest.skip("pitch must be a multiple of 8 elements")
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + K)
    a = torch.randn((K, M) if a_mn else (M, K), device=cuda_device, generator=g).bfloat16()
    b = torch.randn((K, N) if b_mn else (N, K), device=cuda_device, generator=g).bfloat16()
    out = gemm_bf16(a, b, a_mn_major=a_mn, b_mn_major=b_mn)
    _check(out, _ref(a, b, a_mn, b_mn, None), K)


@pytest.mark.parametrize("split", [0, 1, 2, 5])
def test_gemm_splitk_and_addend(cuda_device, split):
    from gpt_from_scratch_b200.ops.gemm import gemm_bf16
    M, N, K = 768, 768, 4096
    g = torch.Generator(device="cuda").manual_seed(5)
    a = torch.randn((K, M), device=cuda_device, generator=g).bfloat16()
    b = torch.randn((K, N), device=cuda_device, generator=g).bfloat16()
    r = torch.randn((M, N), device=cuda_device, generator=g).bfloat16()
    out = r.clone()
    gemm_bf16(a, b, a_mn_major=True, b_mn_major=True, out=out, addend=out, force_split=split)
    _check(out, _ref(a, b, True, True, r), K)
    out2 = r.clone()
    gemm_bf16(a, b, a_mn_major=True, b_mn_major=True, out=out2, addend=out2, force_split=split)
    assert torch.equal(out, out2), "split-K must be deterministic"


def test_gemm_strided_views(cuda_device):
    """Operands and output that are column slices of wider buffers (pitch != width)."""
    from gpt_from_scratch_b200.ops.gemm import gemm_bf16
    g = torch.Generator(device="cuda").manual_seed(11)
    big_a = torch.randn((512, 1024), device=cuda_device, generator=g).bfloat16()
    big_b = torch.randn((640, 1024), device=cuda_device, generator=g).bfloat16()
    a = big_a[:, 256:768]
    b = big_b[:, 128:640]
    big_c = torch.zeros((512, 1280), device=cuda_device, dtype=torch.bfloat16)
    out = big_c[:, 640:]
    gemm_bf16(a, b, out=out)
    _check(out, a.float() @ b.float().t(), 512)
    assert big_c[:, :640].abs().max().item() == 0


def test_gemm_rope_epilogue(cuda_device):
    """Rotary embedding applied by the GEMM epilogue to the q and k thirds of a qkv projection."""
    from gpt_from_scratch_b200.ops.gemm import gemm_bf16
    from gpt_from_scratch_b200.ops.rope import rope_reference
    S, B, nh, D, K = 64, 3, 4, 64, 256
    g = torch.Generator(device="cuda").manual_seed(21)
    x = torch.randn(S * B, K, device=cuda_device, generator=g).bfloat16()
    w = (torch.randn(3 * nh * D, K, device=cuda_device, generator=g) * 0.05).bfloat16()
    ang = torch.rand(S, D // 2, device=cuda_device, generator=g) * 6.28
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    out = gemm_bf16(x, w, rope=(cos, sin, 2 * nh * D, D, B))
    ref = (x.float() @ w.float().t()).view(S, B, 3, nh, D)
    q, k, v = ref.unbind(2)
    ref = torch.stack((rope_reference(q, cos, sin), rope_reference(k, cos, sin), v), dim=2).view(S * B, -1)
    _check(out, ref, K)


@pytest.mark.parametrize("M,N,K", [(256, 256, 64), (512, 768, 256), (1024, 1280, 328), (2000, 520, 1024),
                                   (4096, 2304, 768)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_gemm_cta_pair_kernel(cuda_device, M, N, K, a_mn, b_mn):
    """The cta_group::2 kernel (one 256x256 tile per CTA pair) against the fp32 reference."""
    from gpt_from_scratch_b200.ops.gemm import gemm_bf16
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn((K, M) if a_mn else (M, K), device=cuda_device, generator=g).bfloat16()
    b = torch.randn((K, N) if b_mn else (N, K), device=cuda_device, generator=g).bfloat16()
    r = torch.randn((M, N), device=cuda_device, generator=g).bfloat16()
    out = gemm_bf16(a, b, a_mn_major=a_mn, b_mn_major=b_mn, pair=True)
    _check(out, _ref(a, b, a_mn, b_mn, None), K)
    out2 = r.clone()
    gemm_bf16(a, b, a_mn_major=a_mn, b_mn_major=b_mn, out=out2, addend=out2, pair=True)
    _check(out2, _ref(a, b, a_mn, b_mn, r), K)


def test_grouped_weight_gradients(cuda_device):
    """Several weight-gradient problems in one grouped launch (parked, then flushed) against
    the fp32 reference; one of them accumulates into an existing gradient."""
    from gpt_from_scratch_b200.ops import gemm as gemm_ops

    class Sink:  # the two methods of GradSink the GEMM layer uses, on a plain tensor
        def __init__(self, t, accumulate):
            self.t, self.acc, self.finished = t, accumulate, False

        def target(self):
            return self.t

        def consume_accumulate(self):
            return self.acc

        def done(self):
            self.finished = True

    g = torch.Generator(device="cuda").manual_seed(7)
    T = 1536  # tokens (the contraction)
    shapes = [(768, 768), (2304, 768), (768, 3072), (384, 264)]
    flat = torch.randn(sum(o * i for o, i in shapes), device=cuda_device, generator=g).bfloat16()
    before = flat.clone()
    sinks, operands, off = [], [], 0
    for n, (o, i) in enumerate(shapes):
        dy = torch.randn(T, o, device=cuda_device, generator=g).bfloat16()
        x = torch.randn(T, i, device=cuda_device, generator=g).bfloat16()
        sinks.append(Sink(flat[off:off + o * i].view(o, i), accumulate=(n == 1)))
        operands.append((dy, x))
        off += o * i
    with gemm_ops.pair_min_tiles(10 ** 6):   # park everything until the explicit flush
        for n, ((dy, x), sk) in enumerate(zip(operands, sinks)):
            gemm_ops.linear_wgrad_to_sink(dy, x, sk)
            if n == 2:
                assert not any(s_.finished for s_ in sinks)   # parked, nothing launched yet
        gemm_ops.flush_wgrad()   # (the fourth problem filled the group and launched it already)
    torch.cuda.synchronize()
    off = 0
    for n, ((dy, x), sk, (o, i)) in enumerate(zip(operands, sinks, shapes)):
        assert sk.finished
        ref = dy.float().t() @ x.float()
        if n == 1:
            ref = ref + before[off:off + o * i].view(o, i).float()
        _check(sk.t, ref, T)
        off += o * i


@pytest.mark.parametrize("bn", [64, 128, 256])
@pytest.mark.parametrize("split", [1, 2, 3, 4, 8])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_gemm_tile_kernels(cuda_device, bn, split, a_mn, b_mn):
    """One tile per CTA / CTA pair with K split over the cluster: row, column and K remainders, fewer rows than a
    tile, addend aliasing the output; tolerance as in _check (one bf16 rounding of fp32 sums)."""
    from gpt_from_scratch_b200.ops import _lib
    if bn == 256 and split == 8:
        pytest.skip("four pairs at most")
    g = torch.Generator(device="cuda").manual_seed(bn + split)
    for M, N, K in ((8, 8, 64 * split), (136, 72, 64 * split + 8), (264, 520, 1032)):
        a = torch.randn((K, M) if a_mn else (M, K), device=cuda_device, generator=g).bfloat16()
        b = torch.randn((K, N) if b_mn else (N, K), device=cuda_device, generator=g).bfloat16()
        c = torch.randn(M, N, device=cuda_device, generator=g).bfloat16()
        ref = _ref(a, b, a_mn, b_mn, c)
        kb = (K + 63) // 64
        rc = _lib.lib().gfs_gemm_tile(a.data_ptr(), b.data_ptr(), c.data_ptr(), c.data_ptr(), M, N, K, a.stride(0),
                                      b.stride(0), N, N, int(a_mn), int(b_mn), 0, 0, 0, 0, 1, 0, 0, 0, bn, split,
                                      _lib.stream_ptr())
        if -(-kb // split) * (split - 1) >= kb:
            assert rc == -1       # a CTA would have no K block
            continue
        assert rc == 0
        _check(c, ref, K)


@pytest.mark.parametrize("bn,split", [(64, 1), (64, 3), (128, 2), (256, 1), (256, 2)])
def test_gemm_tile_epilogues(cuda_device, bn, split):
    """Rotary and SwiGLU epilogues and the grouped weight gradients of the tile kernels against fp32."""
    import ctypes
    from gpt_from_scratch_b200.ops import _lib
    lib = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(7 * bn + split)
    rnd = lambda *s: torch.randn(*s, device=cuda_device, generator=g).bfloat16()  # noqa: E731
    S, B, nh, D, K, I = 47, 3, 3, 64, 328, 200
    M = S * B
    x, w = rnd(M, K), rnd(3 * nh * D, K)
    ang = torch.rand(S, D // 2, device=cuda_device, generator=g)
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    out = torch.empty(M, 3 * nh * D, device=cuda_device, dtype=torch.bfloat16)
    assert lib.gfs_gemm_tile(x.data_ptr(), w.data_ptr(), out.data_ptr(), 0, M, 3 * nh * D, K, K, K, out.stride(0), 0, 0, 0,
                             cos.data_ptr(), sin.data_ptr(), 2 * nh * D, D, B, 0, 0, 0, bn, split, _lib.stream_ptr()) == 0
    from gpt_from_scratch_b200.ops.rope import rope_reference
    ref = (x.float() @ w.float().t()).view(S, B, 3 * nh, D)
    ref[:, :, :2 * nh] = rope_reference(ref[:, :, :2 * nh], cos, sin)
    _check(out, ref.view(M, -1), K)

    wg, wd, dy = rnd(2 * I, K) * 0.1, rnd(K, I) * 0.1, rnd(M, K)
    gu, act, dgu = (torch.empty(M, n, device=cuda_device, dtype=torch.bfloat16) for n in (2 * I, I, 2 * I))
    assert lib.gfs_gemm_tile(x.data_ptr(), wg.data_ptr(), gu.data_ptr(), 0, M, I, K, K, K, 2 * I, 0, 0, 0, 0, 0, 0, 0, 1,
                             1, act.data_ptr(), I, bn, split, _lib.stream_ptr()) == 0
    _check(gu, x.float() @ wg.float().t(), K)
    guf = gu.float().requires_grad_()          # act and the gradient are computed from the bf16 projection
    act_ref = torch.nn.functional.silu(guf[:, :I]) * guf[:, I:]
    _check(act, act_ref.detach(), K)
    assert lib.gfs_gemm_tile(dy.data_ptr(), wd.data_ptr(), dgu.data_ptr(), 0, M, I, K, K, I, 2 * I, 0, 0, 1, 0, 0, 0, 0, 1,
                             2, gu.data_ptr(), 2 * I, bn, split, _lib.stream_ptr()) == 0
    act_ref.backward(dy.float() @ wd.float())
    _check(dgu, guf.grad, K)

    shapes = [(72, 64), (264, 136), (128, 8)]
    A, X, C = [rnd(K, m) for m, _ in shapes], [rnd(K, n) for _, n in shapes], [rnd(m, n) for m, n in shapes]
    acc = [0, 1, 1]
    refs = [a.float().t() @ b.float() + (c.float() if f else 0) for a, b, c, f in zip(A, X, C, acc)]
    U, I3 = ctypes.c_ulonglong * 3, ctypes.c_int * 3
    assert lib.gfs_gemm_tile_wgrad_grouped(
        3, U(*[t.data_ptr() for t in A]), U(*[t.data_ptr() for t in X]), U(*[t.data_ptr() for t in C]),
        I3(*[m for m, _ in shapes]), I3(*[n for _, n in shapes]), I3(K, K, K), I3(*[m for m, _ in shapes]),
        I3(*[n for _, n in shapes]), I3(*[n for _, n in shapes]), I3(*acc), bn, split, _lib.stream_ptr()) == 0
    for c, r in zip(C, refs):
        _check(c, r, K)


@pytest.mark.parametrize("M,I,K", [(1, 8, 8), (33, 72, 64), (300, 200, 768), (1000, 1408, 1024), (777, 3080, 256),
                                   (520, 264, 1032), (20000, 136, 192)])
def test_swiglu_backward_on_pairs(cuda_device, M, I, K):
    """Rows and columns that end inside a warp's 32 x 64 box (the last gate columns lie next to the first up
    columns), more chunks than slots, and both sides of the line at K = 1024. Nothing outside the result is
    written. Tolerance: d_act is rounded to bf16 before the epilogue and the result after it."""
    from gpt_from_scratch_b200.ops import _lib
    g = torch.Generator(device="cuda").manual_seed(M + I + K)
    dy = torch.randn(M, K, device=cuda_device, generator=g).bfloat16()
    w = (torch.randn(K, I, device=cuda_device, generator=g) / K ** 0.5).bfloat16()
    gu = torch.randn(M, 2 * I + 16, device=cuda_device, generator=g).bfloat16()
    out = torch.full((M + 1, 2 * I + 8), 7.0, device=cuda_device, dtype=torch.bfloat16)
    rc = _lib.lib().gfs_gemm2_bf16_swiglu(2, dy.data_ptr(), w.data_ptr(), out.data_ptr(), gu.data_ptr(), M, I, K, K, I,
                                          out.stride(0), gu.stride(0), _lib.stream_ptr())
    assert rc == 0
    torch.cuda.synchronize()
    _lib.raise_on_status()
    gate, up = gu[:, :I].double(), gu[:, I:2 * I].double()
    d = (dy.double() @ w.double()).bfloat16().double()
    s = torch.sigmoid(gate)
    ref = torch.cat([d * up * s * (1 + gate * (1 - s)), d * gate * s], dim=1)
    assert (out[M] == 7.0).all() and (out[:, 2 * I:] == 7.0).all()
    rel = (out[:M, :2 * I].double() - ref).norm() / ref.norm()
    assert rel < 5e-3, rel


@pytest.mark.parametrize("N", [8, 120, 128, 136])
@pytest.mark.parametrize("M,K", [(40, 72), (2010, 104), (304, 768), (304, 776), (304, 2200), (19200, 72)])
def test_gemm_few_columns(cuda_device, M, N, K):
    """Around the 128 columns up to which a plain product may stay on the persistent kernel's narrow tiles: one tile, a
    wave with a ragged end, a long K loop, more tiles than SMs; with and without the addend that rules it out."""
    from gpt_from_scratch_b200.ops.gemm import gemm_bf16
    g = torch.Generator(device="cuda").manual_seed(M + N)
    for a_mn, b_mn in ((False, False), (False, True), (True, True)):
        a = torch.randn((K, M) if a_mn else (M, K), device=cuda_device, generator=g).bfloat16()
        if a_mn and M % 8:
            a = torch.nn.functional.pad(a, (0, 8 - M % 8))[:, :M]     # the pitch stays a multiple of 8 elements
        b = torch.randn((K, N) if b_mn else (N, K), device=cuda_device, generator=g).bfloat16()
        c = torch.randn(M, N, device=cuda_device, generator=g).bfloat16()
        _check(gemm_bf16(a, b, a_mn_major=a_mn, b_mn_major=b_mn), _ref(a, b, a_mn, b_mn, None), K)
        _check(gemm_bf16(a, b, a_mn_major=a_mn, b_mn_major=b_mn, addend=c), _ref(a, b, a_mn, b_mn, c), K)


@pytest.mark.parametrize("M,N,K", [(4393, 760, 2544), (623, 2208, 984), (1400, 768, 256), (768, 1288, 4104)])
def test_gemm_below_the_pair_threshold(cuda_device, M, N, K):
    """20 to 59 tiles of 256 x 256: a plain product may go to the persistent pairs, one with an addend may not."""
    from gpt_from_scratch_b200.ops.gemm import gemm_bf16
    g = torch.Generator(device="cuda").manual_seed(M + N)
    for a_mn, b_mn in ((False, False), (False, True), (True, True)):
        if a_mn and M % 8:
            continue
        a = torch.randn((K, M) if a_mn else (M, K), device=cuda_device, generator=g).bfloat16()
        b = torch.randn((K, N) if b_mn else (N, K), device=cuda_device, generator=g).bfloat16()
        c = torch.randn(M, N, device=cuda_device, generator=g).bfloat16()
        _check(gemm_bf16(a, b, a_mn_major=a_mn, b_mn_major=b_mn), _ref(a, b, a_mn, b_mn, None), K)
        _check(gemm_bf16(a, b, a_mn_major=a_mn, b_mn_major=b_mn, addend=c), _ref(a, b, a_mn, b_mn, c), K)


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (33, 72, 64), (95, 264, 392), (700, 1096, 72), (5000, 2056, 256)])
def test_pair_kernel_epilogues_at_edges(cuda_device, M, N, K):
    """Rows, columns and K that end inside a warp's 32 x 64 box of the pair kernel, from one tile to several per CTA: plain,
    with an addend (aliasing the output too), rotary, SwiGLU forward and the row statistics of the LM head. Nothing outside
    the results is written. Tolerance as in _check."""
    from gpt_from_scratch_b200.ops import _lib
    from gpt_from_scratch_b200.ops.rope import rope_reference
    lib, st = _lib.lib(), _lib.stream_ptr()
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rnd = lambda *s: torch.randn(*s, device=cuda_device, generator=g).bfloat16()  # noqa: E731

    def guarded(n):
        return torch.full((M + 1, n + 8), 7.0, device=cuda_device, dtype=torch.bfloat16)

    def outside_untouched(t, n):
        assert (t[M] == 7.0).all() and (t[:, n:] == 7.0).all()

    x, w, r = rnd(M, K), rnd(N, K), rnd(M, N)
    ref = x.float() @ w.float().t()
    for addend in (None, r):
        out = guarded(N)
        assert lib.gfs_gemm2_bf16(x.data_ptr(), w.data_ptr(), out.data_ptr(), _lib.ptr(addend), M, N, K, K, K, out.stride(0),
                                  N if addend is not None else 0, 0, 0, 0, 0, 0, 0, 1, st) == 0
        _check(out[:M, :N], ref if addend is None else ref + addend.float(), K)
        outside_untouched(out, N)
    acc = r.clone()
    assert lib.gfs_gemm2_bf16(x.data_ptr(), w.data_ptr(), acc.data_ptr(), acc.data_ptr(), M, N, K, K, K, N, N, 0, 0, 0, 0, 0,
                              0, 1, st) == 0
    _check(acc, ref + r.float(), K)

    # rotary: heads of 8 columns, the first half of them turned (the line lies inside a box); with an addend too
    B, D = (3, 8) if M % 3 == 0 else (1, 8)
    S, turned = M // B, N // 16 * 8
    ang = torch.rand(S, D // 2, device=cuda_device, generator=g) * 6.28
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    rr = ref.view(S, B, N // 8, 8).clone()
    rr[:, :, :turned // 8] = rope_reference(rr[:, :, :turned // 8], cos, sin)
    for addend in (None, r):
        out = guarded(N)
        assert lib.gfs_gemm2_bf16(x.data_ptr(), w.data_ptr(), out.data_ptr(), _lib.ptr(addend), M, N, K, K, K, out.stride(0),
                                  N if addend is not None else 0, 0, 0, cos.data_ptr(), sin.data_ptr(), turned, D, B,
                                  st) == 0
        _check(out[:M, :N], rr.view(M, N) if addend is None else rr.view(M, N) + addend.float(), K)
        outside_untouched(out, N)

    # SwiGLU forward with I = N
    wg = rnd(2 * N, K) * 0.3
    gu, act = guarded(2 * N), guarded(N)
    assert lib.gfs_gemm2_bf16_swiglu(1, x.data_ptr(), wg.data_ptr(), gu.data_ptr(), act.data_ptr(), M, N, K, K, K,
                                     gu.stride(0), act.stride(0), st) == 0
    _check(gu[:M, :2 * N], x.float() @ wg.float().t(), K)
    gate, up = gu[:M, :N].float(), gu[:M, N:2 * N].float()
    _check(act[:M, :N], torch.nn.functional.silu(gate) * up, K)
    outside_untouched(gu, 2 * N)
    outside_untouched(act, N)

    # row statistics of 128-column slices of the rounded logits (K >= 256 by contract)
    if K >= 256:
        logits = guarded(N)
        parts = torch.full((lib.gfs_gemm2_ce_parts(N), M, 2), 7.0, device=cuda_device)
        assert lib.gfs_gemm2_bf16_ce(x.data_ptr(), w.data_ptr(), logits.data_ptr(), parts.data_ptr(), M, N, K, K, K,
                                     logits.stride(0), st) == 0
        outside_untouched(logits, N)
        m = parts[..., 0].max(dim=0).values
        s = (parts[..., 1] * torch.exp(parts[..., 0] - m)).sum(dim=0)     # empty slices: (-inf, 0)
        assert torch.equal(m, logits[:M, :N].float().max(dim=1).values)
        lse = torch.logsumexp(logits[:M, :N].double(), dim=1)
        # fp32 sums of exponentials of 2^-22 relative error: a few 1e-6 of an lse of the order of its maximum
        assert ((m.double() + s.double().log()) - lse).abs().max() < 1e-5 * lse.abs().max().clamp(min=1)
    torch.cuda.synchronize()
    _lib.raise_on_status()


@pytest.mark.parametrize("M,N,K", [(1, 8, 1032), (95, 264, 1096), (5000, 2056, 1032)])
def test_pair_kernel_epilogues_long_k(cuda_device, M, N, K):
    """The same epilogues behind K loops that keep eight epilogue warps: one tile with rows, columns and K ending inside it, and
    several tiles per CTA."""
    test_pair_kernel_epilogues_at_edges(cuda_device, M, N, K)


@pytest.mark.parametrize("M,N,K", [(2100, 27656, 776), (4200, 17480, 1208)])
def test_pair_kernel_panels(cuda_device, M, N, K):
    """B of more than 40 MB is walked in panels of eight tile rows: a last panel of one row that is cut off, behind one and
    behind two whole panels, with sixteen and with eight epilogue warps."""
    assert 2 * N * K >= 40 << 20
    test_pair_kernel_epilogues_at_edges(cuda_device, M, N, K)


@pytest.mark.parametrize("bn,split", [(64, 1), (128, 2), (256, 1)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
def test_rope_with_addend_and_other_layouts(cuda_device, bn, split, a_mn, b_mn):
    """The rotary epilogue for every operand layout, with and without an addend: tile kernels, the pair kernel and the rule
    that chooses. Against fp32, tolerance as in _check."""
    from gpt_from_scratch_b200.ops import _lib
    from gpt_from_scratch_b200.ops.gemm import gemm_bf16
    from gpt_from_scratch_b200.ops.rope import rope_reference
    S, B, nh, D, K = 46, 4, 3, 64, 328
    M, N = S * B, 3 * nh * D
    g = torch.Generator(device="cuda").manual_seed(bn)
    rnd = lambda *s: torch.randn(*s, device=cuda_device, generator=g).bfloat16()  # noqa: E731
    a, b, r = rnd(K, M) if a_mn else rnd(M, K), rnd(K, N) if b_mn else rnd(N, K), rnd(M, N)
    ang = torch.rand(S, D // 2, device=cuda_device, generator=g) * 6.28
    cos, sin = ang.cos().contiguous(), ang.sin().contiguous()
    ref = _ref(a, b, a_mn, b_mn, None).view(S, B, 3 * nh, D)
    ref = torch.cat((rope_reference(ref[:, :, :2 * nh], cos, sin), ref[:, :, 2 * nh:]), dim=2).view(M, N)
    for addend in (None, r):
        want = ref if addend is None else ref + addend.float()
        out = torch.empty(M, N, device=cuda_device, dtype=torch.bfloat16)
        assert _lib.lib().gfs_gemm_tile(a.data_ptr(), b.data_ptr(), out.data_ptr(), _lib.ptr(addend), M, N, K, a.stride(0),
                                        b.stride(0), N, N if addend is not None else 0, int(a_mn), int(b_mn), cos.data_ptr(),
                                        sin.data_ptr(), 2 * nh * D, D, B, 0, 0, 0, bn, split, _lib.stream_ptr()) == 0
        _check(out, want, K)
        for pair in (None, True):
            _check(gemm_bf16(a, b, a_mn_major=a_mn, b_mn_major=b_mn, addend=addend, rope=(cos, sin, 2 * nh * D, D, B),
                             pair=pair), want, K)


@pytest.mark.parametrize("K", [512, 1032])
def test_pair_kernel_addend_of_one_row(cuda_device, K):
    """An addend whose rows are the same memory (a bias as an expanded view), on both sides of the line in K."""
    from gpt_from_scratch_b200.ops.gemm import gemm_bf16
    g = torch.Generator(device="cuda").manual_seed(K)
    M, N = 600, 520
    a, b, bias = (torch.randn(*s, device=cuda_device, generator=g).bfloat16() for s in ((M, K), (N, K), (N,)))
    _check(gemm_bf16(a, b, addend=bias.expand(M, N), pair=True), _ref(a, b, False, False, bias.expand(M, N)), K)


@pytest.mark.parametrize("K", [640, 648])
@pytest.mark.parametrize("M,N", [(512, 9472), (500, 9480)])
def test_pair_kernel_plain_at_the_lines(cuda_device, M, N, K):
    """Plain products on both sides of the lines between sixteen and eight epilogue warps: K, and a tile per CTA pair (74 on 148
    SMs) or one column of tiles more."""
    from gpt_from_scratch_b200.ops.gemm import gemm_bf16
    g = torch.Generator(device="cuda").manual_seed(K + N)
    for a_mn, b_mn in ((False, False), (False, True), (True, True)):
        m = M - M % 8 if a_mn else M       # the pitch is a multiple of 8 elements
        a = torch.randn((K, m) if a_mn else (m, K), device=cuda_device, generator=g).bfloat16()
        b = torch.randn((K, N) if b_mn else (N, K), device=cuda_device, generator=g).bfloat16()
        _check(gemm_bf16(a, b, a_mn_major=a_mn, b_mn_major=b_mn, pair=True), _ref(a, b, a_mn, b_mn, None), K)


@pytest.mark.parametrize("M,N,K", [(854, 1400, 3032), (1988, 896, 2808), (494, 1536, 2056)])
def test_gemm_long_k_with_odd_pitches(cuda_device, M, N, K):
    """Operands whose rows begin within a 32-byte sector, behind 32 K blocks and more, in every layout."""
    from gpt_from_scratch_b200.ops.gemm import gemm_bf16
    g = torch.Generator(device="cuda").manual_seed(M)
    for a_mn, b_mn in ((False, False), (False, True), (True, True), (True, False)):
        m = M - M % 8 if a_mn else M
        a = torch.randn((K, m) if a_mn else (m, K), device=cuda_device, generator=g).bfloat16()
        b = torch.randn((K, N) if b_mn else (N, K), device=cuda_device, generator=g).bfloat16()
        c = torch.randn(m, N, device=cuda_device, generator=g).bfloat16()
        _check(gemm_bf16(a, b, a_mn_major=a_mn, b_mn_major=b_mn), _ref(a, b, a_mn, b_mn, None), K)
        _check(gemm_bf16(a, b, a_mn_major=a_mn, b_mn_major=b_mn, addend=c), _ref(a, b, a_mn, b_mn, c), K)
