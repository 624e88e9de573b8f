// Whole passes of the model as ONE host call each: the stack of transformer blocks forward and
// backward, and a training step's forward, loss and backward.
//
// A block is eight forward and about thirteen backward kernels of 2-300 us. Launched one by one from
// Python through autograd, a block costs the host about 0.3 ms forward and 0.5 ms backward, more
// than its kernels take at small and ordinary sizes (12 layers, hidden 768, batch 1 x 130 tokens: 4.0 ms
// of host work around 1.0 ms of kernels). Here the same sequence of launches is issued from C, about 2 us
// each, with every intermediate in a workspace whose layout this file defines: the caller allocates
// one buffer per block for what the backward reads (gfs_blocks_act_bytes) and one scratch for the
// backward itself (gfs_blocks_bwd_bytes).
//
// Nothing here computes: the kernels and their selection rules are those of the module-by-module path
// (models/transformer_layer.py). Forward results are its bits. Gradients differ from its by roundings: the weight
// gradients of a block form other groups, for which other tiles and K splits may be chosen (fp32 sums in another order),
// and with dropout the modules round the two gradients of a residual branch one by one.
// Single tensor-parallel rank only (no collectives).
#include <algorithm>
#include <cmath>
#include <memory>
#include <new>

#include "api.h"
#include "common.cuh"

namespace {

enum Weight : int { W_NORM1 = 0, W_QKV, W_OUT, W_NORM2, W_GATE_UP, W_DOWN, W_COUNT };

typedef unsigned long long u64;

}  // namespace

extern "C" {

// Mirrored by ctypes structures in models/native.py.
struct GfsBlockDims {
  int S, B, H, nh, D, I;
  int n_layers;
  int pair_min_tiles;      // 256 x 256 tiles from which a product runs on CTA pairs; < 0: never
  int grouped_wgrad;       // small weight gradients of a block share a launch
  float dropout_p;         // 0: residual adds run in the GEMM epilogues
  float eps_final;
};

struct GfsBlockParams {
  const void* w[W_COUNT];  // norm1, qkv, out, norm2, gate|up, down
  void* g[W_COUNT];        // their gradients (bf16)
  int accumulate[W_COUNT]; // add to the gradient instead of overwriting it
  float eps[2];            // norm1, norm2
  const void* cos_table;   // fp32 [>= S, D/2]
  const void* sin_table;
  u64 seed[2];             // dropout after the attention, after the MLP
};

}  // extern "C"

namespace {

size_t align256(size_t n) { return (n + 255) & ~static_cast<size_t>(255); }

// What the forward of one block leaves behind (byte offsets into the block's buffer).
struct ActLayout {
  size_t y1, rstd1, qkv, attn, lse, x1, y2, rstd2, gu, act, x2, total;
  explicit ActLayout(const GfsBlockDims& d) {
    const size_t T = static_cast<size_t>(d.S) * d.B, H = d.H, I = d.I;
    const size_t s_pad = (static_cast<size_t>(d.S) + 127) / 128 * 128;
    size_t o = 0;
    auto take = [&](size_t bytes) {
      const size_t at = o;
      o += align256(bytes);
      return at;
    };
    y1 = take(2 * T * H);
    rstd1 = take(4 * T);
    qkv = take(2 * T * 3 * H);
    attn = take(2 * T * H);
    lse = take(4 * d.B * d.nh * s_pad);
    x1 = take(2 * T * H);
    y2 = take(2 * T * H);
    rstd2 = take(4 * T);
    gu = take(2 * T * 2 * I);
    act = take(2 * T * I);
    x2 = take(2 * T * H);
    total = o;
  }
};

// Scratch of the backward pass. Reused by every block (stream order), except the column partials of
// the norm weight gradients, which wait for one reduction launch at the end.
struct BwdLayout {
  size_t dgu, dy, dx1, dattn, dqkv, dvec, dmask, dx[2], partial, partial_stride, total;
  explicit BwdLayout(const GfsBlockDims& d) {
    const size_t T = static_cast<size_t>(d.S) * d.B, H = d.H, I = d.I;
    const size_t s_pad = (static_cast<size_t>(d.S) + 127) / 128 * 128;
    size_t o = 0;
    auto take = [&](size_t bytes) {
      const size_t at = o;
      o += align256(bytes);
      return at;
    };
    dgu = take(2 * T * 2 * I);
    dy = take(2 * T * H);
    dx1 = take(2 * T * H);
    dattn = take(2 * T * H);
    dqkv = take(2 * T * 3 * H);
    dvec = take(4 * d.B * d.nh * s_pad);
    dmask = d.dropout_p > 0.f ? take(2 * 2 * T * H) : 0;
    dx[0] = take(2 * T * H);
    dx[1] = take(2 * T * H);
    partial_stride = align256(4 * static_cast<size_t>(gfs_rmsnorm_bwd_parts(static_cast<int>(T))) * H);
    partial = take(partial_stride * (2 * static_cast<size_t>(d.n_layers) + 1));
    total = o;
  }
};

int tiles256(int m, int n) { return ((m + 255) / 256) * ((n + 255) / 256); }

bool use_pair(const GfsBlockDims& d, int tiles) { return d.pair_min_tiles >= 0 && tiles >= d.pair_min_tiles; }

// C[M,N] = op(A) op(B) (+ R), R with the pitch of C. B is a weight, which no kernel of a pass writes.
int product(const GfsBlockDims& d, const void* A, const void* B, void* C, const void* R, int M, int N, int K, int lda,
            int ldb, int ldc, int a_mn, int b_mn, void* stream) {
  const gfs_host::WithHints hints(true, false);
  return gfs_linear(A, B, C, R, M, N, K, lda, ldb, ldc, R != nullptr ? ldc : 0, a_mn, b_mn, nullptr, nullptr, 0, d.D,
                    d.B, d.pair_min_tiles, stream);
}

// The weight gradients of one block that are too small to fill the chip alone share a launch.
struct WgradGroup {
  static constexpr int MAX = 4;
  u64 A[MAX], B[MAX], C[MAX];
  int M[MAX], N[MAX], K[MAX], lda[MAX], ldb[MAX], ldc[MAX], acc[MAX];
  int n = 0, tiles = 0;
  // late: the kernel launched last is a product that writes nothing these read (see launch_hints.h)
  int flush(int* launches, void* stream, bool late) {
    if (n == 0) return 0;
    const gfs_host::WithHints hints(false, late);
    const int rc = gfs_wgrad_grouped(n, A, B, C, M, N, K, lda, ldb, ldc, acc, stream);
    n = tiles = 0;
    ++*launches;
    return rc;
  }
};

// dW[N_out, N_in] (+)= dY[T, N_out]^T X[T, N_in]. Called right after a product of the gradient chain that also reads dY:
// nothing launched here depends on that product, and it may fill the SMs that its last wave leaves idle.
int weight_grad(const GfsBlockDims& d, WgradGroup& grp, const void* dY, const void* X, void* dW, int accumulate, int T,
                int n_out, int n_in, int* launches, void* stream) {
  const int tiles = tiles256(n_out, n_in);
  if (d.grouped_wgrad && d.pair_min_tiles >= 0 && tiles < d.pair_min_tiles) {
    const int i = grp.n++;
    grp.A[i] = reinterpret_cast<u64>(dY);
    grp.B[i] = reinterpret_cast<u64>(X);
    grp.C[i] = reinterpret_cast<u64>(dW);
    grp.M[i] = n_out; grp.N[i] = n_in; grp.K[i] = T;
    grp.lda[i] = n_out; grp.ldb[i] = n_in; grp.ldc[i] = n_in;
    grp.acc[i] = accumulate;
    grp.tiles += tiles;
    if (grp.n == WgradGroup::MAX || grp.tiles >= d.pair_min_tiles) return grp.flush(launches, stream, true);
    return 0;
  }
  ++*launches;
  const gfs_host::WithHints hints(false, true);
  return gfs_linear(dY, X, dW, accumulate ? dW : nullptr, n_out, n_in, T, n_out, n_in, n_in, accumulate ? n_in : 0, 1, 1,
                    nullptr, nullptr, 0, d.D, d.B, d.pair_min_tiles, stream);
}

bool dims_ok(const GfsBlockDims& d) {
  return d.S > 0 && d.B > 0 && d.n_layers >= 0 && (d.D == 64 || d.D == 128) && d.nh * d.D == d.H && d.I > 0 &&
         (d.I & 7) == 0 && d.dropout_p >= 0.f && d.dropout_p < 1.f;
}

}  // namespace

#define GFS_TRY(call)             \
  do {                            \
    const int rc_ = (call);       \
    ++*launches;                  \
    if (rc_ != 0) return rc_;     \
  } while (0)

extern "C" {

// Bytes of one block's saved activations.
size_t gfs_blocks_act_bytes(const GfsBlockDims* d) { return ActLayout(*d).total; }

size_t gfs_blocks_bwd_bytes(const GfsBlockDims* d) { return BwdLayout(*d).total; }

// Forward of all blocks and the final norm. x: [S*B, H] input; act[l]: buffer of block l (one and the
// same buffer for all of them when no backward follows); tmp: [S*B, H] (dropout only); y_final,
// rstd_final: the final norm's output. *launches is increased by the number of kernel launches.
int gfs_blocks_forward(const GfsBlockDims* dp, const GfsBlockParams* layers, const void* w_final, const void* x,
                       const u64* act, void* tmp, void* y_final, void* rstd_final, int* launches, void* stream) {
  const GfsBlockDims& d = *dp;
  if (!dims_ok(d)) return -1;
  const ActLayout a(d);
  const int T = d.S * d.B, H = d.H, I = d.I;
  const float scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(d.D)));
  const bool drop = d.dropout_p > 0.f;
  const long long tok = 3ll * H;   // a token of the packed [S, B, 3, nh, D] projection
  const long long st[12] = {d.B * tok, tok, d.D, d.B * tok, tok, d.D, d.B * tok, tok, d.D,
                            static_cast<long long>(d.B) * H, H, d.D};
  for (int l = 0; l < d.n_layers; ++l) {
    const GfsBlockParams& p = layers[l];
    char* base = reinterpret_cast<char*>(act[l]);
    void *y1 = base + a.y1, *rstd1 = base + a.rstd1, *attn = base + a.attn, *lse = base + a.lse, *x1 = base + a.x1,
         *y2 = base + a.y2, *rstd2 = base + a.rstd2, *gu = base + a.gu, *ac = base + a.act, *x2 = base + a.x2;
    char* qkv = base + a.qkv;
    if (!drop || l == 0) GFS_TRY(gfs_rmsnorm_fwd(x, p.w[W_NORM1], y1, rstd1, T, H, p.eps[0], stream));
    const gfs_host::WithHints hints(true, false);   // (of the products; B is a weight)
    GFS_TRY(gfs_linear(y1, p.w[W_QKV], qkv, nullptr, T, 3 * H, H, H, H, 3 * H, 0, 0, 0, p.cos_table, p.sin_table, 2 * H,
                       d.D, d.B, d.pair_min_tiles, stream));   // q and k leave rotated
    GFS_TRY(gfs_flash_fwd(qkv, qkv + 2 * static_cast<size_t>(H), qkv + 4 * static_cast<size_t>(H), attn, nullptr, lse,
                          d.S, d.B, d.nh, d.D, st, scale, 1, 0, stream));
    if (!drop) {
      GFS_TRY(product(d, attn, p.w[W_OUT], x1, x, T, H, H, H, H, H, 0, 0, stream));
    } else {
      GFS_TRY(product(d, attn, p.w[W_OUT], tmp, nullptr, T, H, H, H, H, H, 0, 0, stream));
      GFS_TRY(gfs_dropout_residual_norm(tmp, x, x1, p.w[W_NORM2], y2, rstd2, T, H, p.eps[1], d.dropout_p, p.seed[0],
                                        stream));
    }
    if (!drop) GFS_TRY(gfs_rmsnorm_fwd(x1, p.w[W_NORM2], y2, rstd2, T, H, p.eps[1], stream));
    GFS_TRY(gfs_linear_swiglu(1, y2, p.w[W_GATE_UP], gu, ac, T, I, H, H, H, 2 * I, I, d.pair_min_tiles, stream));
    if (!drop) {
      GFS_TRY(product(d, ac, p.w[W_DOWN], x2, x1, T, H, I, I, I, H, 0, 0, stream));
    } else {
      GFS_TRY(product(d, ac, p.w[W_DOWN], tmp, nullptr, T, H, I, I, I, H, 0, 0, stream));
      // with the next block's first norm, or the final one
      const bool last = l + 1 == d.n_layers;
      char* next = last ? nullptr : reinterpret_cast<char*>(act[l + 1]);
      GFS_TRY(gfs_dropout_residual_norm(tmp, x1, x2, last ? w_final : layers[l + 1].w[W_NORM1],
                                        last ? y_final : next + a.y1, last ? rstd_final : next + a.rstd1, T, H,
                                        last ? d.eps_final : layers[l + 1].eps[0], d.dropout_p, p.seed[1], stream));
    }
    x = x2;
  }
  if (!drop || d.n_layers == 0) GFS_TRY(gfs_rmsnorm_fwd(x, w_final, y_final, rstd_final, T, H, d.eps_final, stream));
  return 0;
}

// Backward of the final norm and all blocks. dy_final: gradient of the final norm's output; x, act:
// as given to the forward; scratch: gfs_blocks_bwd_bytes bytes; dx: gradient of x (may not alias
// scratch). Weight gradients go to (or are added to) layers[l].g and g_final.
int gfs_blocks_backward(const GfsBlockDims* dp, const GfsBlockParams* layers, const void* w_final, void* g_final,
                        int accumulate_final, const void* x, const u64* act, const void* rstd_final,
                        const void* dy_final, void* scratch, void* dx, int* launches, void* stream) {
  const GfsBlockDims& d = *dp;
  if (!dims_ok(d)) return -1;
  const ActLayout a(d);
  const BwdLayout b(d);
  const int T = d.S * d.B, H = d.H, I = d.I;
  const long long n_el = static_cast<long long>(T) * H;
  const float scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(d.D)));
  const bool drop = d.dropout_p > 0.f;
  const int parts = gfs_rmsnorm_bwd_parts(T);
  const long long tok = 3ll * H;
  const long long q3[3] = {d.B * tok, tok, d.D}, o3[3] = {static_cast<long long>(d.B) * H, H, d.D};
  long long st[24];
  for (int i = 0; i < 3; ++i) {
    st[i] = st[3 + i] = st[6 + i] = st[15 + i] = st[18 + i] = st[21 + i] = q3[i];
    st[9 + i] = st[12 + i] = o3[i];
  }
  char* s = static_cast<char*>(scratch);
  void *dgu = s + b.dgu, *dy = s + b.dy, *dx1 = s + b.dx1, *dattn = s + b.dattn, *dvec = s + b.dvec;
  char* dqkv = s + b.dqkv;

  // one batched reduction of the norm weight gradients at the end
  constexpr int RED = 32;
  u64 red_p[RED], red_g[RED];
  int red_parts[RED], red_acc[RED];
  int n_red = 0, n_partial = 0;
  auto flush_norms = [&]() -> int {
    if (n_red == 0) return 0;
    const int rc = gfs_rmsnorm_dw_reduce_multi(n_red, red_p, red_g, red_parts, red_acc, H, stream);
    n_red = 0;
    ++*launches;
    return rc;
  };
  auto norm_bwd = [&](const void* dyp, const void* xp, const void* w, const void* rstd, const void* dres, void* dxp,
                      void* g, int acc, void* masked, u64 seed) -> int {
    void* part = s + b.partial + b.partial_stride * n_partial++;
    int rc = masked != nullptr ? gfs_rmsnorm_bwd_dropout(dyp, xp, w, rstd, dres, dxp, masked, part, T, H, d.dropout_p,
                                                         seed, stream)
                               : gfs_rmsnorm_bwd(dyp, xp, w, rstd, dres, dxp, nullptr, part, T, H, 0, stream);
    if (rc == 1) {
      rc = gfs_rmsnorm_bwd(dyp, xp, w, rstd, dres, dxp, nullptr, part, T, H, 0, stream);
      if (rc == 0) rc = gfs_dropout_residual(dxp, nullptr, masked, n_el, d.dropout_p, seed, 1, stream);
      ++*launches;
    }
    if (rc != 0) return rc;
    red_p[n_red] = reinterpret_cast<u64>(part);
    red_g[n_red] = reinterpret_cast<u64>(g);
    red_parts[n_red] = parts;
    red_acc[n_red] = acc;
    return ++n_red == RED ? flush_norms() : 0;
  };

  auto input_of = [&](int l) -> const void* {
    return l == 0 ? x : static_cast<const void*>(reinterpret_cast<const char*>(act[l - 1]) + a.x2);
  };
  // gradient of the current block's output; the two buffers alternate
  void* dout = d.n_layers == 0 ? dx : s + b.dx[d.n_layers & 1];
  // with dropout: the gradients of the MLP's and of the attention's output, masked where dout and dx1 are written
  void* m_mlp = drop && d.n_layers > 0 ? s + b.dmask : nullptr;
  void* m_attn = drop ? s + b.dmask + align256(2 * static_cast<size_t>(n_el)) : nullptr;
  GFS_TRY(norm_bwd(dy_final, input_of(d.n_layers), w_final, rstd_final, nullptr, dout, g_final, accumulate_final, m_mlp,
                   m_mlp ? layers[d.n_layers - 1].seed[1] : 0));
  for (int l = d.n_layers - 1; l >= 0; --l) {
    const GfsBlockParams& p = layers[l];
    const char* base = reinterpret_cast<const char*>(act[l]);
    const void *y1 = base + a.y1, *rstd1 = base + a.rstd1, *attn = base + a.attn, *lse = base + a.lse,
               *x1 = base + a.x1, *y2 = base + a.y2, *rstd2 = base + a.rstd2, *gu = base + a.gu, *ac = base + a.act;
    const char* qkv = base + a.qkv;
    WgradGroup grp;
    // gradient of the MLP's output
    const void* dm = drop ? m_mlp : dout;
    {
      const gfs_host::WithHints hints(true, false);
      GFS_TRY(gfs_linear_swiglu(2, dm, p.w[W_DOWN], dgu, const_cast<void*>(gu), T, I, H, H, I, 2 * I, 2 * I,
                                d.pair_min_tiles, stream));
    }
    int rc = weight_grad(d, grp, dm, ac, p.g[W_DOWN], p.accumulate[W_DOWN], T, H, I, launches, stream);
    if (rc != 0) return rc;
    GFS_TRY(product(d, dgu, p.w[W_GATE_UP], dy, nullptr, T, H, 2 * I, 2 * I, H, H, 0, 1, stream));
    rc = weight_grad(d, grp, dgu, y2, p.g[W_GATE_UP], p.accumulate[W_GATE_UP], T, 2 * I, H, launches, stream);
    if (rc != 0) return rc;
    GFS_TRY(norm_bwd(dy, x1, p.w[W_NORM2], rstd2, dout, dx1, p.g[W_NORM2], p.accumulate[W_NORM2], m_attn,
                     p.seed[0]));
    // attention
    const void* da = drop ? m_attn : dx1;
    GFS_TRY(product(d, da, p.w[W_OUT], dattn, nullptr, T, H, H, H, H, H, 0, 1, stream));
    rc = weight_grad(d, grp, da, attn, p.g[W_OUT], p.accumulate[W_OUT], T, H, H, launches, stream);
    if (rc != 0) return rc;
    const size_t h2 = 2 * static_cast<size_t>(H);
    GFS_TRY(gfs_flash_bwd(qkv, qkv + h2, qkv + 2 * h2, attn, dattn, lse, dvec, dqkv, dqkv + h2, dqkv + 2 * h2, d.S, d.B,
                          d.nh, d.D, st, scale, 1, p.cos_table, p.sin_table, nullptr, stream));
    *launches += 2;   // a pre-pass and two main kernels
    GFS_TRY(product(d, dqkv, p.w[W_QKV], dy, nullptr, T, H, 3 * H, 3 * H, H, H, 0, 1, stream));
    const int launched = *launches;
    rc = weight_grad(d, grp, dqkv, y1, p.g[W_QKV], p.accumulate[W_QKV], T, 3 * H, H, launches, stream);
    if (rc != 0) return rc;
    rc = grp.flush(launches, stream, *launches == launched);   // its operands are overwritten by the next block
    if (rc != 0) return rc;
    void* dnext = l == 0 ? dx : s + b.dx[l & 1];
    GFS_TRY(norm_bwd(dy, input_of(l), p.w[W_NORM1], rstd1, dx1, dnext, p.g[W_NORM1], p.accumulate[W_NORM1],
                     l > 0 ? m_mlp : nullptr, l > 0 ? layers[l - 1].seed[1] : 0));
    dout = dnext;
  }
  return flush_norms();
}

// ---------------------------------------------------------------------------
// Forward, mean loss and backward of one micro-batch.
// ---------------------------------------------------------------------------
struct GfsModelTop {
  const void *w_emb, *w_final, *w_out;   // [V, H], [H], [V, H]
  void *g_emb, *g_final, *g_out;
  int acc_emb, acc_final, acc_out;       // add to the gradient instead of overwriting it
  int V;
};

}  // extern "C"

namespace {

// Buffers of a step besides the blocks' activations. The logits are dead when the blocks' backward
// begins, so its scratch lies in the same place.
struct StepLayout {
  size_t acts, x0, y_final, rstd_final, keys, targets, loss_rows, stats, lse, dy, dx0, logits, partials, scratch, total;
  StepLayout(const GfsBlockDims& d, const GfsModelTop& t, const ActLayout& a) {
    const size_t T = static_cast<size_t>(d.S) * d.B, H = d.H, V = t.V;
    size_t o = 0;
    auto take = [&](size_t bytes) {
      const size_t at = o;
      o += align256(bytes);
      return at;
    };
    acts = take(a.total * d.n_layers);
    x0 = take(2 * T * H);
    y_final = take(2 * T * H);
    rstd_final = take(4 * T);
    keys = take(4 * T);
    targets = take(8 * T);
    loss_rows = take(4 * T);
    stats = take(12 * T);
    lse = take(4 * T);
    dy = take(2 * T * H);
    dx0 = take(2 * T * H);
    scratch = o;   // also the dropout's temporary in the forward
    logits = take(2 * T * V);
    partials = take(8 * T * static_cast<size_t>(gfs_gemm2_ce_parts(t.V)));
    total = std::max(o, scratch + std::max(BwdLayout(d).total, align256(2 * T * H)));
  }
};

// The id sort of the embedding backward needs only the ids, the clearing of its gradient nothing: they run beside the
// forward on a stream of their own (one per thread and device, so that neither threads nor captures meet in its events; given back when
// the thread ends).
struct SideStream {
  cudaStream_t stream = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  ~SideStream() {
    if (join != nullptr) cudaEventDestroy(join);
    if (fork != nullptr) cudaEventDestroy(fork);
    if (stream != nullptr) cudaStreamDestroy(stream);
  }
};
SideStream* side_stream() {
  static thread_local SideStream per_dev[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  SideStream& s = per_dev[dev];
  if (s.join == nullptr) {
    if (cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreateWithFlags(&s.fork, cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&s.join, cudaEventDisableTiming) != cudaSuccess)
      return nullptr;
  }
  return &s;
}

// The step without the embedding's backward: logits, loss, and back.
int step_until_embedding(const GfsBlockDims& d, const GfsBlockParams* layers, const GfsModelTop& t, const void* ids,
                         const void* labels, char* m, const StepLayout& lay, const u64* act, void* loss, int* launches,
                         cudaStream_t stream) {
  const int T = d.S * d.B, H = d.H, V = t.V;
  void *x0 = m + lay.x0, *y = m + lay.y_final, *rstd = m + lay.rstd_final, *targets = m + lay.targets,
       *rows = m + lay.loss_rows, *stats = m + lay.stats, *lse = m + lay.lse, *dy = m + lay.dy, *dx0 = m + lay.dx0,
       *logits = m + lay.logits, *partials = m + lay.partials, *scratch = m + lay.scratch;
  GFS_TRY(gfs_embedding_fwd(ids, t.w_emb, x0, d.B, d.S, H, 0, V, 0, d.S, stream));
  int rc = gfs_blocks_forward(&d, layers, t.w_final, x0, act, scratch, y, rstd, launches, stream);
  if (rc != 0) return rc;

  // LM head and loss
  const float g_row = 1.0f / static_cast<float>(T);
  rc = -20;
  if (H >= 256 && use_pair(d, tiles256(T, V))) {
    rc = gfs_gemm2_bf16_ce(y, t.w_out, logits, partials, T, V, H, H, H, V, stream);
    if (rc == 0) {
      *launches += 2;
      rc = gfs_ce_from_partials(partials, logits, labels, stats, lse, rows, gfs_gemm2_ce_parts(V), T, V, V, 0, 1, d.B,
                                targets, stream);
    }
  }
  if (rc == -20) {
    GFS_TRY(product(d, y, t.w_out, logits, nullptr, T, V, H, H, H, V, 0, 0, stream));
    GFS_TRY(gfs_ce_fwd(logits, labels, stats, lse, rows, T, V, V, 0, 1, d.B, targets, stream));
  } else if (rc != 0) {
    return rc;
  }
  GFS_TRY(gfs_mean_f32(rows, loss, T, stream));

  // backward: the logits become their gradient in place
  GFS_TRY(gfs_ce_bwd(logits, lse, targets, nullptr, g_row, T, V, V, 0, stream));
  GFS_TRY(product(d, logits, t.w_out, dy, nullptr, T, H, V, V, H, H, 0, 1, stream));
  WgradGroup grp;
  const int launched = *launches;
  rc = weight_grad(d, grp, logits, y, t.g_out, t.acc_out, T, V, H, launches, stream);
  if (rc == 0) rc = grp.flush(launches, stream, *launches == launched);
  if (rc != 0) return rc;
  return gfs_blocks_backward(&d, layers, t.w_final, t.g_final, t.acc_final, x0, act, rstd, dy, scratch, dx0, launches,
                             stream);
}

}  // namespace

extern "C" {

// 0: the batch does not fit the single-CTA id sort of the embedding backward.
size_t gfs_model_step_bytes(const GfsBlockDims* d, const GfsModelTop* t) {
  if (gfs_embedding_sort_shift(static_cast<long long>(d->B) * d->S, t->V) <= 0) return 0;
  return StepLayout(*d, *t, ActLayout(*d)).total;
}

// One micro-batch: ids, labels int64 [B, S] -> *loss (fp32, mean over all tokens) and all weight
// gradients. arena: gfs_model_step_bytes bytes. Arguments that cannot be served are refused before anything is
// launched; after an error of a launch the caller's stream still waits for the sort, which writes to the arena.
int gfs_model_step(const GfsBlockDims* dp, const GfsBlockParams* layers, const GfsModelTop* tp, const void* ids,
                   const void* labels, void* arena, void* loss, int* launches, void* stream) {
  const GfsBlockDims& d = *dp;
  const GfsModelTop& t = *tp;
  if (!dims_ok(d) || (t.V & 7) || gfs_embedding_sort_shift(static_cast<long long>(d.B) * d.S, t.V) <= 0) return -1;
  const ActLayout a(d);
  const StepLayout lay(d, t, a);
  char* m = static_cast<char*>(arena);
  const std::unique_ptr<u64[]> act(new (std::nothrow) u64[d.n_layers + 1]);
  if (act == nullptr) return -12;
  for (int l = 0; l < d.n_layers; ++l) act[l] = reinterpret_cast<u64>(m + lay.acts + a.total * l);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SideStream* side = side_stream();
  if (side == nullptr) return -10;
  if (cudaEventRecord(side->fork, st) != cudaSuccess || cudaStreamWaitEvent(side->stream, side->fork, 0) != cudaSuccess)
    return -11;
  int shift = gfs_embedding_sort_keys(ids, m + lay.keys, d.B, d.S, 0, t.V, side->stream);
  if (shift >= 0 && !t.acc_emb &&
      cudaMemsetAsync(t.g_emb, 0, 2 * static_cast<size_t>(t.V) * d.H, side->stream) != cudaSuccess)
    shift = -11;
  if (cudaEventRecord(side->join, side->stream) != cudaSuccess) {
    cudaStreamSynchronize(side->stream);
    return -11;
  }
  ++*launches;
  int rc = shift < 0 ? shift : step_until_embedding(d, layers, t, ids, labels, m, lay, act.get(), loss, launches, st);
  if (cudaStreamWaitEvent(st, side->join, 0) != cudaSuccess && rc == 0) rc = -11;
  if (rc != 0) return rc;
  GFS_TRY(gfs_embedding_bwd_keys(m + lay.keys, m + lay.dx0, t.g_emb, d.S * d.B, d.H, shift, stream));
  return 0;
}

}  // extern "C"
