// Which GEMM kernel serves a product, for every caller (ops/gemm.py, ops/mlp_fused.py, model.cu).
//
//   persistent pairs   gemm2.cu   256 x 256 per CTA pair, epilogue of one tile behind the next tile's K loop
//   persistent CTAs    gemm.cu    128 x 256 per CTA
//   one tile per CTA   gemm3.cu   128 x 64, 128 x 128 or 256 x 256 (pair), K split over a cluster
//
// From `pair_min_tiles` (60) tiles of 256 x 256 on, the persistent pairs always win. Below, a product is mostly one
// wave of whatever kernel runs it, and its time is a constant (launch, first TMA, epilogue) plus the K blocks
// one CTA works through. The constants of the persistent kernels were fitted to 110 measured (shape, kernel) pairs on
// B200: M 103 to 4096, N 256 to 50304, K 103 to 50304, every layout, back to back in a CUDA graph; the fits are within 15 %.
// Those of the tiles were fitted again when their epilogues had become shorter: M 64 to 2331, N 128 to 3072, K 256 to 4096,
// every epilogue, and weight gradients over 130 to 8192 rows, each with every tile and split that fits one wave. Of 188
// choices four are more than 4.5 % slower than the best tile, none of those by more than 1.1 us; with the constants before, unsplit 128 x 128 tiles
// lost to the persistent kernel (512 x 3072 x 768 8.7 us there, 7.0 as tiles; 2331 x 768 x 3072 18.5 and 15.1) and small
// K was split (512 x 1024 x 256 4.3 us split in two, 3.9 whole). A step of two blocks of hidden 256 as a graph: 210 -> 201 us.
// us per launch, before (persistent kernels, K split through a workspace and a second launch) -> with this rule:
// 512 x 768 x 256 with rotary epilogue 16.5 -> 5.5, 130 x 768 x 3072 with addend 18.6 -> 7.7,
// 2048 x 768 x 2304 21.4 -> 16.3, weight gradient 768 x 768 x 2331 20.8 -> 9.8.
#include <algorithm>

#include "api.h"
#include "common.cuh"

namespace {

struct Choice {
  enum Kernel { PERSISTENT_CTA, PERSISTENT_PAIR, TILE } kernel;
  int bn, split;
};

// Most CTAs that are resident together when they come in clusters of `c` (148 SMs in GPCs of unequal
// size; counted by where a second wave shows in the measured times).
int wave_of_clusters(int c) {
  switch (c) {
    case 1: return 148;
    case 2: return 148;
    case 3: return 135;
    case 4: return 132;
    case 6: return 108;
    default: return 96;
  }
}

// What a tile's epilogue does beside storing the sums (gemm3.cu)
enum Extra { NONE = 0, ADDEND = 1, ROTATION = 2, SWIGLU = 3, SWIGLU_GRAD = 4 };

struct TileShape {
  int bn;               // columns of the tile
  int cluster;          // CTAs per tile without a split
  float base, per_kblock, split_base, split_cost;   // a split over s CTAs costs split_base + s * split_cost
  float extra[5];       // by Extra, for a whole tile; a CTA of a split tile does its share of the rows
};
// (Operands whose rows begin within a 32-byte sector, pitches of 8 mod 16, are not priced: a K block of a 128 x 128 tile takes
// up to 0.4 us for them. 854 x 1400 x 3032 with addend takes 25 to 27 us there and would take 20 to 21 on 256 x 256 tiles split in two,
// 1988 x 896 x 2808 22.5 and 20; another split sums in another order, so models of such widths would train to other bits.)
constexpr TileShape kShapes[3] = {
    {64, 1, 3.0f, 0.21f, 0.0f, 0.25f, {0.f, 0.2f, 1.3f, 0.6f, 1.2f}},   // 96 cycles per MMA (A and B read for 64 columns)
    {128, 1, 4.0f, 0.225f, 0.5f, 0.3f, {0.f, 0.55f, 3.2f, 1.1f, 2.45f}},   // 128 cycles per MMA: shared-memory reads
    {256, 2, 5.5f, 0.28f, 1.0f, 0.8f, {0.f, 0.85f, 4.4f, 1.2f, 3.5f}},     // tensor-bound, 256 columns per row to store
};

// Best one-wave tile for `tiles(bn)` tiles of 128 (bn = 256: 256) rows. us, or a huge number if none fits.
template <typename Tiles>
float best_tile(Tiles tiles, int kblocks, bool pairs, Extra extra, Choice* c) {
  float best = 1e30f;
  for (const TileShape& s : kShapes) {
    if (s.bn == 256 && !pairs) continue;
    const int n = tiles(s.bn);
    for (int split : {1, 2, 3, 4, 8}) {
      if (split > (s.bn == 256 ? 4 : 8)) break;
      const int per = (kblocks + split - 1) / split;
      if (per * (split - 1) >= kblocks) break;              // a CTA without K blocks
      const int cluster = s.cluster * split;
      if (n * cluster > wave_of_clusters(cluster)) break;
      float t = s.base + s.per_kblock * per + s.extra[extra] / split;
      if (split > 1) t += s.split_base + s.split_cost * split + (extra != NONE ? 0.3f : 0.f);
      if (t < best) {
        best = t;
        *c = Choice{Choice::TILE, s.bn, split};
      }
    }
  }
  return best;
}

int ceil_div(int a, int b) { return (a + b - 1) / b; }

// cols(bn): output columns covered by a tile of bn accumulator columns.
Choice choose(int M, int N, int K, int swi_mode, bool add, bool rope, int pair_min_tiles) {
  auto tiles = [&](int bn) {
    const int cols = swi_mode == 1 ? bn / 2 : bn;
    return ceil_div(M, bn == 256 ? 256 : 128) * ceil_div(N, cols);
  };
  const int kb = ceil_div(K, 64);
  const bool pairs = pair_min_tiles >= 0, plain = swi_mode == 0 && !add && !rope;
  if (pairs && (K >= 256 || swi_mode != 0) && tiles(256) >= pair_min_tiles) return Choice{Choice::PERSISTENT_PAIR, 256, 1};
  Choice c{Choice::PERSISTENT_CTA, 256, 1};
  const Extra extra = swi_mode == 1 ? SWIGLU : swi_mode == 2 ? SWIGLU_GRAD : rope ? ROTATION : add ? ADDEND : NONE;
  const float t_tile = best_tile(tiles, kb, pairs, extra, &c);
  // persistent CTAs: 128 x 256 tiles in waves; the addend, the rotation and the SwiGLU gradient are serial
  // loads in its epilogue. Plain products of up to 128 columns have 128-column tiles and half the epilogue there. Judged
  // by the same line, 27 of 129 measured ones went to kernels more than 5 % slower than the persistent one; with
  // one of their own up to 12 K blocks, one (us, one-tile kernel -> here: 2010 x 48 x 104 5.2 -> 4.0, 3568 x 32 x 104
  // 5.2 -> 4.0, 463 x 32 x 72 4.8 -> 3.7). With more K blocks the split over a cluster is the better one.
  const int waves = ceil_div(ceil_div(M, 128) * ceil_div(N, swi_mode == 1 ? 128 : 256), 148);
  float t_cta = 5.2f + 0.3f * kb * waves + 3.8f * (waves - 1) + (add ? 3.3f : 0.f) + (rope ? 9.5f : 0.f) +
                (swi_mode == 1 ? 2.0f : 0.f) + (swi_mode == 2 ? 6.0f : 0.f);
  if (N <= 128 && kb <= 12 && plain) t_cta = 4.0f + 0.18f * kb * waves + (waves - 1);
  if (t_cta < t_tile) c = Choice{Choice::PERSISTENT_CTA, 256, 1};
  // Persistent pairs from a third of the threshold on, where the K loop is long enough for their rate: 256 x 256 tiles
  // ask least of shared memory and L2 (128 x 128 tiles on all SMs take 0.4 us per K block, not 0.27). Of 439 measured
  // plain products 17 go there, none slower, up to 27 % faster: us, one-tile kernel or persistent CTAs -> here,
  // 4576 x 656 x 8184 53 -> 45, 4393 x 760 x 2544 27 -> 20. (A lone weight gradient of 768 x 3072 x 16384 takes 77 us here and
  // 69 with K split through a workspace, which callers on several streams would share; in a step it is part of a group.)
  if (pairs && plain && K >= 256 && N > 128 && tiles(256) >= pair_min_tiles / 3 && 6.0f + 0.22f * kb < std::min(t_cta, t_tile))
    c = Choice{Choice::PERSISTENT_PAIR, 256, 1};
  return c;
}

}  // namespace

extern "C" {

// C[M,N] = op(A) op(B) (+ R); arguments as gfs_gemm_bf16_rope (R null: no addend). pair_min_tiles: number of
// 256 x 256 tiles from which the persistent pair kernel is always used; < 0: no kernel on CTA pairs.
int gfs_linear(const void* A, const void* B, void* C, const void* R, int M, int N, int K, int lda, int ldb, int ldc,
               int ldr, int a_mn_major, int b_mn_major, const void* rope_cos, const void* rope_sin, int rope_cols,
               int rope_d, int rope_b, int pair_min_tiles, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const Choice c = choose(M, N, K, 0, R != nullptr, rope_cos != nullptr, pair_min_tiles);
  switch (c.kernel) {
    case Choice::PERSISTENT_PAIR:
      return gfs_gemm2_bf16(A, B, C, R, M, N, K, lda, ldb, ldc, ldr, a_mn_major, b_mn_major, rope_cos, rope_sin,
                            rope_cols, rope_d, rope_b, stream);
    case Choice::TILE:
      return gfs_gemm_tile(A, B, C, R, M, N, K, lda, ldb, ldc, ldr, a_mn_major, b_mn_major, rope_cos, rope_sin,
                           rope_cols, rope_d, rope_b, 0, nullptr, 0, c.bn, c.split, stream);
    default:
      return gfs_gemm_bf16_rope(A, B, C, R, M, N, K, lda, ldb, ldc, ldr, a_mn_major, b_mn_major, R != nullptr, nullptr,
                                0, 1, rope_cos, rope_sin, rope_cols, rope_d, rope_b, stream);
  }
}

// The SwiGLU-fused products of the MLP; arguments as gfs_gemm_bf16_swiglu.
int gfs_linear_swiglu(int mode, const void* a, const void* b, void* c, void* extra, int M, int I, int K, int lda,
                      int ldb, int ldc, int ld_extra, int pair_min_tiles, void* stream) {
  if (mode != 1 && mode != 2) return -1;
  if (M <= 0 || I <= 0 || K <= 0) return 0;
  const Choice ch = choose(M, I, K, mode, false, false, pair_min_tiles);
  switch (ch.kernel) {
    case Choice::PERSISTENT_PAIR:
      return gfs_gemm2_bf16_swiglu(mode, a, b, c, extra, M, I, K, lda, ldb, ldc, ld_extra, stream);
    case Choice::TILE:
      return gfs_gemm_tile(a, b, c, nullptr, M, I, K, lda, ldb, ldc, 0, 0, mode == 2, nullptr, nullptr, 0, 0, 1, mode,
                           extra, ld_extra, ch.bn, ch.split, stream);
    default:
      return gfs_gemm_bf16_swiglu(mode, a, b, c, extra, M, I, K, lda, ldb, ldc, ld_extra, stream);
  }
}

// Grouped weight gradients; arguments as gfs_gemm2_wgrad_grouped.
int gfs_wgrad_grouped(int n, const unsigned long long* A, const unsigned long long* B, const unsigned long long* C,
                      const int* M, const int* N, const int* K, const int* lda, const int* ldb, const int* ldc,
                      const int* accumulate, void* stream) {
  if (n <= 0) return 0;
  int kb = 0, kb_min = 1 << 30;
  for (int i = 0; i < n; ++i) {
    kb = std::max(kb, ceil_div(K[i], 64));
    kb_min = std::min(kb_min, ceil_div(K[i], 64));
  }
  auto tiles = [&](int bn) {
    int t = 0;
    for (int i = 0; i < n; ++i) t += ceil_div(M[i], bn == 256 ? 256 : 128) * ceil_div(N[i], bn);
    return t;
  };
  Choice c{Choice::PERSISTENT_PAIR, 256, 1};
  const bool adds = std::any_of(accumulate, accumulate + n, [](int a) { return a != 0; });
  // the persistent grouped kernel: one wave of pairs, an epilogue of four warps, which reads what it adds to late. (Of 122 groups
  // that add to existing gradients, three go to other tiles for it, 4 to 10 % faster: three of hidden 128 and 192.)
  const float t_pair = 6.5f + 0.3f * kb * ceil_div(tiles(256), 74) + (adds ? 2.5f : 0.f);
  // Unsplit 256 x 256 tiles on pairs are that kernel's tiles without its persistence: 95 us instead of 86 for the
  // three small gradients of a block at 16384 tokens (hidden 768, FFN 3072).
  if (kb == kb_min && best_tile(tiles, kb, true, adds ? ADDEND : NONE, &c) < t_pair && c.kernel == Choice::TILE &&
      (c.bn != 256 || c.split > 1))
    return gfs_gemm_tile_wgrad_grouped(n, A, B, C, M, N, K, lda, ldb, ldc, accumulate, c.bn, c.split, stream);
  return gfs_gemm2_wgrad_grouped(n, A, B, C, M, N, K, lda, ldb, ldc, accumulate, stream);
}

}  // extern "C"
