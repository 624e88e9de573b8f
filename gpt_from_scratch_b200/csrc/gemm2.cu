// bf16 GEMM on CTA pairs: tcgen05.mma.cta_group::2 computes one 256 x 256 output tile per
// cluster of two CTAs (each CTA owns 128 rows of A, 128 of the 256 B rows, and the 128 x 256
// half of the accumulator that lands in its own TMEM). Sharing B across the pair halves the
// shared-memory traffic per FLOP, which is what bounds the single-CTA kernel in gemm.cu
// (operand reads plus TMA writes exceed 128 B/clk/SM at full tensor rate).
//
// Roles per CTA: warp 0 TMA producer (loads its own A rows and its half of B into
// its own shared memory; both CTAs' loads complete on the LEADER's "full" barrier), warp 1
// MMA issuer (leader CTA only; both CTAs' warp 1 take part in the paired TMEM allocation),
// then eight or sixteen epilogue warps (each CTA drains its own accumulator half). Barriers that must be seen
// by both CTAs are signalled twice (own address and the peer's address obtained with
// mapa), so no multicast form of any instruction is used. TMA loads are plain per-CTA loads.
//
// Same operand layouts, addend and rotary epilogues as gemm.cu; no split-K. The fused
// collectives of gemm.cu exist here too (template parameter COMM, two extra warps per CTA):
// all-gather of A's row shards before the product (each CTA pushes a slice of the local shard
// to every peer; the producers wait per row chunk for its arrival) and reduce-scatter of the
// product's rows after it (the epilogue stores partial tiles into the owner's staging area,
// the extra warps sum what the peers delivered). Peer traffic is plain loads/stores.
#include <algorithm>
#include <cstdio>

#include "api.h"
#include "common.cuh"

using namespace gfs;

namespace {

constexpr int BM = 128;        // rows per CTA (256 per pair)
constexpr int BNH = 128;       // B rows (output columns) held per CTA
constexpr int BN = 256;        // output columns per tile
constexpr int BK = 64;
constexpr int STAGES = 6;
constexpr int THREADS = 192;
constexpr int COMM_THREADS = 64;
constexpr int MAX_PEERS = 8;
enum CommMode : int { COMM_NONE = 0, COMM_ALLGATHER = 1, COMM_REDUCE_SCATTER = 2 };

struct CommParams {
  int world, rank;
  int rows_per_rank;                    // rows of the sharded dimension per rank (multiple of 256)
  const __nv_bfloat16* ag_src;          // all-gather: local shard [rows_per_rank, ag_cols], pitch ag_ld
  int ag_ld, ag_cols;
  __nv_bfloat16* peer_buf[MAX_PEERS];   // AG: gathered [world*rows_per_rank, ag_cols]; RS: staging [world][rows_per_rank][N]
  __nv_bfloat16* rs_out;                // reduce-scatter: out[rows_per_rank, N] = sum of partial rows (+ residual)
  const __nv_bfloat16* rs_res;
  int rs_ld_out, rs_ld_res;
  __nv_bfloat16* mc_buf;                // all-gather: multicast address of the gathered buffers, or null
  uint32_t* peer_flags[MAX_PEERS];      // flags[p][src]: progress of rank src's writes into rank p
  uint32_t target;                      // value flags[rank][src] must reach in this call
  unsigned long long wait_ns;
};
constexpr int A_BYTES = BM * BK * 2;     // 16 KB
constexpr int B_BYTES = BNH * BK * 2;    // 16 KB
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int EPI_BYTES = 8 * 4096;     // one [32 rows x 128 B] transpose buffer per epilogue warp
// Epilogue warps per CTA (template parameter EW).
// Sixteen, for products without a collective and a K loop of up to 16 blocks: one [32 rows x 64 columns] unit of the CTA's
// 128 x 256 half tile each, results (and the addend) moving by TMA through 4 KB of shared memory per warp. At K = 768 (7,100
// cycles) eight warps with two units each, loads and stores of their own, took longer than the loop as soon as the
// epilogue had anything to compute, and a kernel's last epilogue is never hidden. The price is one of six ring stages
// (SWI == 2: two, for 6 KB per warp: gate | up on the way in and the results on the way out), which a long loop feels.
// Both sides, us, eight -> sixteen warps (SwiGLU backward up to K 1024: eight with TMA boxes of 64 columns, a variant that is
// gone):
//   K                              256         512         768         1024        1152        1280        1536        2048
//   SwiGLU fwd [8192, 2 x 3072]  57 -> 46    72 -> 58    82 -> 69   100 -> 95   108 -> 104  115 -> 116  128 -> 136  164 -> 173
//   SwiGLU bwd [8192, 3072]      56 -> 54    69 -> 66    68 -> 62    84 -> 75    86 -> 78    85 -> 80    92 -> 95   105 -> 118
//   LM head [4096, 32000]       128 -> 97   174 -> 139  213 -> 181  260 -> 244  299 -> 300  279 -> 299  351 -> 374  452 -> 463
//   addend [8192, 2304]          26 -> 19    31 -> 23    35 -> 30    41 -> 38.5  42 -> 41    46 -> 47    51 -> 54    65 -> 69
//   rotary [8192, 2304]          34 -> 19    38 -> 23    43 -> 29    51 -> 38    53 -> 40    55 -> 43    62 -> 51    76 -> 68
// The rotary one always has sixteen. A plain epilogue has nothing to compute, and the line for it lies lower (and above one
// tile per pair: a last epilogue alone is as short with eight, and the CTAs are set up sooner):
//   plain, K                       256         384         512         576         640         768         1024
//   [4096, 1024], 64 tiles        7.3 -> 7.6  8.7 -> 9.0 11.1 -> 11.5 12.0 -> 12.4 12.5 -> 12.8 13.6 -> 14.0 15.5 -> 15.9
//   [8192, 768], 96 tiles         9.6 -> 9.1 10.6 -> 10.1 11.8 -> 11.7 13.8 -> 13.3 12.7 -> 12.7 14.2 -> 14.6 15.4 -> 15.7
//   [8192, 2304], 288 tiles      16.8 -> 14.5 18.3 -> 15.9 19.3 -> 17.7 20.4 -> 19.1 21.0 -> 20.2 23.3 -> 23.0 28.9 -> 29.3
// Eight, for the others (two per TMEM lane quarter, half of the tile's columns each); variants with collectives have two
// more warps for the transfers.
constexpr int EW16_MAX_K = 1024, EW16_PLAIN_MAX_K = 640;
__host__ __device__ constexpr int threads2(int comm, int ew) { return 64 + 32 * ew + (comm != 0 ? 64 : 0); }
__host__ __device__ constexpr int slot_bytes2(int ew, int swi) { return ew == 16 && swi == 2 ? 6144 : 4096; }
__host__ __device__ constexpr int stages2(int ew, int swi) { return ew != 16 ? STAGES : swi == 2 ? 4 : 5; }
__host__ __device__ constexpr int epi_bytes2(int ew, int swi) { return ew * slot_bytes2(ew, swi); }
constexpr int BAR_BYTES = 512;
constexpr int XCH_BYTES = 8 * 32 * 8;   // SWI == 3: a (max, sum) pair per row and 128-column slice
constexpr int SMEM_TOTAL = STAGES * STAGE_BYTES + EPI_BYTES + 256 + 1024;
// (with sixteen warps the base is used as it is, 1024-byte aligned)
__host__ __device__ constexpr int smem2(int ew, int swi) {
  return stages2(ew, swi) * STAGE_BYTES + epi_bytes2(ew, swi) + BAR_BYTES + (ew == 16 ? XCH_BYTES : 1024);
}
static_assert(smem2(16, 0) <= 232448 && smem2(16, 2) <= 232448, "shared memory of an SM");

struct Params2 {
  int M, N, K;
  int ldc, ldr;
  __nv_bfloat16* C;
  const __nv_bfloat16* R;  // addend (may alias C) or null
  int tiles_m, tiles_n, kblocks;
  int group_m;             // see tile_coords
  int early_b, late_wait;  // gfs_host::LaunchHints (without collectives)
  uint32_t* status;
  const float* rope_cos;
  const float* rope_sin;
  int rope_cols, rope_d, rope_b;
  // SwiGLU fusion (template parameter SWI). 1 (forward, B = [gate rows | up rows] of a [2I, K]
  // weight): a tile pairs 128 gate columns (leader CTA's B rows) with the matching 128 up columns
  // (the other CTA's); the epilogue writes both halves of the projection (C, pitch ldc) and
  // act = silu(gate) * up (swi_act, pitch swi_ld). 2 (backward, the product is d_act [M, I]):
  // the epilogue reads gate/up from swi_gu (pitch swi_ld) and writes d_gate | d_up into C
  // ([M, 2I], pitch ldc) instead of d_act.
  int swi_I, swi_ld;
  __nv_bfloat16* swi_act;
  const __nv_bfloat16* swi_gu;
  // SWI == 5: rotary embedding of the first rope_cols columns (sixteen warps; with eight, a run-time switch).
  // SWI == 3 (LM head): besides storing the logits, every epilogue warp writes the online-softmax
  // statistics (max, sum exp(x - max)) of its 128 columns of each row, computed from the
  // bf16-rounded logits: ce_partials[(tile_n * 2 + column half) * M + row]. A small kernel
  // combines them, so the cross entropy needs no pass over the logits in the forward.
  float2* ce_partials;
  // Debugging aid (gfs_gemm2_set_trace): when set, every CTA records SM-clock stamps of its phases
  // in trace[blockIdx.x * 16 + slot] (see TRACE_* below); null in normal operation.
  unsigned long long* trace;
  CommParams comm;
};

enum TraceSlot : int {
  TRACE_GLOBAL_NS = 0,   // globaltimer at kernel entry (to line CTAs up against each other)
  TRACE_ENTRY = 1,       // clock64 at kernel entry; the slots below are clock64 too
  TRACE_SETUP_DONE = 2,  // barriers initialised, TMEM allocated, cluster synchronised
  TRACE_FIRST_TMA = 3,   // producer issued its first load (after the all-gather flag wait, if any)
  TRACE_FIRST_MMA = 4,   // MMA warp committed its first tile
  TRACE_EPI_BEGIN = 5,   // first epilogue warp: first accumulator ready
  TRACE_EPI_FIRST = 6,   //   ... first tile written
  TRACE_EPI_LAST = 7,    //   ... last tile written
  TRACE_RED_BEGIN = 8,   // reduce-scatter: every source's partials have arrived
  TRACE_RED_END = 9,     //   ... this warp's share of the reduction is done
  TRACE_PUSH_DONE = 10,  // all-gather: this warp's share of the push is done
  TRACE_EXIT = 11,       // after the final cluster synchronisation
  TRACE_TILES = 12,      // tiles this CTA pair processed
};
__device__ __forceinline__ void trace_stamp(const Params2& p, int slot) {
  if (p.trace != nullptr) p.trace[blockIdx.x * 16 + slot] = static_cast<unsigned long long>(clock64());
}

// Tile t of a plain product. Row by row, or (group_m > 0) in panels of group_m tile rows, column by column within.
__device__ __forceinline__ void tile_coords(const Params2& p, int t, int& tm, int& tn) {
  if (p.group_m == 0) {
    tm = t / p.tiles_n;
    tn = t - tm * p.tiles_n;
    return;
  }
  const int per_panel = p.group_m * p.tiles_n;
  const int panel = t / per_panel;
  const int rem = t - panel * per_panel;
  const int rows = min(p.group_m, p.tiles_m - panel * p.group_m);
  tn = rem / rows;
  tm = panel * p.group_m + rem - tn * rows;
}

// Tile t -> first row of the pair tile, first column, and (fused collectives) the row chunk.
// The collectives walk the ranks' row chunks in a rotated order: all-gather starts with the
// local chunk (already in place), reduce-scatter ends with it.
template <int COMM>
__device__ __forceinline__ void decode_tile2(const Params2& p, int t, int& m0, int& n0, int& chunk) {
  if (COMM == COMM_NONE) {
    int tm, tn;
    tile_coords(p, t, tm, tn);
    m0 = tm * 256;
    n0 = tn * BN;
    chunk = 0;
  } else {
    const int tiles_per_chunk = (p.comm.rows_per_rank / 256) * p.tiles_n;
    const int ci = t / tiles_per_chunk;
    const int rem = t - ci * tiles_per_chunk;
    chunk = (p.comm.rank + ci + (COMM == COMM_REDUCE_SCATTER ? 1 : 0)) % p.comm.world;
    m0 = chunk * p.comm.rows_per_rank + (rem / p.tiles_n) * 256;
    n0 = (rem % p.tiles_n) * BN;
  }
}

// The epilogue of a warp where there are sixteen: rows [32 q, + 32) and one sixteenth of the columns of each of the
// CTA's half tiles, a row per thread. Results leave through `slot` (4 KB, this warp's) by TMA, which clips what lies
// outside the matrices and writes whole segments; the accumulator is handed back as soon as it has been read.
//   SWI 0  64 columns; + R, which TMA has brought into the slot while the previous tiles were worked on
//   SWI 5  64 columns, rotary embedding
//   SWI 3  64 columns and their share of the row statistics
//   SWI 1  32 gate and 32 up columns -> both and act
//   SWI 2  64 columns of d_act in two chunks: gate | up of a chunk come into the slot one chunk ahead (the next box is asked
//          for as soon as this one is in registers), their gradients leave one after the other through 2 KB behind it
// 64-column boxes are swizzled over 128-byte rows, 32-column ones (SWI 1, 2) over 64-byte rows, so that threads that
// own rows meet no bank conflicts.
template <int SWI>
__device__ __forceinline__ void epilogue16(const Params2& p, const CUtensorMap& tmap_x, const CUtensorMap& tmap_y,
                                               uint8_t* slot, uint64_t* bar, float2* xch_all, uint64_t* tmem_full,
                                               uint64_t* tmem_empty, uint32_t tmem_base, int rank, int pair,
                                               int num_pairs, int total_tiles, int ew, int q, const WaitCtx& wctx) {
  const int lane = threadIdx.x & 31;
  const int cg = ew >> 2;                                      // column group of the tile
  constexpr int COLS = SWI == 1 ? 32 : 64;                     // output columns of this warp (SWI 1: of gate)
  const int col_limit = (SWI == 1 || SWI == 2) ? p.swi_I : p.N;
  const uint32_t sw128 = lane & 7, sw64 = (lane >> 1) & 3;
  uint8_t* const row128 = slot + lane * 128;
  uint8_t* const row64 = slot + lane * 64;
  const bool has_add = SWI == 0 && p.R != nullptr;
  auto tile_origin = [&](int t, int& row0, int& col0) {
    int tm, tn;
    tile_coords(p, t, tm, tn);
    row0 = tm * 256 + rank * BM + q * 32;
    col0 = tn * (SWI == 1 ? BN / 2 : BN) + cg * COLS;
  };
  // loads into the slot, one box ahead: the addend of the next live tile, or the next chunk of gate | up
  uint32_t n_box = 0;
  int pf_t = pair, pf_h = 0;
  auto prefetch = [&]() {
    for (; pf_t < total_tiles; pf_t += num_pairs, pf_h = 0) {
      int row0, col0;
      tile_origin(pf_t, row0, col0);
      col0 += 32 * pf_h;
      if (row0 >= p.M || col0 >= col_limit) continue;
      if (lane == 0) {
        if (SWI != 2) bulk_wait_read_all();   // the slot's previous results have left it
        mbar_arrive_expect_tx(bar, 4096);
        if (SWI == 2) {
          tma_load_3d(slot, &tmap_x, bar, col0, 0, row0);
          tma_load_3d(slot + 2048, &tmap_x, bar, col0, 1, row0);
        } else {
          tma_load_2d(slot, &tmap_x, bar, col0, row0);
        }
      }
      if (SWI == 2 && pf_h == 0) pf_h = 1;
      else { pf_h = 0; pf_t += num_pairs; }
      return;
    }
  };
  if (SWI == 2 || has_add) prefetch();

  int acc = 0;
  uint32_t acc_phase = 0;
  uint32_t n_tile = 0;
  for (int t = pair; t < total_tiles; t += num_pairs, ++n_tile) {
    int row0, col0;
    tile_origin(t, row0, col0);
    const bool live = row0 < p.M && col0 < col_limit;
    // rotary table entries of the vectors that this lane turns, the first half ahead of the accumulator
    float4 cs[4], sn[4];
    const int rrow = lane >> 3, gcol = col0 + (lane & 7) * 8;
    const bool rope = SWI == 5 && live && col0 < p.rope_cols;
    auto load_rope = [&](int i0) {
      const int d2 = (gcol % p.rope_d) >> 1;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int s = min(row0 + (i0 + i) * 4 + rrow, p.M - 1) / p.rope_b;
        const size_t at = static_cast<size_t>(s) * (p.rope_d >> 1) + d2;
        cs[i] = *reinterpret_cast<const float4*>(p.rope_cos + at);
        sn[i] = *reinterpret_cast<const float4*>(p.rope_sin + at);
      }
    };
    if (rope) load_rope(0);
    mbar_wait(&tmem_full[acc], acc_phase, wctx, STATUS_TIMEOUT_TMEM_FULL);
    if (t == pair && ew == 0 && lane == 0) trace_stamp(p, TRACE_EPI_BEGIN);
    tc_fence_after();
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN + cg * COLS;
    auto release = [&]() {      // the accumulator may be overwritten once all epilogue warps of the pair have read it
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&tmem_empty[acc]), 0));
    };
    auto slot_free = [&]() {    // the previous tile's results have left the slot
      if (lane == 0) bulk_wait_read_all();
      __syncwarp();
    };
    float ce_m = -INFINITY, ce_s = 0.f;
    if (!live) {
      release();
    } else if (SWI == 1) {
      uint32_t vg[32], vu[32];
      tmem_ld_32x32(t_row, vg);
      tmem_ld_32x32(t_row + BN / 2, vu);
      slot_free();
      tmem_ld_wait_for(vg);
      tmem_ld_wait_for(vu);
      release();
      uint32_t pg[16], pu[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        pg[e] = pack_bf16x2(__uint_as_float(vg[2 * e]), __uint_as_float(vg[2 * e + 1]));
        pu[e] = pack_bf16x2(__uint_as_float(vu[2 * e]), __uint_as_float(vu[2 * e + 1]));
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint8_t* at = row64 + ((j ^ sw64) << 4);
        *reinterpret_cast<uint4*>(at) = make_uint4(pg[4 * j], pg[4 * j + 1], pg[4 * j + 2], pg[4 * j + 3]);
        *reinterpret_cast<uint4*>(at + 2048) = make_uint4(pu[4 * j], pu[4 * j + 1], pu[4 * j + 2], pu[4 * j + 3]);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_3d(&tmap_y, slot, col0, 0, row0);
        tma_store_3d(&tmap_y, slot + 2048, col0, 1, row0);
        bulk_commit();
      }
      // act from the bf16-rounded projections, silu rounded to bf16 before the product
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const float2 g2 = unpack_bf16x2(pg[e]), u2 = unpack_bf16x2(pu[e]);
        const float s0 = __bfloat162float(__float2bfloat16_rn(g2.x * sigmoid_f(g2.x)));
        const float s1 = __bfloat162float(__float2bfloat16_rn(g2.y * sigmoid_f(g2.y)));
        pg[e] = pack_bf16x2(s0 * u2.x, s1 * u2.y);
      }
      slot_free();
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<uint4*>(row64 + ((j ^ sw64) << 4)) =
            make_uint4(pg[4 * j], pg[4 * j + 1], pg[4 * j + 2], pg[4 * j + 3]);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(&tmap_x, slot, col0, row0);
        bulk_commit();
      }
    } else if (SWI == 2) {
      const uint64_t one2 = pack_f32x2(1.f, 1.f), neg_one2 = pack_f32x2(-1.f, -1.f);
      auto pair_of = [](uint32_t u) {
        const float2 f = unpack_bf16x2(u);
        return pack_f32x2(f.x, f.y);
      };
      auto packed = [](uint64_t v) {
        const float2 f = unpack_f32x2(v);
        return pack_bf16x2(f.x, f.y);
      };
      const int chunks = col0 + 32 < col_limit ? 2 : 1;
#pragma unroll 1
      for (int h = 0; h < chunks; ++h) {
        uint32_t pd[16];    // d_act rounded to bf16, as when it is a tensor of its own
        {
          uint32_t va[32];
          tmem_ld_32x32(t_row + 32 * h, va);
          tmem_ld_wait_for(va);
#pragma unroll
          for (int e = 0; e < 16; ++e)
            pd[e] = pack_bf16x2(__uint_as_float(va[2 * e]), __uint_as_float(va[2 * e + 1]));
        }
        if (h == chunks - 1) release();
        mbar_wait(bar, n_box & 1, wctx, STATUS_TIMEOUT_PIPE_FULL);
        ++n_box;
        uint4 g4[4], u4[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint8_t* at = row64 + ((j ^ sw64) << 4);
          g4[j] = *reinterpret_cast<const uint4*>(at);
          u4[j] = *reinterpret_cast<const uint4*>(at + 2048);
        }
        __syncwarp();
        prefetch();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint32_t *gp = &g4[j].x, *up = &u4[j].x;
#pragma unroll
          for (int e = 0; e < 4; ++e) {   // two columns per instruction of the FMA pipe
            const float2 g = unpack_bf16x2(gp[e]);
            const uint64_t g2 = pack_f32x2(g.x, g.y), d2 = pair_of(pd[4 * j + e]);
            const uint64_t s2 = pack_f32x2(sigmoid_f(g.x), sigmoid_f(g.y));
            // d_gate = d up sigma (1 + gate (1 - sigma)), d_up = d gate sigma
            const uint64_t t2 = fma_f32x2(g2, fma_f32x2(s2, neg_one2, one2), one2);
            up[e] = packed(mul_f32x2(mul_f32x2(mul_f32x2(d2, pair_of(up[e])), s2), t2));
            gp[e] = packed(mul_f32x2(mul_f32x2(d2, g2), s2));
          }
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {      // d_gate (in u4), d_up (in g4)
          slot_free();
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<uint4*>(row64 + 4096 + ((j ^ sw64) << 4)) = half == 0 ? u4[j] : g4[j];
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_3d(&tmap_y, slot + 4096, col0 + 32 * h, half, row0);
            bulk_commit();
          }
        }
      }
    } else {
      uint32_t pk[32];    // this row's 64 columns, rounded to bf16
      {
        uint32_t va[32], vb[32];
        tmem_ld_32x32(t_row, va);
        tmem_ld_32x32(t_row + 32, vb);
        if (!has_add) slot_free();
        tmem_ld_wait_for(va);
        tmem_ld_wait_for(vb);
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          pk[e] = pack_bf16x2(__uint_as_float(va[2 * e]), __uint_as_float(va[2 * e + 1]));
          pk[16 + e] = pack_bf16x2(__uint_as_float(vb[2 * e]), __uint_as_float(vb[2 * e + 1]));
        }
      }
      release();
      if (has_add) {
        mbar_wait(bar, n_box & 1, wctx, STATUS_TIMEOUT_PIPE_FULL);
        ++n_box;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        uint8_t* at = row128 + ((j ^ sw128) << 4);
        uint4 w = make_uint4(pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
        if (has_add) {
          const uint4 r4 = *reinterpret_cast<const uint4*>(at);
          const uint32_t* rp = &r4.x;
          uint32_t* wp = &w.x;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 a = unpack_bf16x2(wp[e]), r = unpack_bf16x2(rp[e]);
            wp[e] = pack_bf16x2(a.x + r.x, a.y + r.y);
          }
        }
        *reinterpret_cast<uint4*>(at) = w;
      }
      if (rope) {
        // Turned in the transposed order, eight lanes to a row: the table's entries are then read as whole
        // segments (by their rows' threads they would be 32 passes through the load / store unit each).
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (i == 4) load_rope(4);
          const int r = i * 4 + rrow;
          uint4* at = reinterpret_cast<uint4*>(slot + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
          if (gcol < p.rope_cols) {
            uint4 w = *at;
            const float2 a0 = unpack_bf16x2(w.x), a1 = unpack_bf16x2(w.y), a2 = unpack_bf16x2(w.z),
                         a3 = unpack_bf16x2(w.w);
            const float4 c = cs[i & 3], s = sn[i & 3];
            float f[8] = {a0.x * c.x - a0.y * s.x, a0.x * s.x + a0.y * c.x, a1.x * c.y - a1.y * s.y,
                          a1.x * s.y + a1.y * c.y, a2.x * c.z - a2.y * s.z, a2.x * s.z + a2.y * c.z,
                          a3.x * c.w - a3.y * s.w, a3.x * s.w + a3.y * c.w};
            w = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]),
                           pack_bf16x2(f[6], f[7]));
            *at = w;
          }
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(&tmap_y, slot, col0, row0);
        bulk_commit();
      }
      if (has_add) prefetch();
      if (SWI == 3) {
        // fold the row's bf16-rounded values into (max, sum exp(x - max)); columns past N only exist in the last tile
        constexpr float L2E = 1.4426950408889634f;
        const int n_valid = p.N - col0;
        if (n_valid < 64) {
#pragma unroll
          for (int e = 0; e < 32; ++e) {
            const uint32_t lo = (2 * e < n_valid) ? (pk[e] & 0xffffu) : 0xff80u;          // bf16 -inf
            const uint32_t hi = (2 * e + 1 < n_valid) ? (pk[e] & 0xffff0000u) : 0xff800000u;
            pk[e] = lo | hi;
          }
        }
        float cm0 = -INFINITY, cm1 = -INFINITY;
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          cm0 = fmaxf(cm0, __uint_as_float(pk[e] << 16));
          cm1 = fmaxf(cm1, __uint_as_float(pk[e] & 0xffff0000u));
        }
        ce_m = fmaxf(cm0, cm1);
        const float off = (ce_m == -INFINITY) ? 0.f : ce_m * L2E;
        float a0 = 0.f, a1 = 0.f;
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          a0 += fast_exp2(fmaf(__uint_as_float(pk[e] << 16), L2E, -off));
          a1 += fast_exp2(fmaf(__uint_as_float(pk[e] & 0xffff0000u), L2E, -off));
        }
        ce_s = a0 + a1;
      }
    }
    if (SWI == 3) {
      // Two warps share a 128-column slice: one hands its pair over, the other one folds and stores. They change
      // parts with every tile, so the buffer is written by the warp that read it last and one barrier is enough.
      float2* xch = xch_all + (q + 4 * (cg >> 1)) * 32 + lane;
      const bool gives = (cg & 1) != static_cast<int>(n_tile & 1);
      if (gives) *xch = make_float2(ce_m, ce_s);
      named_barrier_sync(1 + q + 4 * (cg >> 1), 64);
      const int part = col0 / 128;
      if (!gives && row0 + lane < p.M) {
        constexpr float L2E = 1.4426950408889634f;
        const float2 o = *xch;
        const float m = fmaxf(ce_m, o.x);
        const float off = (m == -INFINITY) ? 0.f : m;
        const float s = ce_s * fast_exp2((ce_m - off) * L2E) + o.y * fast_exp2((o.x - off) * L2E);
        p.ce_partials[static_cast<size_t>(part) * p.M + row0 + lane] = make_float2(m, s);
      }
    }
    if (ew == 0 && lane == 0) {
      if (t == pair) trace_stamp(p, TRACE_EPI_FIRST);
      trace_stamp(p, TRACE_EPI_LAST);
    }
    if (++acc == 2) {
      acc = 0;
      acc_phase ^= 1u;
    }
  }
  settle_copies(wctx);
  if (lane == 0) bulk_wait_all();
}

template <bool A_MN, bool B_MN, int COMM, int SWI, int EW>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(threads2(COMM, EW), 1)
gemm2_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
             const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_y, const Params2 p) {
  // tmap_x, tmap_y: all-gather: the local shard of A, unused; with sixteen epilogue warps: SWI 0 R, C;
  // 1 act, gate | up; 2 gate | up, d_gate | d_up; 3, 5 unused, C
  constexpr int STAGES = stages2(EW, SWI);
  constexpr int EPI_BYTES = epi_bytes2(EW, SWI);
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  if (EW != 16) {
    smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  } else if (smem_u32(smem_raw) & 1023u) {   // both CTAs of a pair see the same offset
    if (threadIdx.x == 0) record_status(p.status, STATUS_BAD_ARGUMENT, 0x5a14u);
    return;
  }
  uint8_t* tiles = smem;
  uint8_t* epi_smem = smem + STAGES * STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi_smem + EPI_BYTES);
  uint64_t* full_bar = bars;                      // [STAGES]  (used in the leader)
  uint64_t* empty_bar = bars + STAGES;            // [STAGES]  (one per CTA)
  uint64_t* tmem_full = bars + 2 * STAGES;        // [2]       (one per CTA)
  uint64_t* tmem_empty = bars + 2 * STAGES + 2;   // [2]       (used in the leader)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);
  uint32_t* rs_sent = tmem_slot + 2;   // [MAX_PEERS] reduce-scatter: (warp, tile) units stored for each peer
  uint64_t* epi_full = reinterpret_cast<uint64_t*>(rs_sent + MAX_PEERS);   // [warp], sixteen of them

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = (rank == 0);

  if (threadIdx.x < MAX_PEERS) rs_sent[threadIdx.x] = 0u;
  if (threadIdx.x == 0) {
    if (p.trace != nullptr) p.trace[blockIdx.x * 16 + TRACE_GLOBAL_NS] = globaltimer_ns();
    trace_stamp(p, TRACE_ENTRY);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], 2 * EW);
    }
    if (EW == 16) {
      for (int i = 0; i < EW; ++i) mbar_init(&epi_full[i], 1);
      tma_prefetch_desc(&tmap_x);
      tma_prefetch_desc(&tmap_y);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    if (COMM == COMM_ALLGATHER) tma_prefetch_desc(&tmap_x);
  }
  __syncthreads();
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  cluster_sync_all();  // barriers of both CTAs initialised, TMEM allocated
  tc_fence_after();
  // Everything above ran while the preceding kernel of the stream may still have been draining. With early_b the TMA warp
  // waits after its first loads of B, with late_wait everybody at the end.
  const bool late_wait = COMM == COMM_NONE && p.late_wait != 0;
  const bool early_b = COMM == COMM_NONE && p.early_b != 0 && !late_wait;
  if (!late_wait && !(early_b && warp == 0)) pdl_wait();
  if (!(early_b && warp == 0)) pdl_trigger();
  const uint32_t tmem_base = *tmem_slot;
  WaitCtx wctx{abort_flag, p.status, GFS_WAIT_LIMIT_NS};

  const int num_pairs = gridDim.x >> 1;
  const int pair = blockIdx.x >> 1;
  const int total_tiles = p.tiles_m * p.tiles_n;
  if (threadIdx.x == 0) {
    trace_stamp(p, TRACE_SETUP_DONE);
    if (p.trace != nullptr)
      p.trace[blockIdx.x * 16 + TRACE_TILES] = (total_tiles - pair + num_pairs - 1) / num_pairs;
  }

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      uint32_t chunk_ready = 0;  // all-gather: chunks whose arrival has been observed
      auto load_b = [&](int st, int k0, int n0) {
        uint8_t* sb = tiles + st * STAGE_BYTES + A_BYTES;
        const uint32_t bar = mapa_u32(smem_u32(&full_bar[st]), 0);
        if (SWI == 1) {
          // n0 counts interleaved tile columns: gate rows [g0, g0 + 128) for the leader, the
          // matching up rows [I + g0, ...) for the other CTA
          const int g0 = (n0 - static_cast<int>(rank) * BNH) >> 1;
          tma_load_2d_pair(sb, &tmap_b, bar, k0, (rank == 0 ? 0 : p.swi_I) + g0);
        } else if (!B_MN) {
          tma_load_2d_pair(sb, &tmap_b, bar, k0, n0);
        } else {
#pragma unroll
          for (int i = 0; i < BNH / 64; ++i) tma_load_2d_pair(sb + i * 8192, &tmap_b, bar, n0 + 64 * i, k0);
        }
      };
      int early = 0;             // stages whose B is on its way
      if (early_b) {
        int m0, n0, chunk;
        decode_tile2<COMM>(p, pair, m0, n0, chunk);
        n0 += static_cast<int>(rank) * BNH;
        early = min(STAGES, p.kblocks);
        for (int kb = 0; kb < early; ++kb) {
          if (leader) mbar_arrive_expect_tx(&full_bar[kb], 2 * STAGE_BYTES);
          load_b(kb, kb * BK, n0);
        }
        pdl_wait();
        pdl_trigger();
      }
      for (int t = pair; t < total_tiles; t += num_pairs) {
        int m0, n0, chunk;
        decode_tile2<COMM>(p, t, m0, n0, chunk);
        m0 += static_cast<int>(rank) * BM;
        n0 += static_cast<int>(rank) * BNH;
        // all-gather: this rank's own chunk is read straight from its shard (tmap_x), so the
        // first tiles start at once; only the peers' chunks wait for their arrival in the gathered buffer
        const bool local_chunk = (COMM == COMM_ALLGATHER) && chunk == p.comm.rank;
        if (COMM == COMM_ALLGATHER && !local_chunk && !((chunk_ready >> chunk) & 1u)) {
          // rows of this chunk are written into our gathered buffer by rank `chunk`
          if (!*abort_flag &&
              !wait_flag_reached(p.comm.peer_flags[p.comm.rank] + chunk, p.comm.target, p.comm.wait_ns, p.status,
                                 0xA7000000u | (chunk << 8) | p.comm.rank))
            *abort_flag = 1u;
          fence_proxy_async_global();  // peer's generic-proxy stores -> our TMA (async proxy) loads
          chunk_ready |= 1u << chunk;
        }
        if (t == pair) trace_stamp(p, TRACE_FIRST_TMA);
        for (int kb = 0; kb < p.kblocks; ++kb) {
          mbar_wait(&empty_bar[stage], phase ^ 1u, wctx, STATUS_TIMEOUT_PIPE_EMPTY);
          uint8_t* sa = tiles + stage * STAGE_BYTES;
          // the leader's barrier counts the bytes of both CTAs
          if (leader && early == 0) mbar_arrive_expect_tx(&full_bar[stage], 2 * STAGE_BYTES);
          const uint32_t bar = mapa_u32(smem_u32(&full_bar[stage]), 0);
          const int k0 = kb * BK;
          if (!A_MN) {
            if (local_chunk) tma_load_2d_pair(sa, &tmap_x, bar, k0, m0 - chunk * p.comm.rows_per_rank);
            else tma_load_2d_pair(sa, &tmap_a, bar, k0, m0);
          } else {
#pragma unroll
            for (int i = 0; i < BM / 64; ++i) tma_load_2d_pair(sa + i * 8192, &tmap_a, bar, m0 + 64 * i, k0);
          }
          if (early == 0) load_b(stage, k0, n0);
          else --early;
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      settle_copies(wctx);
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader only) ------------------------------
    if (leader) {  // whole warp, converged: the MMA / commit helpers elect the issuing lane
      constexpr uint32_t idesc = umma_idesc_bf16(256, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int t = pair; t < total_tiles; t += num_pairs) {
        mbar_wait(&tmem_empty[acc], acc_phase ^ 1u, wctx, STATUS_TIMEOUT_TMEM_EMPTY);
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < p.kblocks; ++kb) {
          mbar_wait(&full_bar[stage], phase, wctx, STATUS_TIMEOUT_PIPE_FULL);
          tc_fence_after();
          const uint32_t sa = smem_u32(tiles + stage * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t adesc = A_MN ? umma_desc_sw128(sa + k * 2048, 8192, 1024)
                                        : umma_desc_sw128(sa + k * 32, 16, 1024);
            const uint64_t bdesc = B_MN ? umma_desc_sw128(sb + k * 2048, 8192, 1024)
                                        : umma_desc_sw128(sb + k * 32, 16, 1024);
            umma_ss_pair(d_tmem, adesc, bdesc, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          }
          // free this stage in both CTAs once the MMAs above have read it
          umma_commit_pair(mapa_u32(smem_u32(&empty_bar[stage]), 0));
          umma_commit_pair(mapa_u32(smem_u32(&empty_bar[stage]), 1));
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        umma_commit_pair(mapa_u32(smem_u32(&tmem_full[acc]), 0));
        umma_commit_pair(mapa_u32(smem_u32(&tmem_full[acc]), 1));
        if (t == pair && lane == 0) trace_stamp(p, TRACE_FIRST_MMA);
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
    }
  } else if (warp < 2 + EW) {
    // ------------------------------ epilogue (both CTAs, own accumulator half) ------------------------------
    if constexpr (EW == 16) {
      epilogue16<SWI>(p, tmap_x, tmap_y, epi_smem + (warp - 2) * slot_bytes2(EW, SWI), &epi_full[warp - 2],
                          reinterpret_cast<float2*>(epi_smem + EPI_BYTES + BAR_BYTES), tmem_full, tmem_empty, tmem_base,
                          static_cast<int>(rank), pair, num_pairs, total_tiles, warp - 2, warp & 3, wctx);
    } else {
      // all-gather variant: until the first accumulator is ready these warps help the two push warps
      if (COMM == COMM_ALLGATHER) {
        ag_push_rows(p.comm, static_cast<int>(threadIdx.x) - 64, COMM_THREADS + 32 * EW, 1);
        if (warp == 2 && lane == 0) trace_stamp(p, TRACE_PUSH_DONE);
      }
      bool rs_handed_over = false;                          // reduce-scatter: remote tiles handed to the signalling warp
      const int q = warp & 3;                               // TMEM lane quarter this warp may access
      const int c_begin = ((warp - 2) >> 2) * (BN / 2);     // this warp's column range of the tile
      const int c_end = c_begin + BN / 2;
      int acc = 0;
      uint32_t acc_phase = 0;
      uint8_t* ebuf = epi_smem + (warp - 2) * 4096;
      const int rrow = lane >> 3;
      const int rch = lane & 7;
      const bool has_add = p.R != nullptr;
      // The addend of a 64-column chunk is fetched one chunk ahead (across tile boundaries too), so
      // its global-memory latency is covered by the previous chunk's work instead of stalling this one.
      uint4 pre[8];
      auto load_addend = [&](uint4 (&dst)[8], int mm0, int col0) {
        const int gc = col0 + rch * 8;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int grow = mm0 + q * 32 + i * 4 + rrow;
          dst[i] = make_uint4(0, 0, 0, 0);
          if (grow < p.M && gc + 8 <= p.N)
            dst[i] = *reinterpret_cast<const uint4*>(p.R + static_cast<size_t>(grow) * p.ldr + gc);
        }
      };
      auto load_addend_of_tile = [&](int t) {   // this warp's first chunk there
        if (t >= total_tiles) return;
        int fm0, fn0, fchunk;
        decode_tile2<COMM>(p, t, fm0, fn0, fchunk);
        load_addend(pre, fm0 + static_cast<int>(rank) * BM, fn0 + c_begin);
      };
      if (has_add) load_addend_of_tile(pair);
      for (int t = pair; t < total_tiles; t += num_pairs) {
        int m0, n0, chunk;
        decode_tile2<COMM>(p, t, m0, n0, chunk);
        m0 += static_cast<int>(rank) * BM;
        mbar_wait(&tmem_full[acc], acc_phase, wctx, STATUS_TIMEOUT_TMEM_FULL);
        if (t == pair && warp == 2 && lane == 0) trace_stamp(p, TRACE_EPI_BEGIN);
        tc_fence_after();
        const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN;
        if (SWI == 1) {
          // accumulator columns [0,128) are gate, [128,256) the matching up columns
          const int g0 = n0 >> 1;  // first gate column of the tile
          const int sc_begin = ((warp - 2) >> 2) * 64;
          const int sc_end = sc_begin + 64;
#pragma unroll 1
          for (int c = sc_begin; c < sc_end; c += 32) {
            if (g0 + c >= p.swi_I) break;
            uint32_t vg[32], vu[32];
            tmem_ld_32x32(t_row + c, vg);
            tmem_ld_32x32(t_row + BN / 2 + c, vu);
            tmem_ld_wait();
            uint32_t pa[16];
            uint8_t* myrow = ebuf + lane * 128;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint4 wg, wu;
              uint32_t* wgp = &wg.x;
              uint32_t* wup = &wu.x;
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                wgp[e] = pack_bf16x2(__uint_as_float(vg[8 * j + 2 * e]), __uint_as_float(vg[8 * j + 2 * e + 1]));
                wup[e] = pack_bf16x2(__uint_as_float(vu[8 * j + 2 * e]), __uint_as_float(vu[8 * j + 2 * e + 1]));
                // act from the bf16-rounded projections, silu rounded to bf16 before the product
                const float2 g2 = unpack_bf16x2(wgp[e]), u2 = unpack_bf16x2(wup[e]);
                const float s0 = __bfloat162float(__float2bfloat16_rn(g2.x * sigmoid_f(g2.x)));
                const float s1 = __bfloat162float(__float2bfloat16_rn(g2.y * sigmoid_f(g2.y)));
                pa[4 * j + e] = pack_bf16x2(s0 * u2.x, s1 * u2.y);
              }
              *reinterpret_cast<uint4*>(myrow + ((j ^ (lane & 7)) << 4)) = wg;
              *reinterpret_cast<uint4*>(myrow + (((4 + j) ^ (lane & 7)) << 4)) = wu;
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 8; ++i) {  // gate | up halves of the projection
              const int r = i * 4 + rrow;
              const int grow = m0 + q * 32 + r;
              const int lc = g0 + c + (rch & 3) * 8;  // column inside [0, I)
              const uint4 w = *reinterpret_cast<const uint4*>(ebuf + r * 128 + ((rch ^ (r & 7)) << 4));
              if (grow < p.M && lc + 8 <= p.swi_I)
                *reinterpret_cast<uint4*>(p.C + static_cast<size_t>(grow) * p.ldc + (rch >= 4 ? p.swi_I : 0) + lc) = w;
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 4; ++j)
              *reinterpret_cast<uint4*>(myrow + ((j ^ (lane & 7)) << 4)) =
                  make_uint4(pa[4 * j], pa[4 * j + 1], pa[4 * j + 2], pa[4 * j + 3]);
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 4; ++i) {  // act: 32 columns per row, 4 lanes per row
              const int r = i * 8 + (lane >> 2);
              const int ch = lane & 3;
              const int grow = m0 + q * 32 + r;
              const int lc = g0 + c + ch * 8;
              const uint4 w = *reinterpret_cast<const uint4*>(ebuf + r * 128 + ((ch ^ (r & 7)) << 4));
              if (grow < p.M && lc + 8 <= p.swi_I)
                *reinterpret_cast<uint4*>(p.swi_act + static_cast<size_t>(grow) * p.swi_ld + lc) = w;
            }
            __syncwarp();
          }
        } else {
          float ce_m = -INFINITY, ce_s = 0.f;   // SWI == 3: running statistics of this lane's row
          if (has_add && n0 + c_begin >= p.N) load_addend_of_tile(t + num_pairs);   // no chunk of this tile does it
#pragma unroll 1
          for (int c = c_begin; c < c_end; c += 64) {
            const int col0 = n0 + c;
            if (col0 >= p.N) break;
            const int gcol = col0 + rch * 8;
            uint4 cur[8];
            uint4 gq[8], uq[8];
            if (SWI == 2) {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const int grow = m0 + q * 32 + i * 4 + rrow;
                gq[i] = make_uint4(0, 0, 0, 0);
                uq[i] = make_uint4(0, 0, 0, 0);
                if (grow < p.M && gcol + 8 <= p.N) {
                  const __nv_bfloat16* gp = p.swi_gu + static_cast<size_t>(grow) * p.swi_ld + gcol;
                  gq[i] = *reinterpret_cast<const uint4*>(gp);
                  uq[i] = *reinterpret_cast<const uint4*>(gp + p.swi_I);
                }
              }
            }
            if (has_add) {
#pragma unroll
              for (int i = 0; i < 8; ++i) cur[i] = pre[i];
              if (c + 64 < c_end && col0 + 64 < p.N) load_addend(pre, m0, col0 + 64);
              else load_addend_of_tile(t + num_pairs);
            }
            uint32_t va[32], vb[32];
            tmem_ld_32x32(t_row + c, va);
            tmem_ld_32x32(t_row + c + 32, vb);
            tmem_ld_wait();
            uint8_t* myrow = ebuf + lane * 128;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint4 w;
              w.x = pack_bf16x2(__uint_as_float(va[8 * j + 0]), __uint_as_float(va[8 * j + 1]));
              w.y = pack_bf16x2(__uint_as_float(va[8 * j + 2]), __uint_as_float(va[8 * j + 3]));
              w.z = pack_bf16x2(__uint_as_float(va[8 * j + 4]), __uint_as_float(va[8 * j + 5]));
              w.w = pack_bf16x2(__uint_as_float(va[8 * j + 6]), __uint_as_float(va[8 * j + 7]));
              *reinterpret_cast<uint4*>(myrow + ((j ^ (lane & 7)) << 4)) = w;
              w.x = pack_bf16x2(__uint_as_float(vb[8 * j + 0]), __uint_as_float(vb[8 * j + 1]));
              w.y = pack_bf16x2(__uint_as_float(vb[8 * j + 2]), __uint_as_float(vb[8 * j + 3]));
              w.z = pack_bf16x2(__uint_as_float(vb[8 * j + 4]), __uint_as_float(vb[8 * j + 5]));
              w.w = pack_bf16x2(__uint_as_float(vb[8 * j + 6]), __uint_as_float(vb[8 * j + 7]));
              *reinterpret_cast<uint4*>(myrow + (((4 + j) ^ (lane & 7)) << 4)) = w;
            }
            if (SWI == 3) {
              // this lane still holds its own row's 64 columns: fold their bf16-rounded values (read
              // back from the words it just wrote for the transpose) into the row's running
              // (max, sum-exp). Columns past N only exist in the last tile (warp-uniform test).
              constexpr float L2E = 1.4426950408889634f;
              const int n_valid = min(64, p.N - col0);
              uint32_t pk[32];
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const uint4 t = *reinterpret_cast<const uint4*>(myrow + ((j ^ (lane & 7)) << 4));
                pk[4 * j + 0] = t.x; pk[4 * j + 1] = t.y; pk[4 * j + 2] = t.z; pk[4 * j + 3] = t.w;
              }
              if (n_valid < 64) {
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                  const uint32_t lo = (2 * e < n_valid) ? (pk[e] & 0xffffu) : 0xff80u;          // bf16 -inf
                  const uint32_t hi = (2 * e + 1 < n_valid) ? (pk[e] & 0xffff0000u) : 0xff800000u;
                  pk[e] = lo | hi;
                }
              }
              float cm0 = -INFINITY, cm1 = -INFINITY;
#pragma unroll
              for (int e = 0; e < 32; ++e) {
                cm0 = fmaxf(cm0, __uint_as_float(pk[e] << 16));
                cm1 = fmaxf(cm1, __uint_as_float(pk[e] & 0xffff0000u));
              }
              const float nm = fmaxf(ce_m, fmaxf(cm0, cm1));
              const float off = (nm == -INFINITY) ? 0.f : nm * L2E;
              float a0 = 0.f, a1 = 0.f;
#pragma unroll
              for (int e = 0; e < 32; ++e) {
                a0 += fast_exp2(fmaf(__uint_as_float(pk[e] << 16), L2E, -off));
                a1 += fast_exp2(fmaf(__uint_as_float(pk[e] & 0xffff0000u), L2E, -off));
              }
              ce_s = ce_s * fast_exp2((ce_m == -INFINITY) ? -INFINITY : (ce_m - nm) * L2E) + (a0 + a1);
              ce_m = nm;
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int r = i * 4 + rrow;
              const int grow = m0 + q * 32 + r;
              uint4 w = *reinterpret_cast<const uint4*>(ebuf + r * 128 + ((rch ^ (r & 7)) << 4));
              if (SWI == 2) {
                // w holds 8 values of d_act; turn them into d_gate and d_up
                if (grow < p.M && gcol + 8 <= p.N) {
                  const uint32_t* dw = &w.x;
                  const uint32_t* gw = &gq[i].x;
                  const uint32_t* uw = &uq[i].x;
                  uint4 og, ou;
                  uint32_t* ogp = &og.x;
                  uint32_t* oup = &ou.x;
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    const float2 d2 = unpack_bf16x2(dw[e]), g2 = unpack_bf16x2(gw[e]), u2 = unpack_bf16x2(uw[e]);
                    const float sg0 = sigmoid_f(g2.x), sg1 = sigmoid_f(g2.y);
                    ogp[e] = pack_bf16x2(d2.x * u2.x * sg0 * (1.f + g2.x * (1.f - sg0)),
                                         d2.y * u2.y * sg1 * (1.f + g2.y * (1.f - sg1)));
                    oup[e] = pack_bf16x2(d2.x * g2.x * sg0, d2.y * g2.y * sg1);
                  }
                  __nv_bfloat16* dst = p.C + static_cast<size_t>(grow) * p.ldc + gcol;
                  *reinterpret_cast<uint4*>(dst) = og;
                  *reinterpret_cast<uint4*>(dst + p.swi_I) = ou;
                }
              } else if (grow < p.M && gcol + 8 <= p.N) {
                if (has_add || p.rope_cos != nullptr) {
                  float f[8];
                  const float2 x0 = unpack_bf16x2(w.x), x1 = unpack_bf16x2(w.y), x2 = unpack_bf16x2(w.z),
                               x3 = unpack_bf16x2(w.w);
                  f[0] = x0.x; f[1] = x0.y; f[2] = x1.x; f[3] = x1.y; f[4] = x2.x; f[5] = x2.y; f[6] = x3.x; f[7] = x3.y;
                  if (p.rope_cos != nullptr && gcol < p.rope_cols) {
                    const int half = p.rope_d >> 1;
                    const size_t ti = static_cast<size_t>(grow / p.rope_b) * half + ((gcol % p.rope_d) >> 1);
                    const float4 cs = *reinterpret_cast<const float4*>(p.rope_cos + ti);
                    const float4 sn = *reinterpret_cast<const float4*>(p.rope_sin + ti);
                    const float a0 = f[0], a1 = f[1], a2 = f[2], a3 = f[3], a4 = f[4], a5 = f[5], a6 = f[6], a7 = f[7];
                    f[0] = a0 * cs.x - a1 * sn.x; f[1] = a0 * sn.x + a1 * cs.x;
                    f[2] = a2 * cs.y - a3 * sn.y; f[3] = a2 * sn.y + a3 * cs.y;
                    f[4] = a4 * cs.z - a5 * sn.z; f[5] = a4 * sn.z + a5 * cs.z;
                    f[6] = a6 * cs.w - a7 * sn.w; f[7] = a6 * sn.w + a7 * cs.w;
                  }
                  if (has_add) {
                    const uint4 rr = cur[i];
                    const float2 r0 = unpack_bf16x2(rr.x), r1 = unpack_bf16x2(rr.y), r2 = unpack_bf16x2(rr.z),
                                 r3 = unpack_bf16x2(rr.w);
                    f[0] += r0.x; f[1] += r0.y; f[2] += r1.x; f[3] += r1.y;
                    f[4] += r2.x; f[5] += r2.y; f[6] += r3.x; f[7] += r3.y;
                  }
                  w.x = pack_bf16x2(f[0], f[1]);
                  w.y = pack_bf16x2(f[2], f[3]);
                  w.z = pack_bf16x2(f[4], f[5]);
                  w.w = pack_bf16x2(f[6], f[7]);
                }
                __nv_bfloat16* dst;
                if (COMM == COMM_REDUCE_SCATTER) {
                  // partial rows go to their owner's staging area, slot of this (source) rank
                  dst = p.comm.peer_buf[chunk] +
                        (static_cast<size_t>(p.comm.rank) * p.comm.rows_per_rank +
                         (grow - chunk * p.comm.rows_per_rank)) * p.N + gcol;
                } else {
                  dst = p.C + static_cast<size_t>(grow) * p.ldc + gcol;
                }
                *reinterpret_cast<uint4*>(dst) = w;
              }
            }
            __syncwarp();
          }
          if (SWI == 3) {
            const int row = m0 + q * 32 + lane;
            const int part = (n0 / BN) * 2 + ((warp - 2) >> 2);
            if (row < p.M) p.ce_partials[static_cast<size_t>(part) * p.M + row] = make_float2(ce_m, ce_s);
          }
        }
        tc_fence_before();
        __syncwarp();
        // the accumulator buffer may be overwritten once all epilogue warps of the pair are done
        if (COMM == COMM_REDUCE_SCATTER) {
          // Signalling the owner needs a system-scope release, which costs several microseconds (it
          // waits for every store in flight). It is therefore not done per tile: tiles for the peers
          // come first in every CTA's order; when this warp moves on to the local chunk (or runs out
          // of tiles) it hands the count to the reduction warps, which signal the owners (one release
          // per destination for the whole CTA) while the epilogue warps work on the local chunk. Local tiles only
          // need device scope.
          if (chunk != p.comm.rank) {
            if (lane == 0) atomicAdd(&rs_sent[chunk], 1u);
          } else {
            if (!rs_handed_over) {
              named_barrier_arrive(2, 32 * EW + COMM_THREADS);
              rs_handed_over = true;
            }
            if (lane == 0) red_release_gpu_add_u32(p.comm.peer_flags[chunk] + p.comm.rank, 1u);
          }
        }
        if (lane == 0) {
          mbar_arrive_cluster(mapa_u32(smem_u32(&tmem_empty[acc]), 0));
          if (warp == 2) {
            if (t == pair) trace_stamp(p, TRACE_EPI_FIRST);
            trace_stamp(p, TRACE_EPI_LAST);
          }
        }
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
      if (COMM == COMM_REDUCE_SCATTER) {
        if (!rs_handed_over) named_barrier_arrive(2, 32 * EW + COMM_THREADS);   // CTAs without local tiles
        // tiles done: join the reduction of this rank's row chunk (second share of the vectors)
        const CommParams& c = p.comm;
        bool ok = true;
        for (int src = 0; src < c.world; ++src)
          ok = wait_flag_reached(c.peer_flags[c.rank] + src, c.target, c.wait_ns, p.status,
                                 0xB8000000u | (src << 8) | c.rank) && ok;
        if (!ok) *abort_flag = 1u;
        constexpr int RED_THREADS = COMM_THREADS + 32 * EW;
        rs_reduce_rows(c.peer_buf[c.rank], c.world, c.rows_per_rank, p.N, c.rs_res, c.rs_ld_res, c.rs_out, c.rs_ld_out,
                       static_cast<size_t>(blockIdx.x) * RED_THREADS + COMM_THREADS + (threadIdx.x - 64),
                       static_cast<size_t>(gridDim.x) * RED_THREADS);
      }
    }
  } else if (COMM == COMM_ALLGATHER) {
    // ------------------------------ all-gather push (the last two warps) ------------------------------
    // Every CTA pushes its slice of the local shard into every rank's gathered buffer
    // (own rank first), then bumps that rank's counter for this source.
    // (the epilogue warps push too, before their first tile: see the top of the epilogue branch)
    ag_push_rows(p.comm, static_cast<int>(threadIdx.x) - (threads2(COMM, EW) - COMM_THREADS) + 32 * EW,
                 COMM_THREADS + 32 * EW, 1);
  } else if (COMM == COMM_REDUCE_SCATTER) {
    // ------------------------------ reduce (the last two warps) ------------------------------
    // Wait until every rank (this one included) has delivered all partial tiles of our row
    // chunk, then sum the staged partials in rank order, add the residual, round once.
    const CommParams& c = p.comm;
    const int ct = threadIdx.x - (threads2(COMM, EW) - COMM_THREADS);
    // every epilogue warp of this CTA has stored its tiles for the peers: the owners learn how many (warp, tile) units this CTA delivered to each of them
    named_barrier_sync(2, 32 * EW + COMM_THREADS);
    if (ct < c.world && ct != c.rank) {
      const uint32_t n = rs_sent[ct];
      if (n != 0u) red_release_sys_add_u32(c.peer_flags[ct] + c.rank, n);   // release: cumulative over the barrier
    }
    bool ok = true;
    for (int src = 0; src < c.world; ++src)
      ok = wait_flag_reached(c.peer_flags[c.rank] + src, c.target, c.wait_ns, p.status,
                             0xB7000000u | (src << 8) | c.rank) && ok;
    if (!ok) *abort_flag = 1u;
    if (ct == 0) trace_stamp(p, TRACE_RED_BEGIN);
    // these 64 threads take the first share of the vectors; the epilogue warps take the rest once
    // their tiles are done (see the end of the epilogue loop)
    constexpr int RED_THREADS = COMM_THREADS + 32 * EW;
    rs_reduce_rows(c.peer_buf[c.rank], c.world, c.rows_per_rank, p.N, c.rs_res, c.rs_ld_res, c.rs_out, c.rs_ld_out,
                   static_cast<size_t>(blockIdx.x) * RED_THREADS + ct, static_cast<size_t>(gridDim.x) * RED_THREADS);
    if (ct == 0) trace_stamp(p, TRACE_RED_END);
  }

  if (late_wait) pdl_wait();
  // nobody leaves while the partner may still touch this CTA's shared memory / barriers
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  if (threadIdx.x == 0) trace_stamp(p, TRACE_EXIT);
  if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

// ---------------------------------------------------------------------------
// Grouped weight-gradient GEMM: up to MAX_GROUP independent problems C_g[M_g, N_g] (+)= A_g^T B_g
// (A_g = [K, M_g], B_g = [K, N_g], both row-major, i.e. MN-major operands) in ONE launch. The
// weight gradients of a transformer layer are many-K, few-tile problems (hidden x hidden
// outputs, K = tokens); one by one they fill a fraction of the SMs, together they fill a wave.
// ---------------------------------------------------------------------------
constexpr int MAX_GROUP = 4;

struct GroupMaps {
  CUtensorMap a[MAX_GROUP];
  CUtensorMap b[MAX_GROUP];
};

struct GroupProblem {
  int M, N, ldc;
  int tiles_n, tile_begin, kblocks;
  int accumulate;        // add the product to C instead of overwriting it
  __nv_bfloat16* C;
};

struct GroupParams {
  int ngroups, total_tiles;
  int late_wait;         // gfs_host::LaunchHints
  GroupProblem g[MAX_GROUP];
  uint32_t* status;
};

__device__ __forceinline__ int group_of_tile(const GroupParams& p, int t) {
  int gi = 0;
#pragma unroll
  for (int i = 1; i < MAX_GROUP; ++i)
    if (i < p.ngroups && t >= p.g[i].tile_begin) gi = i;
  return gi;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
gemm2_grouped_kernel(const __grid_constant__ GroupMaps maps, const __grid_constant__ GroupParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* tiles = smem;
  uint8_t* epi_smem = smem + STAGES * STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(epi_smem + EPI_BYTES);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + STAGES;
  uint64_t* tmem_full = bars + 2 * STAGES;
  uint64_t* tmem_empty = bars + 2 * STAGES + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = (rank == 0);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], 8);
    }
    *abort_flag = 0;
    mbar_fence_init();
    for (int i = 0; i < p.ngroups; ++i) {
      tma_prefetch_desc(&maps.a[i]);
      tma_prefetch_desc(&maps.b[i]);
    }
  }
  __syncthreads();
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  if (p.late_wait == 0) pdl_wait();
  pdl_trigger();
  const uint32_t tmem_base = *tmem_slot;
  WaitCtx wctx{abort_flag, p.status, GFS_WAIT_LIMIT_NS};

  const int num_pairs = gridDim.x >> 1;
  const int pair = blockIdx.x >> 1;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int t = pair; t < p.total_tiles; t += num_pairs) {
        const int gi = group_of_tile(p, t);
        const GroupProblem& g = p.g[gi];
        const int lt = t - g.tile_begin;
        const int m0 = (lt / g.tiles_n) * 256 + static_cast<int>(rank) * BM;
        const int n0 = (lt % g.tiles_n) * BN + static_cast<int>(rank) * BNH;
        for (int kb = 0; kb < g.kblocks; ++kb) {
          mbar_wait(&empty_bar[stage], phase ^ 1u, wctx, STATUS_TIMEOUT_PIPE_EMPTY);
          uint8_t* sa = tiles + stage * STAGE_BYTES;
          uint8_t* sb = sa + A_BYTES;
          if (leader) mbar_arrive_expect_tx(&full_bar[stage], 2 * STAGE_BYTES);
          const uint32_t bar = mapa_u32(smem_u32(&full_bar[stage]), 0);
          const int k0 = kb * BK;
#pragma unroll
          for (int i = 0; i < BM / 64; ++i) tma_load_2d_pair(sa + i * 8192, &maps.a[gi], bar, m0 + 64 * i, k0);
#pragma unroll
          for (int i = 0; i < BNH / 64; ++i) tma_load_2d_pair(sb + i * 8192, &maps.b[gi], bar, n0 + 64 * i, k0);
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      settle_copies(wctx);
    }
  } else if (warp == 1) {
    if (leader) {  // whole warp, converged: the MMA / commit helpers elect the issuing lane
      constexpr uint32_t idesc = umma_idesc_bf16(256, BN, 1, 1);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int t = pair; t < p.total_tiles; t += num_pairs) {
        const int kblocks = p.g[group_of_tile(p, t)].kblocks;
        mbar_wait(&tmem_empty[acc], acc_phase ^ 1u, wctx, STATUS_TIMEOUT_TMEM_EMPTY);
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < kblocks; ++kb) {
          mbar_wait(&full_bar[stage], phase, wctx, STATUS_TIMEOUT_PIPE_FULL);
          tc_fence_after();
          const uint32_t sa = smem_u32(tiles + stage * STAGE_BYTES);
          const uint32_t sb = sa + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint64_t adesc = umma_desc_sw128(sa + k * 2048, 8192, 1024);
            const uint64_t bdesc = umma_desc_sw128(sb + k * 2048, 8192, 1024);
            umma_ss_pair(d_tmem, adesc, bdesc, idesc, (kb > 0 || k > 0) ? 1u : 0u);
          }
          umma_commit_pair(mapa_u32(smem_u32(&empty_bar[stage]), 0));
          umma_commit_pair(mapa_u32(smem_u32(&empty_bar[stage]), 1));
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        umma_commit_pair(mapa_u32(smem_u32(&tmem_full[acc]), 0));
        umma_commit_pair(mapa_u32(smem_u32(&tmem_full[acc]), 1));
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
    }
  } else {
    const int q = warp & 3;
    int acc = 0;
    uint32_t acc_phase = 0;
    uint8_t* ebuf = epi_smem + (warp - 2) * 4096;
    const int rrow = lane >> 3;
    const int rch = lane & 7;
    for (int t = pair; t < p.total_tiles; t += num_pairs) {
      const GroupProblem& g = p.g[group_of_tile(p, t)];
      const int lt = t - g.tile_begin;
      const int m0 = (lt / g.tiles_n) * 256 + static_cast<int>(rank) * BM;
      const int n0 = (lt % g.tiles_n) * BN;
      mbar_wait(&tmem_full[acc], acc_phase, wctx, STATUS_TIMEOUT_TMEM_FULL);
      tc_fence_after();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN;
#pragma unroll 1
      for (int c = 0; c < BN; c += 64) {
        const int col0 = n0 + c;
        if (col0 >= g.N) break;
        const int gcol = col0 + rch * 8;
        uint4 pre[8];
        if (g.accumulate) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int grow = m0 + q * 32 + i * 4 + rrow;
            pre[i] = make_uint4(0, 0, 0, 0);
            if (grow < g.M && gcol + 8 <= g.N)
              pre[i] = *reinterpret_cast<const uint4*>(g.C + static_cast<size_t>(grow) * g.ldc + gcol);
          }
        }
        uint32_t va[32], vb[32];
        tmem_ld_32x32(t_row + c, va);
        tmem_ld_32x32(t_row + c + 32, vb);
        tmem_ld_wait();
        uint8_t* myrow = ebuf + lane * 128;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4 w;
          w.x = pack_bf16x2(__uint_as_float(va[8 * j + 0]), __uint_as_float(va[8 * j + 1]));
          w.y = pack_bf16x2(__uint_as_float(va[8 * j + 2]), __uint_as_float(va[8 * j + 3]));
          w.z = pack_bf16x2(__uint_as_float(va[8 * j + 4]), __uint_as_float(va[8 * j + 5]));
          w.w = pack_bf16x2(__uint_as_float(va[8 * j + 6]), __uint_as_float(va[8 * j + 7]));
          *reinterpret_cast<uint4*>(myrow + ((j ^ (lane & 7)) << 4)) = w;
          w.x = pack_bf16x2(__uint_as_float(vb[8 * j + 0]), __uint_as_float(vb[8 * j + 1]));
          w.y = pack_bf16x2(__uint_as_float(vb[8 * j + 2]), __uint_as_float(vb[8 * j + 3]));
          w.z = pack_bf16x2(__uint_as_float(vb[8 * j + 4]), __uint_as_float(vb[8 * j + 5]));
          w.w = pack_bf16x2(__uint_as_float(vb[8 * j + 6]), __uint_as_float(vb[8 * j + 7]));
          *reinterpret_cast<uint4*>(myrow + (((4 + j) ^ (lane & 7)) << 4)) = w;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = i * 4 + rrow;
          const int grow = m0 + q * 32 + r;
          uint4 w = *reinterpret_cast<const uint4*>(ebuf + r * 128 + ((rch ^ (r & 7)) << 4));
          if (grow < g.M && gcol + 8 <= g.N) {
            if (g.accumulate) {
              const uint4 rr = pre[i];
              const float2 x0 = unpack_bf16x2(w.x), x1 = unpack_bf16x2(w.y), x2 = unpack_bf16x2(w.z),
                           x3 = unpack_bf16x2(w.w);
              const float2 r0 = unpack_bf16x2(rr.x), r1 = unpack_bf16x2(rr.y), r2 = unpack_bf16x2(rr.z),
                           r3 = unpack_bf16x2(rr.w);
              w.x = pack_bf16x2(x0.x + r0.x, x0.y + r0.y);
              w.y = pack_bf16x2(x1.x + r1.x, x1.y + r1.y);
              w.z = pack_bf16x2(x2.x + r2.x, x2.y + r2.y);
              w.w = pack_bf16x2(x3.x + r3.x, x3.y + r3.y);
            }
            *reinterpret_cast<uint4*>(g.C + static_cast<size_t>(grow) * g.ldc + gcol) = w;
          }
        }
        __syncwarp();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&tmem_empty[acc]), 0));
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1u;
      }
    }
  }

  if (p.late_wait) pdl_wait();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  tc_fence_after();
  if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

// Tile rows per panel (see tile_coords). Row by row, every 256 rows read the whole of B again, from HBM once it does not
// stay in L2 beside what streams through; a panel of eight reads it an eighth as often, and eight rows of A stay in L2
// instead. From 40 MB of B on. us, row by row -> panels, with the row statistics: 8192 x 50304 x 768 (77 MB) 567 -> 512,
// 8192 x 50304 x 2048 (206 MB) 1387 -> 1200; nothing changes for smaller ones (SwiGLU, 46 MB: 275 -> 271, 9 MB: 130 -> 133).
int panel_rows(const Params2& p) {
  return static_cast<long long>(p.N) * p.K * 2 >= (40ll << 20) && p.tiles_n >= 16 ? 8 : 0;
}

// Debugging aid: device buffer of 16 uint64 per CTA that the next gemm2_kernel launches fill with
// their phase stamps (TraceSlot); null (the default) switches tracing off.
static unsigned long long* g_trace = nullptr;

template <bool A_MN, bool B_MN, int COMM, int SWI, int EW>
int launch2(const CUtensorMap* ta, const CUtensorMap* tb, const Params2& p, int grid, cudaStream_t stream,
            const CUtensorMap* tx = nullptr, const CUtensorMap* ty = nullptr) {
  auto kern = gemm2_kernel<A_MN, B_MN, COMM, SWI, EW>;
  constexpr int smem = smem2(EW, SWI);
  static gfs_host::SmemLimit limit;
  if (!limit.raise(kern, smem)) return -10;
  Params2 pt = p;
  pt.trace = g_trace;
  if (COMM == COMM_NONE) {
    pt.group_m = panel_rows(p);
    pt.early_b = gfs_host::launch_hints().early_b;
    pt.late_wait = gfs_host::launch_hints().late_wait;
  }
  if (gfs_host::launch_pdl(kern, dim3(grid), dim3(threads2(COMM, EW)), smem, stream, *ta, *tb, tx ? *tx : *ta,
                           ty ? *ty : *ta, pt) != cudaSuccess)
    return -11;
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

}  // namespace

extern "C" {

// Debugging aid: subsequent gemm2_kernel launches (all variants, fused collectives included) write
// their per-CTA phase stamps into `buffer` (device memory, 16 uint64 per CTA of the largest grid;
// slots as in TraceSlot, SM clock cycles). Pass null to switch it off again.
void gfs_gemm2_set_trace(void* buffer) { g_trace = static_cast<unsigned long long*>(buffer); }

// C[M,N] = op(A) op(B) (+R) on CTA pairs. Same conventions as gfs_gemm_bf16; intended for
// problems with at least one full wave of 256 x 256 tiles. Returns a negative value when the
// problem cannot be served (the caller then uses the single-CTA kernel).
int gfs_gemm2_bf16(const void* A, const void* B, void* C, const void* R, int M, int N, int K, int lda, int ldb, int ldc,
                   int ldr, int a_mn_major, int b_mn_major, const void* rope_cos, const void* rope_sin, int rope_cols,
                   int rope_d, int rope_b, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((N & 7) || (lda & 7) || (ldb & 7) || (ldc & 7) || (R && (ldr & 7))) return -1;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C) |
       reinterpret_cast<uintptr_t>(R)) & 15)
    return -2;
  const CUtensorMap* ta = a_mn_major ? gfs_host::tmap_2d_cached(A, K, M, lda, 64, 64)
                                     : gfs_host::tmap_2d_cached(A, M, K, lda, BM, 64);
  const CUtensorMap* tb = b_mn_major ? gfs_host::tmap_2d_cached(B, K, N, ldb, 64, 64)
                                     : gfs_host::tmap_2d_cached(B, N, K, ldb, BNH, 64);
  if (ta == nullptr || tb == nullptr) return -3;
  Params2 p{};
  p.M = M; p.N = N; p.K = K;
  p.ldc = ldc; p.ldr = ldr;
  p.C = static_cast<__nv_bfloat16*>(C);
  p.R = static_cast<const __nv_bfloat16*>(R);
  p.tiles_m = (M + 255) / 256;
  p.tiles_n = (N + BN - 1) / BN;
  p.kblocks = (K + BK - 1) / BK;
  p.status = gfs_host::status_words();
  p.rope_cos = static_cast<const float*>(rope_cos);
  p.rope_sin = static_cast<const float*>(rope_sin);
  p.rope_cols = rope_cols; p.rope_d = rope_d; p.rope_b = rope_b > 0 ? rope_b : 1;
  const int pairs = std::min(p.tiles_m * p.tiles_n, gfs_host::sm_count() / 2);
  const int grid = 2 * pairs;
  // the sixteen-warp rotary epilogue is that of a projection x W^T; the eight-warp kernel rotates by a run-time switch
  const bool projection = !a_mn_major && !b_mn_major && R == nullptr;
  const bool ew16 = rope_cos != nullptr ? projection
                    : R != nullptr      ? K <= EW16_MAX_K
                                        : K <= EW16_PLAIN_MAX_K && p.tiles_m * p.tiles_n > pairs;
  const CUtensorMap* tx = ew16 && R != nullptr ? gfs_host::tmap_2d_cached(R, M, N, ldr, 32, 64) : nullptr;
  const CUtensorMap* ty = ew16 ? gfs_host::tmap_2d_cached(C, M, N, ldc, 32, 64) : nullptr;
  if (ew16 && (ty == nullptr || (R != nullptr && tx == nullptr))) return -3;
  if (ew16 && rope_cos != nullptr) return launch2<false, false, COMM_NONE, 5, 16>(ta, tb, p, grid, stream, tx, ty);
  if (ew16) {
    if (!a_mn_major && !b_mn_major) return launch2<false, false, COMM_NONE, 0, 16>(ta, tb, p, grid, stream, tx, ty);
    if (!a_mn_major && b_mn_major) return launch2<false, true, COMM_NONE, 0, 16>(ta, tb, p, grid, stream, tx, ty);
    if (a_mn_major && b_mn_major) return launch2<true, true, COMM_NONE, 0, 16>(ta, tb, p, grid, stream, tx, ty);
    return launch2<true, false, COMM_NONE, 0, 16>(ta, tb, p, grid, stream, tx, ty);
  }
  if (!a_mn_major && !b_mn_major) return launch2<false, false, COMM_NONE, 0, 8>(ta, tb, p, grid, stream);
  if (!a_mn_major && b_mn_major) return launch2<false, true, COMM_NONE, 0, 8>(ta, tb, p, grid, stream);
  if (a_mn_major && b_mn_major) return launch2<true, true, COMM_NONE, 0, 8>(ta, tb, p, grid, stream);
  return launch2<true, false, COMM_NONE, 0, 8>(ta, tb, p, grid, stream);
}

// LM head with cross-entropy statistics: C[M, N] = A[M, K] @ B[N, K]^T (both K-major) and, per row,
// the (max, sum exp(x - max)) of every 128-column slice of the bf16-rounded logits:
// partials is float2 [gfs_gemm2_ce_parts(N)][M]. Returns -20 if the problem is too small for CTA
// pairs (nothing launched).
int gfs_gemm2_ce_parts(int N) { return 2 * ((N + BN - 1) / BN); }

int gfs_gemm2_bf16_ce(const void* A, const void* B, void* C, void* partials, int M, int N, int K, int lda, int ldb,
                      int ldc, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((N & 7) || (lda & 7) || (ldb & 7) || (ldc & 7)) return -1;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C) |
       reinterpret_cast<uintptr_t>(partials)) & 15)
    return -2;
  if (K < 256) return -20;
  const CUtensorMap* ta = gfs_host::tmap_2d_cached(A, M, K, lda, BM, 64);
  const CUtensorMap* tb = gfs_host::tmap_2d_cached(B, N, K, ldb, BNH, 64);
  const CUtensorMap* ty = gfs_host::tmap_2d_cached(C, M, N, ldc, 32, 64);
  if (ta == nullptr || tb == nullptr || ty == nullptr) return -3;
  Params2 p{};
  p.M = M; p.N = N; p.K = K;
  p.ldc = ldc;
  p.C = static_cast<__nv_bfloat16*>(C);
  p.tiles_m = (M + 255) / 256;
  p.tiles_n = (N + BN - 1) / BN;
  p.kblocks = (K + BK - 1) / BK;
  p.status = gfs_host::status_words();
  p.rope_b = 1;
  p.ce_partials = static_cast<float2*>(partials);
  const int pairs = std::min(p.tiles_m * p.tiles_n, gfs_host::sm_count() / 2);
  if (K > EW16_MAX_K) return launch2<false, false, COMM_NONE, 3, 8>(ta, tb, p, 2 * pairs, stream);
  return launch2<false, false, COMM_NONE, 3, 16>(ta, tb, p, 2 * pairs, stream, nullptr, ty);
}

// SwiGLU-fused products of the MLP on CTA pairs; same contract as gfs_gemm_bf16_swiglu (gemm.cu):
//   mode 1: gu[M, 2I] = x[M, K] @ w_gu[2I, K]^T and act[M, I] = silu(gu[:, :I]) * gu[:, I:]
//           (a = x, b = w_gu, c = gu with pitch ldc, extra = act with pitch ld_extra)
//   mode 2: d_gu[M, 2I] = swiglu_backward(d_act = dy[M, K] @ w_down[K, I], gu)
//           (a = dy, b = w_down stored [K, I], c = d_gu with pitch ldc, extra = gu with pitch ld_extra)
int gfs_gemm2_bf16_swiglu(int mode, const void* a, const void* b, void* c, void* extra, int M, int I, int K, int lda,
                          int ldb, int ldc, int ld_extra, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (mode != 1 && mode != 2) return -1;
  if (M <= 0 || I <= 0 || K <= 0) return 0;
  if ((I & 7) || (K & 7) || (lda & 7) || (ldb & 7) || (ldc & 7) || (ld_extra & 7)) return -1;
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
       reinterpret_cast<uintptr_t>(extra)) & 15)
    return -2;
  Params2 p{};
  p.M = M; p.K = K;
  p.N = (mode == 1) ? 2 * I : I;
  p.C = static_cast<__nv_bfloat16*>(c);
  p.ldc = ldc;
  p.tiles_m = (M + 255) / 256;
  p.tiles_n = (mode == 1) ? (I + BN / 2 - 1) / (BN / 2) : (I + BN - 1) / BN;
  p.kblocks = (K + BK - 1) / BK;
  p.status = gfs_host::status_words();
  p.rope_b = 1;
  p.swi_I = I;
  p.swi_ld = ld_extra;
  if (mode == 1) p.swi_act = static_cast<__nv_bfloat16*>(extra);
  else p.swi_gu = static_cast<const __nv_bfloat16*>(extra);
  const CUtensorMap* ta = gfs_host::tmap_2d_cached(a, M, K, lda, BM, 64);
  const CUtensorMap* tb = (mode == 1) ? gfs_host::tmap_2d_cached(b, 2 * I, K, ldb, BNH, 64)
                                      : gfs_host::tmap_2d_cached(b, K, I, ldb, 64, 64);
  if (ta == nullptr || tb == nullptr) return -3;
  const int pairs = std::min(p.tiles_m * p.tiles_n, gfs_host::sm_count() / 2);
  if (K > EW16_MAX_K)
    return mode == 1 ? launch2<false, false, COMM_NONE, 1, 8>(ta, tb, p, 2 * pairs, stream)
                     : launch2<false, true, COMM_NONE, 2, 8>(ta, tb, p, 2 * pairs, stream);
  // gate | up as [row][half][column] (the last gate columns must not run into up), in boxes of 32 rows x 32 columns
  auto halves = [&](const void* base, int ld) {
    const uint64_t dims[3] = {static_cast<uint64_t>(I), 2, static_cast<uint64_t>(M)};
    const uint64_t strides[3] = {2, static_cast<uint64_t>(I) * 2, static_cast<uint64_t>(ld) * 2};
    const uint32_t box[3] = {32, 1, 32};
    return gfs_host::tmap_nd_cached(base, 3, dims, strides, box);
  };
  const CUtensorMap* ty = halves(c, ldc);
  const CUtensorMap* tx = mode == 1 ? gfs_host::tmap_2d_cached(extra, M, I, ld_extra, 32, 32) : halves(extra, ld_extra);
  if (tx == nullptr || ty == nullptr) return -3;
  if (mode == 1) return launch2<false, false, COMM_NONE, 1, 16>(ta, tb, p, 2 * pairs, stream, tx, ty);
  return launch2<false, true, COMM_NONE, 2, 16>(ta, tb, p, 2 * pairs, stream, tx, ty);
}

// Fused collective + GEMM on CTA pairs; same contract as gfs_gemm_bf16_comm (gemm.cu) with the
// extra requirement that M/world is a multiple of 256. Returns -20 when the problem does not
// qualify, in which case the caller uses the single-CTA kernel (nothing has been launched and
// *target_inout is unchanged).
static int gemm2_comm_impl(int mode, const void* a, int lda, const void* B, int ldb, void* out, int ldo,
                           const void* residual, int ldr, int M, int N, int K, int b_mn_major, int world, int rank,
                           const unsigned long long* peer_bufs, const unsigned long long* peer_flags,
                           unsigned int* target_inout, const void* rope_cos, const void* rope_sin, int rope_cols,
                           int rope_d, int rope_b, long long wait_ns, void* ce_partials, void* stream_,
                           int swi_mode = 0, void* swi_extra = nullptr, int swi_ld = 0) {
  // swi_mode 1 / 2 (all-gather only): the SwiGLU epilogues of gfs_gemm2_bf16_swiglu. Mode 1: N = 2I
  // columns of the [gate | up] projection, out = gu [M, 2I], swi_extra = act [M, I]. Mode 2: N = I
  // columns of d_act, B stored [K, I], out = d_gu [M, 2I], swi_extra = gu [M, 2I].
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (mode != COMM_ALLGATHER && mode != COMM_REDUCE_SCATTER) return -1;
  if (swi_mode != 0 && (mode != COMM_ALLGATHER || ce_partials != nullptr || rope_cos != nullptr || residual ||
                        swi_extra == nullptr || (swi_ld & 7) || (reinterpret_cast<uintptr_t>(swi_extra) & 15) ||
                        b_mn_major != (swi_mode == 2) || (swi_mode == 1 && (N & 15))))
    return -1;
  if (ce_partials != nullptr && (mode != COMM_ALLGATHER || b_mn_major || rope_cos != nullptr)) return -1;
  if (world < 2 || world > MAX_PEERS || rank < 0 || rank >= world) return -1;
  if (M <= 0 || N <= 0 || K <= 0 || (M % world) != 0) return -1;
  if (((M / world) % 256) != 0 || N < 256 || K < 256) return -20;
  if ((N & 7) || (K & 7) || (lda & 7) || (ldb & 7) || (ldo & 7) || (residual && (ldr & 7))) return -1;
  const int rows_per_rank = M / world;
  Params2 p{};
  p.M = M; p.N = N; p.K = K;
  p.tiles_m = M / 256;
  p.tiles_n = (N + BN - 1) / BN;
  p.kblocks = (K + BK - 1) / BK;
  p.status = gfs_host::status_words();
  p.rope_cos = static_cast<const float*>(rope_cos);
  p.rope_sin = static_cast<const float*>(rope_sin);
  p.rope_cols = rope_cols; p.rope_d = rope_d; p.rope_b = rope_b > 0 ? rope_b : 1;
  CommParams& c = p.comm;
  c.world = world; c.rank = rank; c.rows_per_rank = rows_per_rank;
  c.wait_ns = wait_ns > 0 ? static_cast<unsigned long long>(wait_ns) : 20000000000ull;
  for (int i = 0; i < world; ++i) {
    c.peer_buf[i] = reinterpret_cast<__nv_bfloat16*>(peer_bufs[i]);
    c.peer_flags[i] = reinterpret_cast<uint32_t*>(peer_flags[i]);
  }
  // entry `world` of the buffer table: multicast address of the same buffers (0 = none). With two
  // ranks a multicast store saves nothing (one peer) and sends the local copy through the switch
  // as well (measured slower: 8.46 vs 8.28 ms per GPT-124M TP2 step), so it is used from 3 ranks up.
  c.mc_buf = (mode == COMM_ALLGATHER && world > 2) ? reinterpret_cast<__nv_bfloat16*>(peer_bufs[world]) : nullptr;
  const int pairs = std::min(p.tiles_m * p.tiles_n, gfs_host::sm_count() / 2);
  const int grid = 2 * pairs;
  const void* a_base;
  int a_ld;
  unsigned int increment;
  if (mode == COMM_ALLGATHER) {
    c.ag_src = static_cast<const __nv_bfloat16*>(a);
    c.ag_ld = lda;
    c.ag_cols = K;
    a_base = c.peer_buf[rank];   // the GEMM reads the local gathered buffer
    a_ld = K;
    p.C = static_cast<__nv_bfloat16*>(out);
    p.ldc = ldo;
    increment = static_cast<unsigned int>(grid);   // every CTA of a source signals once per destination
  } else {
    a_base = a;
    a_ld = lda;
    c.rs_out = static_cast<__nv_bfloat16*>(out);
    c.rs_ld_out = ldo;
    c.rs_res = static_cast<const __nv_bfloat16*>(residual);
    c.rs_ld_res = ldr;
    increment = static_cast<unsigned int>((rows_per_rank / 256) * p.tiles_n * 2 * 8);  // (warp, tile) units per pair tile
  }
  if ((reinterpret_cast<uintptr_t>(a_base) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(out)) & 15)
    return -2;
  const CUtensorMap* ta = gfs_host::tmap_2d_cached(a_base, M, K, a_ld, BM, 64);
  const CUtensorMap* tb = b_mn_major ? gfs_host::tmap_2d_cached(B, K, N, ldb, 64, 64)
                                     : gfs_host::tmap_2d_cached(B, N, K, ldb, BNH, 64);
  if (ta == nullptr || tb == nullptr) return -3;
  const CUtensorMap* ta_local = nullptr;   // all-gather: this rank's own shard, read in place
  if (mode == COMM_ALLGATHER) {
    if (reinterpret_cast<uintptr_t>(a) & 15) return -2;
    ta_local = gfs_host::tmap_2d_cached(a, rows_per_rank, K, lda, BM, 64);
    if (ta_local == nullptr) return -3;
  }
  if (swi_mode == 1) {
    p.swi_I = N / 2;
    p.tiles_n = (p.swi_I + BN / 2 - 1) / (BN / 2);
    p.swi_ld = swi_ld;
    p.swi_act = static_cast<__nv_bfloat16*>(swi_extra);
  } else if (swi_mode == 2) {
    p.swi_I = N;
    p.swi_ld = swi_ld;
    p.swi_gu = static_cast<const __nv_bfloat16*>(swi_extra);
  }
  *target_inout += increment;
  c.target = *target_inout;
  if (swi_mode == 1) return launch2<false, false, COMM_ALLGATHER, 1, 8>(ta, tb, p, grid, stream, ta_local);
  if (swi_mode == 2) return launch2<false, true, COMM_ALLGATHER, 2, 8>(ta, tb, p, grid, stream, ta_local);
  if (ce_partials != nullptr) {
    p.ce_partials = static_cast<float2*>(ce_partials);
    return launch2<false, false, COMM_ALLGATHER, 3, 8>(ta, tb, p, grid, stream, ta_local);
  }
  if (mode == COMM_ALLGATHER)
    return b_mn_major ? launch2<false, true, COMM_ALLGATHER, 0, 8>(ta, tb, p, grid, stream, ta_local)
                      : launch2<false, false, COMM_ALLGATHER, 0, 8>(ta, tb, p, grid, stream, ta_local);
  return b_mn_major ? launch2<false, true, COMM_REDUCE_SCATTER, 0, 8>(ta, tb, p, grid, stream)
                    : launch2<false, false, COMM_REDUCE_SCATTER, 0, 8>(ta, tb, p, grid, stream);
}

int gfs_gemm2_bf16_comm(int mode, const void* a, int lda, const void* B, int ldb, void* out, int ldo,
                        const void* residual, int ldr, int M, int N, int K, int b_mn_major, int world, int rank,
                        const unsigned long long* peer_bufs, const unsigned long long* peer_flags,
                        unsigned int* target_inout, const void* rope_cos, const void* rope_sin, int rope_cols,
                        int rope_d, int rope_b, long long wait_ns, void* stream_) {
  return gemm2_comm_impl(mode, a, lda, B, ldb, out, ldo, residual, ldr, M, N, K, b_mn_major, world, rank, peer_bufs,
                         peer_flags, target_inout, rope_cos, rope_sin, rope_cols, rope_d, rope_b, wait_ns, nullptr,
                         stream_);
}

// Tensor-parallel SwiGLU MLP under sequence parallelism: the all-gather GEMMs with the SwiGLU
// epilogues of gfs_gemm2_bf16_swiglu.
//   mode 1: a = this rank's shard of x [M/world, K], B = w_gu [2I, K];  out = gu [M, 2I] (pitch ldo),
//           extra = act [M, I] = silu(gate) * up (pitch ld_extra)
//   mode 2: a = this rank's shard of dOut [M/world, K], B = w_down stored [K, I]; out = d_gu [M, 2I],
//           extra = gu [M, 2I] (the forward's projection)
// peer_bufs[p] = rank p's gathered [M, K] buffer. Returns -20 like gfs_gemm2_bf16_comm.
int gfs_gemm2_bf16_comm_swiglu(int swi_mode, const void* a, int lda, const void* B, int ldb, void* out, int ldo,
                               void* extra, int ld_extra, int M, int I, int K, int world, int rank,
                               const unsigned long long* peer_bufs, const unsigned long long* peer_flags,
                               unsigned int* target_inout, long long wait_ns, void* stream_) {
  if (swi_mode != 1 && swi_mode != 2) return -1;
  if ((I & 7) || I < 256) return (I & 7) ? -1 : -20;
  return gemm2_comm_impl(COMM_ALLGATHER, a, lda, B, ldb, out, ldo, nullptr, 0, M, swi_mode == 1 ? 2 * I : I, K,
                         swi_mode == 2 ? 1 : 0, world, rank, peer_bufs, peer_flags, target_inout, nullptr, nullptr, 0, 0,
                         1, wait_ns, nullptr, stream_, swi_mode, extra, ld_extra);
}

// Vocabulary-parallel LM head under sequence parallelism: the all-gather GEMM
// (logits[M, N] = gather(a)[M, K] @ B[N, K]^T, B K-major) whose epilogue also writes the
// cross-entropy statistics of gfs_gemm2_bf16_ce: partials is float2 [gfs_gemm2_ce_parts(N)][M]. Returns -20 like
// gfs_gemm2_bf16_comm.
int gfs_gemm2_bf16_allgather_ce(const void* a, int lda, const void* B, int ldb, void* out, int ldo, void* partials,
                                int M, int N, int K, int world, int rank, const unsigned long long* peer_bufs,
                                const unsigned long long* peer_flags, unsigned int* target_inout, long long wait_ns,
                                void* stream_) {
  if (partials == nullptr || (reinterpret_cast<uintptr_t>(partials) & 15)) return -2;
  return gemm2_comm_impl(COMM_ALLGATHER, a, lda, B, ldb, out, ldo, nullptr, 0, M, N, K, 0, world, rank, peer_bufs,
                         peer_flags, target_inout, nullptr, nullptr, 0, 0, 1, wait_ns, partials, stream_);
}

// Grouped weight gradients: for g < n, C_g[M_g, N_g] (+)= A_g^T B_g with A_g = [K_g, M_g] (pitch lda_g),
// B_g = [K_g, N_g] (pitch ldb_g), all bf16 row-major, fp32 accumulation, one launch. n <= 4.
// accumulate_g != 0 adds the product to the existing C_g (rounded once).
int gfs_gemm2_wgrad_grouped(int n, const unsigned long long* A, const unsigned long long* B,
                            const unsigned long long* C, const int* M, const int* N, const int* K, const int* lda,
                            const int* ldb, const int* ldc, const int* accumulate, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (n <= 0) return 0;
  if (n > MAX_GROUP) return -1;
  GroupMaps maps;
  GroupParams p{};
  p.ngroups = n;
  p.late_wait = gfs_host::launch_hints().late_wait;
  p.status = gfs_host::status_words();
  int total = 0;
  for (int i = 0; i < n; ++i) {
    if (M[i] <= 0 || N[i] <= 0 || K[i] <= 0) return -1;
    if ((N[i] & 7) || (M[i] & 7) || (lda[i] & 7) || (ldb[i] & 7) || (ldc[i] & 7)) return -1;
    if ((A[i] | B[i] | C[i]) & 15) return -2;
    const CUtensorMap* ta = gfs_host::tmap_2d_cached(reinterpret_cast<const void*>(A[i]), K[i], M[i], lda[i], 64, 64);
    const CUtensorMap* tb = gfs_host::tmap_2d_cached(reinterpret_cast<const void*>(B[i]), K[i], N[i], ldb[i], 64, 64);
    if (ta == nullptr || tb == nullptr) return -3;
    maps.a[i] = *ta;
    maps.b[i] = *tb;
    GroupProblem& g = p.g[i];
    g.M = M[i]; g.N = N[i]; g.ldc = ldc[i];
    g.tiles_n = (N[i] + BN - 1) / BN;
    g.tile_begin = total;
    g.kblocks = (K[i] + BK - 1) / BK;
    g.accumulate = accumulate[i];
    g.C = reinterpret_cast<__nv_bfloat16*>(C[i]);
    total += ((M[i] + 255) / 256) * g.tiles_n;
  }
  for (int i = n; i < MAX_GROUP; ++i) {
    maps.a[i] = maps.a[0];
    maps.b[i] = maps.b[0];
    p.g[i] = p.g[0];
    p.g[i].tile_begin = 0x7fffffff;
  }
  p.total_tiles = total;
  static gfs_host::SmemLimit limit;
  if (!limit.raise(gemm2_grouped_kernel, SMEM_TOTAL)) return -10;
  const int pairs = std::min(total, gfs_host::sm_count() / 2);
  if (gfs_host::launch_pdl(gemm2_grouped_kernel, dim3(2 * pairs), dim3(THREADS), SMEM_TOTAL, stream, maps, p) !=
      cudaSuccess)
    return -11;
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

}  // extern "C"
