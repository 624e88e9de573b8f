// Causal flash attention forward and backward for sm_100a (head_dim 64 or 128, bf16).
//
// All matrix products run on tcgen05.mma with fp32 accumulators in TMEM; operands are
// staged by TMA straight out of strided tensors (for the model: the packed
// [S,B,3,nh,D] qkv buffer, so no permute/contiguous copies exist), and the output is
// written directly in [S,B,nh*D] layout.
//
// Forward (persistent; head_dim 64: pairs of 128-row query tiles, 128: two pipelines of 128-row items): per
//   128-key block S = Q K^T -> TMEM; the softmax threads read their row (128: half row) with tcgen05.ld, keep
//   the running max / sum and store P (bf16) in TMEM, from where the MMA warp adds P V to the output
//   accumulator, which stays in TMEM for the whole item. (Few items at head_dim 128: a CTA for each.)
//
// Backward (two kernels from one template, deterministic, no atomics):
//   mode 0: items of 128 keys    -> dK, dV, streaming 64-query tiles
//   mode 1: items of 128 queries -> dQ,     streaming 64-key tiles
//   Both recompute P = exp(S*scale - LSE), dS = P * (dP - D) from two score MMAs
//   (X = R1 T1^T, Y = R2 T2^T), write P / dS (bf16) to TMEM and accumulate dV += P^T dO,
//   dK += dS^T Q (mode 0) or dQ += dS K (mode 1) there. The streamed tile is consumed twice from the same
//   shared-memory bytes: K-major for the score MMA and MN-major for the gradient MMA.
//
// Reference counterparts: core/myFlashAttn.py:460-728 (_attn_fwd), :740-790 (pre-pass),
// :805-1066 (_attn_bwd_LoopQ), :1079-1317 (_attn_bwd_LoopKV).
#include <cuda_fp16.h>

#include <cstdlib>
#include <algorithm>
#include <type_traits>

#include "api.h"
#include "common.cuh"

using namespace gfs;

namespace {

constexpr float LOG2E_F = 1.4426950408889634f;

// three-input maximum (one instruction on sm_100)
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// Classifies a (32-row warp slice) x (column chunk) block of the score matrix against the
// causal / sequence-end mask: 0 = every element alive, 1 = mixed, 2 = every element dead.
// KEY_ROWS: rows are key positions and columns are query positions (dead when col < row);
// otherwise rows are queries and columns are keys (dead when col > row). Warp-uniform.
template <bool KEY_ROWS>
__device__ __forceinline__ int mask_class(int row_min, int row_max, int col_min, int col_max, bool causal, int S) {
  if (col_min >= S) return 2;
  bool all_alive = col_max < S, all_dead = false;
  if (causal) {
    if (KEY_ROWS) {
      all_alive = all_alive && col_min >= row_max;
      all_dead = col_max < row_min;
    } else {
      all_alive = all_alive && col_max <= row_min;
      all_dead = col_min > row_max;
    }
  }
  return all_dead ? 2 : (all_alive ? 0 : 1);
}

// A K-major [rows x K] (64-column blocks a_blk bytes apart), B K-major [N x K] (blocks b_blk apart).
// The shared-memory descriptors are built once per call and advanced by adding the byte offset
// (in 16-byte units) to their start-address field: the tiles are 1024-byte aligned and the
// offsets small, so the 14-bit field never carries. The issuing thread competes with the
// compute warps for issue slots, so every instruction saved per MMA shortens the chain.
template <int KSTEPS>
__device__ __forceinline__ void mma_kk(uint32_t d, uint32_t a, uint32_t a_blk, uint32_t b, uint32_t b_blk,
                                       uint32_t idesc, bool accumulate) {
  const uint64_t ad0 = umma_desc_sw128(a, 16, 1024);
  const uint64_t bd0 = umma_desc_sw128(b, 16, 1024);
#pragma unroll
  for (int ks = 0; ks < KSTEPS; ++ks) {
    const uint64_t ad = ad0 + (((ks >> 2) * a_blk + (ks & 3) * 32) >> 4);
    const uint64_t bd = bd0 + (((ks >> 2) * b_blk + (ks & 3) * 32) >> 4);
    umma_ss_e(d, ad, bd, idesc, (accumulate || ks > 0) ? 1u : 0u);
  }
}
// A K-major; B MN-major: stored as [K rows x N] in 64-column blocks b_blk bytes apart
// (each block: K rows of 128 B).
template <int KSTEPS>
__device__ __forceinline__ void mma_kmn(uint32_t d, uint32_t a, uint32_t a_blk, uint32_t b, uint32_t b_blk,
                                        uint32_t idesc, bool accumulate) {
  const uint64_t ad0 = umma_desc_sw128(a, 16, 1024);
  const uint64_t bd0 = umma_desc_sw128(b, b_blk, 1024);
#pragma unroll
  for (int ks = 0; ks < KSTEPS; ++ks) {
    const uint64_t ad = ad0 + (((ks >> 2) * a_blk + (ks & 3) * 32) >> 4);
    const uint64_t bd = bd0 + ((ks * 2048) >> 4);
    umma_ss_e(d, ad, bd, idesc, (accumulate || ks > 0) ? 1u : 0u);
  }
}

// A in tensor memory (8 columns per 16-wide K step; the second half of the K steps starts HALF columns
// after the first); B MN-major as in mma_kmn.
template <int KSTEPS, int HALF = KSTEPS * 4>
__device__ __forceinline__ void mma_tmn(uint32_t d, uint32_t a_tmem, uint32_t b, uint32_t b_blk, uint32_t idesc,
                                        bool accumulate) {
  const uint64_t bd0 = umma_desc_sw128(b, b_blk, 1024);
#pragma unroll
  for (int ks = 0; ks < KSTEPS; ++ks) {
    const uint64_t bd = bd0 + ((ks * 2048) >> 4);
    const uint32_t a = a_tmem + (ks / (KSTEPS / 2)) * HALF + (ks % (KSTEPS / 2)) * 8;
    umma_ts_e(d, a, bd, idesc, (accumulate || ks > 0) ? 1u : 0u);
  }
}

// ---------------------------------------------------------------------------
// Epilogue stores. An accumulator row lives in one thread, so a direct store instruction writes 16
// bytes to each of 32 different rows: 32 passes through the load/store unit per instruction, which
// made the epilogues of these kernels LSU-bound (about 1,000 cycles per 128 x 64 output tile). The
// rows are therefore transposed through a per-warp staging area in shared memory (XOR-swizzled, free
// of bank conflicts both ways) and leave as whole 64- or 128-byte row segments.
// ---------------------------------------------------------------------------
// 32 rows x 32 bf16 columns; w = this lane's row (16 packed words); stage: 2 KB of this warp.
__device__ __forceinline__ void store_rows_32x32(uint8_t* stage, const uint32_t (&w)[16], int lane,
                                                 __nv_bfloat16* g0, long long row_stride, int rows_valid) {
#pragma unroll
  for (int q4 = 0; q4 < 4; ++q4)
    *reinterpret_cast<uint4*>(stage + lane * 64 + ((q4 ^ ((lane >> 1) & 3)) << 4)) =
        make_uint4(w[4 * q4], w[4 * q4 + 1], w[4 * q4 + 2], w[4 * q4 + 3]);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = (lane >> 2) + 8 * i;
    const uint4 v = *reinterpret_cast<const uint4*>(stage + row * 64 + (((lane & 3) ^ ((row >> 1) & 3)) << 4));
    if (row < rows_valid) *reinterpret_cast<uint4*>(g0 + row * row_stride + (lane & 3) * 8) = v;
  }
  __syncwarp();
}

// 32 rows x 64 bf16 columns; w = this lane's row (32 packed words); stage: 4 KB of this warp.
__device__ __forceinline__ void store_rows_32x64(uint8_t* stage, const uint32_t (&w)[32], int lane,
                                                 __nv_bfloat16* g0, long long row_stride, int rows_valid) {
#pragma unroll
  for (int ch = 0; ch < 8; ++ch)
    *reinterpret_cast<uint4*>(stage + lane * 128 + ((ch ^ (lane & 7)) << 4)) =
        make_uint4(w[4 * ch], w[4 * ch + 1], w[4 * ch + 2], w[4 * ch + 3]);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = (lane >> 3) + 4 * i;
    const uint4 v = *reinterpret_cast<const uint4*>(stage + row * 128 + (((lane & 7) ^ (row & 7)) << 4));
    if (row < rows_valid) *reinterpret_cast<uint4*>(g0 + row * row_stride + (lane & 7) * 8) = v;
  }
  __syncwarp();
}

// Two fp32 values as a 16-bit pair of the output's type. The kernels compute in bf16; tensors of an fp16
// caller are rounded to bf16 on the way in (cast_qkv_kernel, attn_dvec_kernel) and results leave as fp16
// straight from fp32, so an fp16 call costs one launch more than a bf16 one and no pass over its results.
__device__ __forceinline__ uint32_t pack_out(float lo, float hi, int f16) {
  if (f16) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
  return pack_bf16x2(lo, hi);
}

// ---------------------------------------------------------------------------
// Forward
// ---------------------------------------------------------------------------
struct FwdParams {
  __nv_bfloat16* O;            // 16-bit elements; fp16 when o_f16 is set
  long long o_copy;            // element offset from O to a second copy of the output; 0: none
  long long o_ss, o_bs, o_hs;  // element strides: sequence, batch, head
  float* lse;                  // [B, nh, S_pad], log2 of the row's sum of exponentials (base e scores)
  int o_f16;
  int S, S_pad, B, nh;
  float scale;
  int causal;
  uint32_t* status;
};

// ---------------------------------------------------------------------------
// Forward, head_dim 128, few items: one CTA per 128 query rows, four softmax warps (a row per thread). A lone chain of
// blocks is what bounds such a problem, and here S, P and P V are double buffered (P through shared memory, the
// output folded into registers), so the next block's scores are ready when the softmax gets there; the
// pipelines of the kernel below hide each other's waits instead.
// ---------------------------------------------------------------------------
constexpr int FWD128S_THREADS = 192;
constexpr int FWD128S_SMEM = 5 * 32768 + 2 * 32768 + 256;

// Which of the two serves nb query tiles of B * nh heads. Up to one item per SM, this one: us, here -> two pipelines,
// [1, 1, 1024, 128] 24 -> 27, [4, 2, 2048] 39 -> 43, [1, 4, 4096] 68 -> 76, [1, 2, 8192] 123 -> 137 (up to 300
// tokens they are equal). A few more items change nothing as long as they find room behind short causal ones:
// [1, 5, 4096] 70 -> 80, [1, 6, 4096] 78 -> 84, [1, 3, 8192] 130 -> 152, [1, 10, 2048] 41 -> 47, [1, 12, 2048] 49 -> 50,
// [1, 19, 1024] 27 -> 31; past that two pipelines per SM win: [1, 7, 4096] 91 -> 86, [1, 13, 2048] 55 -> 51,
// [1, 20, 1024] 33 -> 31, [1, 40, 512] 25 -> 23, [1, 32, 4096] 294 -> 182; without a mask [1, 9, 2048] 41 -> 45,
// [1, 10, 2048] 68 -> 57. The line is the share of the SMs' time that the blocks take if none works longer than the
// longest item; a second item costs an SM a launch, which short items feel more.
bool fwd128_few_items(int nb, long long heads, bool causal, int sms) {
  if (nb * heads <= sms) return true;
  const long long blocks = causal ? heads * nb * (nb + 1) / 2 : heads * nb * nb;
  return blocks * 100 <= static_cast<long long>(sms) * nb * (nb >= 16 ? 70 : 59);
}

__global__ void __launch_bounds__(FWD128S_THREADS, 1)
flash_fwd128_small_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                          const __grid_constant__ CUtensorMap tv, const FwdParams p) {
  constexpr int D = 128;
  constexpr int DB = D / 64;
  constexpr int TILE_BYTES = DB * 16384;  // [128 x D] bf16 as DB swizzled blocks
  constexpr int P_BYTES = 32768;          // [128 x 128] bf16 as 2 swizzled blocks
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t OP_COL = 256;        // PV tiles start after the S tiles
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;  // the launcher requests exactly the bytes used; the base must be 1024-aligned
  uint8_t* Qs = smem;
  uint8_t* Ks = Qs + TILE_BYTES;
  uint8_t* Vs = Ks + 2 * TILE_BYTES;
  uint8_t* Ps = Vs + 2 * TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(Ps + 2 * P_BYTES);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;
  uint64_t* k_empty = bars + 3;
  uint64_t* v_full = bars + 5;
  uint64_t* v_empty = bars + 7;
  uint64_t* s_full = bars + 9;
  uint64_t* s_empty = bars + 11;
  uint64_t* p_full = bars + 13;
  uint64_t* p_empty = bars + 15;
  uint64_t* o_full = bars + 17;
  uint64_t* o_empty = bars + 19;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 21);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if (smem_u32(smem_raw) & 1023u) {  // swizzled tiles need a 1024-byte aligned base
    if (threadIdx.x == 0) record_status(p.status, STATUS_BAD_ARGUMENT, 0x5a11u);
    return;
  }
  const int qt = gridDim.x - 1 - blockIdx.x;  // heaviest (most key blocks) first
  const int bh = blockIdx.y;
  const int b = bh / p.nh;
  const int h = bh % p.nh;
  const int n_blocks_all = (p.S + 127) >> 7;
  const int n_kv = p.causal ? min(qt + 1, n_blocks_all) : n_blocks_all;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&s_empty[i], 4);
      mbar_init(&p_full[i], 4);
      mbar_init(&p_empty[i], 1);
      mbar_init(&o_full[i], 1);
      mbar_init(&o_empty[i], 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tq);
    tma_prefetch_desc(&tk);
    tma_prefetch_desc(&tv);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();       // set-up above may overlap the tail of the preceding kernel (programmatic launch)
  pdl_trigger();
  const uint32_t tmem_base = *tmem_slot;
  WaitCtx wctx{abort_flag, p.status, GFS_WAIT_LIMIT_NS};

  if (warp == 0) {
    if (lane == 0) {
      mbar_arrive_expect_tx(q_full, TILE_BYTES);
#pragma unroll
      for (int db = 0; db < DB; ++db) tma_load_4d(Qs + db * 16384, &tq, q_full, db * 64, qt * 128, h, b);
      for (int j = 0; j < n_kv; ++j) {
        const int st = j & 1;
        const uint32_t par = ((j >> 1) & 1) ^ 1u;
        mbar_wait(&k_empty[st], par, wctx, STATUS_TIMEOUT_PIPE_EMPTY);
        mbar_arrive_expect_tx(&k_full[st], TILE_BYTES);
#pragma unroll
        for (int db = 0; db < DB; ++db)
          tma_load_4d(Ks + st * TILE_BYTES + db * 16384, &tk, &k_full[st], db * 64, j * 128, h, b);
        mbar_wait(&v_empty[st], par, wctx, STATUS_TIMEOUT_PIPE_EMPTY);
        mbar_arrive_expect_tx(&v_full[st], TILE_BYTES);
#pragma unroll
        for (int db = 0; db < DB; ++db)
          tma_load_4d(Vs + st * TILE_BYTES + db * 16384, &tv, &v_full[st], db * 64, j * 128, h, b);
      }
      settle_copies(wctx);
    }
  } else if (warp == 1) {
    {  // whole warp, converged: the MMA / commit helpers elect the issuing lane
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, 0, 0);
      constexpr uint32_t idesc_o = umma_idesc_bf16(128, D, 0, 1);
      const uint32_t q_addr = smem_u32(Qs);
      mbar_wait(q_full, 0, wctx, STATUS_TIMEOUT_PIPE_FULL);
      auto issue_s = [&](int j) {
        const int st = j & 1;                       // K/V stage
        const uint32_t par = (j >> 1) & 1;
        const int sb = j & 1;   // S / P / PV buffer
        const uint32_t spar = (j >> 1) & 1;
        mbar_wait(&k_full[st], par, wctx, STATUS_TIMEOUT_PIPE_FULL);
        mbar_wait(&s_empty[sb], spar ^ 1u, wctx, STATUS_TIMEOUT_SOFTMAX);
        tc_fence_after();
        mma_kk<D / 16>(tmem_base + sb * 128, q_addr, 16384, smem_u32(Ks + st * TILE_BYTES), 16384, idesc_s, false);
        umma_commit_e(&s_full[sb]);
        umma_commit_e(&k_empty[st]);
      };
      issue_s(0);
      for (int j = 0; j < n_kv; ++j) {
        if (j + 1 < n_kv) issue_s(j + 1);
        const int st = j & 1;
        const uint32_t par = (j >> 1) & 1;
        const int sb = j & 1;
        const uint32_t spar = (j >> 1) & 1;
        mbar_wait(&p_full[sb], spar, wctx, STATUS_TIMEOUT_SOFTMAX);
        mbar_wait(&v_full[st], par, wctx, STATUS_TIMEOUT_PIPE_FULL);
        mbar_wait(&o_empty[sb], spar ^ 1u, wctx, STATUS_TIMEOUT_SOFTMAX);
        tc_fence_after();
        mma_kmn<8>(tmem_base + OP_COL + sb * D, smem_u32(Ps + sb * P_BYTES), 16384, smem_u32(Vs + st * TILE_BYTES),
                   16384, idesc_o, false);
        umma_commit_e(&o_full[sb]);
        umma_commit_e(&v_empty[st]);
        umma_commit_e(&p_empty[sb]);
      }
    }
  } else {
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;       // row inside the query tile
    const int row_g = qt * 128 + r;          // query position
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const float sl2 = p.scale * LOG2E_F;
    float m = -INFINITY, l = 0.f, alpha_prev = 0.f;
    float o[D];
#pragma unroll
    for (int i = 0; i < D; ++i) o[i] = 0.f;

    auto fold_pv = [&](int j, float alpha) {
      const int st = j & 1;
      mbar_wait(&o_full[st], (j >> 1) & 1, wctx, STATUS_TIMEOUT_SOFTMAX);
      tc_fence_after();
      const uint32_t o_addr = tmem_base + lane_base + OP_COL + st * D;
      uint32_t wa[32], wb[32];
      tmem_ld_32x32(o_addr, wa);
#pragma unroll
      for (int c = 0; c < D; c += 64) {
        tmem_ld_wait_for(wa);
        tmem_ld_32x32(o_addr + c + 32, wb);
#pragma unroll
        for (int e = 0; e < 32; ++e) o[c + e] = fmaf(o[c + e], alpha, __uint_as_float(wa[e]));
        tmem_ld_wait_for(wb);
        if (c + 64 < D) tmem_ld_32x32(o_addr + c + 64, wa);
#pragma unroll
        for (int e = 0; e < 32; ++e) o[c + 32 + e] = fmaf(o[c + 32 + e], alpha, __uint_as_float(wb[e]));
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&o_empty[st]);
    };

    for (int j = 0; j < n_kv; ++j) {
      const int st = j & 1;
      const uint32_t par = (j >> 1) & 1;
      const bool need_mask = (p.causal && j == qt) || ((j + 1) * 128 > p.S);
      mbar_wait(&s_full[st], par, wctx, STATUS_TIMEOUT_SOFTMAX);
      tc_fence_after();
      const uint32_t s_addr = tmem_base + lane_base + st * 128;
      // pass 1: row maximum (TMEM loads double buffered against the arithmetic)
      float mx = -INFINITY;
      uint32_t va[32], vb[32];
      // Diagonal / tail block: dead scores become -inf in the registers and the block runs the same
      // max / exponential code as every other block (a separate masked copy of that code executes
      // once per CTA from a cold instruction cache and cost more than two unmasked blocks).
      auto mask_chunk = [&](uint32_t (&v)[32], int c) {
        if (need_mask) {
          const int lim_c = p.causal ? row_g - j * 128 - c : 0x7fffffff;   // last live column of the chunk
          const int lim = min(lim_c, p.S - 1 - j * 128 - c);
#pragma unroll
          for (int e = 0; e < 32; ++e) v[e] = (e > lim) ? 0xff800000u : v[e];
        }
      };
      auto max_chunk = [&](uint32_t (&v)[32], int c) {
        mask_chunk(v, c);
#pragma unroll
        for (int e = 0; e < 32; ++e) mx = fmaxf(mx, __uint_as_float(v[e]));
      };
      tmem_ld_32x32(s_addr + 0, va);
      tmem_ld_wait_for(va);
      tmem_ld_32x32(s_addr + 32, vb);
      max_chunk(va, 0);
      tmem_ld_wait_for(vb);
      tmem_ld_32x32(s_addr + 64, va);
      max_chunk(vb, 32);
      tmem_ld_wait_for(va);
      tmem_ld_32x32(s_addr + 96, vb);
      max_chunk(va, 64);
      tmem_ld_wait_for(vb);
      tmem_ld_32x32(s_addr + 0, va);  // first chunk of pass 2
      max_chunk(vb, 96);
      const float m_new = fmaxf(m, mx);
      const float m_use = (m_new == -INFINITY) ? 0.f : m_new;  // row with no live key so far
      const float alpha = fast_exp2((m - m_use) * sl2);
      const float moff = m_use * sl2;
      mbar_wait(&p_empty[st], par ^ 1u, wctx, STATUS_TIMEOUT_SOFTMAX);
      // pass 2: probabilities -> shared memory (bf16, swizzled K-major), row sum
      float rs = 0.f;
      uint8_t* prow = Ps + st * P_BYTES + r * 128;
      auto prob_chunk = [&](uint32_t (&v)[32], int c) {
        mask_chunk(v, c);
        uint32_t packed[16];
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          const float x0 = fast_exp2(fmaf(__uint_as_float(v[e]), sl2, -moff));
          const float x1 = fast_exp2(fmaf(__uint_as_float(v[e + 1]), sl2, -moff));
          rs += x0 + x1;
          packed[e >> 1] = pack_bf16x2(x0, x1);
        }
        uint8_t* blk = prow + (c >> 6) * 16384;
        const int chunk0 = (c & 63) >> 3;
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          const uint4 w = make_uint4(packed[4 * q4], packed[4 * q4 + 1], packed[4 * q4 + 2], packed[4 * q4 + 3]);
          *reinterpret_cast<uint4*>(blk + ((((chunk0 + q4) ^ (r & 7)) & 7) << 4)) = w;
        }
      };
      tmem_ld_wait_for(va);
      tmem_ld_32x32(s_addr + 32, vb);
      prob_chunk(va, 0);
      tmem_ld_wait_for(vb);
      tmem_ld_32x32(s_addr + 64, va);
      prob_chunk(vb, 32);
      tmem_ld_wait_for(va);
      tmem_ld_32x32(s_addr + 96, vb);
      prob_chunk(va, 64);
      tmem_ld_wait_for(vb);
      prob_chunk(vb, 96);
      l = l * alpha + rs;
      m = m_new;
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&s_empty[st]);
        mbar_arrive(&p_full[st]);
      }
      if (j > 0) fold_pv(j - 1, alpha_prev);
      alpha_prev = alpha;
    }
    fold_pv(n_kv - 1, alpha_prev);

    const float inv_l = (l > 0.f) ? 1.f / l : 0.f;
    {
      // every P V MMA has completed (the last fold waited for it): the P buffer serves as staging
      uint8_t* stage = Ps + (r >> 5) * 4096;
      const int row0 = row_g - lane;
      __nv_bfloat16* g0 = p.O + row0 * p.o_ss + b * p.o_bs + h * p.o_hs;
      // twice when a copy is wanted (rolled, to keep the registers of the loop above)
#pragma unroll 1
      for (int n_out = p.o_copy != 0 ? 2 : 1; n_out > 0; --n_out, g0 += p.o_copy) {
#pragma unroll
        for (int hf = 0; hf < D / 64; ++hf) {
          uint32_t ow[32];
#pragma unroll
          for (int e = 0; e < 32; ++e)
            ow[e] = pack_out(o[hf * 64 + 2 * e] * inv_l, o[hf * 64 + 2 * e + 1] * inv_l, p.o_f16);
          store_rows_32x64(stage, ow, lane, g0 + hf * 64, p.o_ss, p.S - row0);
        }
      }
    }
    if (row_g < p.S_pad) {
      const float mm = (m == -INFINITY) ? 0.f : m;
      p.lse[static_cast<size_t>(bh) * p.S_pad + row_g] = mm * sl2 + log2f(fmaxf(l, 1e-37f));
    }
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

constexpr int FWD128_CW = 8;                           // softmax warps of a pipeline
constexpr int FWD128_FIRST_CW = 4;                     // warps 0, 1: TMA; 2, 3: MMAs (one each per pipeline)
constexpr int FWD128_THREADS = 32 * (FWD128_FIRST_CW + 2 * FWD128_CW);

constexpr int FWD128_TILE = 128 * 256;              // [128 x 128] bf16
constexpr int FWD128_PIPE = 3 * FWD128_TILE;        // Q, K, V of a pipeline
constexpr int FWD128_XCH = 2 * 2 * 2 * 128 * 4;     // [pipeline][parity][half][row] fp32
constexpr int FWD128_SMEM = 2 * FWD128_PIPE + FWD128_XCH + 512;

// head_dim 128: two independent pipelines per CTA, each with its own work items (128 query rows of one (batch, head)),
// TMA warp, MMA warp, eight softmax warps and half of the tensor memory: S | O. What one pipeline loses
// while it waits for its MMAs and at an item's end the other one's exponentials fill. Two warps share the 32
// rows of a quarter, 64 of a block's 128 keys each, and exchange their row maxima through shared memory.
// There are no columns left for P: it overwrites the scores it was made from, and the next block's scores
// wait for its P V.
//
// The output accumulates in tensor memory and is rescaled there when the running maximum grows. (Raising the
// maximum only when it grows by more than 2^8 saves 7 to 12 % of the time, but the largest probability of a row, exactly 1
// with the true maximum, is then rounded to bf16 like the others: the output's error against 64 bits
// was 2 % larger for scores of unit variance and 8 to 25 % for a standard deviation of 4.)
//
// Persistent: items are dealt heaviest first in a snake (left to right, then right to left), which evens
// out the totals; all barrier parities run on counters that continue across items.
//
// us, the kernel above -> this: [1, 8, 4096, 128] causal 100 -> 88, [1, 32, 4096, 128] 290 -> 182, [2, 16, 2048, 128]
// without a mask 138 -> 105. At head_dim 64, where a block's products are
// half as long, the kernel below is the faster one (75 against 78 us at [16, 12, 1024, 64]): its two tiles share
// the K and V loads.
__global__ void __launch_bounds__(FWD128_THREADS, 1)
flash_fwd128_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                 const __grid_constant__ CUtensorMap tv, const FwdParams p, int nb, int n_items) {
  constexpr int D = 128, DB = D / 64, TILE = FWD128_TILE;
  constexpr uint32_t O_COL = 128;
  constexpr uint32_t P_HALF = 64;                   // columns from the first to the second half of P (over S)
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  float* xch = reinterpret_cast<float*>(smem_raw + 2 * FWD128_PIPE);
  uint64_t* bars0 = reinterpret_cast<uint64_t*>(smem_raw + 2 * FWD128_PIPE + FWD128_XCH);
  constexpr int N_BARS = 10;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars0 + 2 * N_BARS);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if (smem_u32(smem_raw) & 1023u) {
    if (threadIdx.x == 0) record_status(p.status, STATUS_BAD_ARGUMENT, 0x5a12u);
    return;
  }
  const int BH = p.B * p.nh;
  const int x = warp < FWD128_FIRST_CW ? (warp & 1) : (warp - FWD128_FIRST_CW) / FWD128_CW;   // this warp's pipeline
  uint8_t* Qs = smem_raw + x * FWD128_PIPE;   // [128 x D], 64-column blocks
  uint8_t* Ks = Qs + TILE;
  uint8_t* Vs = Ks + TILE;
  uint64_t* q_full = bars0 + x * N_BARS;
  uint64_t* q_empty = q_full + 1;
  uint64_t* k_full = q_full + 2;
  uint64_t* k_empty = q_full + 3;
  uint64_t* v_full = q_full + 4;
  uint64_t* v_empty = q_full + 5;
  uint64_t* s_full = q_full + 6;
  uint64_t* o_full = q_full + 7;
  uint64_t* p_full = q_full + 8;
  uint64_t* o_empty = q_full + 9;

  if (threadIdx.x == 0) {
    for (int pipe = 0; pipe < 2; ++pipe) {
      uint64_t* b = bars0 + pipe * N_BARS;
      for (int i = 0; i < N_BARS; ++i) mbar_init(&b[i], i < 8 ? 1 : FWD128_CW);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tq);
    tma_prefetch_desc(&tk);
    tma_prefetch_desc(&tv);
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();       // set-up above may overlap the tail of the preceding kernel (programmatic launch)
  pdl_trigger();
  const uint32_t tmem_base = *tmem_slot + x * 256;
  WaitCtx wctx{abort_flag, p.status, GFS_WAIT_LIMIT_NS};

  // pipeline 1 of a CTA comes after pipeline 0 of all CTAs: with few items every SM has one
  const int W = 2 * static_cast<int>(gridDim.x);
  const int wk = x * static_cast<int>(gridDim.x) + static_cast<int>(blockIdx.x);
  auto snake = [&](int rnd) { return rnd * W + ((rnd & 1) ? W - 1 - wk : wk); };
  // query tile, batch * head and number of key blocks (at least one) of work item w
  auto decode = [&](int w, int& qt, int& bh, int& n) {
    qt = nb - 1 - w / BH;
    bh = w % BH;
    n = p.causal ? qt + 1 : nb;
  };

  if (warp < 2) {
    if (lane == 0) {
      // in the order of the MMAs: K of block g + 1, then V of block g
      auto load = [&](uint8_t* dst, const CUtensorMap& map, uint64_t* full, uint64_t* empty, int n_loaded, int row,
                      int bh) {
        mbar_wait(empty, (n_loaded & 1) ^ 1u, wctx, STATUS_TIMEOUT_PIPE_EMPTY);
        mbar_arrive_expect_tx(full, TILE);
#pragma unroll
        for (int db = 0; db < DB; ++db)    // rows past S: zeros
          tma_load_4d(dst + db * 16384, &map, full, db * 64, row, bh % p.nh, bh / p.nh);
      };
      int v_prev = -1, bh_prev = 0;        // the V block that is still to be loaded
      int gk = 0, gv = 0;
      for (int rnd = 0; rnd * W < n_items; ++rnd) {
        const int w = snake(rnd);
        if (w >= n_items) break;
        int qt, bh, n;
        decode(w, qt, bh, n);
        for (int j = 0; j < n; ++j) {
          if (j == 0) load(Qs, tq, q_full, q_empty, rnd, qt * 128, bh);
          load(Ks, tk, k_full, k_empty, gk++, j * 128, bh);
          if (v_prev >= 0) load(Vs, tv, v_full, v_empty, gv++, v_prev * 128, bh_prev);
          v_prev = j;
          bh_prev = bh;
        }
      }
      if (v_prev >= 0) load(Vs, tv, v_full, v_empty, gv++, v_prev * 128, bh_prev);
      settle_copies(wctx);
    }
  } else if (warp < FWD128_FIRST_CW) {
    // whole warp, converged: the MMA / commit helpers elect the issuing lane. The blocks of all items are one
    // sequence g = 0, 1, ...: P V of block g, then, when it has read P, the scores of block g + 1.
    constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, 0, 0);
    constexpr uint32_t idesc_o = umma_idesc_bf16(128, D, 0, 1);
    int s_rnd = 0, s_j = 0, s_n = 0, s_g = 0;     // next block whose scores are issued
    auto open_item = [&]() {
      s_n = 0;
      s_j = 0;
      if (s_rnd * W < n_items) {
        const int w = snake(s_rnd);
        int qt, bh;
        if (w < n_items) decode(w, qt, bh, s_n);
      }
    };
    open_item();
    auto issue_s = [&]() {
      if (s_n == 0) return;
      if (s_j == 0) mbar_wait(q_full, s_rnd & 1, wctx, STATUS_TIMEOUT_PIPE_FULL);
      mbar_wait(k_full, s_g & 1, wctx, STATUS_TIMEOUT_PIPE_FULL);
      tc_fence_after();
      mma_kk<D / 16>(tmem_base, smem_u32(Qs), 16384, smem_u32(Ks), 16384, idesc_s, false);
      umma_commit_e(s_full);
      umma_commit_e(k_empty);
      ++s_g;
      if (++s_j == s_n) {
        umma_commit_e(q_empty);
        ++s_rnd;
        open_item();
      }
    };
    issue_s();
    int g = 0;
    for (int rnd = 0; rnd * W < n_items; ++rnd) {
      const int w = snake(rnd);
      if (w >= n_items) break;
      int qt, bh, n;
      decode(w, qt, bh, n);
      for (int j = 0; j < n; ++j, ++g) {
        mbar_wait(v_full, g & 1, wctx, STATUS_TIMEOUT_PIPE_FULL);
        mbar_wait(p_full, g & 1, wctx, STATUS_TIMEOUT_SOFTMAX);
        // the accumulator is overwritten once per item: the previous item's result has been read out of it
        if (j == 0) mbar_wait(o_empty, (rnd & 1) ^ 1u, wctx, STATUS_TIMEOUT_SOFTMAX);
        tc_fence_after();
        mma_tmn<8, P_HALF>(tmem_base + O_COL, tmem_base, smem_u32(Vs), 16384, idesc_o, j > 0);
        umma_commit_e(o_full);
        umma_commit_e(v_empty);
        if (s_n > 0) mbar_wait(o_full, g & 1, wctx, STATUS_TIMEOUT_TMEM_FULL);
        issue_s();
      }
    }
  } else {
    const int half = ((warp - FWD128_FIRST_CW) >> 2) & 1;   // keys [64 half, + 64) of every block
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t s_addr = tmem_base + lane_base + half * 64;
    const uint32_t o_addr = tmem_base + lane_base + O_COL + half * (D / 2);
    const uint32_t p_addr = tmem_base + lane_base + half * P_HALF;
    const int bar_id = 1 + x * 4 + quarter;              // the two warps that share these rows
    float* const xch_own = xch + x * 512 + half * 128 + r;          // + 256 * parity
    const float* const xch_other = xch + x * 512 + (half ^ 1) * 128 + r;
    const float sl2 = p.scale * LOG2E_F;
    const uint64_t sl2_2 = pack_f32x2(sl2, sl2);
    int g = 0;
    uint32_t xpar = 0;                                   // parity of the exchange buffer
    auto exchange = [&](float v) {
      xch_own[xpar * 256] = v;
      named_barrier_sync(bar_id, 64);
      const float o = xch_other[xpar * 256];
      xpar ^= 1u;
      return o;
    };
    for (int rnd = 0; rnd * W < n_items; ++rnd) {
      const int w = snake(rnd);
      if (w >= n_items) break;
      int qt, bh, n;
      decode(w, qt, bh, n);
      const int b = bh / p.nh, h = bh % p.nh;
      const int row_g = qt * 128 + r;
      float m = -INFINITY;
      uint64_t l2 = 0;                                   // two partial sums of this thread's exponentials
      for (int j = 0; j < n; ++j, ++g) {
        const int col0 = j * 128 + half * 64;
        const bool need_mask = (p.causal && j == qt) || ((j + 1) * 128 > p.S);
        mbar_wait(s_full, g & 1, wctx, STATUS_TIMEOUT_SOFTMAX);
        tc_fence_after();
        uint32_t v[2][32];
        float mx0 = -INFINITY, mx1 = -INFINITY;
        tmem_ld_32x32(s_addr, v[0]);
        tmem_ld_32x32(s_addr + 32, v[1]);
        tmem_ld_wait_for(v[0]);
        tmem_ld_wait_for(v[1]);
        if (need_mask) {
          // Diagonal block (causal) or the block that crosses the end of the sequence: dead scores
          // become -inf in the registers, then the block takes the same code as every other one
          // (exp2(-inf) = 0, max ignores -inf).
          const int lim = min(p.causal ? row_g - col0 : 0x7fffffff, p.S - 1 - col0);   // last live column
#pragma unroll
          for (int e = 0; e < 64; ++e) v[e >> 5][e & 31] = (e > lim) ? 0xff800000u : v[e >> 5][e & 31];
        }
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          mx0 = fmax3(mx0, __uint_as_float(v[0][e]), __uint_as_float(v[0][e + 1]));
          mx1 = fmax3(mx1, __uint_as_float(v[1][e]), __uint_as_float(v[1][e + 1]));
        }
        const float mx = fmaxf(mx0, mx1);
        const float m_new = fmax3(m, mx, exchange(mx));
        // the maximum of all keys so far: both threads of a row raise it alike
        const bool grow = m_new > m;
        float alpha = 1.f;
        if (grow) {
          alpha = (m == -INFINITY) ? 0.f : fast_exp2((m - m_new) * sl2);
          l2 = mul_f32x2(l2, pack_f32x2(alpha, alpha));
          m = m_new;
        }
        const float moff = ((m == -INFINITY) ? 0.f : m) * sl2;
        const uint64_t moff2 = pack_f32x2(-moff, -moff);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t pk[16];
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            const float2 a = unpack_f32x2(fma_f32x2(pack_u32x2(v[c][e], v[c][e + 1]), sl2_2, moff2));
            const float p0 = fast_exp2(a.x), p1 = fast_exp2(a.y);
            l2 = add_f32x2(l2, pack_f32x2(p0, p1));
            pk[e >> 1] = pack_bf16x2(p0, p1);
          }
          tmem_st_32x16(p_addr + 16 * c, pk);
        }
        if (j > 0 && __any_sync(0xffffffffu, grow)) {
          // rescale this warp's 32 accumulator rows in tensor memory (warp-collective accesses; rows whose
          // maximum stays get factor 1), its half of the columns, while the registers of the scores are free. P V of
          // the previous block is done: this block's scores were issued after it.
          mbar_wait(o_full, (g - 1) & 1, wctx, STATUS_TIMEOUT_SOFTMAX);
          tc_fence_after();
          uint32_t wv[4][16];
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld_32x16(o_addr + 16 * c, wv[c]);
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld_wait_for16(wv[c]);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
#pragma unroll
            for (int e = 0; e < 16; ++e) wv[c][e] = __float_as_uint(__uint_as_float(wv[c][e]) * alpha);
            tmem_st_32x16(o_addr + 16 * c, wv[c]);
          }
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
      }
      const float2 lp = unpack_f32x2(l2);
      float l = lp.x + lp.y;
      l += exchange(l);
      const float inv_l = (l > 0.f) ? 1.f / l : 0.f;
      mbar_wait(o_full, (g - 1) & 1, wctx, STATUS_TIMEOUT_SOFTMAX);
      tc_fence_after();
      __nv_bfloat16* dst = p.O + row_g * p.o_ss + b * p.o_bs + h * p.o_hs + half * (D / 2);
      uint32_t o[D / 64][32];
#pragma unroll
      for (int c = 0; c < D / 64; ++c) tmem_ld_32x32(o_addr + 32 * c, o[c]);
#pragma unroll
      for (int c = 0; c < D / 64; ++c) tmem_ld_wait_for(o[c]);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(o_empty);   // the next item's first P V may overwrite the accumulator
      // twice when a copy is wanted (rolled: a second store beside the first one cost 12 bytes of spills)
#pragma unroll 1
      for (int n_out = row_g >= p.S ? 0 : (p.o_copy != 0 ? 2 : 1); n_out > 0; --n_out, dst += p.o_copy) {
#pragma unroll
        for (int c = 0; c < D / 64; ++c) {
#pragma unroll
          for (int e = 0; e < 32; e += 8) {
            uint4 wv;
            wv.x = pack_out(__uint_as_float(o[c][e + 0]) * inv_l, __uint_as_float(o[c][e + 1]) * inv_l, p.o_f16);
            wv.y = pack_out(__uint_as_float(o[c][e + 2]) * inv_l, __uint_as_float(o[c][e + 3]) * inv_l, p.o_f16);
            wv.z = pack_out(__uint_as_float(o[c][e + 4]) * inv_l, __uint_as_float(o[c][e + 5]) * inv_l, p.o_f16);
            wv.w = pack_out(__uint_as_float(o[c][e + 6]) * inv_l, __uint_as_float(o[c][e + 7]) * inv_l, p.o_f16);
            *reinterpret_cast<uint4*>(dst + 32 * c + e) = wv;
          }
        }
      }
      if (half == 0 && row_g < p.S_pad) {
        const float mm = (m == -INFINITY) ? 0.f : m;
        p.lse[static_cast<size_t>(bh) * p.S_pad + row_g] = mm * sl2 + log2f(fmaxf(l, 1e-37f));
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 2) tmem_dealloc(*tmem_slot, 512);
}

// ---------------------------------------------------------------------------
// Forward, head_dim 64: two 128-row query tiles per CTA.
//
// One CTA per SM; warps 4-7 run the softmax of tile A and warps 8-11 that of tile B (one thread
// per query row, so no cross-thread reductions), which gives every scheduler two independent
// softmax warps while K/V tiles are fetched once for 256 query rows. S, P V and P each live
// in tensor memory (S_A S_B | PV_A PV_B | P_A P_B = 512 columns): the probabilities are
// handed to the P V MMA as its TMEM A operand, nothing of the softmax goes through shared
// memory. K/V use a 4-stage ring (three: 111.1 us, four: 109.4 us at the GPT-124M shape with an
// earlier version; six stages measured 1.5 % slower than four with this one).
// ---------------------------------------------------------------------------
constexpr int FWD64_FIRST_SW = 4;                   // warps 0: TMA, 1: MMAs, 2 and 3: idle; then the softmax warps
constexpr int FWD64_THREADS = 32 * (FWD64_FIRST_SW + 8);
// Registers: 384 threads x 168 at the launch = 128 x 72 + 256 x 216. A softmax thread holds the 128 scores of its row and
// their packed probabilities; with 168 the exponentials' sums and products could not be paired (spills). us, 168 registers
// and scalar arithmetic -> this: [16, 12, 1024, 64] 64.4 -> 59.3, [8, 12, 2048, 64] 94.3 -> 89.0,
// [4, 12, 4096, 64] 163 -> 155, [3, 12, 777, 64] 15.7 -> 15.0, [2, 4, 256, 64] 7.6 -> 7.4.
constexpr int FWD64_REGS_IO = 72, FWD64_REGS_SOFTMAX = 216;
constexpr int FWD64_KS = 4;
constexpr int FWD64_SMEM = 2 * 16384 + FWD64_KS * 32768 + 512;

// Persistent: each CTA walks work items (pair of query tiles, batch*head), heaviest pairs
// first, so barrier set-up, the TMEM allocation and the CTA launch gap are paid once per SM
// instead of once per item (at sequence length 1024 they were ~45 % of the kernel's time).
// All barrier parities therefore run on counters that continue across items.
//
// The output accumulates in tensor memory (P V issued with accumulate) instead of being
// folded into registers after every key block, and the running maximum is only raised when it
// grows by more than 2^8 (any consistent offset gives the same softmax; the stale one keeps
// exp2 arguments <= 8). Raising it rescales the accumulator in tensor memory, which after the
// first blocks is rare. This frees the 64 accumulator registers per thread, so a block's 128
// scores are loaded once and stay in registers for both the maximum and the exponentials.
__global__ void __launch_bounds__(FWD64_THREADS, 1)
flash_fwd64_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                   const __grid_constant__ CUtensorMap tv, const FwdParams p, int n_pairs, int n_items) {
  constexpr int D = 64;
  constexpr int KS = FWD64_KS;
  constexpr uint32_t S_COL = 0, OP_COL = 256, P_COL = 384;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* Qs = smem_raw;                    // [2][128 x 64]
  uint8_t* Ks = Qs + 2 * 16384;              // [KS][128 x 64]
  uint8_t* Vs = Ks + KS * 16384;             // [KS][128 x 64]
  uint64_t* bars = reinterpret_cast<uint64_t*>(Vs + KS * 16384);
  uint64_t* q_full = bars;
  uint64_t* q_empty = bars + 1;
  uint64_t* k_full = bars + 2;               // [KS]
  uint64_t* k_empty = k_full + KS;
  uint64_t* v_full = k_empty + KS;
  uint64_t* v_empty = v_full + KS;
  uint64_t* s_full = v_empty + KS;           // [2] per query tile
  uint64_t* p_full = s_full + 2;
  uint64_t* o_full = p_full + 2;
  uint64_t* o_empty = o_full + 2;
  uint64_t* s_free = o_empty + 2;            // [2] the tile's scores have been read out of tensor memory
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_free + 2);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if (smem_u32(smem_raw) & 1023u) {
    if (threadIdx.x == 0) record_status(p.status, STATUS_BAD_ARGUMENT, 0x5a12u);
    return;
  }
  const int nb = (p.S + 127) >> 7;
  const int BH = p.B * p.nh;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    for (int i = 0; i < KS; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);
      mbar_init(&o_full[i], 1);
      mbar_init(&o_empty[i], 4);
      mbar_init(&s_free[i], 4);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tq);
    tma_prefetch_desc(&tk);
    tma_prefetch_desc(&tv);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_wait();       // set-up above may overlap the tail of the preceding kernel (programmatic launch)
  pdl_trigger();
  const uint32_t tmem_base = *tmem_slot;
  WaitCtx wctx{abort_flag, p.status, GFS_WAIT_LIMIT_NS};

  // Work items are dealt to the CTAs in a snake (left to right, then right to left), which
  // evens out the per-CTA totals of the descending item weights; an item past the end can
  // only occur in a CTA's last round.
  const int G = static_cast<int>(gridDim.x);
  auto snake = [&](int rnd) {
    return rnd * G + ((rnd & 1) ? G - 1 - static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x));
  };
  // decode of work item w: pairs in descending order (most key blocks first), then batch*head
  auto decode = [&](int w, int& qp, int& bh, int& na, int& nbk) {
    qp = n_pairs - 1 - w / BH;
    bh = w % BH;
    const int qa = 2 * qp, qb = 2 * qp + 1;
    na = p.causal ? min(qa + 1, nb) : nb;
    nbk = (qb < nb) ? (p.causal ? min(qb + 1, nb) : nb) : 0;
  };

  if (warp < FWD64_FIRST_SW) {
    setmaxnreg_dec<FWD64_REGS_IO>();
    if (warp == 0) {
      if (lane == 0) {
        int g = 0;      // key blocks loaded so far (ring position)
        for (int rnd = 0; rnd * G < n_items; ++rnd) {
          const int w = snake(rnd);
          if (w >= n_items) break;
          const int item = rnd;
          int qp, bh, na, nbk;
          decode(w, qp, bh, na, nbk);
          const int b = bh / p.nh, h = bh % p.nh;
          const int n_kv = max(na, nbk);
          mbar_wait(q_empty, (item & 1) ^ 1u, wctx, STATUS_TIMEOUT_PIPE_EMPTY);  // previous item's S MMAs done
          mbar_arrive_expect_tx(q_full, 2 * 16384);
          tma_load_4d(Qs, &tq, q_full, 0, (2 * qp) * 128, h, b);
          tma_load_4d(Qs + 16384, &tq, q_full, 0, (2 * qp + 1) * 128, h, b);   // rows past S are zero-filled
          for (int j = 0; j < n_kv; ++j, ++g) {
            const int st = g % KS;
            const uint32_t par = ((g / KS) & 1) ^ 1u;
            mbar_wait(&k_empty[st], par, wctx, STATUS_TIMEOUT_PIPE_EMPTY);
            mbar_arrive_expect_tx(&k_full[st], 16384);
            tma_load_4d(Ks + st * 16384, &tk, &k_full[st], 0, j * 128, h, b);
            mbar_wait(&v_empty[st], par, wctx, STATUS_TIMEOUT_PIPE_EMPTY);
            mbar_arrive_expect_tx(&v_full[st], 16384);
            tma_load_4d(Vs + st * 16384, &tv, &v_full[st], 0, j * 128, h, b);
          }
        }
        settle_copies(wctx);
      }
    } else if (warp == 1) {
      {  // whole warp, converged: the MMA / commit helpers elect the issuing lane
        constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, 0, 0);
        constexpr uint32_t idesc_o = umma_idesc_bf16(128, D, 0, 1);
        int g0 = 0;            // ring position of this item's first key block
        int cx[2] = {0, 0};    // blocks processed so far per query tile (barrier phase counters)
        int it[2] = {0, 0};    // items in which the tile had blocks (phase of o_empty)
        for (int rnd = 0; rnd * G < n_items; ++rnd) {
          const int w = snake(rnd);
          if (w >= n_items) break;
          const int item = rnd;
          int qp, bh, n_x[2];
          decode(w, qp, bh, n_x[0], n_x[1]);
          const int n_kv = max(n_x[0], n_x[1]);
          mbar_wait(q_full, item & 1, wctx, STATUS_TIMEOUT_PIPE_FULL);
          auto issue_s = [&](int x, int j) {
            const int g = g0 + j;
            mbar_wait(&k_full[g % KS], (g / KS) & 1, wctx, STATUS_TIMEOUT_PIPE_FULL);
            tc_fence_after();
            mma_kk<D / 16>(tmem_base + S_COL + x * 128, smem_u32(Qs + x * 16384), 0, smem_u32(Ks + (g % KS) * 16384),
                           0, idesc_s, false);
            umma_commit_e(&s_full[x]);
          };
          // S(0) of this item may only overwrite S once the softmax has consumed the previous
          // item's last block of that tile; that is guaranteed because the previous item's last
          // P V of the tile was issued after its p_full, and we issue in program order.
          if (n_x[0] > 0) issue_s(0, 0);
          if (n_x[1] > 0) issue_s(1, 0);
          if (n_kv > 0) umma_commit_e(&k_empty[g0 % KS]);
          if (n_kv == 1) umma_commit_e(q_empty);
          // Event loop over both query tiles. Two kinds of events per tile: "scores read out"
          // (s_free: the softmax warps hold block j's scores in registers) lets S(j+1) be issued
          // into the same columns while the exponentials of block j are still being computed, so
          // the next scores are ready when the softmax gets there; "probabilities stored" (p_full)
          // lets P V(j) be issued. Every wait here is a poll, so a tile that is ahead (bounded by
          // the K/V ring, whose stages are released when both tiles have used a
          // block) never blocks the warp that the other tile needs.
          int s_iss[2] = {n_x[0] > 0 ? 1 : 0, n_x[1] > 0 ? 1 : 0};   // S MMAs issued per tile
          int pv_iss[2] = {0, 0};                                     // P V MMAs issued per tile
          uint32_t spins = 0;
          uint64_t spin_t0 = 0;
          bool dead = false;
          while ((pv_iss[0] < n_x[0] || pv_iss[1] < n_x[1]) && !dead) {
            bool progressed = false;
#pragma unroll
            for (int x = 0; x < 2; ++x) {
              const int ot = x ^ 1;
              const int bn = s_iss[x];          // next block whose S is to be issued
              if (bn > 0 && bn < n_x[x]) {
                const int gb = g0 + bn;
                if (mbar_try_wait(&s_free[x], (cx[x] + bn - 1) & 1) &&
                    mbar_try_wait(&k_full[gb % KS], (gb / KS) & 1)) {
                  tc_fence_after();
                  mma_kk<D / 16>(tmem_base + S_COL + x * 128, smem_u32(Qs + x * 16384), 0,
                                 smem_u32(Ks + (gb % KS) * 16384), 0, idesc_s, false);
                  umma_commit_e(&s_full[x]);
                  s_iss[x] = bn + 1;
                  // the K block is free once both tiles' S MMAs on it have been issued
                  if (s_iss[ot] > bn || bn >= n_x[ot]) umma_commit_e(&k_empty[gb % KS]);
                  if (s_iss[0] >= n_x[0] && s_iss[1] >= n_x[1]) umma_commit_e(q_empty);   // the item's last S
                  progressed = true;
                }
              }
              const int j = pv_iss[x];
              if (j < n_x[x]) {
                const int c = cx[x] + j;
                const int g = g0 + j;
                if (mbar_try_wait(&p_full[x], c & 1) && mbar_try_wait(&v_full[g % KS], (g / KS) & 1)) {
                  // the accumulator is overwritten once per item: wait until the softmax warps
                  // have read the previous item's result out of it
                  if (j == 0) mbar_wait(&o_empty[x], (it[x] & 1) ^ 1u, wctx, STATUS_TIMEOUT_SOFTMAX);
                  tc_fence_after();
                  mma_tmn<8>(tmem_base + OP_COL + x * 64, tmem_base + P_COL + x * 64, smem_u32(Vs + (g % KS) * 16384),
                             0, idesc_o, j > 0);
                  umma_commit_e(&o_full[x]);
                  pv_iss[x] = j + 1;
                  if (pv_iss[ot] > j || j >= n_x[ot]) umma_commit_e(&v_empty[g % KS]);
                  progressed = true;
                }
              }
            }
            if (progressed) {
              spins = 0;
              spin_t0 = 0;
            } else if (((++spins) & 0xfffu) == 0u) {
              // bounded like mbar_wait: give up (status recorded) when nothing becomes ready in time
              if (*abort_flag) {
                dead = true;
              } else {
                const uint64_t now = globaltimer_ns();
                if (spin_t0 == 0) {
                  spin_t0 = now;
                } else if (now - spin_t0 > GFS_WAIT_LIMIT_NS) {
                  *abort_flag = 1u;
                  record_status(p.status, STATUS_TIMEOUT_SOFTMAX, (blockIdx.x << 8) | 0xE1u);
                  dead = true;
                }
              }
            }
          }
          g0 += n_kv;
          cx[0] += n_x[0];
          cx[1] += n_x[1];
          it[0] += n_x[0] > 0;
          it[1] += n_x[1] > 0;
        }
      }
    }
  } else {
    setmaxnreg_inc<FWD64_REGS_SOFTMAX>();
    const int x = (warp - FWD64_FIRST_SW) >> 2;   // query tile of this warp
    const int quarter = warp & 3;
    const int r = quarter * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t s_addr = tmem_base + lane_base + S_COL + x * 128;
    const uint32_t o_addr = tmem_base + lane_base + OP_COL + x * 64;
    const uint32_t p_addr = tmem_base + lane_base + P_COL + x * 64;
    const float sl2 = p.scale * LOG2E_F;
    const uint64_t sl2_2 = pack_f32x2(sl2, sl2);
    int cdone = 0;  // blocks of this tile processed in earlier items
    {
      for (int rnd = 0; rnd * G < n_items; ++rnd) {
        const int w = snake(rnd);
        if (w >= n_items) break;
        int qp, bh, na, nbk;
        decode(w, qp, bh, na, nbk);
        const int b = bh / p.nh, h = bh % p.nh;
        const int qtx = 2 * qp + x;
        const int row_g = qtx * 128 + r;
        const int n_mine = x == 0 ? na : nbk;
        float m = -INFINITY, l = 0.f;
        for (int j = 0; j < n_mine; ++j) {
          const int c = cdone + j;
          const bool need_mask = (p.causal && j == qtx) || ((j + 1) * 128 > p.S);
          mbar_wait(&s_full[x], c & 1, wctx, STATUS_TIMEOUT_SOFTMAX);
          tc_fence_after();
          uint32_t v0[32], v1[32], v2[32], v3[32];
          tmem_ld_32x32(s_addr + 0, v0);
          tmem_ld_32x32(s_addr + 32, v1);
          tmem_ld_32x32(s_addr + 64, v2);
          tmem_ld_32x32(s_addr + 96, v3);
          float mx0 = -INFINITY, mx1 = -INFINITY;
          tmem_ld_wait_for(v0);
          tmem_ld_wait_for(v1);
          tmem_ld_wait_for(v2);
          tmem_ld_wait_for(v3);
          // all 128 scores are in registers: the MMA warp may overwrite S with the next block's
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&s_free[x]);
          if (need_mask) {
            // Diagonal block (causal) or the block that crosses the end of the sequence: dead scores
            // become -inf in the registers, then the block takes the same code as every other one
            // (exp2(-inf) = 0, max ignores -inf). A separate masked copy of the max / exponential code
            // ran once per work item from a cold instruction cache: 6500 cycles for that block
            // against 2450 for an unmasked one.
            auto mask_chunk = [&](uint32_t (&v)[32], int cc) {
              const int lim_c = p.causal ? row_g - j * 128 - cc : 0x7fffffff;   // last live column of the chunk
              const int lim = min(lim_c, p.S - 1 - j * 128 - cc);
#pragma unroll
              for (int e = 0; e < 32; ++e) v[e] = (e > lim) ? 0xff800000u : v[e];
            };
            mask_chunk(v0, 0);
            mask_chunk(v1, 32);
            mask_chunk(v2, 64);
            mask_chunk(v3, 96);
          }
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            mx0 = fmax3(mx0, __uint_as_float(v0[e]), __uint_as_float(v0[e + 1]));
            mx1 = fmax3(mx1, __uint_as_float(v1[e]), __uint_as_float(v1[e + 1]));
            mx0 = fmax3(mx0, __uint_as_float(v2[e]), __uint_as_float(v2[e + 1]));
            mx1 = fmax3(mx1, __uint_as_float(v3[e]), __uint_as_float(v3[e + 1]));
          }
          const float m_new = fmaxf(m, fmaxf(mx0, mx1));
          // raise the running maximum only when it grew by more than 2^8 (or was still -inf)
          bool grow = false;
          float alpha = 1.f;
          if (m_new > m && (m == -INFINITY || (m_new - m) * sl2 > 8.f)) {
            grow = true;
            alpha = (m == -INFINITY) ? 0.f : fast_exp2((m - m_new) * sl2);
          }
          if (j > 0 && __any_sync(0xffffffffu, grow)) {
            // rescale this warp's 32 accumulator rows in tensor memory (warp-collective accesses;
            // rows whose maximum stays get factor 1). P V of the previous block must be done.
            mbar_wait(&o_full[x], (c - 1) & 1, wctx, STATUS_TIMEOUT_SOFTMAX);
            tc_fence_after();
            const float a = grow ? alpha : 1.f;
#pragma unroll 1
            for (int cc = 0; cc < D; cc += 16) {
              uint32_t wv[16];
              tmem_ld_32x16(o_addr + cc, wv);
              tmem_ld_wait_for16(wv);
#pragma unroll
              for (int e = 0; e < 16; ++e) wv[e] = __float_as_uint(__uint_as_float(wv[e]) * a);
              tmem_st_32x16(o_addr + cc, wv);
            }
            tmem_st_wait();
          }
          if (grow) {
            l *= alpha;
            m = m_new;
          }
          const float moff = ((m == -INFINITY) ? 0.f : m) * sl2;
          const uint64_t moff2 = pack_f32x2(-moff, -moff);
          uint64_t rs2 = 0;                        // two columns per instruction of the FMA pipe
          auto prob_chunk = [&](const uint32_t (&v)[32], uint32_t (&packed)[16]) {
#pragma unroll
            for (int e = 0; e < 32; e += 2) {
              const float2 y = unpack_f32x2(fma_f32x2(pack_u32x2(v[e], v[e + 1]), sl2_2, moff2));
              const float x0 = fast_exp2(y.x), x1 = fast_exp2(y.y);
              rs2 = add_f32x2(rs2, pack_f32x2(x0, x1));
              packed[e >> 1] = pack_bf16x2(x0, x1);
            }
          };
          uint32_t p0[16], p1[16], p2[16], p3[16];
          prob_chunk(v0, p0);
          prob_chunk(v1, p1);
          prob_chunk(v2, p2);
          prob_chunk(v3, p3);
          const float2 rs = unpack_f32x2(rs2);
          l += rs.x + rs.y;
          // P of the previous block is read by its P V MMA: overwrite it only when that is done
          if (j > 0) {
            mbar_wait(&o_full[x], (c - 1) & 1, wctx, STATUS_TIMEOUT_SOFTMAX);
            tc_fence_after();
          }
          tmem_st_32x16(p_addr + 0, p0);
          tmem_st_32x16(p_addr + 16, p1);
          tmem_st_32x16(p_addr + 32, p2);
          tmem_st_32x16(p_addr + 48, p3);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&p_full[x]);
        }
        if (n_mine > 0) {
          mbar_wait(&o_full[x], (cdone + n_mine - 1) & 1, wctx, STATUS_TIMEOUT_SOFTMAX);
          tc_fence_after();
          uint32_t wa[32], wb[32];
          tmem_ld_32x32(o_addr, wa);
          tmem_ld_32x32(o_addr + 32, wb);
          tmem_ld_wait_for(wa);
          tmem_ld_wait_for(wb);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&o_empty[x]);   // the next item's first P V may overwrite the accumulator
          const float inv_l = (l > 0.f) ? 1.f / l : 0.f;
          if (row_g < p.S) {
            __nv_bfloat16* dst = p.O + row_g * p.o_ss + b * p.o_bs + h * p.o_hs;
#pragma unroll
            for (int cc = 0; cc < 32; cc += 8) {
              uint4 wv;
              wv.x = pack_out(__uint_as_float(wa[cc + 0]) * inv_l, __uint_as_float(wa[cc + 1]) * inv_l, p.o_f16);
              wv.y = pack_out(__uint_as_float(wa[cc + 2]) * inv_l, __uint_as_float(wa[cc + 3]) * inv_l, p.o_f16);
              wv.z = pack_out(__uint_as_float(wa[cc + 4]) * inv_l, __uint_as_float(wa[cc + 5]) * inv_l, p.o_f16);
              wv.w = pack_out(__uint_as_float(wa[cc + 6]) * inv_l, __uint_as_float(wa[cc + 7]) * inv_l, p.o_f16);
              *reinterpret_cast<uint4*>(dst + cc) = wv;
              if (p.o_copy != 0) *reinterpret_cast<uint4*>(dst + p.o_copy + cc) = wv;
              wv.x = pack_out(__uint_as_float(wb[cc + 0]) * inv_l, __uint_as_float(wb[cc + 1]) * inv_l, p.o_f16);
              wv.y = pack_out(__uint_as_float(wb[cc + 2]) * inv_l, __uint_as_float(wb[cc + 3]) * inv_l, p.o_f16);
              wv.z = pack_out(__uint_as_float(wb[cc + 4]) * inv_l, __uint_as_float(wb[cc + 5]) * inv_l, p.o_f16);
              wv.w = pack_out(__uint_as_float(wb[cc + 6]) * inv_l, __uint_as_float(wb[cc + 7]) * inv_l, p.o_f16);
              *reinterpret_cast<uint4*>(dst + 32 + cc) = wv;
              if (p.o_copy != 0) *reinterpret_cast<uint4*>(dst + p.o_copy + 32 + cc) = wv;
            }
          }
          if (row_g < p.S_pad) {
            const float mm = (m == -INFINITY) ? 0.f : m;
            p.lse[static_cast<size_t>(bh) * p.S_pad + row_g] = mm * sl2 + log2f(fmaxf(l, 1e-37f));
          }
        }
        cdone += n_mine;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

// ---------------------------------------------------------------------------
// fp16 callers: q, k, v ([B, nh, S, D] views with any strides) rounded to bf16, contiguous, one launch.
// ---------------------------------------------------------------------------
struct CastArgs {
  const __half* src[3];
  long long ss[3], bs[3], hs[3];   // element strides: sequence, batch, head
};
__global__ void cast_qkv_kernel(const CastArgs a, __nv_bfloat16* __restrict__ dst, int S, int B, int nh, int D) {
  const int vpr = D >> 3;
  const long long n = static_cast<long long>(B) * nh * S * vpr;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(i % vpr) * 8;
    const long long row = i / vpr;
    const int s = static_cast<int>(row % S);
    const long long bh = row / S;
    const int h = static_cast<int>(bh % nh), b = static_cast<int>(bh / nh);
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      const uint4 x = *reinterpret_cast<const uint4*>(a.src[t] + s * a.ss[t] + b * a.bs[t] + h * a.hs[t] + c);
      const uint32_t w[4] = {x.x, x.y, x.z, x.w};
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[e]));
        o[e] = pack_bf16x2(f.x, f.y);
      }
      *reinterpret_cast<uint4*>(dst + (t * n + i) * 8) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// ---------------------------------------------------------------------------
// Backward pre-pass: dvec[b,h,s] = sum_d dO[s,b,h,d] * O[s,b,h,d]. F16: dO and O are fp16, and dO is also
// written rounded to bf16 ([B, nh, S, D] contiguous), the form the gradient products read (and the
// one the sum uses, so that it matches them).
//
// Bound by memory latency, not bandwidth: 50 MB at the GPT-124M shape (batch 16) took 25 us with one row
// chunk (two 16-byte loads) per thread; four rows per thread with all loads issued first, and
// no second pass over the LSE (the forward now writes it in the form the backward wants).
// ---------------------------------------------------------------------------
constexpr int DVEC_ROWS = 4;
template <bool F16>
__global__ void __launch_bounds__(256)
attn_dvec_kernel(const void* dO_, const void* O_, float* __restrict__ dvec,
                 __nv_bfloat16* __restrict__ dO_bf16, int S, int S_pad, int B, int nh, int D, long long do_ss,
                 long long do_bs, long long do_hs, long long o_ss, long long o_bs, long long o_hs, int s_fastest) {
  pdl_wait();
  pdl_trigger();
  const uint16_t* dO = static_cast<const uint16_t*>(dO_);
  const uint16_t* O = static_cast<const uint16_t*>(O_);
  // D/8 threads per (s, b, h) row, 16-byte loads; rows in memory order ([S,B,nh,D]: h fastest, [B,nh,S,D]: s fastest)
  const int tpr = D >> 3;                       // 8 or 16 threads per row
  const int rows_per_pass = blockDim.x / tpr;
  const int sub = threadIdx.x % tpr;
  const unsigned total = static_cast<unsigned>(S) * B * nh;
  const unsigned row0 = blockIdx.x * static_cast<unsigned>(rows_per_pass * DVEC_ROWS) + threadIdx.x / tpr;
  uint4 x[DVEC_ROWS], y[DVEC_ROWS];
  unsigned at[DVEC_ROWS];                       // b * nh + h, s
  int sq[DVEC_ROWS];
#pragma unroll
  for (int i = 0; i < DVEC_ROWS; ++i) {
    const unsigned row = row0 + i * rows_per_pass;
    x[i] = make_uint4(0, 0, 0, 0);
    y[i] = x[i];
    unsigned h, b, s;
    if (s_fastest) {
      s = row % S;
      const unsigned bh = row / S;
      h = bh % nh;
      b = bh / nh;
    } else {
      h = row % nh;
      const unsigned sb = row / nh;
      b = sb % B;
      s = sb / B;
    }
    at[i] = b * nh + h;
    sq[i] = static_cast<int>(s);
    if (row < total) {
      x[i] = *reinterpret_cast<const uint4*>(dO + s * do_ss + b * do_bs + h * do_hs + sub * 8);
      y[i] = *reinterpret_cast<const uint4*>(O + s * o_ss + b * o_bs + h * o_hs + sub * 8);
    }
  }
#pragma unroll
  for (int i = 0; i < DVEC_ROWS; ++i) {
    const unsigned row = row0 + i * rows_per_pass;
    uint32_t xw[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
    const uint32_t yw[4] = {y[i].x, y[i].y, y[i].z, y[i].w};
    float acc = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float2 b2;
      if (F16) {
        const float2 a2 = __half22float2(*reinterpret_cast<const __half2*>(&xw[e]));
        xw[e] = pack_bf16x2(a2.x, a2.y);
        b2 = __half22float2(*reinterpret_cast<const __half2*>(&yw[e]));
      } else {
        b2 = unpack_bf16x2(yw[e]);
      }
      const float2 a2 = unpack_bf16x2(xw[e]);
      acc += a2.x * b2.x + a2.y * b2.y;
    }
    if (F16 && row < total)
      *reinterpret_cast<uint4*>(dO_bf16 + (static_cast<size_t>(at[i]) * S + sq[i]) * D + sub * 8) =
          make_uint4(xw[0], xw[1], xw[2], xw[3]);
    for (int o = tpr >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (row < total && sub == 0) dvec[static_cast<size_t>(at[i]) * S_pad + sq[i]] = acc;
  }
  // rows S .. S_pad-1 of every head: zeros (the backward multiplies them by probabilities that are 0)
  const unsigned pad = S_pad - S;
  const unsigned pad_total = pad * B * nh;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < pad_total; i += gridDim.x * blockDim.x)
    dvec[static_cast<size_t>(i / pad) * S_pad + S + (i % pad)] = 0.f;
}

// ---------------------------------------------------------------------------
// Backward main kernel
// ---------------------------------------------------------------------------
struct BwdParams {
  __nv_bfloat16* out1;  // mode 0: dK, mode 1: dQ
  __nv_bfloat16* out2;  // mode 0: dV
  long long o1_ss, o1_bs, o1_hs;
  long long o2_ss, o2_bs, o2_hs;
  const float* lse;   // [B, nh, S_pad], base 2
  const float* dvec;  // [B, nh, S_pad]
  int S, S_pad, B, nh;
  float scale;
  int causal;
  uint32_t* status;
  // optional: inverse rotary embedding applied to dQ and dK rows before they are stored
  const float* rope_cos;
  const float* rope_sin;
  int out_f16;        // dQ, dK, dV are stored as fp16
};

constexpr int BWD_CW = 16;                          // compute warps
constexpr int BWD_FIRST_CW = 4;                     // warps 0-2: TMA, score MMAs, gradient MMAs; 3: idle
constexpr int BWD_THREADS = 32 * (BWD_FIRST_CW + BWD_CW);

template <int D, int MODE>
struct BwdShape {
  // Stages of the streamed-tile ring. A stage is only released when the gradient MMAs that read it have
  // finished and the score MMAs run two tiles ahead, so the TMA of a tile has (TS - 2) tile periods to land.
  static constexpr int TS = D == 64 ? 7 : 4;
  // epilogue, per compute warp: 2 KB to transpose through; at head_dim 64 the rotary table's entries before that
  static constexpr bool ROPE_STAGED = D == 64;
  static constexpr int STAGE_BYTES = ROPE_STAGED ? 4096 : 2048;
  static constexpr int STAGING = BWD_CW * STAGE_BYTES;
  static constexpr int SMEM = 2 * (D / 64) * 16384 + 2 * TS * (D / 64) * 8192 + STAGING + (MODE == 0 ? TS * 512 : 0) + 256;
};

// Bound by the chain of a streamed tile in the compute warps (barrier test, tensor-memory loads, ~ 10
// instructions per score element, tensor-memory store, arrive), not by a unit, so what counts is how many
// chains are in flight: sixteen compute warps, four per scheduler. Two groups of eight take alternate
// streamed tiles (group = X/Y buffer); within a group two warps share the 32 rows of a quarter, 32 streamed
// columns each (no exchange is needed: the row / column statistics are inputs). The MMAs are issued by two
// warps (1: scores, 2: gradients), so neither order waits for the other. P / dS (bf16) go to the gradient
// MMAs as their tensor-memory A operand: in columns of their own where there is room, for dK / dV at
// head_dim 128 in the columns of the scores they were made from (then a score buffer is free again when
// the gradient MMAs have read it).
// us per backward (pre-pass, dK / dV, dQ), eight compute warps (at head_dim 128 with P / dS in shared memory)
// -> this: [16, 12, 1024, 64] causal 211 -> 173, [4, 2, 2048, 128] 92 -> 76, [1, 8, 4096, 128] 166 -> 136.
template <int D, int MODE>
__global__ void __launch_bounds__(BWD_THREADS, 1)
flash_bwd_kernel(const __grid_constant__ CUtensorMap tr1, const __grid_constant__ CUtensorMap tr2,
                 const __grid_constant__ CUtensorMap tt1, const __grid_constant__ CUtensorMap tt2,
                 const BwdParams p, int n_rt, int n_items) {
  constexpr int DB = D / 64;
  constexpr int TS = BwdShape<D, MODE>::TS;
  constexpr int R_BYTES = DB * 16384;  // resident [128 x D]
  constexpr int T_BYTES = DB * 8192;   // streamed [64 x D]
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t Y_COL = 128;      // X tiles at [0, 128), Y tiles after them
  constexpr uint32_t ACC1 = 256, ACC2 = 256 + D;
  constexpr bool OVERLAY = (D == 128 && MODE == 0);   // P over X, dS over Y
  constexpr uint32_t PT_COL = 384;     // else: [buffer][P 32 cols | dS 32 cols]
  constexpr int EPI_WARPS = (MODE == 1 && D == 64) ? BWD_CW / 2 : BWD_CW;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* R1 = smem_raw;
  uint8_t* R2 = R1 + R_BYTES;
  uint8_t* T1 = R2 + R_BYTES;
  uint8_t* T2 = T1 + TS * T_BYTES;
  uint8_t* staging = T2 + TS * T_BYTES;
  float* stats = reinterpret_cast<float*>(staging + BwdShape<D, MODE>::STAGING);  // mode 0: [TS stages][lse 64 | dvec 64]
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(stats) + (MODE == 0 ? TS * 512 : 0));
  uint64_t* r_full = bars;
  uint64_t* t_full = bars + 1;             // [TS]
  uint64_t* t_empty = t_full + TS;         // [TS]
  uint64_t* xy_full = t_empty + TS;
  uint64_t* xy_empty = xy_full + 2;
  uint64_t* m_full = xy_empty + 2;
  uint64_t* m_empty = m_full + 2;
  uint64_t* acc_full = m_empty + 2;
  uint64_t* acc_empty = acc_full + 1;
  uint64_t* r_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 3);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if (smem_u32(smem_raw) & 1023u) {
    if (threadIdx.x == 0) record_status(p.status, STATUS_BAD_ARGUMENT, 0x5a13u);
    return;
  }
  const int n_small = (p.S + 63) >> 6;  // number of 64-row streamed tiles in the sequence
  const int BH = p.B * p.nh;
  // Persistent: a CTA walks work items (resident tile, batch*head), heaviest resident tiles
  // first, dealt in a snake over the CTAs; barrier phases run on counters that continue
  // across items, so set-up and the TMEM allocation are paid once and the next item's loads
  // and first score MMAs overlap the current item's epilogue.
  const int G = static_cast<int>(gridDim.x);
  auto snake = [&](int rnd) {
    return rnd * G + ((rnd & 1) ? G - 1 - static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x));
  };
  // resident tile index and range of streamed tiles of work item w (at least one tile)
  auto decode = [&](int w, int& rt, int& bh, int& t_begin, int& n_t) {
    const int level = w / BH;
    bh = w % BH;
    int t_end;
    if (MODE == 0) {
      rt = level;  // key tile; the first ones have the most query tiles
      t_begin = p.causal ? 2 * rt : 0;
      t_end = n_small;
    } else {
      rt = n_rt - 1 - level;  // query tile; the last ones have the most key tiles
      t_begin = 0;
      t_end = p.causal ? min(n_small, 2 * rt + 2) : n_small;
    }
    n_t = max(t_end - t_begin, 0);
  };

  if (threadIdx.x == 0) {
    mbar_init(r_full, 1);
    for (int i = 0; i < TS; ++i) {
      mbar_init(&t_full[i], 1);
      mbar_init(&t_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&xy_full[i], 1);
      mbar_init(&xy_empty[i], BWD_CW / 2);
      mbar_init(&m_full[i], BWD_CW / 2);
      mbar_init(&m_empty[i], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, EPI_WARPS);
    mbar_init(r_empty, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tr1);
    tma_prefetch_desc(&tr2);
    tma_prefetch_desc(&tt1);
    tma_prefetch_desc(&tt2);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // Set-up above may overlap the tail of the preceding kernel (programmatic launch). The dQ kernel reads nothing that the
  // preceding dK / dV kernel writes, and that one had waited for everything before it when it let this one start: it
  // waits at its end, so that its completion means that of both. us per backward: [1, 12, 130, 64] 14.0 -> 12.2,
  // [2, 4, 256, 64] 14.9 -> 13.1, [3, 12, 777, 64] 32.2 -> 31.3, [16, 12, 1024, 64] 163.6 -> 162.4. (launch_hints.h has
  // what this means for the kernel that follows.)
  if (MODE == 0) pdl_wait();
  pdl_trigger();
  const uint32_t tmem_base = *tmem_slot;
  WaitCtx wctx{abort_flag, p.status, GFS_WAIT_LIMIT_NS};

  if (warp == 0) {
    if (lane == 0) {
      int g = 0;  // streamed tiles loaded so far (ring position)
      for (int it = 0; it * G < n_items; ++it) {
        const int w = snake(it);
        if (w >= n_items) break;
        int rt, bh, t_begin, n_t;
        decode(w, rt, bh, t_begin, n_t);
        const int b = bh / p.nh, h = bh % p.nh;
        mbar_wait(r_empty, (it & 1) ^ 1u, wctx, STATUS_TIMEOUT_PIPE_EMPTY);  // previous item's score MMAs done
        mbar_arrive_expect_tx(r_full, 2 * R_BYTES);
#pragma unroll
        for (int db = 0; db < DB; ++db) {
          tma_load_4d(R1 + db * 16384, &tr1, r_full, db * 64, rt * 128, h, b);
          tma_load_4d(R2 + db * 16384, &tr2, r_full, db * 64, rt * 128, h, b);
        }
        for (int t = 0; t < n_t; ++t, ++g) {
          const int st = g % TS;
          const int ti = t_begin + t;
          mbar_wait(&t_empty[st], ((g / TS) & 1) ^ 1u, wctx, STATUS_TIMEOUT_PIPE_EMPTY);
          mbar_arrive_expect_tx(&t_full[st], 2 * T_BYTES + (MODE == 0 ? 512 : 0));
#pragma unroll
          for (int db = 0; db < DB; ++db) {
            tma_load_4d(T1 + st * T_BYTES + db * 8192, &tt1, &t_full[st], db * 64, ti * 64, h, b);
            tma_load_4d(T2 + st * T_BYTES + db * 8192, &tt2, &t_full[st], db * 64, ti * 64, h, b);
          }
          if (MODE == 0) {
            const size_t off = static_cast<size_t>(bh) * p.S_pad + ti * 64;
            bulk_load_1d(stats + st * 128, p.lse + off, 256, &t_full[st]);
            bulk_load_1d(stats + st * 128 + 64, p.dvec + off, 256, &t_full[st]);
          }
        }
      }
      settle_copies(wctx);
    }
  } else if (warp == 1) {
    // Score MMAs (whole warp, converged: the MMA / commit helpers elect the issuing lane); runs ahead as
    // far as the X/Y buffers and the streamed-tile ring allow.
    constexpr uint32_t idesc_xy = umma_idesc_bf16(128, 64, 0, 0);
    const uint32_t r1 = smem_u32(R1), r2 = smem_u32(R2);
    int g = 0;
    for (int it = 0; it * G < n_items; ++it) {
      const int w = snake(it);
      if (w >= n_items) break;
      int rt, bh, t_begin, n_t;
      decode(w, rt, bh, t_begin, n_t);
      mbar_wait(r_full, it & 1, wctx, STATUS_TIMEOUT_PIPE_FULL);
      for (int t = 0; t < n_t; ++t, ++g) {
        const int st = g % TS, sb = g & 1;
        mbar_wait(&t_full[st], (g / TS) & 1, wctx, STATUS_TIMEOUT_PIPE_FULL);
        mbar_wait(OVERLAY ? &m_empty[sb] : &xy_empty[sb], ((g >> 1) & 1) ^ 1u, wctx, STATUS_TIMEOUT_SOFTMAX);
        tc_fence_after();
        mma_kk<D / 16>(tmem_base + sb * 64, r1, 16384, smem_u32(T1 + st * T_BYTES), 8192, idesc_xy, false);
        mma_kk<D / 16>(tmem_base + Y_COL + sb * 64, r2, 16384, smem_u32(T2 + st * T_BYTES), 8192, idesc_xy, false);
        umma_commit_e(&xy_full[sb]);
      }
      umma_commit_e(r_empty);
    }
  } else if (warp == 2) {
    // gradient MMAs
    constexpr uint32_t idesc_acc = umma_idesc_bf16(128, D, 0, 1);
    int g = 0;
    for (int it = 0; it * G < n_items; ++it) {
      const int w = snake(it);
      if (w >= n_items) break;
      int rt, bh, t_begin, n_t;
      decode(w, rt, bh, t_begin, n_t);
      for (int t = 0; t < n_t; ++t, ++g) {
        const int st = g % TS, sb = g & 1;
        mbar_wait(&m_full[sb], (g >> 1) & 1, wctx, STATUS_TIMEOUT_SOFTMAX);
        if (t == 0) mbar_wait(acc_empty, (it & 1) ^ 1u, wctx, STATUS_TIMEOUT_TMEM_EMPTY);  // previous epilogue done
        tc_fence_after();
        const uint32_t pt = tmem_base + (OVERLAY ? sb * 64 : PT_COL + sb * 64);
        const uint32_t ds = OVERLAY ? pt + Y_COL : pt + 32;
        constexpr int HALF = OVERLAY ? 32 : 16;   // columns from the first to the second half of P / dS
        if (MODE == 0) {
          mma_tmn<4, HALF>(tmem_base + ACC1, pt, smem_u32(T2 + st * T_BYTES), 8192, idesc_acc, t > 0);   // dV += P^T dO
          mma_tmn<4, HALF>(tmem_base + ACC2, ds, smem_u32(T1 + st * T_BYTES), 8192, idesc_acc, t > 0);   // dK += dS^T Q
        } else {
          mma_tmn<4, HALF>(tmem_base + ACC1, ds, smem_u32(T1 + st * T_BYTES), 8192, idesc_acc, t > 0);   // dQ += dS K
        }
        umma_commit_e(&t_empty[st]);
        umma_commit_e(&m_empty[sb]);
      }
      umma_commit_e(acc_full);
    }
  } else if (warp >= BWD_FIRST_CW) {
    const int cw = warp - BWD_FIRST_CW;
    const int quarter = warp & 3;
    const int half = (cw >> 2) & 1;     // 32 of the 64 streamed columns
    const int group = cw >> 3;          // parity of the streamed tiles of this warp
    const int r = quarter * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const float sl2 = p.scale * LOG2E_F;
    const uint64_t neg_sl2 = pack_f32x2(-sl2, -sl2), neg_one = pack_f32x2(-1.f, -1.f);
    const uint32_t x_addr = tmem_base + lane_base + group * 64 + half * 32;
    const uint32_t y_addr = x_addr + Y_COL;
    const uint32_t p_addr = OVERLAY ? x_addr : tmem_base + lane_base + PT_COL + group * 64 + half * 16;
    const uint32_t ds_addr = OVERLAY ? y_addr : p_addr + 32;
    uint8_t* stage = staging + cw * BwdShape<D, MODE>::STAGE_BYTES;
    bool acc_pending = false;           // the previous item's acc_full phase has not been waited for
    int g0 = 0;
    for (int it = 0; it * G < n_items; ++it) {
      const int w = snake(it);
      if (w >= n_items) break;
      int rt, bh, t_begin, n_t;
      decode(w, rt, bh, t_begin, n_t);
      const int b = bh / p.nh, h = bh % p.nh;
      const int row_g = rt * 128 + r;  // mode 0: key position, mode 1: query position
      float row_lse = 0.f, row_dvec = 0.f;
      if (MODE == 1 && row_g < p.S_pad) {
        row_lse = p.lse[static_cast<size_t>(bh) * p.S_pad + row_g];
        row_dvec = p.dvec[static_cast<size_t>(bh) * p.S_pad + row_g];
      }
      for (int t = (g0 + group) & 1; t < n_t; t += 2) {
        const int g = g0 + t;
        const int st = g % TS;                      // streamed-tile stage (for the column statistics)
        const uint32_t par = (g >> 1) & 1;
        const int ti = t_begin + t;
        const int col0 = ti * 64 + half * 32;       // position of this warp's first column
        bool need_mask;
        if (MODE == 0) need_mask = (p.causal && ti < 2 * rt + 2) || ((ti + 1) * 64 > p.S);
        else need_mask = (p.causal && ti >= 2 * rt) || ((ti + 1) * 64 > p.S);
        // alive / mixed / dead for this warp's 32 rows x 32 columns; a dead chunk costs no math
        const int row_lo = rt * 128 + quarter * 32;
        const int kind = need_mask ? mask_class<MODE == 0>(row_lo, row_lo + 31, col0, col0 + 31, p.causal != 0, p.S) : 0;
        mbar_wait(&xy_full[group], par, wctx, STATUS_TIMEOUT_SOFTMAX);
        tc_fence_after();
        uint32_t pp[16], dd[16];
        if (kind == 2) {
#pragma unroll
          for (int e = 0; e < 16; ++e) pp[e] = dd[e] = 0u;
          if (!OVERLAY && lane == 0) mbar_arrive(&xy_empty[group]);
        } else {
          uint32_t xv[32], yv[32];
          tmem_ld_32x32(x_addr, xv);
          tmem_ld_32x32(y_addr, yv);
          tmem_ld_wait_for(xv);
          tmem_ld_wait_for(yv);
          if (!OVERLAY) {
            // X / Y are in registers: hand the buffer back now so the next scores can be computed
            // into it while this block's math runs
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&xy_empty[group]);
          }
          // Masked tiles (the diagonal, the sequence tail) turn their dead scores into -inf in the
          // registers, which makes both P and dS exact zeros (dvec and dP are finite everywhere, the
          // padding rows of dvec are written as zeros), and then run the same code as every other tile.
          if (kind == 1) {
            const int hi = p.S - col0;                                   // first column past the sequence
            if (MODE == 0) {                                             // col = query, row = key
              const int lo = p.causal ? row_g - col0 : -0x7fffffff;      // queries before the key are dead
#pragma unroll
              for (int e = 0; e < 32; ++e) xv[e] = (e < lo || e >= hi) ? 0xff800000u : xv[e];
            } else {                                                     // col = key, row = query
              const int lim = min(p.causal ? row_g - col0 : 0x7fffffff, hi - 1);
#pragma unroll
              for (int e = 0; e < 32; ++e) xv[e] = (e > lim) ? 0xff800000u : xv[e];
            }
          }
          const float* st_lse = stats + st * 128 + half * 32;
          const float* st_dv = st_lse + 64;
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            uint64_t ls[2], dv[2];
            if (MODE == 0) {   // per-column statistics of the streamed query tile (same address in all lanes)
              const float4 l4 = *reinterpret_cast<const float4*>(st_lse + e);
              const float4 d4 = *reinterpret_cast<const float4*>(st_dv + e);
              ls[0] = pack_f32x2(l4.x, l4.y); ls[1] = pack_f32x2(l4.z, l4.w);
              dv[0] = pack_f32x2(d4.x, d4.y); dv[1] = pack_f32x2(d4.z, d4.w);
            } else {
              ls[0] = ls[1] = pack_f32x2(row_lse, row_lse);
              dv[0] = dv[1] = pack_f32x2(row_dvec, row_dvec);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              // P = 2^(x scale log2(e) - lse), dS = P (y - dvec), two columns per instruction. The first
              // sum is formed negated; the exponential turns the sign back.
              const float2 a = unpack_f32x2(fma_f32x2(pack_u32x2(xv[e + 2 * u], xv[e + 2 * u + 1]), neg_sl2, ls[u]));
              const float p0 = fast_exp2(-a.x), p1 = fast_exp2(-a.y);
              const uint64_t dy = fma_f32x2(dv[u], neg_one, pack_u32x2(yv[e + 2 * u], yv[e + 2 * u + 1]));
              const float2 d = unpack_f32x2(mul_f32x2(pack_f32x2(p0, p1), dy));
              if (MODE == 0) pp[(e >> 1) + u] = pack_bf16x2(p0, p1);
              dd[(e >> 1) + u] = pack_bf16x2(d.x, d.y);
            }
          }
        }
        // columns of this row -> 16 packed columns of the P / dS tensor-memory tiles
        if (!OVERLAY) {
          mbar_wait(&m_empty[group], par ^ 1u, wctx, STATUS_TIMEOUT_SOFTMAX);
          tc_fence_after();
        }
        if (MODE == 0) tmem_st_32x16(p_addr, pp);
        tmem_st_32x16(ds_addr, dd);
        if (acc_pending) {   // before the arrival that lets the next phase of acc_full complete
          mbar_wait(acc_full, (it - 1) & 1, wctx, STATUS_TIMEOUT_TMEM_FULL);
          acc_pending = false;
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&m_full[group]);
      }
      g0 += n_t;
      // Epilogue: accumulators -> global. dK / dV: one group of warps each, a half of the columns per warp.
      // dQ: a quarter of the columns per warp at head_dim 128; at head_dim 64 the group that does not own
      // the next item's first tile does it all and the other one goes on.
      if (EPI_WARPS != BWD_CW && group == (g0 & 1)) {
        acc_pending = true;
        continue;
      }
      constexpr int NC = (MODE == 0) ? D / 64 : 1;    // 32-column chunks per warp
      const int c0 = (MODE == 0) ? half * (D / 2) : (D == 128 ? group * 64 + half * 32 : half * 32);
      const bool is_dv = MODE == 0 && group == 1;
      const bool rope_on = !is_dv && p.rope_cos != nullptr && row_g < p.S;
      const float out_scale = is_dv ? 1.f : p.scale;
      const int row0 = rt * 128 + quarter * 32;
      const long long o_ss = is_dv ? p.o2_ss : p.o1_ss;
      __nv_bfloat16* out = is_dv ? p.out2 + row0 * p.o2_ss + b * p.o2_bs + h * p.o2_hs
                                 : p.out1 + row0 * p.o1_ss + b * p.o1_bs + h * p.o1_hs;
      const uint32_t acc = tmem_base + lane_base + (MODE == 0 && !is_dv ? ACC2 : ACC1);
      constexpr bool ROPE_STAGED = BwdShape<D, MODE>::ROPE_STAGED;
      if (ROPE_STAGED && p.rope_cos != nullptr && !is_dv) {
        // The rotary table's entries of the 32 rows come into shared memory as whole 64-byte segments while the
        // item's last gradient MMAs finish: read by their rows' threads they would be 256 passes through the
        // load / store unit after the wait.
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = (lane >> 2) + 8 * i, ch = lane & 3;
          if (row0 + row < p.S) {
            const size_t at = static_cast<size_t>(row0 + row) * (D / 2) + (c0 >> 1) + ch * 4;
            uint8_t* dst = stage + row * 64 + ((ch ^ ((row >> 1) & 3)) << 4);
            cp_async_16(dst, p.rope_cos + at);
            cp_async_16(dst + 2048, p.rope_sin + at);
          }
        }
      }
#pragma unroll
      for (int ci = 0; ci < NC; ++ci) {
        const int c = c0 + 32 * ci;
        if (ci == 0) {
          mbar_wait(acc_full, it & 1, wctx, STATUS_TIMEOUT_TMEM_FULL);
          tc_fence_after();
        }
        uint32_t v[32], wv[16];
        tmem_ld_32x32(acc + c, v);
        tmem_ld_wait_for(v);
        if (ci == NC - 1) {      // the accumulators may be overwritten by the next item
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_empty);
        }
        if (ROPE_STAGED) {
          cp_async_wait_all();
          __syncwarp();
        }
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          float f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(v[8 * q4 + e]) * out_scale;
          if (rope_on) {  // inverse rotation: sin -> -sin
            float4 cs, sn;
            if (ROPE_STAGED) {
              const uint8_t* src = stage + lane * 64 + ((q4 ^ ((lane >> 1) & 3)) << 4);
              cs = *reinterpret_cast<const float4*>(src);
              sn = *reinterpret_cast<const float4*>(src + 2048);
            } else {
              const size_t at = static_cast<size_t>(row_g) * (D / 2) + ((c + 8 * q4) >> 1);
              cs = *reinterpret_cast<const float4*>(p.rope_cos + at);
              sn = *reinterpret_cast<const float4*>(p.rope_sin + at);
            }
            const float a0 = f[0], a1 = f[1], a2 = f[2], a3 = f[3], a4 = f[4], a5 = f[5], a6 = f[6], a7 = f[7];
            f[0] = a0 * cs.x + a1 * sn.x; f[1] = a1 * cs.x - a0 * sn.x;
            f[2] = a2 * cs.y + a3 * sn.y; f[3] = a3 * cs.y - a2 * sn.y;
            f[4] = a4 * cs.z + a5 * sn.z; f[5] = a5 * cs.z - a4 * sn.z;
            f[6] = a6 * cs.w + a7 * sn.w; f[7] = a7 * cs.w - a6 * sn.w;
          }
          wv[4 * q4 + 0] = pack_out(f[0], f[1], p.out_f16);
          wv[4 * q4 + 1] = pack_out(f[2], f[3], p.out_f16);
          wv[4 * q4 + 2] = pack_out(f[4], f[5], p.out_f16);
          wv[4 * q4 + 3] = pack_out(f[6], f[7], p.out_f16);
        }
        if (ROPE_STAGED) __syncwarp();   // every row's entries have been read
        store_rows_32x32(stage, wv, lane, out + c, o_ss, p.S - row0);
      }
    }
  }

  if (MODE == 1) pdl_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

const CUtensorMap* make_map(const void* base, int D, int S, int nh, int B, const long long* st, uint32_t box_rows) {
  // st = {seq, batch, head} element strides
  uint64_t dims[4] = {static_cast<uint64_t>(D), static_cast<uint64_t>(S), static_cast<uint64_t>(nh),
                      static_cast<uint64_t>(B)};
  uint64_t strides[4] = {2, static_cast<uint64_t>(st[0]) * 2, static_cast<uint64_t>(st[2]) * 2,
                         static_cast<uint64_t>(st[1]) * 2};
  uint32_t box[4] = {64, box_rows, 1, 1};
  return gfs_host::tmap_nd_cached(base, 4, dims, strides, box);
}


bool strides_ok(const long long* st, int n) {
  for (int i = 0; i < n; ++i)
    if (st[i] & 7) return false;
  return true;
}

}  // namespace

extern "C" {

// fp16 q, k, v -> bf16 copies in dst (3 x [B, nh, S, D], contiguous). strides: 9 element strides
// {q_seq, q_batch, q_head, k_.., v_..}.
int gfs_attn_cast_qkv(const void* q, const void* k, const void* v, void* dst, int S, int B, int nh, int D,
                      const long long* strides, void* stream_) {
  if (D & 7) return -1;
  if (!strides_ok(strides, 9)) return -1;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(dst)) & 15)
    return -2;
  const long long n = static_cast<long long>(B) * nh * S * (D >> 3);
  if (n <= 0) return 0;
  CastArgs a;
  const void* src[3] = {q, k, v};
  for (int t = 0; t < 3; ++t) {
    a.src[t] = static_cast<const __half*>(src[t]);
    a.ss[t] = strides[3 * t]; a.bs[t] = strides[3 * t + 1]; a.hs[t] = strides[3 * t + 2];
  }
  const int blocks = static_cast<int>(std::min<long long>((n + 255) / 256, gfs_host::sm_count() * 16));
  cast_qkv_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream_)>>>(a, static_cast<__nv_bfloat16*>(dst), S, B, nh,
                                                                          D);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// strides: 12 element strides {q_seq,q_batch,q_head, k_.., v_.., o_..}. lse: fp32 [B, nh, S_pad] (base 2),
// S_pad = S rounded up to a multiple of 128. o_f16: store the output as fp16. o_copy: null, or where to store the
// output a second time, with the same strides (for a backward whose caller may write to the first copy).
int gfs_flash_fwd(const void* q, const void* k, const void* v, void* o, void* o_copy, void* lse, int S, int B, int nh,
                  int D, const long long* strides, float scale, int causal, int o_f16, void* stream_) {
  if (D != 64 && D != 128) return -1;
  if (!strides_ok(strides, 12)) return -1;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(o_copy)) & 15)
    return -2;
  if (S <= 0 || B <= 0 || nh <= 0) return 0;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const CUtensorMap* tq = make_map(q, D, S, nh, B, strides + 0, 128);
  const CUtensorMap* tk = make_map(k, D, S, nh, B, strides + 3, 128);
  const CUtensorMap* tv = make_map(v, D, S, nh, B, strides + 6, 128);
  if (!tq || !tk || !tv) return -3;
  FwdParams p;
  p.O = static_cast<__nv_bfloat16*>(o);
  p.o_copy = o_copy != nullptr ? (static_cast<char*>(o_copy) - static_cast<char*>(o)) / 2 : 0;
  p.o_ss = strides[9]; p.o_bs = strides[10]; p.o_hs = strides[11];
  p.lse = static_cast<float*>(lse);
  p.S = S; p.S_pad = ((S + 127) / 128) * 128; p.B = B; p.nh = nh;
  p.scale = scale; p.causal = causal; p.o_f16 = o_f16;
  p.status = gfs_host::status_words();
  const int nb = (S + 127) / 128;
  static gfs_host::SmemLimit limit64, limit128, limit128s;
  if (D == 64) {
    if (!limit64.raise(flash_fwd64_kernel, FWD64_SMEM)) return -10;
    const int n_pairs = (nb + 1) / 2;
    const int n_items = n_pairs * B * nh;
    const int ctas = std::min(n_items, gfs_host::sm_count());
    gfs_host::launch_pdl(flash_fwd64_kernel, dim3(ctas), dim3(FWD64_THREADS), FWD64_SMEM, stream, *tq, *tk, *tv, p,
                         n_pairs, n_items);
  } else {
    const int n_items = nb * B * nh;
    if (fwd128_few_items(nb, static_cast<long long>(B) * nh, causal != 0, gfs_host::sm_count())) {
      if (!limit128s.raise(flash_fwd128_small_kernel, FWD128S_SMEM)) return -10;
      gfs_host::launch_pdl(flash_fwd128_small_kernel, dim3(nb, B * nh), dim3(FWD128S_THREADS), FWD128S_SMEM, stream, *tq,
                           *tk, *tv, p);
      return cudaGetLastError() == cudaSuccess ? 0 : -11;
    }
    if (!limit128.raise(flash_fwd128_kernel, FWD128_SMEM)) return -10;
    const int ctas = std::min(n_items, gfs_host::sm_count());
    gfs_host::launch_pdl(flash_fwd128_kernel, dim3(ctas), dim3(FWD128_THREADS), FWD128_SMEM, stream, *tq, *tk, *tv, p, nb,
                         n_items);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// strides: 24 element strides for {q, k, v, o, do, dq, dk, dv} x {seq, batch, head}.
// lse (from the forward), dvec: fp32 [B, nh, S_pad]; dvec is scratch written by the pre-pass.
// rope_cos / rope_sin (optional, fp32 [>=S, D/2]): when given, dq and dk are rotated back
// (inverse rotary embedding) as they are written, i.e. they are gradients w.r.t. the
// un-rotated projections.
// do_bf16: null for bf16 tensors; otherwise o, dO, dq, dk and dv are fp16 (q, k, v stay bf16) and this is
// scratch for a contiguous bf16 [B, nh, S, D] copy of dO.
// dq shares no memory with anything that is read for dk and dv, nor with them: its kernel runs beside theirs.
int gfs_flash_bwd(const void* q, const void* k, const void* v, const void* o, const void* dO, const void* lse,
                  void* dvec, void* dq, void* dk, void* dv, int S, int B, int nh, int D, const long long* strides,
                  float scale, int causal, const void* rope_cos, const void* rope_sin, void* do_bf16, void* stream_) {
  if (D != 64 && D != 128) return -1;
  if (!strides_ok(strides, 24)) return -1;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(dO) | reinterpret_cast<uintptr_t>(dq) |
       reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv) | reinterpret_cast<uintptr_t>(do_bf16)) & 15)
    return -2;
  if (S <= 0 || B <= 0 || nh <= 0) return 0;
  if (static_cast<long long>(S) * B * nh > 0x3fffffffll) return -1;   // 32-bit row numbers in the pre-pass
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int S_pad = ((S + 127) / 128) * 128;
  const long long *sq = strides, *sk = strides + 3, *sv = strides + 6, *so = strides + 9, *sdo = strides + 12,
                  *sdq = strides + 15, *sdk = strides + 18, *sdv = strides + 21;
  long long sdo16[3];
  {
    const long long rows = static_cast<long long>(S) * B * nh;
    const int threads = 256;
    const int rows_per_block = threads / (D >> 3) * DVEC_ROWS;
    const dim3 grid(static_cast<unsigned>((rows + rows_per_block - 1) / rows_per_block));
    const int s_fastest = so[0] < so[2] ? 1 : 0;
    auto kern = do_bf16 != nullptr ? attn_dvec_kernel<true> : attn_dvec_kernel<false>;
    gfs_host::launch_pdl(kern, grid, dim3(threads), 0, stream, dO, o, static_cast<float*>(dvec),
                         static_cast<__nv_bfloat16*>(do_bf16), S, S_pad, B, nh, D, sdo[0], sdo[1], sdo[2], so[0], so[1],
                         so[2], s_fastest);
    if (cudaGetLastError() != cudaSuccess) return -11;
    if (do_bf16 != nullptr) {
      dO = do_bf16;
      sdo16[0] = D;
      sdo16[2] = static_cast<long long>(S) * D;
      sdo16[1] = nh * sdo16[2];
      sdo = sdo16;
    }
  }
  const CUtensorMap* q128 = make_map(q, D, S, nh, B, sq, 128);
  const CUtensorMap* k128 = make_map(k, D, S, nh, B, sk, 128);
  const CUtensorMap* v128 = make_map(v, D, S, nh, B, sv, 128);
  const CUtensorMap* do128 = make_map(dO, D, S, nh, B, sdo, 128);
  const CUtensorMap* q64 = make_map(q, D, S, nh, B, sq, 64);
  const CUtensorMap* k64 = make_map(k, D, S, nh, B, sk, 64);
  const CUtensorMap* v64 = make_map(v, D, S, nh, B, sv, 64);
  const CUtensorMap* do64 = make_map(dO, D, S, nh, B, sdo, 64);
  if (!q128 || !k128 || !v128 || !do128 || !q64 || !k64 || !v64 || !do64) return -3;
  BwdParams p;
  p.lse = static_cast<const float*>(lse);
  p.out_f16 = do_bf16 != nullptr ? 1 : 0;
  p.dvec = static_cast<const float*>(dvec);
  p.S = S; p.S_pad = S_pad; p.B = B; p.nh = nh; p.scale = scale; p.causal = causal;
  p.status = gfs_host::status_words();
  p.rope_cos = static_cast<const float*>(rope_cos);
  p.rope_sin = static_cast<const float*>(rope_sin);
  const int n_rt = (S + 127) / 128;
  const int n_items = n_rt * B * nh;
  const int ctas = std::min(n_items, gfs_host::sm_count());
  static gfs_host::SmemLimit limits[4];
  // mode 0: dK, dV
  BwdParams p0 = p;
  p0.out1 = static_cast<__nv_bfloat16*>(dk); p0.o1_ss = sdk[0]; p0.o1_bs = sdk[1]; p0.o1_hs = sdk[2];
  p0.out2 = static_cast<__nv_bfloat16*>(dv); p0.o2_ss = sdv[0]; p0.o2_bs = sdv[1]; p0.o2_hs = sdv[2];
  BwdParams p1 = p;
  p1.out1 = static_cast<__nv_bfloat16*>(dq); p1.o1_ss = sdq[0]; p1.o1_bs = sdq[1]; p1.o1_hs = sdq[2];
  p1.out2 = nullptr; p1.o2_ss = p1.o2_bs = p1.o2_hs = 0;
  if (D == 64) {
    constexpr int smem0 = BwdShape<64, 0>::SMEM;
    if (!limits[0].raise(flash_bwd_kernel<64, 0>, smem0)) return -10;
    gfs_host::launch_pdl(flash_bwd_kernel<64, 0>, dim3(ctas), dim3(BWD_THREADS), smem0, stream, *k128, *v128,
                         *q64, *do64, p0, n_rt, n_items);
    if (cudaGetLastError() != cudaSuccess) return -12;
    constexpr int smem1 = BwdShape<64, 1>::SMEM;
    if (!limits[1].raise(flash_bwd_kernel<64, 1>, smem1)) return -10;
    gfs_host::launch_pdl(flash_bwd_kernel<64, 1>, dim3(ctas), dim3(BWD_THREADS), smem1, stream, *q128, *do128,
                         *k64, *v64, p1, n_rt, n_items);
  } else {
    constexpr int smem0 = BwdShape<128, 0>::SMEM;
    if (!limits[2].raise(flash_bwd_kernel<128, 0>, smem0)) return -10;
    gfs_host::launch_pdl(flash_bwd_kernel<128, 0>, dim3(ctas), dim3(BWD_THREADS), smem0, stream, *k128, *v128,
                         *q64, *do64, p0, n_rt, n_items);
    if (cudaGetLastError() != cudaSuccess) return -12;
    constexpr int smem1 = BwdShape<128, 1>::SMEM;
    if (!limits[3].raise(flash_bwd_kernel<128, 1>, smem1)) return -10;
    gfs_host::launch_pdl(flash_bwd_kernel<128, 1>, dim3(ctas), dim3(BWD_THREADS), smem1, stream, *q128, *do128,
                         *k64, *v64, p1, n_rt, n_items);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -13;
}

}  // extern "C"
