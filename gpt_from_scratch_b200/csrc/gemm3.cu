// bf16 GEMM for problems that do not fill the chip with the persistent kernels' tiles (gemm.cu: 128 x 256,
// gemm2.cu: 256 x 256 per CTA pair): one 128 x BN output tile (BN = 64 or 128) per CTA, and a cluster of
// up to eight CTAs may share a tile by splitting K, reducing through distributed shared memory. A second kernel
// does the same with 256 x 256 tiles on CTA pairs.
//
// What bounds such a problem is the chain launch -> first TMA -> K loop -> epilogue of one CTA, not a
// unit of the chip. A 512 x 768 x 256 product is 12 tiles of 128 x 256 on 148 SMs and took 11 us; a
// 130 x 768 x 3072 one took 20 us (2 x 3 tiles, split along K through a workspace and a second
// launch). Narrow tiles shorten the epilogue (64 instead of 256 columns per row) and put more SMs to work, and
// the split inside the cluster shortens the K loop without the second launch.
//
// Roles (6 warps): warp 0 TMA producer, warp 1 MMA issuer, warps 2-5 move the accumulator from tensor
// memory to the fp32 staging tile; then all warps apply the epilogue to vectors of eight columns read
// from staging, so global accesses are coalesced and every thread has epilogue work.
//
// Split K over a cluster of s CTAs: CTA r of the cluster owns rows [r * 128/s, +128/s) of the tile. Every
// CTA writes the rows of its partial tile into their owners' staging areas (st.shared::cluster), one
// cluster barrier, and the owner sums the s partials in rank order (deterministic) in its epilogue. The staging
// area is s x (128/s) rows whatever s is. (Bulk copies out of the dead operand ring, counted on a barrier of the owner's,
// instead of the threads' scattered stores: 6.0 against 5.3 us at 130 x 768 x 768, split 4.)
//
// A kernel of a few microseconds executes its code once, so what counts in the epilogue is how much of it there is: every
// kind (EPI_*) is a variant of its own, and vectors past the end skip theirs. One epilogue for all kinds, six
// vectors unrolled, took 3,700 of the 12,500 cycles of an unsplit 512 x 256 x 256 product for the 5 vectors of a thread.
// us in a chain of products, that -> this: 512 x 256 x 256 5.5 -> 4.1, 130 x 768 x 768 unsplit 7.2 -> 5.8. What
// an epilogue reads (addend, rotation table, gate and up) is fetched six vectors at a time, the first six before the
// accumulator is ready; read where it is used, each vector waited for memory: 1040 x 768 x 768 with the SwiGLU gradient
// 9.0 -> 7.1, with the rotation 8.2 -> 7.2.
//
// Operand layouts, addend, rotary and SwiGLU epilogues as in gemm.cu; values are rounded once, from fp32.
#include <algorithm>
#include <climits>

#include "api.h"
#include "common.cuh"

using namespace gfs;

namespace {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int THREADS = 192;
constexpr int MAX_GROUP = 4;
// Epilogues: (+ addend) / SwiGLU forward / SwiGLU backward / rotary embedding (+ addend)
enum Epi : int { EPI_PLAIN = 0, EPI_SWIGLU = 1, EPI_SWIGLU_BWD = 2, EPI_ROPE = 3 };

struct TileProblem {
  int M, N;
  int kblocks, per_split;   // K blocks in all, and per CTA of the cluster
  int tiles_n, tile_begin;
  int ldc, ldr;
  __nv_bfloat16* C;
  const __nv_bfloat16* R;   // addend (may alias C) or null
};

template <int NG>
struct TileMaps {
  CUtensorMap a[NG], b[NG];
};

template <int NG>
struct TileParams {
  TileProblem g[NG];
  int ngroups, split;
  int early_b, late_wait;   // gfs_host::LaunchHints
  uint32_t* status;
  const float* rope_cos;    // rotary embedding of the first rope_cols columns (see gemm.cu)
  const float* rope_sin;
  int rope_cols, rope_d, rope_b;
  int swi_I, swi_ld;             // SwiGLU, as in gemm.cu
  __nv_bfloat16* swi_act;
  const __nv_bfloat16* swi_gu;
};

template <int BN>
struct Cfg {
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = BN == 64 ? 7 : 4;
  static constexpr int PITCH = BN + 4;
  static constexpr int STAGING = (BM + 1) * PITCH * 4;   // split 3: 3 x 43 rows
  static constexpr int TOTAL = STAGES * STAGE_BYTES + STAGING + 256 + 1024;
};

__device__ __forceinline__ void cluster_sync() {
  __syncwarp();   // the aligned barrier wants whole warps
  cluster_sync_all();
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d)
               : "memory");
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
}

// The epilogue of one CTA, called by all its threads: rows [rank * rows_per_cta, ...) of the tile at (m0, n0)
// are the sums of `split` fp32 slabs in `staging`. `sync` makes the slabs visible; the addends of the first
// vectors are fetched before it, while the K loop still runs.
template <int BN, int NT, int EPI, int NG, typename Sync>
__device__ __forceinline__ void tile_epilogue(const TileParams<NG>& p, const TileProblem& g, const float* staging,
                                              int split, int rank, int m0, int n0, Sync sync) {
  constexpr int PITCH = BN + 4;   // floats per staging row: 16-byte chunks of consecutive rows hit different banks
  const int rows_per_cta = (BM + split - 1) / split;
  const int rows_here = min(BM, (rank + 1) * rows_per_cta) - rank * rows_per_cta;
  const int row_base = m0 + rank * rows_per_cta;
  if constexpr (EPI == EPI_SWIGLU) {
    constexpr int VPR = BN / 16;   // vectors of gate columns per row
    sync();
#pragma unroll 1
    for (int v = threadIdx.x; v < rows_here * VPR; v += NT) {
      const int lr = v / VPR, c = (v % VPR) * 8;
      const int row = row_base + lr, col = (n0 >> 1) + c;
      if (row >= g.M || col + 8 > p.swi_I) continue;
      float gt[8] = {0, 0, 0, 0, 0, 0, 0, 0}, up[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 1
      for (int r = 0; r < split; ++r) {
        const float* src = staging + (r * rows_per_cta + lr) * PITCH + c;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          gt[e] += src[e];
          up[e] += src[BN / 2 + e];
        }
      }
      const uint4 wg = pack8(gt), wu = pack8(up);
      unpack8(wg, gt);   // act from the bf16-rounded projections, silu rounded to bf16 before the product
      unpack8(wu, up);
      float a[8];
#pragma unroll
      for (int e = 0; e < 8; ++e)
        a[e] = __bfloat162float(__float2bfloat16_rn(gt[e] * sigmoid_f(gt[e]))) * up[e];
      __nv_bfloat16* dst = g.C + static_cast<size_t>(row) * g.ldc + col;
      *reinterpret_cast<uint4*>(dst) = wg;
      *reinterpret_cast<uint4*>(dst + p.swi_I) = wu;
      *reinterpret_cast<uint4*>(p.swi_act + static_cast<size_t>(row) * p.swi_ld + col) = pack8(a);
    }
  } else {
    constexpr int VPR = BN / 8;
    constexpr int NPRE = 6;        // vectors of a thread whose operands are fetched together, the first before the wait
    constexpr bool TABLE = EPI == EPI_SWIGLU_BWD || EPI == EPI_ROPE;
    uint4 pre[NPRE], aux[TABLE ? NPRE : 1], aux2[TABLE ? NPRE : 1];   // addend; gate and up, or cos and sin
    const bool has_add = EPI != EPI_SWIGLU_BWD && g.R != nullptr;
    static_assert(NT % VPR == 0, "a thread's vectors lie in the same columns");
    const int c = (threadIdx.x % VPR) * 8, col = n0 + c;
    const int rope_col = EPI == EPI_ROPE ? (col % p.rope_d) >> 1 : 0;
    auto fetch = [&](int v0) {
#pragma unroll
      for (int i = 0; i < NPRE; ++i) {
        const int lr = v0 / VPR + i * (NT / VPR), row = row_base + lr;
        if (lr >= rows_here || row >= g.M || col + 8 > g.N) continue;
        if (has_add) pre[i] = *reinterpret_cast<const uint4*>(g.R + static_cast<size_t>(row) * g.ldr + col);
        if constexpr (EPI == EPI_SWIGLU_BWD) {
          const __nv_bfloat16* gp = p.swi_gu + static_cast<size_t>(row) * p.swi_ld + col;
          aux[i] = *reinterpret_cast<const uint4*>(gp);
          aux2[i] = *reinterpret_cast<const uint4*>(gp + p.swi_I);
        }
        if (EPI == EPI_ROPE && col < p.rope_cols) {
          const size_t ti = static_cast<size_t>(row / p.rope_b) * (p.rope_d >> 1) + rope_col;
          aux[i] = *reinterpret_cast<const uint4*>(p.rope_cos + ti);
          aux2[i] = *reinterpret_cast<const uint4*>(p.rope_sin + ti);
        }
      }
    };
    const bool fetches = TABLE || has_add;
    if (fetches) fetch(threadIdx.x);
    sync();
    auto finish = [&](int v, const uint4& addend, const uint4& t0, const uint4& t1) {
      const int lr = v / VPR, row = row_base + lr;
      if (lr >= rows_here || row >= g.M || col + 8 > g.N) return;
      float f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 1
      for (int r = 0; r < split; ++r) {
        const float4* src = reinterpret_cast<const float4*>(staging + (r * rows_per_cta + lr) * PITCH + c);
        const float4 a = src[0], b = src[1];
        f[0] += a.x; f[1] += a.y; f[2] += a.z; f[3] += a.w;
        f[4] += b.x; f[5] += b.y; f[6] += b.z; f[7] += b.w;
      }
      if constexpr (EPI == EPI_SWIGLU_BWD) {
        // f holds d_act; turn it into d_gate and d_up
        float gt[8], up[8], dg[8], du[8];
        unpack8(t0, gt);
        unpack8(t1, up);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float sg = sigmoid_f(gt[e]);
          dg[e] = f[e] * up[e] * sg * (1.f + gt[e] * (1.f - sg));
          du[e] = f[e] * gt[e] * sg;
        }
        __nv_bfloat16* dst = g.C + static_cast<size_t>(row) * g.ldc + col;
        *reinterpret_cast<uint4*>(dst) = pack8(dg);
        *reinterpret_cast<uint4*>(dst + p.swi_I) = pack8(du);
        return;
      }
      if (EPI == EPI_ROPE && col < p.rope_cols) {
        const float4 cs = make_float4(__uint_as_float(t0.x), __uint_as_float(t0.y), __uint_as_float(t0.z), __uint_as_float(t0.w));
        const float4 sn = make_float4(__uint_as_float(t1.x), __uint_as_float(t1.y), __uint_as_float(t1.z), __uint_as_float(t1.w));
        const float a0 = f[0], a1 = f[1], a2 = f[2], a3 = f[3], a4 = f[4], a5 = f[5], a6 = f[6], a7 = f[7];
        f[0] = a0 * cs.x - a1 * sn.x; f[1] = a0 * sn.x + a1 * cs.x;
        f[2] = a2 * cs.y - a3 * sn.y; f[3] = a2 * sn.y + a3 * cs.y;
        f[4] = a4 * cs.z - a5 * sn.z; f[5] = a4 * sn.z + a5 * cs.z;
        f[6] = a6 * cs.w - a7 * sn.w; f[7] = a6 * sn.w + a7 * cs.w;
      }
      if (has_add) {
        float r8[8];
        unpack8(addend, r8);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] += r8[e];
      }
      *reinterpret_cast<uint4*>(g.C + static_cast<size_t>(row) * g.ldc + col) = pack8(f);
    };
    const int n_vec = rows_here * VPR;
    int v = threadIdx.x;
    if (!fetches) {
      const uint4 none = make_uint4(0, 0, 0, 0);
#pragma unroll 1
      for (; v < n_vec; v += NT) finish(v, none, none, none);
      return;
    }
#pragma unroll 1
    while (true) {
#pragma unroll
      for (int i = 0; i < NPRE; ++i, v += NT) {
        if (v >= n_vec) return;
        finish(v, pre[i], aux[TABLE ? i : 0], aux2[TABLE ? i : 0]);
      }
      if (v >= n_vec) return;
      fetch(v);
    }
  }
}

// One accumulator row (this lane's) from tensor memory to the staging area of the CTA that owns it. `owner`:
// cluster rank of that CTA; `slab`: which of its slabs; columns [c0, c1).
template <int PITCH>
__device__ __forceinline__ void stage_row(uint32_t t_row, float* staging, int slab, int rows_per_cta, int row_in_owner,
                                          bool remote, uint32_t owner, int c0, int c1) {
  float* local = staging + (slab * rows_per_cta + row_in_owner) * PITCH;
  uint32_t dst = smem_u32(local);
  if (remote) dst = mapa_u32(dst, owner);
  uint32_t va[32], vb[32];
#pragma unroll 1
  for (int c = c0; c < c1; c += 64) {
    tmem_ld_32x32(t_row + c, va);
    tmem_ld_32x32(t_row + c + 32, vb);
    tmem_ld_wait_for(va);
    tmem_ld_wait_for(vb);
    if (remote) {
#pragma unroll
      for (int j = 0; j < 8; ++j) st_cluster_v4(dst + (c + 4 * j) * 4, va[4 * j], va[4 * j + 1], va[4 * j + 2], va[4 * j + 3]);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        st_cluster_v4(dst + (c + 32 + 4 * j) * 4, vb[4 * j], vb[4 * j + 1], vb[4 * j + 2], vb[4 * j + 3]);
    } else {
      uint4* out = reinterpret_cast<uint4*>(local + c);
#pragma unroll
      for (int j = 0; j < 8; ++j) out[j] = make_uint4(va[4 * j], va[4 * j + 1], va[4 * j + 2], va[4 * j + 3]);
#pragma unroll
      for (int j = 0; j < 8; ++j) out[8 + j] = make_uint4(vb[4 * j], vb[4 * j + 1], vb[4 * j + 2], vb[4 * j + 3]);
    }
  }
}

template <bool A_MN, bool B_MN, int BN, int NG, int EPI>
__global__ void __launch_bounds__(THREADS, 1)
gemm_tile_kernel(const __grid_constant__ TileMaps<NG> maps, const __grid_constant__ TileParams<NG> p) {
  using C_ = Cfg<BN>;
  constexpr int STAGES = C_::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* tiles = smem;
  float* staging = reinterpret_cast<float*>(smem + STAGES * C_::STAGE_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * C_::STAGE_BYTES + C_::STAGING);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + STAGES;
  uint64_t* tmem_full = bars + 2 * STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 1);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int split = p.split;
  const int rank = split > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int tile = static_cast<int>(blockIdx.x) / split;
  int gi = 0;
  if (NG > 1) {
#pragma unroll
    for (int i = 1; i < NG; ++i)
      if (i < p.ngroups && tile >= p.g[i].tile_begin) gi = i;
  }
  const TileProblem& g = p.g[gi];
  const int lt = tile - g.tile_begin;
  const int m0 = (lt / g.tiles_n) * BM;
  const int n0 = (lt % g.tiles_n) * BN;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(tmem_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&maps.a[gi]);
    tma_prefetch_desc(&maps.b[gi]);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  tc_fence_before();
  if (split > 1) cluster_sync();   // also: every CTA of the cluster runs before its shared memory is written
  else __syncthreads();
  tc_fence_after();
  // Set-up above may overlap the tail of the preceding kernel (programmatic launch). With early_b the TMA warp waits after
  // its first loads of B, with late_wait everybody at the end.
  const bool early_b = p.early_b != 0 && p.late_wait == 0;
  if (p.late_wait == 0 && !(early_b && warp == 0)) pdl_wait();
  if (!(early_b && warp == 0)) pdl_trigger();
  const uint32_t tmem_base = *tmem_slot;
  WaitCtx wctx{abort_flag, p.status, GFS_WAIT_LIMIT_NS};
  const int kb0 = rank * g.per_split;
  const int kb1 = min(g.kblocks, kb0 + g.per_split);

  if (warp == 0) {
    if (lane == 0) {
      auto load_b = [&](int stage, int k0) {
        uint8_t* sb = tiles + stage * C_::STAGE_BYTES + C_::A_BYTES;
        if (!B_MN) {
          if (EPI == EPI_SWIGLU) {   // BN/2 gate rows + the matching up rows (tensor map box = BN/2 rows)
            tma_load_2d(sb, &maps.b[gi], &full_bar[stage], k0, n0 >> 1);
            tma_load_2d(sb + (BN / 2) * 128, &maps.b[gi], &full_bar[stage], k0, p.swi_I + (n0 >> 1));
          } else {
            tma_load_2d(sb, &maps.b[gi], &full_bar[stage], k0, n0);
          }
        } else {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j) tma_load_2d(sb + j * 8192, &maps.b[gi], &full_bar[stage], n0 + 64 * j, k0);
        }
      };
      auto load_a = [&](int stage, int k0) {
        uint8_t* sa = tiles + stage * C_::STAGE_BYTES;
        if (!A_MN) {
          tma_load_2d(sa, &maps.a[gi], &full_bar[stage], k0, m0);
        } else {
#pragma unroll
          for (int j = 0; j < BM / 64; ++j) tma_load_2d(sa + j * 8192, &maps.a[gi], &full_bar[stage], m0 + 64 * j, k0);
        }
      };
      int i = 0;
      if (early_b) {
        const int n = min(STAGES, kb1 - kb0);
        for (int e = 0; e < n; ++e) {
          mbar_arrive_expect_tx(&full_bar[e], C_::STAGE_BYTES);
          load_b(e, (kb0 + e) * BK);
        }
        pdl_wait();
        pdl_trigger();
        for (; i < n; ++i) load_a(i, (kb0 + i) * BK);
      }
      for (; i < kb1 - kb0; ++i) {
        const int stage = i % STAGES, k0 = (kb0 + i) * BK;
        mbar_wait(&empty_bar[stage], ((i / STAGES) & 1) ^ 1u, wctx, STATUS_TIMEOUT_PIPE_EMPTY);
        mbar_arrive_expect_tx(&full_bar[stage], C_::STAGE_BYTES);
        load_a(stage, k0);
        load_b(stage, k0);
      }
      settle_copies(wctx);
    }
    __syncwarp();
  } else if (warp == 1) {   // whole warp, converged: the MMA / commit helpers elect the issuing lane
    constexpr uint32_t idesc = umma_idesc_bf16(BM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
    for (int kb = kb0; kb < kb1; ++kb) {
      const int i = kb - kb0, stage = i % STAGES;
      mbar_wait(&full_bar[stage], (i / STAGES) & 1, wctx, STATUS_TIMEOUT_PIPE_FULL);
      tc_fence_after();
      const uint32_t sa = smem_u32(tiles + stage * C_::STAGE_BYTES);
      const uint32_t sb = sa + C_::A_BYTES;
#pragma unroll
      for (int k = 0; k < BK / 16; ++k) {
        const uint64_t adesc = A_MN ? umma_desc_sw128(sa + k * 2048, 8192, 1024) : umma_desc_sw128(sa + k * 32, 16, 1024);
        const uint64_t bdesc = B_MN ? umma_desc_sw128(sb + k * 2048, 8192, 1024) : umma_desc_sw128(sb + k * 32, 16, 1024);
        umma_ss_e(tmem_base, adesc, bdesc, idesc, (i > 0 || k > 0) ? 1u : 0u);
      }
      umma_commit_e(&empty_bar[stage]);
    }
    umma_commit_e(tmem_full);
  } else {
    const int row = (warp & 3) * 32 + lane;
    const int rows_per_cta = (BM + split - 1) / split;
    const int owner = row / rows_per_cta;
    mbar_wait(tmem_full, 0, wctx, STATUS_TIMEOUT_TMEM_FULL);
    tc_fence_after();
    stage_row<C_::PITCH>(tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16), staging, rank, rows_per_cta,
                         row - owner * rows_per_cta, split > 1, static_cast<uint32_t>(owner), 0, BN);
    tc_fence_before();
  }

  tile_epilogue<BN, THREADS, EPI>(p, g, staging, split, rank, m0, n0, [&]() {
    if (split > 1) cluster_sync();
    else __syncthreads();
  });

  if (p.late_wait) pdl_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, BN);
}

// ---------------------------------------------------------------------------
// The same on CTA pairs: a 256 x 256 tile per pair (cta_group::2, operands as in gemm2.cu), `split` pairs per
// tile along K in one cluster. For products whose 256 x 256 tiles leave most pairs idle but whose K loop is
// long enough to be bound by operand traffic: sharing B across the pair needs 128 bytes of shared memory per
// clock, a single CTA's 128 x 128 tile 256 (2048 x 768 x 2304: 24 tiles, 21 us on single CTAs with split
// K through a workspace). The staging area lies over the operand ring, which is dead once
// every CTA of the cluster has finished its products (one more cluster barrier when K is split).
// ---------------------------------------------------------------------------
constexpr int PAIR_STAGES = 6;
constexpr int PAIR_STAGE_BYTES = 32768;
constexpr int PAIR_THREADS = 320;   // TMA, MMA, eight warps that drain the accumulator
constexpr int PAIR_TOTAL = PAIR_STAGES * PAIR_STAGE_BYTES + 256 + 1024;
static_assert((BM + 1) * 260 * 4 <= PAIR_STAGES * PAIR_STAGE_BYTES, "staging fits the ring");

template <bool A_MN, bool B_MN, int NG, int EPI>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
gemm_pair_tile_kernel(const __grid_constant__ TileMaps<NG> maps, const __grid_constant__ TileParams<NG> p) {
  constexpr int BN = 256, BNH = 128, PITCH = BN + 4;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* tiles = smem;
  float* staging = reinterpret_cast<float*>(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + PAIR_STAGES * PAIR_STAGE_BYTES);
  uint64_t* full_bar = bars;                    // (used in the pair's leader)
  uint64_t* empty_bar = bars + PAIR_STAGES;     // (one per CTA)
  uint64_t* tmem_full = bars + 2 * PAIR_STAGES; // (one per CTA)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * PAIR_STAGES + 1);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int split = p.split;
  const uint32_t crank = cluster_ctarank();
  const int half = static_cast<int>(crank & 1u);     // rows / columns half of this CTA in its pair
  const int z = static_cast<int>(crank >> 1);        // K slice of the pair
  const uint32_t lead = crank & ~1u;
  const bool leader = half == 0;
  const int tile = static_cast<int>(blockIdx.x) / (2 * split);
  int gi = 0;
  if (NG > 1) {
#pragma unroll
    for (int i = 1; i < NG; ++i)
      if (i < p.ngroups && tile >= p.g[i].tile_begin) gi = i;
  }
  const TileProblem& g = p.g[gi];
  const int lt = tile - g.tile_begin;
  const int m0 = (lt / g.tiles_n) * 256 + half * BM;   // this CTA's rows
  const int n0 = (lt % g.tiles_n) * BN;

  if (threadIdx.x == 0) {
    for (int s = 0; s < PAIR_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(tmem_full, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&maps.a[gi]);
    tma_prefetch_desc(&maps.b[gi]);
  }
  __syncthreads();
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, BN);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  cluster_sync();   // barriers of all CTAs initialised, TMEM allocated
  tc_fence_after();
  const bool early_b = p.early_b != 0 && p.late_wait == 0;   // as above
  if (p.late_wait == 0 && !(early_b && warp == 0)) pdl_wait();
  if (!(early_b && warp == 0)) pdl_trigger();
  const uint32_t tmem_base = *tmem_slot;
  WaitCtx wctx{abort_flag, p.status, GFS_WAIT_LIMIT_NS};
  const int kb0 = z * g.per_split;
  const int kb1 = min(g.kblocks, kb0 + g.per_split);

  if (warp == 0) {
    if (lane == 0) {
      const int nb = n0 + half * BNH;
      auto begin = [&](int stage) {      // the leader's barrier counts the bytes of both CTAs
        if (leader) mbar_arrive_expect_tx(&full_bar[stage], 2 * PAIR_STAGE_BYTES);
      };
      auto load_b = [&](int stage, int k0) {
        uint8_t* sb = tiles + stage * PAIR_STAGE_BYTES + 16384;
        const uint32_t bar = mapa_u32(smem_u32(&full_bar[stage]), lead);
        if (!B_MN) {
          // SwiGLU forward: 128 gate rows for the leader, the matching up rows for the other CTA
          tma_load_2d_pair(sb, &maps.b[gi], bar, k0, EPI == EPI_SWIGLU ? half * p.swi_I + (n0 >> 1) : nb);
        } else {
#pragma unroll
          for (int j = 0; j < 2; ++j) tma_load_2d_pair(sb + j * 8192, &maps.b[gi], bar, nb + 64 * j, k0);
        }
      };
      auto load_a = [&](int stage, int k0) {
        uint8_t* sa = tiles + stage * PAIR_STAGE_BYTES;
        const uint32_t bar = mapa_u32(smem_u32(&full_bar[stage]), lead);
        if (!A_MN) {
          tma_load_2d_pair(sa, &maps.a[gi], bar, k0, m0);
        } else {
#pragma unroll
          for (int j = 0; j < 2; ++j) tma_load_2d_pair(sa + j * 8192, &maps.a[gi], bar, m0 + 64 * j, k0);
        }
      };
      int i = 0;
      if (early_b) {
        const int n = min(PAIR_STAGES, kb1 - kb0);
        for (int e = 0; e < n; ++e) {
          begin(e);
          load_b(e, (kb0 + e) * BK);
        }
        pdl_wait();
        pdl_trigger();
        for (; i < n; ++i) load_a(i, (kb0 + i) * BK);
      }
      for (; i < kb1 - kb0; ++i) {
        const int stage = i % PAIR_STAGES, k0 = (kb0 + i) * BK;
        mbar_wait(&empty_bar[stage], ((i / PAIR_STAGES) & 1) ^ 1u, wctx, STATUS_TIMEOUT_PIPE_EMPTY);
        begin(stage);
        load_a(stage, k0);
        load_b(stage, k0);
      }
      settle_copies(wctx);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (leader) {
      constexpr uint32_t idesc = umma_idesc_bf16(256, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
      for (int kb = kb0; kb < kb1; ++kb) {
        const int i = kb - kb0, stage = i % PAIR_STAGES;
        mbar_wait(&full_bar[stage], (i / PAIR_STAGES) & 1, wctx, STATUS_TIMEOUT_PIPE_FULL);
        tc_fence_after();
        const uint32_t sa = smem_u32(tiles + stage * PAIR_STAGE_BYTES);
        const uint32_t sb = sa + 16384;
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {
          const uint64_t adesc = A_MN ? umma_desc_sw128(sa + k * 2048, 8192, 1024) : umma_desc_sw128(sa + k * 32, 16, 1024);
          const uint64_t bdesc = B_MN ? umma_desc_sw128(sb + k * 2048, 8192, 1024) : umma_desc_sw128(sb + k * 32, 16, 1024);
          umma_ss_pair(tmem_base, adesc, bdesc, idesc, (i > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit_pair(mapa_u32(smem_u32(&empty_bar[stage]), lead));
        umma_commit_pair(mapa_u32(smem_u32(&empty_bar[stage]), lead | 1u));
      }
      umma_commit_pair(mapa_u32(smem_u32(tmem_full), lead));
      umma_commit_pair(mapa_u32(smem_u32(tmem_full), lead | 1u));
    }
  }
  // every product of this pair is done (both halves of the ring have been read)
  if (warp >= 2) {
    mbar_wait(tmem_full, 0, wctx, STATUS_TIMEOUT_TMEM_FULL);
    tc_fence_after();
  }
  if (split > 1) cluster_sync();   // ... and of every other pair whose ring is about to be written
  if (warp >= 2) {
    const int row = (warp & 3) * 32 + lane;
    const int rows_per_cta = (BM + split - 1) / split;
    const int owner = row / rows_per_cta;
    const int c0 = ((warp - 2) >> 2) * BNH;
    stage_row<PITCH>(tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16), staging, z, rows_per_cta,
                     row - owner * rows_per_cta, split > 1, static_cast<uint32_t>(2 * owner + half), c0, c0 + BNH);
    tc_fence_before();
  }
  tile_epilogue<BN, PAIR_THREADS, EPI>(p, g, staging, split, z, m0, n0, [&]() {
    if (split > 1) cluster_sync();
    else __syncthreads();
  });

  if (p.late_wait) pdl_wait();
  // nobody leaves while the partner may still touch this CTA's shared memory / barriers
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  if (warp == 1) tmem_dealloc_pair(tmem_base, BN);
}

// Launch with `cluster` CTAs per cluster (and programmatic stream serialization).
template <typename Kern, typename Maps, typename Params>
int launch_clustered(Kern kern, int threads, int smem, int cluster, const Maps& maps, const Params& p, int ctas,
                     cudaStream_t stream, gfs_host::SmemLimit& limit) {
  if (!limit.raise(kern, smem)) return -10;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = gfs_host::pdl_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, maps, p);
  gfs_host::launch_hints().late_wait = false;
  return e == cudaSuccess ? 0 : -11;
}

template <bool A_MN, bool B_MN, int NG, int EPI>
int launch_tile(int bn, const TileMaps<NG>& maps, const TileParams<NG>& p, int ctas, cudaStream_t stream) {
  static gfs_host::SmemLimit limit64, limit128, limit256;
  if (bn == 64)
    return launch_clustered(gemm_tile_kernel<A_MN, B_MN, 64, NG, EPI>, THREADS, Cfg<64>::TOTAL, p.split, maps, p, ctas,
                            stream, limit64);
  if (bn == 128)
    return launch_clustered(gemm_tile_kernel<A_MN, B_MN, 128, NG, EPI>, THREADS, Cfg<128>::TOTAL, p.split, maps, p, ctas,
                            stream, limit128);
  return launch_clustered(gemm_pair_tile_kernel<A_MN, B_MN, NG, EPI>, PAIR_THREADS, PAIR_TOTAL, 2 * p.split, maps, p,
                          2 * ctas, stream, limit256);
}

template <int EPI>
int launch_layout(int a_mn, int b_mn, int bn, const TileMaps<1>& maps, const TileParams<1>& p, int ctas,
                  cudaStream_t stream) {
  if (!a_mn) return b_mn ? launch_tile<false, true, 1, EPI>(bn, maps, p, ctas, stream)
                         : launch_tile<false, false, 1, EPI>(bn, maps, p, ctas, stream);
  return b_mn ? launch_tile<true, true, 1, EPI>(bn, maps, p, ctas, stream)
              : launch_tile<true, false, 1, EPI>(bn, maps, p, ctas, stream);
}

// Splits 5 to 7 round the rows of a CTA up so far that `split` slabs of them exceed the staging area's 129 rows.
int bad_shape(int bn, int split) {
  if (bn != 64 && bn != 128 && bn != 256) return 1;
  return split < 1 || split > (bn == 256 ? 4 : 8) || (BM + split - 1) / split * split > BM + 1;
}

}  // namespace

extern "C" {

// C[M,N] = op(A) op(B) (+ R) on one tile per CTA (bn = 64, 128: 128 x bn) or per CTA pair (bn = 256: 256 x 256),
// `split` CTAs (1 to 4 or 8) or pairs (1 to 4) per tile along K, each of which has to get a 64-wide K block. Arguments
// otherwise as gfs_gemm_bf16_rope;
// swi_mode 1 / 2 with swi_extra as gfs_gemm_bf16_swiglu (then N is I: columns of act, resp. d_act).
int gfs_gemm_tile(const void* A, const void* B, void* C, const void* R, int M, int N, int K, int lda, int ldb, int ldc,
                  int ldr, int a_mn_major, int b_mn_major, const void* rope_cos, const void* rope_sin, int rope_cols,
                  int rope_d, int rope_b, int swi_mode, void* swi_extra, int swi_ld, int bn, int split, void* stream_) {
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if ((N & 7) || (lda & 7) || (ldb & 7) || (ldc & 7) || (R && (ldr & 7))) return -1;
  if (bad_shape(bn, split)) return -1;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C) |
       reinterpret_cast<uintptr_t>(R) | reinterpret_cast<uintptr_t>(swi_extra)) & 15)
    return -2;
  if (rope_cos != nullptr && ((rope_d & 7) || (rope_cols & 7) || rope_b <= 0)) return -1;
  if (swi_mode != 0 && (swi_mode < 0 || swi_mode > 2 || swi_extra == nullptr || (swi_ld & 7) || a_mn_major ||
                        b_mn_major != (swi_mode == 2) || R != nullptr || rope_cos != nullptr))
    return -1;
  const CUtensorMap* ta = a_mn_major ? gfs_host::tmap_2d_cached(A, K, M, lda, 64, 64)
                                     : gfs_host::tmap_2d_cached(A, M, K, lda, BM, 64);
  const int brows = bn == 256 ? 128 : bn;   // a CTA of a pair holds half of B
  const CUtensorMap* tb = swi_mode == 1 ? gfs_host::tmap_2d_cached(B, 2ull * N, K, ldb, bn / 2, 64)
                          : b_mn_major  ? gfs_host::tmap_2d_cached(B, K, N, ldb, 64, 64)
                                        : gfs_host::tmap_2d_cached(B, N, K, ldb, brows, 64);
  if (ta == nullptr || tb == nullptr) return -3;
  TileMaps<1> maps;
  maps.a[0] = *ta;
  maps.b[0] = *tb;
  TileParams<1> p{};
  p.ngroups = 1;
  p.split = split;
  p.early_b = gfs_host::launch_hints().early_b;
  p.late_wait = gfs_host::launch_hints().late_wait;
  p.status = gfs_host::status_words();
  p.rope_cos = static_cast<const float*>(rope_cos);
  p.rope_sin = static_cast<const float*>(rope_sin);
  p.rope_cols = rope_cols; p.rope_d = rope_d; p.rope_b = rope_b > 0 ? rope_b : 1;
  p.swi_I = N; p.swi_ld = swi_ld;
  if (swi_mode == 1) p.swi_act = static_cast<__nv_bfloat16*>(swi_extra);
  if (swi_mode == 2) p.swi_gu = static_cast<const __nv_bfloat16*>(swi_extra);
  TileProblem& g = p.g[0];
  g.M = M; g.N = swi_mode == 1 ? 2 * N : N;
  g.kblocks = (K + BK - 1) / BK;
  g.per_split = (g.kblocks + split - 1) / split;
  if (g.per_split * (split - 1) >= g.kblocks) return -1;   // a CTA without K blocks
  const int cols = swi_mode == 1 ? bn / 2 : bn;            // output columns (of N) per tile
  g.tiles_n = (N + cols - 1) / cols;
  g.tile_begin = 0;
  g.ldc = ldc; g.ldr = ldr;
  g.C = static_cast<__nv_bfloat16*>(C);
  g.R = static_cast<const __nv_bfloat16*>(R);
  const int bm = bn == 256 ? 256 : BM;
  const int ctas = (M + bm - 1) / bm * g.tiles_n * split;
  if (swi_mode == 1) return launch_tile<false, false, 1, EPI_SWIGLU>(bn, maps, p, ctas, stream);
  if (swi_mode == 2) return launch_tile<false, true, 1, EPI_SWIGLU_BWD>(bn, maps, p, ctas, stream);
  return rope_cos != nullptr ? launch_layout<EPI_ROPE>(a_mn_major, b_mn_major, bn, maps, p, ctas, stream)
                             : launch_layout<EPI_PLAIN>(a_mn_major, b_mn_major, bn, maps, p, ctas, stream);
}

// Grouped weight gradients with this kernel: same contract as gfs_gemm2_wgrad_grouped.
int gfs_gemm_tile_wgrad_grouped(int n, const unsigned long long* A, const unsigned long long* B,
                                const unsigned long long* C, const int* M, const int* N, const int* K, const int* lda,
                                const int* ldb, const int* ldc, const int* accumulate, int bn, int split,
                                void* stream_) {
  if (n <= 0) return 0;
  if (n > MAX_GROUP) return -1;
  if (bad_shape(bn, split)) return -1;
  TileMaps<MAX_GROUP> maps;
  TileParams<MAX_GROUP> p{};
  p.ngroups = n;
  p.split = split;
  p.early_b = gfs_host::launch_hints().early_b;
  p.late_wait = gfs_host::launch_hints().late_wait;
  p.status = gfs_host::status_words();
  p.rope_b = 1;
  int total = 0;
  const int bm = bn == 256 ? 256 : BM;
  for (int i = 0; i < n; ++i) {
    if (M[i] <= 0 || N[i] <= 0 || K[i] <= 0) return -1;
    if ((N[i] & 7) || (M[i] & 7) || (lda[i] & 7) || (ldb[i] & 7) || (ldc[i] & 7)) return -1;
    if ((A[i] | B[i] | C[i]) & 15) return -2;
    const CUtensorMap* ta = gfs_host::tmap_2d_cached(reinterpret_cast<const void*>(A[i]), K[i], M[i], lda[i], 64, 64);
    const CUtensorMap* tb = gfs_host::tmap_2d_cached(reinterpret_cast<const void*>(B[i]), K[i], N[i], ldb[i], 64, 64);
    if (ta == nullptr || tb == nullptr) return -3;
    maps.a[i] = *ta;
    maps.b[i] = *tb;
    TileProblem& g = p.g[i];
    g.M = M[i]; g.N = N[i];
    g.kblocks = (K[i] + BK - 1) / BK;
    g.per_split = (g.kblocks + split - 1) / split;
    if (g.per_split * (split - 1) >= g.kblocks) return -1;
    g.tiles_n = (N[i] + bn - 1) / bn;
    g.tile_begin = total;
    g.ldc = ldc[i]; g.ldr = ldc[i];
    g.C = reinterpret_cast<__nv_bfloat16*>(C[i]);
    g.R = accumulate[i] ? g.C : nullptr;
    total += (M[i] + bm - 1) / bm * g.tiles_n;
  }
  for (int i = n; i < MAX_GROUP; ++i) {
    maps.a[i] = maps.a[0];
    maps.b[i] = maps.b[0];
    p.g[i] = p.g[0];
    p.g[i].tile_begin = INT_MAX;
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  return launch_tile<true, true, MAX_GROUP, EPI_PLAIN>(bn, maps, p, total * split, stream);
}

}  // extern "C"
