// Memory-bound kernels of the training step: RMSNorm fwd/bwd, rotary embedding,
// SwiGLU fwd/bwd, embedding lookup fwd/bwd. Each replaces a chain of ATen kernels of
// the reference with one pass over the data (16-byte vector accesses, fp32 math).
//
// Reference counterparts: core/normalization.py:13-25 (RMSNorm), core/rope_triton.py:74-141
// (RoPE), core/mlp.py:25-28 (SwiGLU), core/tensor_parallel/layers.py:117-134 (embedding).
#include <algorithm>
#include <type_traits>

#include "api.h"
#include "common.cuh"

using namespace gfs;

namespace {

constexpr int NORM_WARPS = 4;

__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&f)[8]) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const float (&f)[8]) {
  uint4 o;
  o.x = pack_bf16x2(f[0], f[1]);
  o.y = pack_bf16x2(f[2], f[3]);
  o.z = pack_bf16x2(f[4], f[5]);
  o.w = pack_bf16x2(f[6], f[7]);
  *reinterpret_cast<uint4*>(p) = o;
}
__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// ---------------------------------------------------------------------------
// Dropout. Counter-based generator: one 64-bit mix of (seed, vector index) yields the eight 8-bit thresholds of a
// vector of 8 elements, so the keep probability is quantised to 1/256 and no mask tensor exists.
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
struct Dropout {
  float p;
  unsigned long long seed;
};
// f: vector v of the tensor; dropped elements become 0, the others are scaled
__device__ __forceinline__ void drop8(float (&f)[8], long long v, const Dropout& d) {
  const unsigned int drop_below = static_cast<unsigned int>(d.p * 256.f + 0.5f);  // byte < drop_below -> dropped
  const float scale = 256.f / static_cast<float>(256u - drop_below);             // 1 / (realised keep probability)
  const unsigned long long bits = mix64(d.seed ^ (static_cast<unsigned long long>(v) * 0xd1342543de82ef95ull));
#pragma unroll
  for (int e = 0; e < 8; ++e) f[e] = ((bits >> (8 * e)) & 0xffull) >= drop_below ? f[e] * scale : 0.f;
}

// ---------------------------------------------------------------------------
// RMSNorm forward: y = bf16(x * rstd) * w, rstd = rsqrt(mean(x^2) + eps). One warp per row.
// ---------------------------------------------------------------------------
// NORM_MAXV = vectors of 8 bf16 cached per lane (covers H <= 256 * NORM_MAXV without a second
// read); a template parameter so that small hidden sizes do not pay for 64 cache registers.
// DROP: x is not read but made, x = residual + dropout(z), and written beside y: a pass over x and a launch less
// (bits as from the two kernels). A step of the 124M model at 4 x 512 tokens, dropout 0.1, with the backward's counterpart below,
// which masks the gradient that it writes: 4229 -> 4172 us.
struct DropResidual {
  const __nv_bfloat16 *z, *residual;
  __nv_bfloat16* x;
  Dropout drop;
};
template <int NORM_MAXV, bool DROP>
__global__ void __launch_bounds__(NORM_WARPS * 32)
rmsnorm_fwd_kernel(const __nv_bfloat16* x, const __nv_bfloat16* w, __nv_bfloat16* __restrict__ y,
                   float* __restrict__ rstd_out, int rows, int H, float eps, const DropResidual dr) {
  pdl_wait();       // launched programmatically: the preceding kernel's output is complete from here on
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * NORM_WARPS + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int nvec = H >> 3;
  const __nv_bfloat16* xr = (DROP ? dr.x : x) + static_cast<size_t>(row) * H;
  auto load = [&](int v) -> uint4 {
    if constexpr (!DROP) {
      return *reinterpret_cast<const uint4*>(xr + 8 * v);
    } else {
      const size_t at = static_cast<size_t>(row) * H + 8 * v;
      float f[8], r[8];
      load8(dr.z + at, f);
      load8(dr.residual + at, r);
      drop8(f, static_cast<long long>(at >> 3), dr.drop);
#pragma unroll
      for (int e = 0; e < 8; ++e) r[e] += round_bf16(f[e]);
      const uint4 o = make_uint4(pack_bf16x2(r[0], r[1]), pack_bf16x2(r[2], r[3]), pack_bf16x2(r[4], r[5]),
                                 pack_bf16x2(r[6], r[7]));
      *reinterpret_cast<uint4*>(dr.x + at) = o;
      return o;
    }
  };
  __nv_bfloat16* yr = y + static_cast<size_t>(row) * H;
  uint4 cache[NORM_MAXV];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < NORM_MAXV; ++i) {
    const int v = lane + 32 * i;
    if (v < nvec) {
      cache[i] = load(v);
      const float2 a = unpack_bf16x2(cache[i].x), b = unpack_bf16x2(cache[i].y), c = unpack_bf16x2(cache[i].z),
                   d = unpack_bf16x2(cache[i].w);
      ss += a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y + c.x * c.x + c.y * c.y + d.x * d.x + d.y * d.y;
    }
  }
  for (int v = lane + 32 * NORM_MAXV; v < nvec; v += 32) {
    float f[8];
    if (DROP) load(v);
    load8(xr + 8 * v, f);
#pragma unroll
    for (int e = 0; e < 8; ++e) ss += f[e] * f[e];
  }
  ss = warp_sum(ss);
  const float rstd = rsqrtf(ss / static_cast<float>(H) + eps);
  if (lane == 0 && rstd_out != nullptr) rstd_out[row] = rstd;
#pragma unroll
  for (int i = 0; i < NORM_MAXV; ++i) {
    const int v = lane + 32 * i;
    if (v < nvec) {
      float f[8], g[8];
      const float2 a = unpack_bf16x2(cache[i].x), b = unpack_bf16x2(cache[i].y), c = unpack_bf16x2(cache[i].z),
                   d = unpack_bf16x2(cache[i].w);
      f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
      load8(w + 8 * v, g);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] = round_bf16(f[e] * rstd) * g[e];
      store8(yr + 8 * v, f);
    }
  }
  for (int v = lane + 32 * NORM_MAXV; v < nvec; v += 32) {
    float f[8], g[8];
    load8(xr + 8 * v, f);
    load8(w + 8 * v, g);
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = round_bf16(f[e] * rstd) * g[e];
    store8(yr + 8 * v, f);
  }
}

// ---------------------------------------------------------------------------
// RMSNorm backward. Each CTA owns a contiguous block of rows; every warp keeps the
// weight-gradient partial of the rows it handled in its own shared-memory row, so dw
// needs no atomics: per-CTA partials [gridDim.x, H] are summed by a second kernel.
//   g = dy * w;  dx = rstd * g - x * rstd^3 * mean(g * x)  (+ dres);  dw += dy * bf16(x * rstd)
// ---------------------------------------------------------------------------
constexpr int NB_WARPS = 8;

// Register path, for few rows (H <= 256 * NV): every lane keeps the row values it needs for the second
// pass and its dw partial sums in registers; shared memory is only used once at the end.
template <int NV>
__global__ void __launch_bounds__(NB_WARPS * 32, NV <= 4 ? 2 : 1)
rmsnorm_bwd_reg_kernel(const __nv_bfloat16* dy, const __nv_bfloat16* x,
                       const __nv_bfloat16* w, const float* rstd,
                       const __nv_bfloat16* dres, __nv_bfloat16* __restrict__ dx,
                       float* __restrict__ dw_partial, int rows, int H, int rows_per_cta) {
  extern __shared__ float red[];  // [warps][H]
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  const int nvec = H >> 3;
  const int r0 = blockIdx.x * rows_per_cta;
  const int r1 = min(rows, r0 + rows_per_cta);
  float wv[NV][8];
  float dwacc[NV][8];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = lane + 32 * i;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      dwacc[i][e] = 0.f;
      wv[i][e] = 0.f;
    }
    if (v < nvec) load8(w + 8 * v, wv[i]);
  }
  for (int row = r0 + warp; row < r1; row += nwarps) {
    const __nv_bfloat16* dyr = dy + static_cast<size_t>(row) * H;
    const __nv_bfloat16* xr = x + static_cast<size_t>(row) * H;
    const float rs = rstd[row];
    uint4 cdy[NV], cx[NV], cres[NV];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = lane + 32 * i;
      if (v < nvec) {
        cdy[i] = *reinterpret_cast<const uint4*>(dyr + 8 * v);
        cx[i] = *reinterpret_cast<const uint4*>(xr + 8 * v);
        if (dres != nullptr) cres[i] = *reinterpret_cast<const uint4*>(dres + static_cast<size_t>(row) * H + 8 * v);
      }
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = lane + 32 * i;
      if (v < nvec) {
        const float2 a0 = unpack_bf16x2(cdy[i].x), a1 = unpack_bf16x2(cdy[i].y), a2 = unpack_bf16x2(cdy[i].z),
                     a3 = unpack_bf16x2(cdy[i].w);
        const float2 b0 = unpack_bf16x2(cx[i].x), b1 = unpack_bf16x2(cx[i].y), b2 = unpack_bf16x2(cx[i].z),
                     b3 = unpack_bf16x2(cx[i].w);
        dot += a0.x * wv[i][0] * b0.x + a0.y * wv[i][1] * b0.y + a1.x * wv[i][2] * b1.x + a1.y * wv[i][3] * b1.y +
               a2.x * wv[i][4] * b2.x + a2.y * wv[i][5] * b2.y + a3.x * wv[i][6] * b3.x + a3.y * wv[i][7] * b3.y;
      }
    }
    dot = warp_sum(dot);
    const float coef = dot * rs * rs * rs / static_cast<float>(H);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = lane + 32 * i;
      if (v < nvec) {
        float a[8], b[8], o[8];
        const float2 a0 = unpack_bf16x2(cdy[i].x), a1 = unpack_bf16x2(cdy[i].y), a2 = unpack_bf16x2(cdy[i].z),
                     a3 = unpack_bf16x2(cdy[i].w);
        const float2 b0 = unpack_bf16x2(cx[i].x), b1 = unpack_bf16x2(cx[i].y), b2 = unpack_bf16x2(cx[i].z),
                     b3 = unpack_bf16x2(cx[i].w);
        a[0] = a0.x; a[1] = a0.y; a[2] = a1.x; a[3] = a1.y; a[4] = a2.x; a[5] = a2.y; a[6] = a3.x; a[7] = a3.y;
        b[0] = b0.x; b[1] = b0.y; b[2] = b1.x; b[3] = b1.y; b[4] = b2.x; b[5] = b2.y; b[6] = b3.x; b[7] = b3.y;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          o[e] = rs * a[e] * wv[i][e] - b[e] * coef;
          dwacc[i][e] += a[e] * round_bf16(b[e] * rs);
        }
        if (dres != nullptr) {
          const float2 d0 = unpack_bf16x2(cres[i].x), d1 = unpack_bf16x2(cres[i].y), d2 = unpack_bf16x2(cres[i].z),
                       d3 = unpack_bf16x2(cres[i].w);
          o[0] += d0.x; o[1] += d0.y; o[2] += d1.x; o[3] += d1.y; o[4] += d2.x; o[5] += d2.y; o[6] += d3.x; o[7] += d3.y;
        }
        store8(dx + static_cast<size_t>(row) * H + 8 * v, o);
      }
    }
  }
  float* my_red = red + static_cast<size_t>(warp) * H;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = lane + 32 * i;
    if (v < nvec) {
#pragma unroll
      for (int e = 0; e < 8; ++e) my_red[8 * v + e] = dwacc[i][e];
    }
  }
  __syncthreads();
  float* outp = dw_partial + static_cast<size_t>(blockIdx.x) * H;
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    float s = 0.f;
    for (int wv2 = 0; wv2 < nwarps; ++wv2) s += red[static_cast<size_t>(wv2) * H + i];
    outp[i] = s;
  }
}

// Ring path (H <= 256 * NV): bound by memory, 8 bytes per element. Every warp works through rows of its own, which bulk
// copies bring into its two slots of shared memory (dy | x | dres, one row each) two rows ahead, so the memory system is
// busy while the warps compute. (With the rows loaded into registers as they were needed, nothing was in
// flight between a row's loads and its results, and at H 2048 only eight warps fitted on an SM.) The dw partial sums stay
// in registers; the slots hold them at the end for the sum over the CTA's
// warps. us in a training step, registers -> this: [16384, 768] 30.6 -> 21.6, [8192, 768] 17.8 -> 12.8, [2331, 768] 7.3 -> 5.8,
// [8192, 2048] 53 -> 31 (134 MB: 21 at copy bandwidth).
template <int NV>
struct NormBwdShape {
  static constexpr int WARPS = NV <= 4 ? 8 : 4;       // two CTAs per SM: 96 KB of slots each at most
  static constexpr int SLOTS = 2;
  static int smem(int H) { return WARPS * SLOTS * (3 * 2 * H) + 256; }
};

// DROP: dmask = dropout's gradient of the (rounded) dx, for the branch whose output was dropped
template <int NV, bool DROP>
__global__ void __launch_bounds__(NormBwdShape<NV>::WARPS * 32, 2)
rmsnorm_bwd_ring_kernel(const __nv_bfloat16* dy, const __nv_bfloat16* x,
                        const __nv_bfloat16* w, const float* rstd,
                        const __nv_bfloat16* dres, __nv_bfloat16* __restrict__ dx,
                        float* __restrict__ dw_partial, int rows, int H, int rows_per_cta, uint32_t* status,
                        __nv_bfloat16* __restrict__ dmask, const Dropout drop) {
  constexpr int WARPS = NormBwdShape<NV>::WARPS, SLOTS = NormBwdShape<NV>::SLOTS;
  extern __shared__ __align__(128) uint8_t ring_smem[];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const uint32_t row_bytes = 2u * H;
  uint8_t* ring = ring_smem + warp * (SLOTS * 3 * row_bytes);
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring_smem + WARPS * SLOTS * 3 * row_bytes);
  uint64_t* full = bars + warp * SLOTS;
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(bars + WARPS * SLOTS);
  if (threadIdx.x == 0) {
    for (int i = 0; i < WARPS * SLOTS; ++i) mbar_init(&bars[i], 1);
    *abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  WaitCtx wctx{abort_flag, status, GFS_WAIT_LIMIT_NS};
  const int nvec = H >> 3;
  const int r0 = blockIdx.x * rows_per_cta + warp;
  const int r1 = min(rows, (static_cast<int>(blockIdx.x) + 1) * rows_per_cta);
  auto fetch = [&](int row, int slot) {     // lane 0
    uint8_t* dst = ring + slot * (3 * row_bytes);
    const size_t at = static_cast<size_t>(row) * H;
    mbar_arrive_expect_tx(&full[slot], (dres != nullptr ? 3 : 2) * row_bytes);
    bulk_load_1d(dst, dy + at, row_bytes, &full[slot]);
    bulk_load_1d(dst + row_bytes, x + at, row_bytes, &full[slot]);
    if (dres != nullptr) bulk_load_1d(dst + 2 * row_bytes, dres + at, row_bytes, &full[slot]);
  };
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < SLOTS; ++i)
      if (r0 + i * WARPS < r1) fetch(r0 + i * WARPS, i);
  }
  uint4 wv[NV];
  uint64_t dwacc[NV][4];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = lane + 32 * i;
    wv[i] = v < nvec ? *reinterpret_cast<const uint4*>(w + 8 * v) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int e = 0; e < 4; ++e) dwacc[i][e] = 0;
  }
  auto pair_of = [](uint32_t u) {
    const float2 f = unpack_bf16x2(u);
    return pack_f32x2(f.x, f.y);
  };
  const float inv_h = 1.f / static_cast<float>(H);
  float rs_lane = 0.f;
  int k = 0;
  for (int row = r0; row < r1; row += WARPS, ++k) {
    if ((k & 31) == 0) {                    // lane i: the row i after this one
      const int at = row + lane * WARPS;
      rs_lane = at < r1 ? rstd[at] : 0.f;
    }
    const float rs = __shfl_sync(0xffffffffu, rs_lane, k & 31);
    const int slot = k % SLOTS;
    const uint8_t* src = ring + slot * (3 * row_bytes);
    if (!__all_sync(0xffffffffu, mbar_wait(&full[slot], (k / SLOTS) & 1, wctx, STATUS_TIMEOUT_PIPE_FULL))) break;
    uint64_t dot2 = 0;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = lane + 32 * i;
      if (v < nvec) {
        const uint4 a = *reinterpret_cast<const uint4*>(src + 16 * v);
        const uint4 b = *reinterpret_cast<const uint4*>(src + row_bytes + 16 * v);
        const uint32_t *ap = &a.x, *bp = &b.x, *wp = &wv[i].x;
#pragma unroll
        for (int e = 0; e < 4; ++e)
          dot2 = fma_f32x2(mul_f32x2(pair_of(ap[e]), pair_of(wp[e])), pair_of(bp[e]), dot2);
      }
    }
    const float2 d2 = unpack_f32x2(dot2);
    const float coef = warp_sum(d2.x + d2.y) * rs * rs * rs * inv_h;
    const uint64_t rs2 = pack_f32x2(rs, rs), nc2 = pack_f32x2(-coef, -coef);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int v = lane + 32 * i;
      if (v < nvec) {
        const uint4 a = *reinterpret_cast<const uint4*>(src + 16 * v);
        const uint4 b = *reinterpret_cast<const uint4*>(src + row_bytes + 16 * v);
        uint4 c = make_uint4(0, 0, 0, 0);
        if (dres != nullptr) c = *reinterpret_cast<const uint4*>(src + 2 * row_bytes + 16 * v);
        const uint32_t *ap = &a.x, *bp = &b.x, *wp = &wv[i].x;
        uint32_t* cp = &c.x;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint64_t a2 = pair_of(ap[e]), b2 = pair_of(bp[e]);
          const float2 n = unpack_f32x2(mul_f32x2(b2, rs2));
          dwacc[i][e] = fma_f32x2(a2, pair_of(pack_bf16x2(n.x, n.y)), dwacc[i][e]);
          const uint64_t g = fma_f32x2(mul_f32x2(rs2, a2), pair_of(wp[e]), mul_f32x2(b2, nc2));
          const float2 o = unpack_f32x2(add_f32x2(g, pair_of(cp[e])));
          cp[e] = pack_bf16x2(o.x, o.y);
        }
        const size_t at = static_cast<size_t>(row) * H + 8 * v;
        *reinterpret_cast<uint4*>(dx + at) = c;
        if constexpr (DROP) {
          float f[8];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 o = unpack_bf16x2(cp[e]);
            f[2 * e] = o.x;
            f[2 * e + 1] = o.y;
          }
          drop8(f, static_cast<long long>(at >> 3), drop);
          store8(dmask + at, f);
        }
      }
    }
    __syncwarp();                           // the slot has been read
    if (lane == 0 && row + SLOTS * WARPS < r1) fetch(row + SLOTS * WARPS, slot);
  }
  settle_copies(wctx);
  __syncthreads();                          // all rows of all warps: the ring is free
  float* red = reinterpret_cast<float*>(ring_smem);   // [WARPS][H]
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int v = lane + 32 * i;
    if (v < nvec) {
      float* at = red + warp * H + 8 * v;
#pragma unroll
      for (int e = 0; e < 4; ++e) *reinterpret_cast<float2*>(at + 2 * e) = unpack_f32x2(dwacc[i][e]);
    }
  }
  __syncthreads();
  float* outp = dw_partial + static_cast<size_t>(blockIdx.x) * H;
  for (int i = threadIdx.x; i < H; i += WARPS * 32) {
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < WARPS; ++j) s += red[j * H + i];
    outp[i] = s;
  }
}

// Generic path (any H that is a multiple of 8): partial sums live in shared memory.
__global__ void __launch_bounds__(NB_WARPS * 32)
rmsnorm_bwd_kernel(const __nv_bfloat16* dy, const __nv_bfloat16* x,
                   const __nv_bfloat16* w, const float* rstd,
                   const __nv_bfloat16* dres, __nv_bfloat16* __restrict__ dx,
                   float* __restrict__ dw_partial, int rows, int H, int rows_per_cta) {
  extern __shared__ float red[];  // [warps][H]
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  const int nvec = H >> 3;
  const int r0 = blockIdx.x * rows_per_cta;
  const int r1 = min(rows, r0 + rows_per_cta);
  float* my_red = red + static_cast<size_t>(warp) * H;
  for (int i = lane; i < H; i += 32) my_red[i] = 0.f;
  __syncwarp();

  for (int row = r0 + warp; row < r1; row += nwarps) {
    const __nv_bfloat16* dyr = dy + static_cast<size_t>(row) * H;
    const __nv_bfloat16* xr = x + static_cast<size_t>(row) * H;
    __nv_bfloat16* dxr = dx + static_cast<size_t>(row) * H;
    const float rs = rstd[row];
    float dot = 0.f;
    for (int v = lane; v < nvec; v += 32) {
      float a[8], b[8], c[8];
      load8(dyr + 8 * v, a);
      load8(xr + 8 * v, b);
      load8(w + 8 * v, c);
#pragma unroll
      for (int e = 0; e < 8; ++e) dot += a[e] * c[e] * b[e];
    }
    dot = warp_sum(dot);
    const float coef = dot * rs * rs * rs / static_cast<float>(H);
    for (int v = lane; v < nvec; v += 32) {
      float a[8], b[8], c[8], o[8];
      load8(dyr + 8 * v, a);
      load8(xr + 8 * v, b);
      load8(w + 8 * v, c);
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = rs * a[e] * c[e] - b[e] * coef;
      if (dres != nullptr) {
        float d[8];
        load8(dres + static_cast<size_t>(row) * H + 8 * v, d);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] += d[e];
      }
      store8(dxr + 8 * v, o);
      float* acc = my_red + 8 * v;
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += a[e] * round_bf16(b[e] * rs);
    }
  }
  __syncthreads();
  float* outp = dw_partial + static_cast<size_t>(blockIdx.x) * H;
  for (int i = threadIdx.x; i < H; i += blockDim.x) {
    float s = 0.f;
    for (int wv = 0; wv < nwarps; ++wv) s += red[static_cast<size_t>(wv) * H + i];
    outp[i] = s;
  }
}

// blockDim = (32, 32): 32 columns per block, the partial rows are split over 32 thread rows and
// combined through shared memory in a fixed order (deterministic).
__global__ void rmsnorm_dw_reduce_kernel(const float* __restrict__ partial, __nv_bfloat16* __restrict__ dw, int parts,
                                         int H, int accumulate) {
  __shared__ float sm[32][33];
  const int i = blockIdx.x * 32 + threadIdx.x;
  float s = 0.f;
  if (i < H) {
    for (int p = threadIdx.y; p < parts; p += 32) s += partial[static_cast<size_t>(p) * H + i];
  }
  sm[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && i < H) {
    float t = 0.f;
#pragma unroll
    for (int y = 0; y < 32; ++y) t += sm[y][threadIdx.x];
    if (accumulate) t += __bfloat162float(dw[i]);
    dw[i] = __float2bfloat16_rn(t);
  }
}

// The same reduction for several RMSNorm layers in one launch (blockIdx.y = layer): the
// per-layer reductions are tiny, so a backward pass parks them and runs them together.
constexpr int DW_MULTI_MAX = 32;
struct DwReduceBatch {
  const float* partial[DW_MULTI_MAX];
  __nv_bfloat16* dw[DW_MULTI_MAX];
  int parts[DW_MULTI_MAX];
  int accumulate[DW_MULTI_MAX];
};

__global__ void rmsnorm_dw_reduce_multi_kernel(const __grid_constant__ DwReduceBatch b, int H) {
  __shared__ float sm[32][33];
  pdl_wait();
  pdl_trigger();
  const int l = blockIdx.y;
  const float* partial = b.partial[l];
  __nv_bfloat16* __restrict__ dw = b.dw[l];
  const int parts = b.parts[l];
  const int i = blockIdx.x * 32 + threadIdx.x;
  float s = 0.f;
  if (i < H) {
    for (int p = threadIdx.y; p < parts; p += 32) s += partial[static_cast<size_t>(p) * H + i];
  }
  sm[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && i < H) {
    float t = 0.f;
#pragma unroll
    for (int y = 0; y < 32; ++y) t += sm[y][threadIdx.x];
    if (b.accumulate[l]) t += __bfloat162float(dw[i]);
    dw[i] = __float2bfloat16_rn(t);
  }
}

// ---------------------------------------------------------------------------
// Rotary embedding, interleaved pairs, in place on `parts` consecutive [nh*D] blocks
// of every token (parts = 2: the q and k thirds of a [S,B,3,nh,D] buffer).
//   x'[2i] = x[2i] cos - x[2i+1] sin ; x'[2i+1] = x[2i] sin + x[2i+1] cos ; backward: sin -> -sin
// ---------------------------------------------------------------------------
__global__ void rope_kernel(__nv_bfloat16* __restrict__ x, const float* __restrict__ cosb,
                            const float* __restrict__ sinb, int S, int B, int nhD, int D, int parts,
                            long token_stride, int backward, int s_offset) {
  const int vec_per_token = (parts * nhD) >> 3;
  const size_t total = static_cast<size_t>(S) * B * vec_per_token;
  for (size_t v = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; v < total;
       v += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t token = v / vec_per_token;
    const int e0 = static_cast<int>(v % vec_per_token) << 3;
    const int s = static_cast<int>(token / B) + s_offset;
    const int d = e0 % D;
    __nv_bfloat16* p = x + token * token_stride + e0;
    float f[8];
    load8(p, f);
    const float4 c = *reinterpret_cast<const float4*>(cosb + static_cast<size_t>(s) * (D >> 1) + (d >> 1));
    float4 sn = *reinterpret_cast<const float4*>(sinb + static_cast<size_t>(s) * (D >> 1) + (d >> 1));
    if (backward) {
      sn.x = -sn.x; sn.y = -sn.y; sn.z = -sn.z; sn.w = -sn.w;
    }
    float o[8];
    o[0] = f[0] * c.x - f[1] * sn.x; o[1] = f[0] * sn.x + f[1] * c.x;
    o[2] = f[2] * c.y - f[3] * sn.y; o[3] = f[2] * sn.y + f[3] * c.y;
    o[4] = f[4] * c.z - f[5] * sn.z; o[5] = f[4] * sn.z + f[5] * c.z;
    o[6] = f[6] * c.w - f[7] * sn.w; o[7] = f[6] * sn.w + f[7] * c.w;
    store8(p, o);
  }
}

// ---------------------------------------------------------------------------
// Dropout fused with the residual add (the reference's `residual + dropout(x)`,
// core/transformer_layer.py:97,103); the native passes have it in the RMSNorm kernels.
// ---------------------------------------------------------------------------
__global__ void dropout_residual_kernel(const __nv_bfloat16* x, const __nv_bfloat16* residual,
                                        __nv_bfloat16* __restrict__ out, long long nvec, Dropout drop, int backward) {
  pdl_wait();
  pdl_trigger();
  for (long long v = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; v < nvec;
       v += static_cast<long long>(gridDim.x) * blockDim.x) {
    float f[8], r[8];
    load8(x + 8 * v, f);
    const bool add = !backward && residual != nullptr;
    if (add) load8(residual + 8 * v, r);
    drop8(f, v, drop);
    if (add) {
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] = r[e] + round_bf16(f[e]);
    }
    store8(out + 8 * v, f);
  }
}

// ---------------------------------------------------------------------------
// SwiGLU on a [M, 2I] buffer whose first I columns are the gate and last I the up half.
// ---------------------------------------------------------------------------
// Grid: x covers the 8-column vectors of a row, y strides over rows (no integer divisions).
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ act, int M, int I) {
  const int vec_per_row = I >> 3;
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= vec_per_row) return;
  const int c = v << 3;
  for (int row = blockIdx.y; row < M; row += gridDim.y) {
    const __nv_bfloat16* base = gu + static_cast<size_t>(row) * 2 * I;
    float g[8], u[8], o[8];
    load8(base + c, g);
    load8(base + I + c, u);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float sg = sigmoid_f(g[e]);
      // silu rounded to bf16 before the product, as two separate bf16 ops would do
      o[e] = round_bf16(g[e] * sg) * u[e];
    }
    store8(act + static_cast<size_t>(row) * I + c, o);
  }
}

__global__ void swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dact, const __nv_bfloat16* __restrict__ gu,
                                  __nv_bfloat16* __restrict__ dgu, int M, int I) {
  const int vec_per_row = I >> 3;
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= vec_per_row) return;
  const int c = v << 3;
  for (int row = blockIdx.y; row < M; row += gridDim.y) {
    const size_t rb = static_cast<size_t>(row) * 2 * I;
    float g[8], u[8], d[8], dg[8], du[8];
    load8(gu + rb + c, g);
    load8(gu + rb + I + c, u);
    load8(dact + static_cast<size_t>(row) * I + c, d);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float sg = sigmoid_f(g[e]);
      const float silu = g[e] * sg;
      dg[e] = d[e] * u[e] * sg * (1.f + g[e] * (1.f - sg));
      du[e] = d[e] * silu;
    }
    store8(dgu + rb + c, dg);
    store8(dgu + rb + I + c, du);
  }
}

// ---------------------------------------------------------------------------
// Embedding forward: out[s - s0, b, :] = W[id - v0] if v0 <= id < v1 else 0, ids are [B, S].
// One warp per output row.
// ---------------------------------------------------------------------------
__global__ void embedding_fwd_kernel(const long long* ids, const __nv_bfloat16* W,
                                     __nv_bfloat16* __restrict__ out, int B, int S, int H, int v0, int v1, int s0,
                                     int s_count) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (r >= s_count * B) return;
  const int s = s0 + r / B;
  const int b = r % B;
  const long long id = ids[static_cast<size_t>(b) * S + s];
  __nv_bfloat16* o = out + static_cast<size_t>(r) * H;
  const int nvec = H >> 3;
  if (id >= v0 && id < v1) {
    const __nv_bfloat16* src = W + static_cast<size_t>(id - v0) * H;
    for (int v = lane; v < nvec; v += 32)
      *reinterpret_cast<uint4*>(o + 8 * v) = *reinterpret_cast<const uint4*>(src + 8 * v);
  } else {
    for (int v = lane; v < nvec; v += 32) *reinterpret_cast<uint4*>(o + 8 * v) = make_uint4(0, 0, 0, 0);
  }
}

// Embedding backward over token ids sorted ascending (perm gives each sorted position's
// row in dout). A warp owns one run of equal ids and sums its rows in sorted order,
// so the result is deterministic; dW rows are accumulated (bf16, fp32 sum).
__global__ void embedding_bwd_kernel(const long long* __restrict__ sorted_ids, const long long* __restrict__ perm,
                                     const __nv_bfloat16* __restrict__ dout, __nv_bfloat16* __restrict__ dW, int n,
                                     int H, int v0, int v1) {
  const int lane = threadIdx.x & 31;
  const int p = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (p >= n) return;
  const long long id = sorted_ids[p];
  if (id < v0 || id >= v1) return;
  if (p > 0 && sorted_ids[p - 1] == id) return;  // not the start of a run
  int q_end = p + 1;
  while (q_end < n && sorted_ids[q_end] == id) ++q_end;
  __nv_bfloat16* dst = dW + static_cast<size_t>(id - v0) * H;
  const int nvec = H >> 3;
  for (int v = lane; v < nvec; v += 32) {
    float acc[8];
    load8(dst + 8 * v, acc);
    for (int q = p; q < q_end; ++q) {
      float f[8];
      load8(dout + static_cast<size_t>(perm[q]) * H + 8 * v, f);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += f[e];
    }
    store8(dst + 8 * v, acc);
  }
}

// Embedding backward without a library sort: the token ids of one micro-batch (n <= 32768) are
// sorted by ONE CTA in shared memory. Key = (local vocabulary row << shift) | dout row index, so
// keys are unique and ascending order is "by row, then by position" - the order a stable sort
// gives, hence the same bitwise result as summing in sorted order. Ids owned by other ranks get
// the all-ones key and end up behind the valid ones. Bitonic network on npow2 keys.
constexpr int SORT_THREADS = 1024;
__global__ void __launch_bounds__(SORT_THREADS)
embedding_sort_kernel(const long long* __restrict__ ids_bs, uint32_t* __restrict__ keys_out, int n, int npow2,
                      int shift, int B, int S, int v0, int v1) {
  extern __shared__ uint32_t sk[];
  for (int i = threadIdx.x; i < npow2; i += SORT_THREADS) {
    uint32_t key = 0xFFFFFFFFu;
    if (i < n) {
      const long long id = ids_bs[static_cast<size_t>(i % B) * S + i / B];   // dout row i = (s, b) = (i / B, i % B)
      if (id >= v0 && id < v1) key = (static_cast<uint32_t>(id - v0) << shift) | static_cast<uint32_t>(i);
    }
    sk[i] = key;
  }
  __syncthreads();
  for (int k = 2; k <= npow2; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int c = threadIdx.x; c < (npow2 >> 1); c += SORT_THREADS) {
        const int a = ((c & ~(j - 1)) << 1) | (c & (j - 1));
        const int b = a | j;
        const uint32_t x = sk[a], y = sk[b];
        const bool ascending = (a & k) == 0;
        if ((x > y) == ascending) {
          sk[a] = y;
          sk[b] = x;
        }
      }
      __syncthreads();
    }
  }
  for (int i = threadIdx.x; i < n; i += SORT_THREADS) keys_out[i] = sk[i];
}

// Segmented sum over the sorted keys, dout rows added in key order (deterministic); dW rows are accumulated (bf16, fp32
// sum). A warp per position; the first warps of a run of equal vocabulary rows share its columns, 256 at a time. The longest
// run bounds the time of a text (its commonest token is some 3 % of it, 245 rows of 8192 tokens), so its column blocks are
// worked on side by side, with EMB_AHEAD rows in flight and 32 keys per load. Uniform tokens are runs of one or two rows,
// and what counts there is the number of warps and what each does before its first row: the keys around its
// position come in one load, from which it knows its run, and two column blocks are in flight together. Few positions leave the chip
// idle: then several warps (blockIdx.y) stand for one.
// us, a warp per run -> a warp per run and column block -> this: 16384 uniform tokens at H 768 11.5 -> 18.3 -> 9.9, at 2048
// 53 -> 62 -> 38; 8192 tokens of text at 768 108 -> 28 -> 20. (EMB_AHEAD 16 takes 14 for the text, but 14.6 for the uniform
// tokens: fewer warps fit.)
constexpr int EMB_AHEAD = 8;
// A load that stays where it is written: the compiler would move each one down to its addition, one latency after the other.
__device__ __forceinline__ uint4 load_now(const __nv_bfloat16* p) {
  uint4 x;
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "l"(p));
  return x;
}
constexpr int EMB_BACK = 15;                           // keys ahead of the position in a warp's first load
__global__ void embedding_bwd_keys_kernel(const uint32_t* __restrict__ keys, const __nv_bfloat16* __restrict__ dout,
                                          __nv_bfloat16* __restrict__ dW, int n, int H, int shift) {
  const int lane = threadIdx.x & 31;
  const int p = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (p >= n) return;
  const int near = p - EMB_BACK + lane;
  const uint32_t k0 = near >= 0 && near < n ? keys[near] : 0xFFFFFFFFu;
  const uint32_t key = __shfl_sync(0xffffffffu, k0, EMB_BACK);
  if (key == 0xFFFFFFFFu) return;
  const uint32_t row = key >> shift, mask = (1u << shift) - 1u;
  auto run_lanes = [&](uint32_t k) { return __ballot_sync(0xffffffffu, k != 0xFFFFFFFFu && (k >> shift) == row); };
  const uint32_t same = run_lanes(k0);
  const uint32_t other = ~same & ((1u << EMB_BACK) - 1u);
  const int back = other != 0u ? __clz(other) - (32 - EMB_BACK) : EMB_BACK;   // rows of the run ahead of this one (or more)
  const int here = __ffs(~(same >> EMB_BACK)) - 1;     // and from this one on, as far as the load reaches
  const int nvec = H >> 3, blocks = (nvec + 31) >> 5;
  const int sharers = min(min(blocks, EMB_BACK), back + here);
  if (back >= sharers) return;
  const int cb0 = back * gridDim.y + blockIdx.y, cb_step = sharers * gridDim.y;   // this warp's column blocks
  __nv_bfloat16* const dst = dW + static_cast<size_t>(row) * H;
  auto add = [](float (&acc)[8], const uint4& x) {
    const float2 a = unpack_bf16x2(x.x), b = unpack_bf16x2(x.y), c = unpack_bf16x2(x.z), d = unpack_bf16x2(x.w);
    acc[0] += a.x; acc[1] += a.y; acc[2] += b.x; acc[3] += b.y;
    acc[4] += c.x; acc[5] += c.y; acc[6] += d.x; acc[7] += d.y;
  };
  const int first = EMB_BACK - back;                   // lane of the run's first key
  if (back + here <= 2) {
    const uint32_t r0 = __shfl_sync(0xffffffffu, k0, first) & mask;
    const uint32_t r1 = __shfl_sync(0xffffffffu, k0, first + back + here - 1) & mask;
    const bool two = back + here == 2;
    const __nv_bfloat16 *s0 = dout + static_cast<size_t>(r0) * H, *s1 = dout + static_cast<size_t>(r1) * H;
    for (int cb = cb0; cb < blocks; cb += 2 * cb_step) {
      uint4 old[2], x0[2], x1[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int v = (cb + u * cb_step) * 32 + lane;
        old[u] = x0[u] = x1[u] = make_uint4(0, 0, 0, 0);
        if (v >= nvec) continue;
        old[u] = *reinterpret_cast<const uint4*>(dst + 8 * v);
        x0[u] = *reinterpret_cast<const uint4*>(s0 + 8 * v);
        if (two) x1[u] = *reinterpret_cast<const uint4*>(s1 + 8 * v);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int v = (cb + u * cb_step) * 32 + lane;
        if (v >= nvec) continue;
        const float2 a = unpack_bf16x2(old[u].x), b = unpack_bf16x2(old[u].y), c = unpack_bf16x2(old[u].z),
                     d = unpack_bf16x2(old[u].w);
        float acc[8] = {a.x, a.y, b.x, b.y, c.x, c.y, d.x, d.y};
        add(acc, x0[u]);
        if (two) add(acc, x1[u]);
        store8(dst + 8 * v, acc);
      }
    }
    return;
  }
  for (int cb = cb0; cb < blocks; cb += cb_step) {
    const int v = cb * 32 + lane;
    const __nv_bfloat16* src = dout + 8 * min(v, nvec - 1);   // (idle lanes read what others read: no branch per load)
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (v < nvec) load8(dst + 8 * v, acc);
    uint32_t k = k0;
    for (int from = first, cnt = back + here, q = p + here;; q += 32) {   // rows of lanes [from, from + cnt)
      const bool more = from + cnt == 32;              // the run may go on behind these keys
      const uint32_t next = more && q + lane < n ? keys[q + lane] : 0xFFFFFFFFu;
      for (int i = 0; i < cnt; i += EMB_AHEAD) {
        uint4 x[EMB_AHEAD];
#pragma unroll
        for (int u = 0; u < EMB_AHEAD; ++u) {
          const uint32_t r = __shfl_sync(0xffffffffu, k, from + min(i + u, cnt - 1)) & mask;
          x[u] = load_now(src + static_cast<size_t>(r) * H);
        }
        if (i + EMB_AHEAD <= cnt) {
#pragma unroll
          for (int u = 0; u < EMB_AHEAD; ++u) add(acc, x[u]);
        } else {
#pragma unroll
          for (int u = 0; u < EMB_AHEAD - 1; ++u)
            if (i + u < cnt) add(acc, x[u]);
        }
      }
      if (!more) break;
      const uint32_t in_run = run_lanes(next);
      from = 0;
      cnt = in_run == 0xffffffffu ? 32 : __ffs(~in_run) - 1;
      k = next;
    }
    if (v < nvec) store8(dst + 8 * v, acc);
  }
}

inline int grid_for(size_t work_items, int threads, int max_blocks_per_sm = 16) {
  const size_t blocks = (work_items + threads - 1) / threads;
  const size_t cap = static_cast<size_t>(gfs_host::sm_count()) * max_blocks_per_sm;
  return static_cast<int>(std::max<size_t>(1, std::min(blocks, cap)));
}

}  // namespace

extern "C" {

static int rmsnorm_fwd_any(const void* x, const void* w, void* y, void* rstd, int rows, int H, float eps,
                           const DropResidual& dr, void* stream) {
  if (H & 7) return -1;
  if (rows == 0) return 0;
  const __nv_bfloat16* xp = static_cast<const __nv_bfloat16*>(x);
  const __nv_bfloat16* wp = static_cast<const __nv_bfloat16*>(w);
  __nv_bfloat16* yp = static_cast<__nv_bfloat16*>(y);
  float* rp = static_cast<float*>(rstd);
  auto launch = [&](auto kern) {
    gfs_host::launch_pdl(kern, dim3((rows + NORM_WARPS - 1) / NORM_WARPS), dim3(NORM_WARPS * 32), 0,
                         static_cast<cudaStream_t>(stream), xp, wp, yp, rp, rows, H, eps, dr);
  };
  const bool drop = dr.x != nullptr;
  if (H <= 1024) drop ? launch(rmsnorm_fwd_kernel<4, true>) : launch(rmsnorm_fwd_kernel<4, false>);
  else if (H <= 2048) drop ? launch(rmsnorm_fwd_kernel<8, true>) : launch(rmsnorm_fwd_kernel<8, false>);
  else drop ? launch(rmsnorm_fwd_kernel<16, true>) : launch(rmsnorm_fwd_kernel<16, false>);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

int gfs_rmsnorm_fwd(const void* x, const void* w, void* y, void* rstd, int rows, int H, float eps, void* stream) {
  return rmsnorm_fwd_any(x, w, y, rstd, rows, H, eps, DropResidual{}, stream);
}

// x = residual + dropout(z, p), then y = rmsnorm(x) and rstd: the bits of gfs_dropout_residual and gfs_rmsnorm_fwd.
int gfs_dropout_residual_norm(const void* z, const void* residual, void* x, const void* w, void* y, void* rstd, int rows,
                              int H, float eps, float p, unsigned long long seed, void* stream) {
  if (!(p >= 0.f) || p >= 1.f || x == nullptr) return -1;
  const DropResidual dr{static_cast<const __nv_bfloat16*>(z), static_cast<const __nv_bfloat16*>(residual),
                        static_cast<__nv_bfloat16*>(x), Dropout{p, seed}};
  return rmsnorm_fwd_any(nullptr, w, y, rstd, rows, H, eps, dr, stream);
}

// Number of fp32 elements the backward needs in `partial`: parts * H with parts from this call.
int gfs_rmsnorm_bwd_parts(int rows) {
  const int sms = gfs_host::sm_count();
  const int want = sms * 2;   // one resident wave (two CTAs per SM): 39 -> 34 us at 16384 x 768
  const int rows_per_cta = std::max(NB_WARPS, (rows + want - 1) / want);
  return (rows + rows_per_cta - 1) / rows_per_cta;
}

// (dmask null: no dropout. Few rows or H > 2048 with one: 1, nothing launched)
static int rmsnorm_bwd_any(const void* dy, const void* x, const void* w, const void* rstd, const void* dres, void* dx,
                           void* dw, void* partial, int rows, int H, int accumulate_dw, void* dmask, const Dropout& drop,
                           void* stream_) {
  if (H & 7) return -1;
  if (rows == 0) return 0;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int parts = gfs_rmsnorm_bwd_parts(rows);
  const int rows_per_cta = (rows + parts - 1) / parts;
  int warps = NB_WARPS;
  while (warps > 1 && static_cast<size_t>(warps) * H * sizeof(float) > 200 * 1024) warps >>= 1;
  const size_t smem = static_cast<size_t>(warps) * H * sizeof(float);
  if (smem > 200 * 1024) return -1;
  const __nv_bfloat16* a_dy = static_cast<const __nv_bfloat16*>(dy);
  const __nv_bfloat16* a_x = static_cast<const __nv_bfloat16*>(x);
  const __nv_bfloat16* a_w = static_cast<const __nv_bfloat16*>(w);
  const float* a_rstd = static_cast<const float*>(rstd);
  const __nv_bfloat16* a_res = static_cast<const __nv_bfloat16*>(dres);
  __nv_bfloat16* a_dx = static_cast<__nv_bfloat16*>(dx);
  float* a_part = static_cast<float*>(partial);
  auto too_much = [&](auto kern, gfs_host::SmemLimit& limit) {
    return smem > 48 * 1024 && !limit.raise(kern, 200 * 1024);
  };
  static gfs_host::SmemLimit limit_gen, limit_r4, limit_r8;
  auto ring = [&](auto nv, auto with_drop) -> int {
    constexpr int NV = decltype(nv)::value;
    constexpr bool DROP = decltype(with_drop)::value;
    static gfs_host::SmemLimit limit;
    auto kern = rmsnorm_bwd_ring_kernel<NV, DROP>;
    if (!limit.raise(kern, NormBwdShape<NV>::smem(256 * NV))) return -10;
    gfs_host::launch_pdl(kern, dim3(parts), dim3(NormBwdShape<NV>::WARPS * 32), NormBwdShape<NV>::smem(H), stream, a_dy,
                         a_x, a_w, a_rstd, a_res, a_dx, a_part, rows, H, rows_per_cta, gfs_host::status_words(),
                         static_cast<__nv_bfloat16*>(dmask), drop);
    return 0;
  };
  // Up to a row per warp and a CTA per SM nothing streams, and a row's loads into registers are there sooner than bulk
  // copies: 2.9 against 3.2 us at 512 x 256.
  const bool few = parts <= gfs_host::sm_count();
  if (dmask != nullptr && (few || H > 2048)) return 1;
  if (!few && H <= 1024) {
    const std::integral_constant<int, 4> nv;
    if (const int rc = dmask ? ring(nv, std::true_type{}) : ring(nv, std::false_type{})) return rc;
  } else if (!few && H <= 2048) {
    const std::integral_constant<int, 8> nv;
    if (const int rc = dmask ? ring(nv, std::true_type{}) : ring(nv, std::false_type{})) return rc;
  } else if (H <= 1024) {
    if (too_much(rmsnorm_bwd_reg_kernel<4>, limit_r4)) return -10;
    gfs_host::launch_pdl(rmsnorm_bwd_reg_kernel<4>, dim3(parts), dim3(warps * 32), smem, stream, a_dy, a_x, a_w, a_rstd,
                         a_res, a_dx, a_part, rows, H, rows_per_cta);
  } else if (H <= 2048) {
    if (too_much(rmsnorm_bwd_reg_kernel<8>, limit_r8)) return -10;
    gfs_host::launch_pdl(rmsnorm_bwd_reg_kernel<8>, dim3(parts), dim3(warps * 32), smem, stream, a_dy, a_x, a_w, a_rstd,
                         a_res, a_dx, a_part, rows, H, rows_per_cta);
  } else {
    if (too_much(rmsnorm_bwd_kernel, limit_gen)) return -10;
    gfs_host::launch_pdl(rmsnorm_bwd_kernel, dim3(parts), dim3(warps * 32), smem, stream, a_dy, a_x, a_w, a_rstd, a_res,
                         a_dx, a_part, rows, H, rows_per_cta);
  }
  if (cudaGetLastError() != cudaSuccess) return -11;
  if (dw == nullptr) return 0;   // the caller reduces `partial` later (gfs_rmsnorm_dw_reduce_multi)
  rmsnorm_dw_reduce_kernel<<<(H + 31) / 32, dim3(32, 32), 0, stream>>>(static_cast<const float*>(partial),
                                                              static_cast<__nv_bfloat16*>(dw), parts, H,
                                                              accumulate_dw);
  return cudaGetLastError() == cudaSuccess ? 0 : -12;
}

// dx = rmsnorm backward (+ dres); dw (bf16 [H]) written or accumulated. partial: fp32 scratch [parts*H].
int gfs_rmsnorm_bwd(const void* dy, const void* x, const void* w, const void* rstd, const void* dres, void* dx,
                    void* dw, void* partial, int rows, int H, int accumulate_dw, void* stream) {
  return rmsnorm_bwd_any(dy, x, w, rstd, dres, dx, dw, partial, rows, H, accumulate_dw, nullptr, Dropout{0.f, 0}, stream);
}

// The same, dw left in `partial`, and dmask = the gradient through dropout(p, seed) of dx: the bits of gfs_rmsnorm_bwd
// and gfs_dropout_residual. Returns 1 without a launch where only the two serve the shape.
int gfs_rmsnorm_bwd_dropout(const void* dy, const void* x, const void* w, const void* rstd, const void* dres, void* dx,
                            void* dmask, void* partial, int rows, int H, float p, unsigned long long seed, void* stream) {
  if (!(p >= 0.f) || p >= 1.f || dmask == nullptr) return -1;
  return rmsnorm_bwd_any(dy, x, w, rstd, dres, dx, nullptr, partial, rows, H, 0, dmask, Dropout{p, seed}, stream);
}

// Weight-gradient reductions of n RMSNorm layers (n <= 32) that ran gfs_rmsnorm_bwd with dw == null:
// dw_l (bf16 [H]) = (or +=) column sums of partial_l (fp32 [parts_l, H]).
int gfs_rmsnorm_dw_reduce_multi(int n, const unsigned long long* partial, const unsigned long long* dw,
                                const int* parts, const int* accumulate, int H, void* stream) {
  if (n <= 0) return 0;
  if (n > DW_MULTI_MAX) return -1;
  DwReduceBatch b{};
  for (int i = 0; i < n; ++i) {
    b.partial[i] = reinterpret_cast<const float*>(partial[i]);
    b.dw[i] = reinterpret_cast<__nv_bfloat16*>(dw[i]);
    b.parts[i] = parts[i];
    b.accumulate[i] = accumulate[i];
  }
  gfs_host::launch_pdl(rmsnorm_dw_reduce_multi_kernel, dim3((H + 31) / 32, n), dim3(32, 32), 0,
                       static_cast<cudaStream_t>(stream), b, H);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

int gfs_rope(void* x, const void* cosb, const void* sinb, int S, int B, int nh, int D, int parts, long token_stride,
             int backward, int s_offset, void* stream) {
  if ((D & 7) || (token_stride & 7)) return -1;
  const size_t total = static_cast<size_t>(S) * B * ((static_cast<size_t>(parts) * nh * D) >> 3);
  if (total == 0) return 0;
  rope_kernel<<<grid_for(total, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<__nv_bfloat16*>(x), static_cast<const float*>(cosb), static_cast<const float*>(sinb), S, B, nh * D,
      D, parts, token_stride, backward, s_offset);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// out = residual + dropout(x, p) (forward) or dx = dy * keep / (1 - p) (backward, mode 1). The keep
// mask is a pure function of (seed, element index), so the backward regenerates it instead of
// storing it; n is a multiple of 8.
int gfs_dropout_residual(const void* x, const void* residual, void* out, long long n, float p, unsigned long long seed,
                         int backward, void* stream) {
  if (n & 7) return -1;
  if (n == 0) return 0;
  if (!(p >= 0.f) || p >= 1.f) return -1;
  const long long nvec = n >> 3;
  const int blocks = static_cast<int>(std::min<long long>((nvec + 255) / 256, static_cast<long long>(gfs_host::sm_count()) * 16));
  gfs_host::launch_pdl(dropout_residual_kernel, dim3(blocks), dim3(256), 0,
                       static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(x),
                       static_cast<const __nv_bfloat16*>(residual), static_cast<__nv_bfloat16*>(out), nvec, Dropout{p, seed},
                       backward);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

int gfs_swiglu_fwd(const void* gu, void* act, int M, int I, void* stream) {
  if (I & 7) return -1;
  if (M == 0 || I == 0) return 0;
  const dim3 grid(((I >> 3) + 127) / 128, std::min(M, 32768));
  swiglu_fwd_kernel<<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(gu), static_cast<__nv_bfloat16*>(act), M, I);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

int gfs_swiglu_bwd(const void* dact, const void* gu, void* dgu, int M, int I, void* stream) {
  if (I & 7) return -1;
  if (M == 0 || I == 0) return 0;
  const dim3 grid(((I >> 3) + 127) / 128, std::min(M, 32768));
  swiglu_bwd_kernel<<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(dact), static_cast<const __nv_bfloat16*>(gu),
      static_cast<__nv_bfloat16*>(dgu), M, I);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

int gfs_embedding_fwd(const void* ids, const void* W, void* out, int B, int S, int H, int v0, int v1, int s0,
                      int s_count, void* stream) {
  if (H & 7) return -1;
  const int rows = s_count * B;
  if (rows == 0) return 0;
  const int warps = 8;
  gfs_host::launch_pdl(embedding_fwd_kernel, dim3((rows + warps - 1) / warps), dim3(warps *
                       32), 0, static_cast<cudaStream_t>(stream), static_cast<const long long*>(ids),
                       static_cast<const __nv_bfloat16*>(W), static_cast<__nv_bfloat16*>(out), B, S, H, v0, v1, s0,
                       s_count);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

int gfs_embedding_bwd(const void* sorted_ids, const void* perm, const void* dout, void* dW, int n, int H, int v0,
                      int v1, void* stream) {
  if (H & 7) return -1;
  if (n == 0) return 0;
  const int warps = 8;
  embedding_bwd_kernel<<<(n + warps - 1) / warps, warps * 32, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const long long*>(sorted_ids), static_cast<const long long*>(perm),
      static_cast<const __nv_bfloat16*>(dout), static_cast<__nv_bfloat16*>(dW), n, H, v0, v1);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

// Embedding backward with the in-library sort, in two calls so that the sort (one CTA, tens of
// microseconds, needs only the token ids) can run on a side stream during the forward pass:
//   gfs_embedding_sort_keys  ids [B, S] (int64) -> keys [S * B] uint32, sorted; returns the key
//                            shift (> 0), or -20 when the problem does not fit the single-CTA sort
//                            (n > 32768 or the key does not fit 32 bits: the caller then sorts
//                            elsewhere and uses gfs_embedding_bwd)
//   gfs_embedding_bwd_keys   dW [v1 - v0, H] += segmented sum of dout [S, B, H] in key order
//   gfs_embedding_sort_shift what the first one would return for n tokens and a vocabulary of v rows
int gfs_embedding_sort_shift(long long n, int v) {
  if (n <= 0 || v < 0) return -1;
  if (n > 32768) return -20;
  int npow2 = 2, shift = 1;
  while (npow2 < n) { npow2 <<= 1; ++shift; }
  return (static_cast<unsigned long long>(v) << shift) >= 0xFFFFFFFFull ? -20 : shift;
}

int gfs_embedding_sort_keys(const void* ids_bs, void* keys, int B, int S, int v0, int v1, void* stream_) {
  const long long n64 = static_cast<long long>(B) * S;
  const int shift = gfs_embedding_sort_shift(n64, v1 - v0);
  if (shift < 0) return shift;
  const int n = static_cast<int>(n64), npow2 = 1 << shift;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  static gfs_host::SmemLimit limit;
  if (!limit.raise(embedding_sort_kernel, 32768 * 4)) return -10;
  embedding_sort_kernel<<<1, SORT_THREADS, npow2 * sizeof(uint32_t), stream>>>(
      static_cast<const long long*>(ids_bs), static_cast<uint32_t*>(keys), n, npow2, shift, B, S, v0, v1);
  return cudaGetLastError() == cudaSuccess ? shift : -11;
}

int gfs_embedding_bwd_keys(const void* keys, const void* dout, void* dW, int n, int H, int shift, void* stream_) {
  if ((H & 7) || shift <= 0 || shift > 31) return -1;
  if (n == 0) return 0;
  const int warps = 8;
  // as many warps per position as one wave of the chip (32 per SM) has room for, and columns for
  const int share = std::max(1, std::min((H / 8 + 31) / 32, gfs_host::sm_count() * 32 / n));
  embedding_bwd_keys_kernel<<<dim3((n + warps - 1) / warps, share), warps * 32, 0, static_cast<cudaStream_t>(stream_)>>>(
      static_cast<const uint32_t*>(keys), static_cast<const __nv_bfloat16*>(dout), static_cast<__nv_bfloat16*>(dW), n, H,
      shift);
  return cudaGetLastError() == cudaSuccess ? 0 : -11;
}

}  // extern "C"
