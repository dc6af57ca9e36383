// RMSNorm forward (+ fused residual add) and backward for sm_100a, contiguous rows or the heads of a
// strided projection.
//
// Both directions move each row once and are bound by memory; what the forms below differ in is how the
// row's bytes are kept in flight.
//   rows of up to 512 channels    a warp (or 8 or 16 lanes of one) per row, the row in registers, the
//                                 next row's loads issued before this one's reduction
//   longer rows                   a 256-thread block per row; bulk copies bring the block's next rows
//                                 into a ring in shared memory, so the reduction and its barrier never
//                                 wait for memory latency
// The weight gradient is summed in registers over all rows of a thread, then over the block in shared
// memory, and leaves as one 16-byte vector reduction per four columns and block: scalar atomics with a
// 32-byte stride between lanes cost more than the rows themselves (37 us for 768 x 256).
//
// Measured (one B200, kernel durations with the L2 flushed before each launch; before: one 256-thread block per
// row, next row prefetched in registers):
//   forward   8192 x 4096           33 -> 26 us (5.1 TB/s)    + residual add     52 -> 47 us (5.7 TB/s)
//   backward  8192 x 4096           89 -> 41 us (4.9 TB/s)    added to dx       110 -> 47 us (5.7 TB/s)
//   backward   768 x 256            37 -> 3.3 us              1999 x 2048        43 -> 13 us
//   1999 x 16 rows of 128, forward  68 -> 7 us                backward           92 -> 8 us
// Heads of a projection are normalised where they lie: no copy to contiguous rows and back.
//
// The math follows the reference's pure-PyTorch definition
// (packages/workloads/src/shadowspill_workloads/models/shared/decoder.py:18).
#include "sm100_ptx.cuh"
#include "launchers.h"

#include <stdint.h>

namespace ss {

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ void norm_unpack8(const uint4& u, float (&f)[8]) {
  const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), c = unpack_bf16(u.z), d = unpack_bf16(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 norm_pack8(const float (&f)[8]) {
  return make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
}
template <int LANES>
__device__ __forceinline__ float lanes_sum(float v) {
#pragma unroll
  for (int o = LANES / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// Four neighbouring columns of a weight gradient; off a 16-byte boundary one by one.
__device__ __forceinline__ void red_add_v4(float* p, float4 v) {
  if (reinterpret_cast<uintptr_t>(p) & 15) {
    atomicAdd(p, v.x); atomicAdd(p + 1, v.y); atomicAdd(p + 2, v.z); atomicAdd(p + 3, v.w);
    return;
  }
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
               : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_dst), "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ uint4 ld_shared_u4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}

constexpr int NORM_THREADS = 256;
constexpr int NORM_MAX_SMEM = 226 * 1024;   // the block also has some static shared memory
// rows in flight per block of the long-row form; three where four rows of three tensors do not fit
__host__ __device__ constexpr int norm_ring(int vpt) { return vpt > 4 ? 3 : 4; }

// ============================================================================ rows of <= 512 channels
// Row r of a tensor is head r % heads of token r / heads: `ld` elements between tokens, D between heads.
struct NormRows {
  bf16* x; long long ldx;
  bf16* y; long long ldy;               // normalised rows, or dx
  const bf16* z; long long ldz;         // backward: gy
  bf16* raw; long long ldraw;           // forward: a copy of the input rows, optional
  const bf16* delta;                    // forward: folded into x first; x is rewritten (rows of one head)
  const bf16* w;
  float* rstd;                          // [rows]
  float* dw;                            // [D] fp32, accumulated; optional
  long long rows;
  int heads, D, zero_centered, accumulate;
  float eps;
  __device__ __forceinline__ long long at(long long r, long long ld) const {
    if (heads == 1) return r * ld;
    const unsigned t = static_cast<unsigned>(r) / static_cast<unsigned>(heads);
    return t * ld + (static_cast<unsigned>(r) - t * heads) * static_cast<long long>(D);
  }
};

// The row's sum is formed the same way with and without DELTA, so a residual add that one caller fuses and
// another does not gives both the same bits.
template <int LANES, int VPT, bool DELTA>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_fwd_short_kernel(const NormRows p) {
  chain_wait();
  chain_release();
  const int lane = threadIdx.x & (LANES - 1), nv = p.D >> 3;
  const float wofs = p.zero_centered ? 1.f : 0.f;
  uint4 wq[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = lane + i * LANES;
    wq[i] = c < nv ? reinterpret_cast<const uint4*>(p.w)[c] : make_uint4(0, 0, 0, 0);
  }
  const long long step = static_cast<long long>(gridDim.x) * (NORM_THREADS / LANES);
  uint4 xq[VPT], xn[VPT], dq[VPT], dn[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) xq[i] = xn[i] = dq[i] = dn[i] = make_uint4(0, 0, 0, 0);
  auto fetch = [&](long long r, uint4 (&o)[VPT], uint4 (&d)[VPT]) {
    const uint4* xr = reinterpret_cast<const uint4*>(p.x + p.at(r, p.ldx));
    const uint4* er = DELTA ? reinterpret_cast<const uint4*>(p.delta + r * p.D) : nullptr;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      if (lane + i * LANES >= nv) continue;
      o[i] = xr[lane + i * LANES];
      if (DELTA) d[i] = er[lane + i * LANES];
    }
  };
  const long long r0 = blockIdx.x * static_cast<long long>(NORM_THREADS / LANES) + threadIdx.x / LANES;
  if (r0 < p.rows) fetch(r0, xq, dq);
  // a warp's lanes stay together through the shuffles: rows past the end are computed and not stored
  for (long long r = r0, base = blockIdx.x * static_cast<long long>(NORM_THREADS / LANES); base < p.rows;
       r += step, base += step) {
    if (r + step < p.rows) fetch(r + step, xn, dn);
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      float v[8];
      norm_unpack8(xq[i], v);
      if (DELTA) {
        float d[8];
        norm_unpack8(dq[i], d);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] += d[e];
        // The residual stream is kept in bf16: round once here so that the
        // normalised value and the stored stream agree.
        xq[i] = norm_pack8(v);
        norm_unpack8(xq[i], v);
        if (r < p.rows && lane + i * LANES < nv)
          reinterpret_cast<uint4*>(p.x + p.at(r, p.ldx))[lane + i * LANES] = xq[i];
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += v[e] * v[e];
    }
    const float rs = rsqrtf(lanes_sum<LANES>(ss) / static_cast<float>(p.D) + p.eps);
    if (r < p.rows) {
      if (lane == 0 && p.rstd) p.rstd[r] = rs;
      uint4* yr = reinterpret_cast<uint4*>(p.y + p.at(r, p.ldy));
      uint4* rr = p.raw ? reinterpret_cast<uint4*>(p.raw + p.at(r, p.ldraw)) : nullptr;
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        const int c = lane + i * LANES;
        if (c >= nv) continue;
        float v[8], ww[8], o[8];
        norm_unpack8(xq[i], v);
        norm_unpack8(wq[i], ww);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = v[e] * rs * (ww[e] + wofs);
        yr[c] = norm_pack8(o);
        if (rr) rr[c] = xq[i];
      }
    }
#pragma unroll
    for (int i = 0; i < VPT; ++i) { xq[i] = xn[i]; dq[i] = dn[i]; }
  }
}

// dx = rstd * (g*w - xhat * mean(g*w*xhat)),  dw += sum_t g * xhat; dx is ADDED to its old value when
// `accumulate` (the residual stream's gradient).
template <int LANES, int VPT>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_bwd_short_kernel(const NormRows p) {
  chain_wait();
  chain_release();
  constexpr int GROUPS = NORM_THREADS / LANES;
  __shared__ __align__(16) float s_dw[GROUPS * LANES * VPT * 8];
  const int lane = threadIdx.x & (LANES - 1), nv = p.D >> 3;
  const float wofs = p.zero_centered ? 1.f : 0.f;
  uint4 wq[VPT];
  float acc[VPT][8];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = lane + i * LANES;
    wq[i] = c < nv ? reinterpret_cast<const uint4*>(p.w)[c] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[i][e] = 0.f;
  }
  const long long step = static_cast<long long>(gridDim.x) * GROUPS;
  uint4 xq[VPT], gq[VPT], xn[VPT], gn[VPT];
  float rs = 0.f, rn = 0.f;
#pragma unroll
  for (int i = 0; i < VPT; ++i) xq[i] = gq[i] = xn[i] = gn[i] = make_uint4(0, 0, 0, 0);
  auto fetch = [&](long long r, uint4 (&xo)[VPT], uint4 (&go)[VPT], float& ro) {
    const uint4* xr = reinterpret_cast<const uint4*>(p.x + p.at(r, p.ldx));
    const uint4* gr = reinterpret_cast<const uint4*>(p.z + p.at(r, p.ldz));
    ro = p.rstd[r];
#pragma unroll
    for (int i = 0; i < VPT; ++i)
      if (lane + i * LANES < nv) { xo[i] = xr[lane + i * LANES]; go[i] = gr[lane + i * LANES]; }
  };
  const long long r0 = blockIdx.x * static_cast<long long>(GROUPS) + threadIdx.x / LANES;
  if (r0 < p.rows) fetch(r0, xq, gq, rs);
  for (long long r = r0, base = blockIdx.x * static_cast<long long>(GROUPS); base < p.rows; r += step, base += step) {
    if (r + step < p.rows) fetch(r + step, xn, gn, rn);
    const bool in = r < p.rows;
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      float xv[8], gv[8], ww[8];
      norm_unpack8(xq[i], xv);
      norm_unpack8(gq[i], gv);
      norm_unpack8(wq[i], ww);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float xh = xv[e] * rs;
        if (in) acc[i][e] += gv[e] * xh;
        dot += gv[e] * (ww[e] + wofs) * xh;
      }
    }
    const float mean = lanes_sum<LANES>(dot) / static_cast<float>(p.D);
    if (in) {
      uint4* dr = reinterpret_cast<uint4*>(p.y + p.at(r, p.ldy));
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        const int c = lane + i * LANES;
        if (c >= nv) continue;
        float xv[8], gv[8], ww[8], o[8];
        norm_unpack8(xq[i], xv);
        norm_unpack8(gq[i], gv);
        norm_unpack8(wq[i], ww);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = rs * (gv[e] * (ww[e] + wofs) - xv[e] * rs * mean);
        if (p.accumulate) {
          float prev[8];
          norm_unpack8(dr[c], prev);
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] += prev[e];
        }
        dr[c] = norm_pack8(o);
      }
    }
    rs = rn;
#pragma unroll
    for (int i = 0; i < VPT; ++i) { xq[i] = xn[i]; gq[i] = gn[i]; }
  }
  if (p.dw == nullptr) return;
  float* mine = s_dw + (threadIdx.x / LANES) * (LANES * VPT * 8);
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = lane + i * LANES;
    *reinterpret_cast<float4*>(mine + c * 8) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    *reinterpret_cast<float4*>(mine + c * 8 + 4) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
  }
  __syncthreads();
  for (int q = threadIdx.x; q < (p.D >> 2); q += NORM_THREADS) {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int g = 0; g < GROUPS; ++g) {
      const float4 v = *reinterpret_cast<const float4*>(s_dw + g * (LANES * VPT * 8) + q * 4);
      t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
    }
    red_add_v4(p.dw + q * 4, t);
  }
}

// ============================================================================ longer rows
// Sum over the block of one value per thread; `red` has two sets of eight, used in turn, so one barrier
// per row is enough. After it every thread has also read its part of the row from the ring. False for the
// whole block where a thread's wait for the row ran out (`ok`).
__device__ __forceinline__ bool row_sum(bool ok, float v, float (*red)[8], int turn, float& sum) {
  v = lanes_sum<32>(v);
  if ((threadIdx.x & 31) == 0) red[turn][threadIdx.x >> 5] = v;
  ok = __syncthreads_and(ok);
  const float4 a = *reinterpret_cast<const float4*>(red[turn]), b = *reinterpret_cast<const float4*>(red[turn] + 4);
  sum = ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w));
  return ok;
}

// The ring of one block: `parts` tensors of D channels each per row.
struct NormRing {
  uint32_t base;
  uint64_t* full;
  int D, parts;
  long long T;
  int* status;
  __device__ __forceinline__ uint32_t part(int s, int k) const { return base + (s * parts + k) * (D * 2); }
  __device__ __forceinline__ void load(int s, long long row, const bf16* a, const bf16* b, const bf16* c) const {
    if (row >= T) return;
    mbar_expect_tx(&full[s], parts * D * 2);
    bulk_load(part(s, 0), a + row * D, D * 2, &full[s]);
    if (parts > 1) bulk_load(part(s, 1), b + row * D, D * 2, &full[s]);
    if (parts > 2) bulk_load(part(s, 2), c + row * D, D * 2, &full[s]);
  }
  // Row `it` of the block has arrived.
  template <int STAGES>
  __device__ __forceinline__ bool wait(int it) const {
    return mbar_wait(&full[it % STAGES], (it / STAGES) & 1, status, KS_TIMEOUT_FULL);
  }
  // The copies in flight when row `it` (global row `row`) failed get one more bounded wait, so that none lands
  // in memory that another block has been given.
  template <int STAGES>
  __device__ __forceinline__ void drain(int it, long long row) const {
#pragma unroll 1
    for (int i = 0; i < STAGES && row < T; ++i, ++it, row += gridDim.x) wait<STAGES>(it);
    __syncthreads();
  }
};

template <int VPT>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_fwd_long_kernel(bf16* x, const bf16* delta, const bf16* w, bf16* y, float* rstd,
                        long long T, int D, float eps, int zero_centered, int* status) {
  chain_wait();
  chain_release();
  extern __shared__ __align__(128) uint8_t ring_smem[];
  __shared__ __align__(16) float red[2][8];
  constexpr int NORM_RING = norm_ring(VPT);
  __shared__ __align__(8) uint64_t full[NORM_RING];
  const int nv = D >> 3;
  const float wofs = zero_centered ? 1.f : 0.f;
  const NormRing ring{smem_u32(ring_smem), full, D, delta ? 2 : 1, T, status};
  if (threadIdx.x == 0) {
    for (int s = 0; s < NORM_RING; ++s) mbar_init(&full[s], 1);
    mbar_fence_init();
    fence_async_proxy();
    for (int s = 0; s < NORM_RING; ++s)
      ring.load(s, blockIdx.x + static_cast<long long>(s) * gridDim.x, x, delta, nullptr);
  }
  uint4 wq[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = threadIdx.x + i * NORM_THREADS;
    wq[i] = c < nv ? reinterpret_cast<const uint4*>(w)[c] : make_uint4(0, 0, 0, 0);
  }
  __syncthreads();
  int it = 0;
  for (long long row = blockIdx.x; row < T; row += gridDim.x, ++it) {
    const int s = it % NORM_RING;
    const bool ok = ring.wait<NORM_RING>(it);
    uint4 xq[VPT];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = threadIdx.x + i * NORM_THREADS;
      xq[i] = make_uint4(0, 0, 0, 0);
      if (c >= nv) continue;
      xq[i] = ld_shared_u4(ring.part(s, 0) + c * 16);
      float v[8];
      norm_unpack8(xq[i], v);
      if (delta) {
        float d[8];
        norm_unpack8(ld_shared_u4(ring.part(s, 1) + c * 16), d);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] += d[e];
        // The residual stream is kept in bf16: round once here so that the
        // normalised value and the stored stream agree.
        xq[i] = norm_pack8(v);
        norm_unpack8(xq[i], v);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) ss += v[e] * v[e];
    }
    float sum;
    if (!row_sum(ok, ss, red, it & 1, sum)) return ring.drain<NORM_RING>(it, row);   // reported; this row is not stored
    const float rs = rsqrtf(sum / static_cast<float>(D) + eps);
    if (threadIdx.x == 0) {
      ring.load(s, row + static_cast<long long>(NORM_RING) * gridDim.x, x, delta, nullptr);
      if (rstd) rstd[row] = rs;
    }
    uint4* yr = reinterpret_cast<uint4*>(y + row * D);
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = threadIdx.x + i * NORM_THREADS;
      if (c >= nv) continue;
      float v[8], ww[8], o[8];
      norm_unpack8(xq[i], v);
      norm_unpack8(wq[i], ww);
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = v[e] * rs * (ww[e] + wofs);
      if (delta) reinterpret_cast<uint4*>(x + row * D)[c] = xq[i];
      yr[c] = norm_pack8(o);
    }
  }
}

template <int VPT>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_bwd_long_kernel(const bf16* x, const bf16* w, const bf16* gy, const float* rstd,
                        bf16* dx, float* dw, long long T, int D, int zero_centered, int accumulate,
                        int* status) {
  chain_wait();
  chain_release();
  extern __shared__ __align__(128) uint8_t ring_smem[];
  __shared__ __align__(16) float red[2][8];
  constexpr int NORM_RING = norm_ring(VPT);
  __shared__ __align__(8) uint64_t full[NORM_RING];
  const int nv = D >> 3;
  const float wofs = zero_centered ? 1.f : 0.f;
  const NormRing ring{smem_u32(ring_smem), full, D, accumulate ? 3 : 2, T, status};
  if (threadIdx.x == 0) {
    for (int s = 0; s < NORM_RING; ++s) mbar_init(&full[s], 1);
    mbar_fence_init();
    fence_async_proxy();
    for (int s = 0; s < NORM_RING; ++s)
      ring.load(s, blockIdx.x + static_cast<long long>(s) * gridDim.x, x, gy, dx);
  }
  uint4 wq[VPT];
  float acc[VPT][8];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = threadIdx.x + i * NORM_THREADS;
    wq[i] = c < nv ? reinterpret_cast<const uint4*>(w)[c] : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[i][e] = 0.f;
  }
  __syncthreads();
  int it = 0;
  float rn = blockIdx.x < T ? rstd[blockIdx.x] : 0.f;
  for (long long row = blockIdx.x; row < T; row += gridDim.x, ++it) {
    const int s = it % NORM_RING;
    const float rs = rn;
    if (row + gridDim.x < T) rn = rstd[row + gridDim.x];
    const bool ok = ring.wait<NORM_RING>(it);
    uint4 xq[VPT], gq[VPT], pq[VPT];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = threadIdx.x + i * NORM_THREADS;
      if (c >= nv) continue;
      xq[i] = ld_shared_u4(ring.part(s, 0) + c * 16);
      gq[i] = ld_shared_u4(ring.part(s, 1) + c * 16);
      if (accumulate) pq[i] = ld_shared_u4(ring.part(s, 2) + c * 16);
      float xv[8], gv[8], ww[8];
      norm_unpack8(xq[i], xv);
      norm_unpack8(gq[i], gv);
      norm_unpack8(wq[i], ww);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float xh = xv[e] * rs;
        acc[i][e] += gv[e] * xh;
        dot += gv[e] * (ww[e] + wofs) * xh;
      }
    }
    float sum;
    if (!row_sum(ok, dot, red, it & 1, sum)) return ring.drain<NORM_RING>(it, row);  // reported; neither row nor dw is stored
    const float mean = sum / static_cast<float>(D);
    if (threadIdx.x == 0) ring.load(s, row + static_cast<long long>(NORM_RING) * gridDim.x, x, gy, dx);
    uint4* dr = reinterpret_cast<uint4*>(dx + row * D);
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int c = threadIdx.x + i * NORM_THREADS;
      if (c >= nv) continue;
      float xv[8], gv[8], ww[8], o[8];
      norm_unpack8(xq[i], xv);
      norm_unpack8(gq[i], gv);
      norm_unpack8(wq[i], ww);
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = rs * (gv[e] * (ww[e] + wofs) - xv[e] * rs * mean);
      if (accumulate) {
        float prev[8];
        norm_unpack8(pq[i], prev);
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] += prev[e];
      }
      dr[c] = norm_pack8(o);
    }
  }
  if (dw == nullptr || it == 0) return;
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int c = threadIdx.x + i * NORM_THREADS;
    if (c >= nv) continue;
    red_add_v4(dw + c * 8, make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
    red_add_v4(dw + c * 8 + 4, make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]));
  }
}

// ============================================================================ launchers
static inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Shared memory and grid of the long-row form: as many blocks per SM as the rings fit, up to `most`, and
// `rows` rows or more to each block beyond one per SM.
struct LongShape {
  int smem, grid;
  LongShape(long long T, int D, int parts, int ring, int most, int rows) : smem(ring * parts * D * 2) {
    int per_sm = 220 * 1024 / smem;
    per_sm = per_sm < 1 ? 1 : per_sm > most ? most : per_sm;
    long long blocks = T / rows < 148 ? 148 : T / rows;
    if (blocks > 148 * per_sm) blocks = 148 * per_sm;
    grid = static_cast<int>(T < blocks ? T : blocks);
  }
};

enum { FWD, FWD_DELTA, BWD };
template <int KIND, int LANES, int VPT>
static int launch_short_as(const NormRows& p, cudaStream_t s) {
  const long long per = NORM_THREADS / LANES, blocks = (p.rows + per - 1) / per;
  const long long cap = 148 * (KIND == BWD ? 4 : 8);
  const int grid = static_cast<int>(blocks < cap ? blocks : cap);
  if constexpr (KIND == BWD) launch_chained(rmsnorm_bwd_short_kernel<LANES, VPT>, grid, NORM_THREADS, 0, s, p);
  else launch_chained(rmsnorm_fwd_short_kernel<LANES, VPT, KIND == FWD_DELTA>, grid, NORM_THREADS, 0, s, p);
  return static_cast<int>(cudaGetLastError());
}
template <int KIND>
static int launch_short(const NormRows& p, cudaStream_t s) {
  if (p.D <= 64) return launch_short_as<KIND, 8, 1>(p, s);
  if (p.D <= 128) return launch_short_as<KIND, 16, 1>(p, s);
  if (p.D <= 256) return launch_short_as<KIND, 32, 1>(p, s);
  return launch_short_as<KIND, 32, 2>(p, s);
}

}  // namespace ss

extern "C" {
using namespace ss;

int ss_rmsnorm_fwd(void* x, const void* delta, const void* w, void* y, float* rstd, int T, int D,
                   float eps, int zero_centered, int* status, void* stream) {
  if (D % 8 || D <= 0 || D > 8192) return -2;
  if (!aligned16(x) || !aligned16(delta) || !aligned16(w) || !aligned16(y)) return -2;
  if (T <= 0) return 0;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (D <= 512) {
    NormRows p{};
    p.x = (bf16*)x; p.delta = (const bf16*)delta; p.y = (bf16*)y; p.w = (const bf16*)w; p.rstd = rstd;
    p.ldx = p.ldy = D; p.rows = T; p.heads = 1; p.D = D; p.zero_centered = zero_centered; p.eps = eps;
    return delta ? launch_short<FWD_DELTA>(p, s) : launch_short<FWD>(p, s);
  }
  auto go = [&](auto kern, SmemOptIn& opt_in, int vpt) -> int {
    const LongShape shape(T, D, delta ? 2 : 1, norm_ring(vpt), 4, 1);
    if (int e = opt_in.ensure(kern, NORM_MAX_SMEM)) return e;
    launch_chained(kern, shape.grid, NORM_THREADS, shape.smem, s, (bf16*)x, (const bf16*)delta, (const bf16*)w, (bf16*)y,
                   rstd, T, D, eps, zero_centered, status);
    return static_cast<int>(cudaGetLastError());
  };
  static SmemOptIn o1, o2, o4;
  if (D <= 2048) return go(rmsnorm_fwd_long_kernel<1>, o1, 1);
  if (D <= 4096) return go(rmsnorm_fwd_long_kernel<2>, o2, 2);
  return go(rmsnorm_fwd_long_kernel<4>, o4, 4);
}

int ss_rmsnorm_bwd(const void* x, const void* w, const void* gy, const float* rstd, void* dx,
                   float* dw, int T, int D, int zero_centered, int accumulate, int* status, void* stream) {
  if (D % 8 || D <= 0 || D > 12288) return -2;
  if (!aligned16(x) || !aligned16(w) || !aligned16(gy) || !aligned16(dx)) return -2;
  if (T <= 0) return 0;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (D <= 512) {
    NormRows p{};
    p.x = (bf16*)x; p.z = (const bf16*)gy; p.y = (bf16*)dx; p.w = (const bf16*)w;
    p.rstd = const_cast<float*>(rstd); p.dw = dw;
    p.ldx = p.ldy = p.ldz = D; p.rows = T; p.heads = 1; p.D = D; p.zero_centered = zero_centered;
    p.accumulate = accumulate;
    return launch_short<BWD>(p, s);
  }
  auto go = [&](auto kern, SmemOptIn& opt_in, int vpt) -> int {
    const LongShape shape(T, D, accumulate ? 3 : 2, norm_ring(vpt), 4, 8);   // eight rows to a weight-gradient flush
    if (int e = opt_in.ensure(kern, NORM_MAX_SMEM)) return e;
    launch_chained(kern, shape.grid, NORM_THREADS, shape.smem, s, (const bf16*)x, (const bf16*)w, (const bf16*)gy, rstd,
                   (bf16*)dx, dw, T, D, zero_centered, accumulate, status);
    return static_cast<int>(cudaGetLastError());
  };
  static SmemOptIn o1, o2, o4, o6;
  if (D <= 2048) return go(rmsnorm_bwd_long_kernel<1>, o1, 1);
  if (D <= 4096) return go(rmsnorm_bwd_long_kernel<2>, o2, 2);
  if (D <= 8192) return go(rmsnorm_bwd_long_kernel<4>, o4, 4);
  return go(rmsnorm_bwd_long_kernel<6>, o6, 6);
}

// RMSNorm of `heads` adjacent heads of D channels in every row of a [T, ld] buffer, one weight for all
// heads. x and y may be the same buffer; `raw` (optional) receives a copy of the input heads.
// rstd is [T * heads].
int ss_headnorm_fwd(const void* x, long long ldx, const void* w, void* y, long long ldy, void* raw, long long ldraw,
                    float* rstd, int T, int heads, int D, float eps, int zero_centered, void* stream) {
  if (D % 8 || D <= 0 || D > 512 || heads <= 0 || ldx % 8 || ldy % 8 || ldraw % 8) return -2;
  if (!aligned16(x) || !aligned16(w) || !aligned16(y) || !aligned16(raw)) return -2;
  if (static_cast<long long>(T) * heads > 0x7fffffffLL) return -2;
  if (T <= 0) return 0;
  NormRows p{};
  p.x = (bf16*)x; p.ldx = ldx; p.y = (bf16*)y; p.ldy = ldy; p.raw = (bf16*)raw; p.ldraw = ldraw;
  p.w = (const bf16*)w; p.rstd = rstd; p.rows = static_cast<long long>(T) * heads; p.heads = heads; p.D = D;
  p.zero_centered = zero_centered; p.eps = eps;
  return launch_short<FWD>(p, reinterpret_cast<cudaStream_t>(stream));
}

// Backward of ss_headnorm_fwd; dx may be gy. dw (fp32 [D]) is accumulated.
int ss_headnorm_bwd(const void* x, long long ldx, const void* w, const void* gy, long long ldg, const float* rstd,
                    void* dx, long long lddx, float* dw, int T, int heads, int D, int zero_centered, void* stream) {
  if (D % 8 || D <= 0 || D > 512 || heads <= 0 || ldx % 8 || ldg % 8 || lddx % 8) return -2;
  if (!aligned16(x) || !aligned16(w) || !aligned16(gy) || !aligned16(dx)) return -2;
  if (static_cast<long long>(T) * heads > 0x7fffffffLL) return -2;
  if (T <= 0) return 0;
  NormRows p{};
  p.x = (bf16*)x; p.ldx = ldx; p.z = (const bf16*)gy; p.ldz = ldg; p.y = (bf16*)dx; p.ldy = lddx;
  p.w = (const bf16*)w; p.rstd = const_cast<float*>(rstd); p.dw = dw;
  p.rows = static_cast<long long>(T) * heads; p.heads = heads; p.D = D; p.zero_centered = zero_centered;
  return launch_short<BWD>(p, reinterpret_cast<cudaStream_t>(stream));
}

}  // extern "C"
