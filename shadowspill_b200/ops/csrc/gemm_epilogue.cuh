// Epilogue store of the tcgen05 GEMMs: 32 accumulator rows x 32 columns per warp and step.
//
// A thread owns an accumulator row, so stores straight from its registers put 16 bytes into each of 32
// lines per instruction; a 128 x 256 bf16 tile then takes 4096 line requests. The block goes through
// 2 KiB of XOR-swizzled shared memory instead, and every instruction moves whole 32-byte sectors (bf16)
// or 64-byte runs (fp32) of eight rows. It stays fp32 up to the final rounding, also where the old C is
// added. Eight warps share a tile: with four the chain of TMEM read, staging and store of 256 columns
// outlasts a short contraction.
// Measured against four warps storing from registers: head weight gradient 128256 x 4096 over 2 x 2048 rows,
// second added to the first 3.38 -> 2.68 ms; four weight gradients of a 2048-wide layer over 1999 rows, added,
// 306 -> 185 us; expert weight gradients of 128 experts with 62 rows each 513 -> 410 us; 63 products of a
// 256-wide model 707 -> 634 us. (Staging with four warps was slower than no staging: 687 us and 862 us.)
#pragma once
#include "sm100_ptx.cuh"

namespace ss {

constexpr int EPI_WARPS = 8;
constexpr int EPI_WARP_STAGE = 32 * 64;       // bytes of staging per epilogue warp

// C(row0 + [0,32), col0 + [0,32)) (+)= alpha * r; rows >= M and columns >= N are not touched (N % 8 == 0).
// `stage`: this warp's staging bytes (shared::cta address, 128-byte aligned). All 32 lanes call it.
template <typename OUT>
__device__ __forceinline__ void epilogue_store_32x32(uint32_t stage, const uint32_t (&r)[32], OUT* C, int accumulate,
                                                     float alpha, long long ldc, int row0, int M, int col0, int N) {
  constexpr bool F32 = sizeof(OUT) == 4;
  const int lane = threadIdx.x & 31;
  const int sub = lane >> 2, chunk = lane & 3;            // this lane's row in a group of eight, its 4 columns
  OUT* dst = C + static_cast<long long>(row0 + sub) * ldc + col0 + chunk * 4;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const bool col_in = col0 + h * 16 + chunk * 4 < N;
    float4 old[4];
    if (accumulate) {                                     // in flight while the block is staged
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        old[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!col_in || row0 + sub + i * 8 >= M) continue;
        const OUT* src = dst + static_cast<long long>(i) * 8 * ldc + h * 16;
        if constexpr (F32) {
          old[i] = *reinterpret_cast<const float4*>(src);
        } else {
          const uint2 o = *reinterpret_cast<const uint2*>(src);
          const float2 a = unpack_bf16(o.x), b = unpack_bf16(o.y);
          old[i] = make_float4(a.x, a.y, b.x, b.y);
        }
      }
    }
    __syncwarp();                                         // the half before this one has been read
#pragma unroll
    for (int i = 0; i < 4; ++i)
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage + lane * 64 + ((i ^ ((lane >> 1) & 3)) << 4)),
                   "r"(r[h * 16 + 4 * i]), "r"(r[h * 16 + 4 * i + 1]), "r"(r[h * 16 + 4 * i + 2]),
                   "r"(r[h * 16 + 4 * i + 3])
                   : "memory");
    __syncwarp();
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int srow = i * 8 + sub;
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                   : "=f"(v[i].x), "=f"(v[i].y), "=f"(v[i].z), "=f"(v[i].w)
                   : "r"(stage + srow * 64 + ((chunk ^ ((srow >> 1) & 3)) << 4)) : "memory");
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[i].x *= alpha; v[i].y *= alpha; v[i].z *= alpha; v[i].w *= alpha;
      if (accumulate) { v[i].x += old[i].x; v[i].y += old[i].y; v[i].z += old[i].z; v[i].w += old[i].w; }
      if (!col_in || row0 + sub + i * 8 >= M) continue;
      OUT* to = dst + static_cast<long long>(i) * 8 * ldc + h * 16;
      if constexpr (F32) *reinterpret_cast<float4*>(to) = v[i];
      else *reinterpret_cast<uint2*>(to) = make_uint2(pack_bf16(v[i].x, v[i].y), pack_bf16(v[i].z, v[i].w));
    }
  }
}

}  // namespace ss
