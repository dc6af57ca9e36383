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
#include "swiglu_math.cuh"

namespace ss {

//
// A bf16 output that nothing is added to leaves by TMA instead, 64 columns of the tile's 128 rows at a time from a
// swizzled block of shared memory: half the shared-memory passes, whole 128-byte lines, and no address or edge
// arithmetic in the warps. Expert weight gradients as above 402 -> 250 us (1.2 GB at 4.8 TB/s); for 64 experts with
// 1,024 rows each 749 -> 710 us.
constexpr int EPI_WARPS = 8;
constexpr int EPI_WARP_STAGE = 32 * 64;       // bytes of staging per epilogue warp
constexpr int EPI_BLOCK = 128 * 128;          // 128 rows of 64 bf16
constexpr int EPI_STAGE = 2 * EPI_BLOCK;      // one block for each half of a tile's columns, or the warps' staging
static_assert(EPI_WARPS * EPI_WARP_STAGE <= EPI_STAGE, "the warps' staging is the smaller");

// What a GEMM does with its products besides storing them.
//   EPI_PLAIN       C (+)= alpha * product; the values added are read from `src` (C itself, or a residual of C's shape)
//   EPI_SWIGLU      B holds the rows of a gate matrix and those of an up matrix F rows behind: a tile takes as many of
//                   the one as of the other, and what leaves is h = silu(gate) * up [M, F] and, unless C is null, the
//                   two themselves, [M, 2F]
//   EPI_SWIGLU_BWD  the products are the gradient of h; with gate and up read from `src` [M, 2F], what leaves is
//                   their gradient, C [M, 2F]
// h and the gradients take gate, up and dh rounded to bf16, so that they have the bits of the separate kernels.
// Those moved 6 bytes a value of h forward and 10 backward beside the GEMMs' own (8,192 tokens, 14,336 wide:
// 135 and 202 us), and without gate and up kept the GEMM stores a third.
enum : int { EPI_PLAIN = 0, EPI_SWIGLU = 1, EPI_SWIGLU_BWD = 2 };

struct EpiArgs {
  const void* src;
  long long ldsrc;
  __nv_bfloat16* h;
  long long ldh;
};

// Half h of a warp's 32 x 32 block through its staging bytes: a thread's row in, for each of four groups of eight rows
// the four columns of chunk (lane & 3) of row (lane >> 2) out.
__device__ __forceinline__ void stage_half(uint32_t stage, const uint32_t (&r)[32], int h, float4 (&v)[4]) {
  const int lane = threadIdx.x & 31, sub = lane >> 2, chunk = lane & 3;
  __syncwarp();                                           // what was staged before has been read
#pragma unroll
  for (int i = 0; i < 4; ++i)
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(stage + lane * 64 + ((i ^ ((lane >> 1) & 3)) << 4)),
                 "r"(r[h * 16 + 4 * i]), "r"(r[h * 16 + 4 * i + 1]), "r"(r[h * 16 + 4 * i + 2]),
                 "r"(r[h * 16 + 4 * i + 3])
                 : "memory");
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int srow = i * 8 + sub;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[i].x), "=f"(v[i].y), "=f"(v[i].z), "=f"(v[i].w)
                 : "r"(stage + srow * 64 + ((chunk ^ ((srow >> 1) & 3)) << 4)) : "memory");
  }
}

// C(row0 + [0,32), col0 + [0,32)) = alpha * r, plus `add` there where `accumulate` is set; rows >= M and columns >= N are
// not touched (N % 8 == 0). The flag is the kernel's parameter: as a pointer that is null or not, 768 x 1024 over 256 in
// bf16 took 7.9 us, and takes 7.15.
// `stage`: this warp's staging bytes (shared::cta address, 128-byte aligned). All 32 lanes call it.
template <typename OUT>
__device__ __forceinline__ void epilogue_store_32x32(uint32_t stage, const uint32_t (&r)[32], OUT* C, int accumulate,
                                                     const OUT* add, long long ldadd, float alpha, long long ldc,
                                                     int row0, int M, int col0, int N) {
  constexpr bool F32 = sizeof(OUT) == 4;
  const int lane = threadIdx.x & 31;
  const int sub = lane >> 2, chunk = lane & 3;            // this lane's row in a group of eight, its 4 columns
  OUT* dst = C + static_cast<long long>(row0 + sub) * ldc + col0 + chunk * 4;
  add += static_cast<long long>(row0 + sub) * ldadd + col0 + chunk * 4;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const bool col_in = col0 + h * 16 + chunk * 4 < N;
    float4 old[4];
    if (accumulate) {                                     // in flight while the block is staged
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        old[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!col_in || row0 + sub + i * 8 >= M) continue;
        const OUT* src = add + static_cast<long long>(i) * 8 * ldadd + h * 16;
        if constexpr (F32) {
          old[i] = *reinterpret_cast<const float4*>(src);
        } else {
          const uint2 o = *reinterpret_cast<const uint2*>(src);
          const float2 a = unpack_bf16(o.x), b = unpack_bf16(o.y);
          old[i] = make_float4(a.x, a.y, b.x, b.y);
        }
      }
    }
    float4 v[4];
    stage_half(stage, r, h, v);
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

// Columns col0.. of a tile's 128 rows for the four warps of one half of its columns (`part`; `row` is the thread's):
// `blocks` times 64 accumulator columns from taddr on, through `block` (1024-byte aligned) to (x, row0, z) of `out`.
// `drained` is called by every warp once its accumulators have been read. The thread with `issuer` set waits for its
// stores before the kernel ends. Rows from M on and columns from N on are clipped by the map.
__device__ __forceinline__ void epilogue_part_sync(int part) {
  if (part == 0) asm volatile("bar.sync 3, 128;" ::: "memory");
  else asm volatile("bar.sync 4, 128;" ::: "memory");
}
// Have all four warps of a part what they waited for? A wait gives up in each warp by itself (once the status word is
// set it may do so in one warp and succeed in the next), and none may be left alone at the barriers of epilogue_tma:
// they enter it, or leave their loop, together (0.1 us of a launch of one wave, 4.9 -> 5.0 for 768 x 1024 over 256).
__device__ __forceinline__ bool epilogue_part_agree(int part, bool ok) {
  uint32_t all;
  if (part == 0)
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, 3, 128, p;\n\t"
                 "selp.u32 %0, 1, 0, q;\n\t}" : "=r"(all) : "r"(static_cast<uint32_t>(ok)) : "memory");
  else
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, 4, 128, p;\n\t"
                 "selp.u32 %0, 1, 0, q;\n\t}" : "=r"(all) : "r"(static_cast<uint32_t>(ok)) : "memory");
  return all != 0;
}
template <class F>
__device__ __forceinline__ void epilogue_tma(uint8_t* block, uint32_t taddr, int blocks, int part, int row, bool issuer,
                                             const CUtensorMap* out, float alpha, int col0, int N, int row0, int M, int z,
                                             F drained) {
#pragma unroll 1
  for (int b = 0; b < blocks; ++b) {
    const int col = col0 + b * 64;
    const bool last = b + 1 == blocks || col + 64 >= N;
    if (col < N) {
      uint32_t pk[32];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t r[32];
        tmem_ld_32x32(taddr + b * 64 + h * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; ++e)
          pk[h * 16 + e] = pack_bf16(__uint_as_float(r[2 * e]) * alpha, __uint_as_float(r[2 * e + 1]) * alpha);
      }
      if (last) drained();
      if (issuer) tma_store_wait_read<0>();
      epilogue_part_sync(part);                            // the block before has left
#pragma unroll
      for (int q = 0; q < 8; ++q)
        *reinterpret_cast<uint4*>(block + row * 128 + ((q ^ (row & 7)) << 4)) =
            make_uint4(pk[4 * q], pk[4 * q + 1], pk[4 * q + 2], pk[4 * q + 3]);
      fence_async_proxy();
      epilogue_part_sync(part);
      if (issuer && row0 < M) {
        tma_store_3d(out, block, col, row0, z);
        tma_store_commit();
      }
    } else if (b == 0) {
      drained();
    }
    if (last) break;
  }
}

// EPI_SWIGLU: gate and up of the same 32 rows and 32 columns. C is null where gate and up are not kept.
__device__ __forceinline__ void epilogue_swiglu_32x32(uint32_t stage, const uint32_t (&g)[32], const uint32_t (&u)[32],
                                                      __nv_bfloat16* C, long long ldc, const EpiArgs& e, int row0, int M,
                                                      int col0, int F) {
  uint32_t h[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const float gb = __bfloat162float(__float2bfloat16_rn(__uint_as_float(g[i])));
    const float ub = __bfloat162float(__float2bfloat16_rn(__uint_as_float(u[i])));
    h[i] = __float_as_uint(swiglu_value(gb, ub));
  }
  const __nv_bfloat16* none = nullptr;
  if (C != nullptr) {
    epilogue_store_32x32(stage, g, C, 0, none, 0, 1.f, ldc, row0, M, col0, F);
    epilogue_store_32x32(stage, u, C + F, 0, none, 0, 1.f, ldc, row0, M, col0, F);
  }
  epilogue_store_32x32(stage, h, e.h, 0, none, 0, 1.f, e.ldh, row0, M, col0, F);
}

// EPI_SWIGLU_BWD: r is the gradient of h at columns col0.. of F; C and e.src have 2F columns.
__device__ __forceinline__ void epilogue_swiglu_bwd_32x32(uint32_t stage, const uint32_t (&r)[32], __nv_bfloat16* C,
                                                          long long ldc, const EpiArgs& e, int row0, int M, int col0,
                                                          int F) {
  const int lane = threadIdx.x & 31, sub = lane >> 2, chunk = lane & 3;
  const __nv_bfloat16* gu = reinterpret_cast<const __nv_bfloat16*>(e.src);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int col = col0 + h * 16 + chunk * 4;
    uint2 gv[4], uv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {                           // in flight while the block is staged
      gv[i] = uv[i] = make_uint2(0, 0);
      const int row = row0 + sub + i * 8;
      if (col >= F || row >= M) continue;
      gv[i] = *reinterpret_cast<const uint2*>(gu + row * e.ldsrc + col);
      uv[i] = *reinterpret_cast<const uint2*>(gu + row * e.ldsrc + F + col);
    }
    float4 v[4];
    stage_half(stage, r, h, v);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = row0 + sub + i * 8;
      if (col >= F || row >= M) continue;
      const float2 d0 = unpack_bf16(pack_bf16(v[i].x, v[i].y)), d1 = unpack_bf16(pack_bf16(v[i].z, v[i].w));
      const float2 g0 = unpack_bf16(gv[i].x), g1 = unpack_bf16(gv[i].y);
      const float2 u0 = unpack_bf16(uv[i].x), u1 = unpack_bf16(uv[i].y);
      float4 dg, du;
      swiglu_grad(g0.x, u0.x, d0.x, dg.x, du.x);
      swiglu_grad(g0.y, u0.y, d0.y, dg.y, du.y);
      swiglu_grad(g1.x, u1.x, d1.x, dg.z, du.z);
      swiglu_grad(g1.y, u1.y, d1.y, dg.w, du.w);
      __nv_bfloat16* to = C + row * ldc + col;
      *reinterpret_cast<uint2*>(to) = make_uint2(pack_bf16(dg.x, dg.y), pack_bf16(dg.z, dg.w));
      *reinterpret_cast<uint2*>(to + F) = make_uint2(pack_bf16(du.x, du.y), pack_bf16(du.z, du.w));
    }
  }
}

}  // namespace ss
