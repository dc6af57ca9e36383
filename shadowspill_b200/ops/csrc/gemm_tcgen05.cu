// Persistent bf16 GEMM for sm_100a: TMA -> 128B-swizzled shared memory ->
// tcgen05.mma (accumulators in TMEM) -> tcgen05.ld epilogue.
//
//   C[M,N] (=|+=) op(A) * op(B)      fp32 accumulation, C in bf16 or fp32
//
// Operand storage (row-major, element pitch lda/ldb):
//   a_mn = 0 : A stored [M,K]  (contraction contiguous, "K-major")
//   a_mn = 1 : A stored [K,M]  (M contiguous, "MN-major")      -> C = A^T * ...
//   b_mn = 0 : B stored [N,K]  (K-major)                       -> C = A * B^T
//   b_mn = 1 : B stored [K,N]  (MN-major)                      -> C = A * B
// which covers forward (0,0), data-gradient (0,1) and weight-gradient (1,1)
// without materialising a transpose. `accumulate` folds the existing C into the
// result in the epilogue; this is the in-place weight-gradient accumulation the
// reference expresses as shadowspill::accumulate_matmul_
// (packages/engine/src/shadowspill/pytorch/operations.py:15).
//
// One CTA per SM, 192 threads:
//   warp 0      TMA producer (one elected lane)
//   warp 1      TMEM allocator + MMA issuer (one elected lane)
//   warps 2..9  epilogue; warp w owns TMEM lanes 32*(w%4)..+31
// Two 128x256 fp32 accumulators (2 x 256 TMEM columns) let the epilogue of tile
// i overlap the main loop of tile i+1.
#include "sm100_ptx.cuh"
#include "gemm_epilogue.cuh"
#include "launchers.h"

#include <cudaTypedefs.h>
#include <stdio.h>

namespace ss {

constexpr int BM = 128;
constexpr int BK = 64;  // 64 bf16 = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int GEMM_THREADS = 64 + EPI_WARPS * 32;

template <int BN>
struct GemmCfg {
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = (BN == 256) ? 4 : 6;
  static constexpr int OFF_EPI = STAGES * STAGE_BYTES;      // epilogue staging, then barriers
  static constexpr int SMEM = OFF_EPI + EPI_STAGE + 256 /*barriers*/ + 1024 /*align*/;
  // scatter epilogue only: per epilogue warp a 32-row x 128-column bf16 staging tile, so that
  // rows leave the SM as whole 256-byte runs (peer stores want full lines, not 16-byte pieces)
  static constexpr int SCATTER_STAGE = 4 * 32 * 256;
  static_assert(SCATTER_STAGE <= EPI_STAGE, "it is the epilogue's staging");
  static constexpr int TMEM_COLS = 2 * BN;  // 512 or 256
};

// Grouped (mixture-of-experts) forms share the kernel:
//   mode 1  rows of A/C are grouped by expert in 128-row-aligned segments; the B
//           operand of a tile is expert tile_expert[m-block] of a [E, ., .] bank
//           (forward and data-gradient of an expert bank).
//   mode 2  one output matrix per expert, contracted over that expert's padded row
//           segment [expert_offset[e], expert_offset[e+1]) (weight gradient of a bank).
// With row_dst (mode 1, bf16 output) the epilogue writes output row r to the address
// row_dst[r] instead of C + r*ldc; 0 drops the row. Addresses may point into another
// GPU's memory (plain peer stores), which is how an expert bank's output rows go
// straight back to the ranks that own their tokens: the combine transfer of expert
// parallelism rides in this kernel's epilogue, overlapped with the next tile's MMAs.
struct GroupInfo {
  int mode;
  const int* tile_expert;     // mode 1: [ceil(M/128)], -1 = tile past the used rows
  const int* expert_offset;   // mode 2: [E+1], multiples of 128
  const int* expert_rows;     // mode 2, optional: [E] rows of each segment that are not padding
  int n_experts;
  long long c_expert_stride;  // mode 2: elements between experts' outputs
  const long long* row_dst;   // mode 1, optional: per-row destination addresses (bytes)
};

struct GemmParams {
  void* C;
  int M, N, K;
  long long ldc;
  int c_f32;
  int accumulate;
  int tma_out;                // the products leave by TMA through tmC
  const int* used;            // optional: of the M rows those up to *used - used_from are in use
  int used_from;
  int a_mn, b_mn;
  int* status;
  float alpha;
  GroupInfo g;
  EpiArgs e;
};

struct TileWork {
  int mb, nb, expert, kb0, nkb;
  long long c_off;
  bool skip;
};

__device__ __forceinline__ void tile_coords(int t, int num_m, int num_n, int& mb, int& nb) {
  constexpr int GROUP_M = 16;
  const int per_group = GROUP_M * num_n;
  const int g = t / per_group;
  const int first_m = g * GROUP_M;
  const int gm = min(GROUP_M, num_m - first_m);
  const int r = t - g * per_group;
  mb = first_m + (r % gm);
  nb = r / gm;
}

__device__ __forceinline__ TileWork decode_tile(const GemmParams& p, int t, int num_m, int num_n,
                                                int num_kb) {
  TileWork w;
  w.expert = 0; w.kb0 = 0; w.nkb = num_kb; w.c_off = 0; w.skip = false;
  if (p.g.mode == 2) {
    const int per = num_m * num_n;
    w.expert = t / per;
    tile_coords(t - w.expert * per, num_m, num_n, w.mb, w.nb);
    const int lo = p.g.expert_offset[w.expert], hi = p.g.expert_offset[w.expert + 1];
    w.kb0 = lo / BK;
    w.nkb = (hi - lo) / BK;
    // Blocks that are all padding add nothing: a segment of up to 64 rows needs one block of its two
    // (128 experts, 62 rows each on average, both bank gradients: 410 -> 402 us, when their stores bound them).
    if (p.g.expert_rows) w.nkb = min(w.nkb, (p.g.expert_rows[w.expert] + BK - 1) / BK);
    w.c_off = static_cast<long long>(w.expert) * p.g.c_expert_stride;
  } else {
    tile_coords(t, num_m, num_n, w.mb, w.nb);
    if (p.g.mode == 1) {
      w.expert = p.g.tile_expert[w.mb];
      w.skip = w.expert < 0;
    }
  }
  return w;
}

template <int BN, bool A_MN, bool B_MN, int EPI>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmC, const GemmParams p) {
  using Cfg = GemmCfg<BN>;
  // columns of p.N that a tile takes: with gate and up side by side half of its own
  constexpr int TILE_N = EPI == EPI_SWIGLU ? BN / 2 : BN;
  extern __shared__ uint8_t smem_raw[];
  // 1024-byte alignment: the 128B swizzle pattern repeats every 8 rows = 1024 B.
  uint8_t* smem = align_smem_1024(smem_raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_EPI + EPI_STAGE);
  uint64_t* full = bars;
  uint64_t* empty = bars + Cfg::STAGES;
  uint64_t* tfull = bars + 2 * Cfg::STAGES;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);

  const int warp = static_cast<int>(warp_uniform(threadIdx.x >> 5));
  const int lane = threadIdx.x & 31;
  int num_m = (p.M + BM - 1) / BM;
  const int num_n = (p.N + TILE_N - 1) / TILE_N;
  const int num_kb = (p.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], EPI_WARPS);  // one arrival per epilogue warp
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  chain_wait();
  chain_release();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  if (p.used != nullptr) num_m = (max(0, min(p.M, *p.used - p.used_from)) + BM - 1) / BM;
  const int num_tiles = num_m * num_n * (p.g.mode == 2 ? p.g.n_experts : 1);

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
        const TileWork w = decode_tile(p, t, num_m, num_n, num_kb);
        if (w.skip) continue;
        const int mb = w.mb, nb = w.nb;
        for (int kr = 0; kr < w.nkb; ++kr) {
          const int kb = w.kb0 + kr;
          if (!mbar_wait(&empty[stage], phase ^ 1, p.status, KS_TIMEOUT_EMPTY)) {
            ok = false;
            break;
          }
          uint8_t* sa = smem + stage * Cfg::STAGE_BYTES;
          uint8_t* sb = sa + Cfg::A_BYTES;
          mbar_expect_tx(&full[stage], Cfg::STAGE_BYTES);
          if (!A_MN) {
            tma_load_2d(sa, &tmA, &full[stage], kb * BK, mb * BM);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j)
              tma_load_2d(sa + j * (BK * 128), &tmA, &full[stage], mb * BM + j * 64, kb * BK);
          }
          // B is always described by a 3-D map [expert, rows, cols]; plain GEMMs have one expert
          const int bz = p.g.mode == 1 ? w.expert : 0;
          if (EPI == EPI_SWIGLU) {
            tma_load_3d(sb, &tmB, &full[stage], kb * BK, nb * TILE_N, bz);
            tma_load_3d(sb + TILE_N * 128, &tmB, &full[stage], kb * BK, p.N + nb * TILE_N, bz);
          } else if (!B_MN) {
            tma_load_3d(sb, &tmB, &full[stage], kb * BK, nb * BN, bz);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j)
              tma_load_3d(sb + j * (BK * 128), &tmB, &full[stage], nb * BN + j * 64, kb * BK, bz);
          }
          if (++stage == Cfg::STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    const uint32_t leader = elect_one();
    constexpr uint32_t idesc = umma_idesc_bf16(BM, BN, A_MN, B_MN);
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
      const TileWork w = decode_tile(p, t, num_m, num_n, num_kb);
      if (w.skip || w.nkb == 0) continue;
      if (!mbar_wait(&tempty[acc], acc_phase ^ 1, p.status, KS_TIMEOUT_TMEM_EMPTY)) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
      for (int kb = 0; kb < w.nkb; ++kb) {
        if (!mbar_wait(&full[stage], phase, p.status, KS_TIMEOUT_FULL)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + stage * Cfg::STAGE_BYTES);
        const uint32_t sb = sa + Cfg::A_BYTES;
#pragma unroll
        for (int kk = 0; kk < BK / UMMA_K; ++kk) {
          const uint64_t adesc = A_MN ? umma_smem_desc(sa + kk * (UMMA_K * 128), BK * 128, 1024)
                                      : umma_smem_desc(sa + kk * (UMMA_K * 2), 16, 1024);
          const uint64_t bdesc = B_MN ? umma_smem_desc(sb + kk * (UMMA_K * 128), BK * 128, 1024)
                                      : umma_smem_desc(sb + kk * (UMMA_K * 2), 16, 1024);
          umma_bf16_if(leader, d_tmem, adesc, bdesc, idesc, (kb | kk) != 0 ? 1u : 0u);
        }
        umma_commit_if(leader, &empty[stage]);  // stage reusable once these MMAs retire
        if (++stage == Cfg::STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
      if (!ok) break;
      umma_commit_if(leader, &tfull[acc]);
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3;  // TMEM lane quarter this warp may touch
    const int part = (warp - 2) >> 2;    // the left or the right half of the tile's columns
    const uint32_t stage_out = smem_u32(smem + Cfg::OFF_EPI) + (warp - 2) * EPI_WARP_STAGE;
    const bool issuer = ((warp - 2) & 3) == 0 && lane == 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
      const TileWork w = decode_tile(p, t, num_m, num_n, num_kb);
      if (w.skip) continue;
      const int mb = w.mb, nb = w.nb;
      if (w.nkb == 0) {
        // an expert without rows: its gradient tile is zero (nothing to add when accumulating)
        if (!p.accumulate) {
          const int zr = mb * BM + q * 32 + lane;
          for (int c = nb * BN + part * (BN / 2); zr < p.M && c < min(p.N, nb * BN + (part + 1) * (BN / 2)); c += 8) {
            if (p.c_f32) {
              float* d = reinterpret_cast<float*>(p.C) + w.c_off + static_cast<long long>(zr) * p.ldc + c;
              *reinterpret_cast<float4*>(d) = make_float4(0, 0, 0, 0);
              *reinterpret_cast<float4*>(d + 4) = make_float4(0, 0, 0, 0);
            } else {
              uint2* d = reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.C) + w.c_off +
                                                  static_cast<long long>(zr) * p.ldc + c);
              d[0] = d[1] = make_uint2(0, 0);
            }
          }
        }
        continue;
      }
      bool ok = mbar_wait(&tfull[acc], acc_phase, p.status, KS_TIMEOUT_TMEM_FULL);
      if (EPI == EPI_PLAIN && p.tma_out) ok = epilogue_part_agree(part, ok);
      if (!ok) break;
      tc_fence_after();
      const int row = mb * BM + q * 32 + lane;
      const uint32_t taddr =
          tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(acc * BN);
      if (p.g.row_dst != nullptr) {
        // Scatter epilogue. Each thread owns one accumulator row; the rows are transposed
        // through an XOR-swizzled staging tile so that 16 lanes store one row's 256
        // contiguous bytes at its destination address.
        uint8_t* stg = smem + Cfg::OFF_EPI + q * (32 * 256);
        const long long my_dst = (row < p.M) ? p.g.row_dst[row] : 0;
#pragma unroll 1
        for (int half = 0; half < (part == 0 ? BN / 128 : 0); ++half) {   // one staging tile per lane quarter
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t r[32];
            tmem_ld_32x32(taddr + half * 128 + c * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint4 v;
              v.x = pack_bf16(__uint_as_float(r[8 * i + 0]) * p.alpha, __uint_as_float(r[8 * i + 1]) * p.alpha);
              v.y = pack_bf16(__uint_as_float(r[8 * i + 2]) * p.alpha, __uint_as_float(r[8 * i + 3]) * p.alpha);
              v.z = pack_bf16(__uint_as_float(r[8 * i + 4]) * p.alpha, __uint_as_float(r[8 * i + 5]) * p.alpha);
              v.w = pack_bf16(__uint_as_float(r[8 * i + 6]) * p.alpha, __uint_as_float(r[8 * i + 7]) * p.alpha);
              const int chunk = c * 4 + i;
              *reinterpret_cast<uint4*>(stg + lane * 256 + ((chunk ^ (lane & 15)) << 4)) = v;
            }
          }
          __syncwarp();
#pragma unroll 1
          for (int rr = 0; rr < 16; ++rr) {
            const int srow = rr * 2 + (lane >> 4);
            const int chunk = lane & 15;
            const long long where = __shfl_sync(0xffffffffu, my_dst, srow);
            const int col = nb * BN + half * 128 + chunk * 8;
            if (where != 0 && col < p.N) {
              const uint4 v = *reinterpret_cast<const uint4*>(stg + srow * 256 + ((chunk ^ (srow & 15)) << 4));
              *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(where) + col) = v;
            }
          }
          __syncwarp();
        }
      } else if (EPI == EPI_PLAIN && p.tma_out) {
        epilogue_tma(smem + Cfg::OFF_EPI + part * EPI_BLOCK, taddr + part * (BN / 2), BN / 128, part, q * 32 + lane, issuer,
                     &tmC, p.alpha, nb * BN + part * (BN / 2), p.N, mb * BM, p.M,
                     p.g.mode == 2 ? w.expert : 0, [&] {
                       tc_fence_before();
                       __syncwarp();
                       if (lane == 0) mbar_arrive(&tempty[acc]);
                     });
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1;
        }
        continue;
      } else
#pragma unroll 1
      for (int c = part * (TILE_N / 64); c < (part + 1) * (TILE_N / 64); ++c) {
        const int col0 = nb * TILE_N + c * 32, row0 = mb * BM + q * 32;
        if (col0 >= p.N) break;
        uint32_t r[32];
        tmem_ld_32x32(taddr + c * 32, r);
        if constexpr (EPI == EPI_SWIGLU) {
          uint32_t up[32];
          tmem_ld_32x32(taddr + TILE_N + c * 32, up);
          tmem_ld_wait();
          epilogue_swiglu_32x32(stage_out, r, up, reinterpret_cast<__nv_bfloat16*>(p.C), p.ldc, p.e, row0, p.M, col0, p.N);
        } else if constexpr (EPI == EPI_SWIGLU_BWD) {
          tmem_ld_wait();
          epilogue_swiglu_bwd_32x32(stage_out, r, reinterpret_cast<__nv_bfloat16*>(p.C), p.ldc, p.e, row0, p.M, col0, p.N);
        } else {
          tmem_ld_wait();
          if (p.c_f32)
            epilogue_store_32x32(stage_out, r, reinterpret_cast<float*>(p.C) + w.c_off,
                                 p.accumulate, reinterpret_cast<const float*>(p.e.src) + w.c_off, p.e.ldsrc,
                                 p.alpha, p.ldc, row0, p.M, col0, p.N);
          else
            epilogue_store_32x32(stage_out, r, reinterpret_cast<__nv_bfloat16*>(p.C) + w.c_off,
                                 p.accumulate, reinterpret_cast<const __nv_bfloat16*>(p.e.src) + w.c_off,
                                 p.e.ldsrc, p.alpha, p.ldc, row0, p.M, col0, p.N);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[acc]);
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
    if (issuer && p.tma_out) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// ---------------------------------------------------------------- host side
static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
  }
  return fn;
}

// 2-D bf16 row-major [rows, cols] with element pitch ld; box = [box_rows, 64 cols], 128B swizzle.
// The tensor-map encoder is a driver entry point and needs this thread to have a
// current context. Framework worker threads (for example an autograd engine thread)
// may not have touched the runtime yet, so bind the device that owns the operand.
static void bind_device_of(const void* ptr) {
  cudaPointerAttributes attr;
  if (cudaPointerGetAttributes(&attr, ptr) == cudaSuccess && attr.type == cudaMemoryTypeDevice)
    cudaSetDevice(attr.device);
  else
    cudaGetLastError();   // clear the sticky "invalid value" of a non-CUDA pointer
}

int make_tmap_bf16(CUtensorMap* map, const void* base, long long rows, long long cols,
                   long long ld, int box_rows) {
  bind_device_of(base);
  auto fn = encode_fn();
  if (fn == nullptr) return -1;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
  cuuint32_t box[2] = {64, static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

// 3-D bf16 [experts, rows, cols] with row pitch ld and expert pitch `expert_rows * ld`.
int make_tmap3_bf16(CUtensorMap* map, const void* base, long long experts, long long rows,
                    long long cols, long long ld, long long expert_pitch_elems, int box_rows) {
  bind_device_of(base);
  auto fn = encode_fn();
  if (fn == nullptr) return -1;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows),
                        static_cast<cuuint64_t>(experts)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld) * 2,
                           static_cast<cuuint64_t>(expert_pitch_elems) * 2};
  cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box_rows), 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

template <int BN, bool A_MN, bool B_MN, int EPI = EPI_PLAIN>
static int launch(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& params, int num_sms,
                  cudaStream_t stream) {
  using Cfg = GemmCfg<BN>;
  GemmParams p = params;
  CUtensorMap tc = ta;                                       // unused unless tma_out
  // TMA stores from 16-byte boundaries on, the staged stores from 8-byte ones
  p.tma_out = EPI == EPI_PLAIN && !p.c_f32 && !p.accumulate && p.g.row_dst == nullptr &&
              (reinterpret_cast<uintptr_t>(p.C) & 15) == 0;
  if (p.tma_out) {
    const long long matrices = p.g.mode == 2 ? p.g.n_experts : 1;
    if (int r = make_tmap3_bf16(&tc, p.C, matrices, p.M, p.N, p.ldc,
                                p.g.mode == 2 ? p.g.c_expert_stride : static_cast<long long>(p.M) * p.ldc, BM))
      return r;
  }
  static SmemOptIn opt_in;
  auto kern = gemm_bf16_kernel<BN, A_MN, B_MN, EPI>;
  constexpr int TILE_N = EPI == EPI_SWIGLU ? BN / 2 : BN;
  if (int e = opt_in.ensure(kern, Cfg::SMEM)) return e;
  const int smem_bytes = Cfg::SMEM;
  const long long tiles = static_cast<long long>((p.M + BM - 1) / BM) * ((p.N + TILE_N - 1) / TILE_N) *
                          (p.g.mode == 2 ? p.g.n_experts : 1);
  const int grid = tiles < num_sms ? static_cast<int>(tiles) : num_sms;
  // Not the expert banks: chaining them and the kernels around them cost 5 % (64 experts, 8,192 tokens,
  // forward and backward 2883 -> 3034 us) and gave nothing for 128 experts and 1,000 tokens.
  if (p.g.mode == 0) launch_chained(kern, grid, GEMM_THREADS, smem_bytes, stream, ta, tb, tc, p);
  else kern<<<grid, GEMM_THREADS, smem_bytes, stream>>>(ta, tb, tc, p);
  return static_cast<int>(cudaGetLastError());
}

static int dispatch(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int bn,
                    int num_sms, cudaStream_t s) {
  const bool a_mn = p.a_mn, b_mn = p.b_mn;
#define SS_DISPATCH(BN_)                                                              \
  do {                                                                                \
    if (!a_mn && !b_mn) return launch<BN_, false, false>(ta, tb, p, num_sms, s);      \
    if (!a_mn && b_mn) return launch<BN_, false, true>(ta, tb, p, num_sms, s);        \
    if (a_mn && b_mn) return launch<BN_, true, true>(ta, tb, p, num_sms, s);          \
    return launch<BN_, true, false>(ta, tb, p, num_sms, s);                           \
  } while (0)
  if (bn == 256) SS_DISPATCH(256);
  SS_DISPATCH(128);
#undef SS_DISPATCH
}

// Do the 128x128 tiles of an output fit one wave? Such a tile takes about half the time of a 128x256 one
// or of a CTA pair's 256x256 one (512 x 2048 over 2048: 9.9 us against 15.2 and 16.0; 1024 x 2048 over
// 6144: 21.4 against 33.3 and 34.1; 768 x 256 over 256: 5.1 against 7.0 and 7.7), so wider tiles only pay
// once there is more than one wave of them (1999 x 4096 over 2048: 30.3 against 26.8 and 26.3).
bool gemm_fits_one_wave(int M, int N, int num_sms) {
  return N <= 128 || static_cast<long long>((M + 127) / 128) * ((N + 127) / 128) <= num_sms;
}

int gemm_from(const void* A, const void* B, const void* src, void* C, long long ldsrc, int M, int N, int K, long long lda,
              long long ldb, long long ldc, int a_mn, int b_mn, int c_f32, int accumulate, float alpha, int bn,
              int num_sms, int* status, void* stream, const int* used = nullptr, int used_from = 0);

static int sm_count() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

}  // namespace ss

extern "C" {

// Returns 0 on success, a CUDA/driver error code otherwise, -2 for bad arguments.
// `status` is an int32 in device (or mapped pinned) memory that receives a
// ss::KernelStatus if a bounded wait inside the kernel gave up; it may be null.
int ss_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                 long long ldb, long long ldc, int a_mn, int b_mn, int c_f32, int accumulate,
                 float alpha, int bn, int num_sms, int* status, void* stream) {
  return ss::gemm_from(A, B, C, C, ldc, M, N, K, lda, ldb, ldc, a_mn, b_mn, c_f32, accumulate, alpha, bn, num_sms, status,
                       stream);
}

}  // extern "C"

namespace ss {

// ss_gemm_bf16 whose `accumulate` adds `src` [M, N] (pitch `ldsrc`, C's type) to the products; with `used` (not for a_mn)
// of the first `*used - used_from` rows only, in whole tiles.
int gemm_from(const void* A, const void* B, const void* src, void* C, long long ldsrc, int M, int N, int K, long long lda,
              long long ldb, long long ldc, int a_mn, int b_mn, int c_f32, int accumulate, float alpha, int bn,
              int num_sms, int* status, void* stream, const int* used, int used_from) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (accumulate && ((ldsrc % (c_f32 ? 4 : 8)) || (reinterpret_cast<uintptr_t>(src) & 15))) return -2;
  if ((lda % 8) || (ldb % 8) || (ldc % (c_f32 ? 4 : 8)) || (N % 8) ||
      (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) ||
      (reinterpret_cast<uintptr_t>(C) & 15))
    return -2;
  if (num_sms <= 0) num_sms = sm_count();
  if (bn != 128 && bn != 256) bn = gemm_fits_one_wave(M, N, num_sms) ? 128 : 256;
  CUtensorMap ta, tb;
  int r;
  if (!a_mn) r = make_tmap_bf16(&ta, A, M, K, lda, BM);
  else       r = make_tmap_bf16(&ta, A, K, M, lda, BK);
  if (r) return r;
  if (!b_mn) r = make_tmap3_bf16(&tb, B, 1, N, K, ldb, static_cast<long long>(N) * ldb, bn);
  else       r = make_tmap3_bf16(&tb, B, 1, K, N, ldb, static_cast<long long>(K) * ldb, BK);
  if (r) return r;
  GemmParams p{};
  p.C = C; p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.c_f32 = c_f32; p.accumulate = accumulate;
  p.a_mn = a_mn; p.b_mn = b_mn; p.status = status; p.alpha = alpha;
  p.e.src = src; p.e.ldsrc = ldsrc; p.used = used; p.used_from = used_from;
  p.g.mode = 0;
  return dispatch(ta, tb, p, bn, num_sms, reinterpret_cast<cudaStream_t>(stream));
}

}  // namespace ss

extern "C" {

// Expert-bank GEMMs over token rows sorted by expert into 128-row-aligned segments.
//   mode 1, b_mn = 0: C[R,N]  = A[R,K] @ bank[e][N,K]^T     (forward through the bank)
//   mode 1, b_mn = 1: C[R,N]  = A[R,K] @ bank[e][K,N]        (data gradient)
//   mode 2          : C[e][M,N] (+)= A[rows_e, M]^T @ B[rows_e, N]   (weight gradient)
// R = padded row count; `tile_expert` (mode 1), `expert_offset` and `expert_rows` (mode 2; null: contract
// the padding too) are device arrays.
int ss_gemm_grouped_bf16(const void* A, const void* B, void* C, int mode, int rows, int M, int N,
                         int K, int n_experts, long long lda, long long ldb, long long ldc,
                         int b_mn, int c_f32, int accumulate, const int* tile_expert,
                         const int* expert_offset, const int* expert_rows, int bn, int* status,
                         void* stream) {
  using namespace ss;
  if (rows <= 0 || n_experts <= 0) return 0;
  if ((lda % 8) || (ldb % 8) || (ldc % (c_f32 ? 4 : 8)) || (N % 8) || (rows % BM) ||
      (reinterpret_cast<uintptr_t>(C) & (c_f32 ? 15 : 7)))
    return -2;
  if (bn != 128 && bn != 256) bn = (N <= 128) ? 128 : 256;
  CUtensorMap ta, tb;
  GemmParams p{};
  int r;
  if (mode == 1) {
    if (tile_expert == nullptr) return -2;
    if ((r = make_tmap_bf16(&ta, A, rows, K, lda, BM))) return r;
    if (!b_mn) r = make_tmap3_bf16(&tb, B, n_experts, N, K, ldb, static_cast<long long>(N) * ldb, bn);
    else       r = make_tmap3_bf16(&tb, B, n_experts, K, N, ldb, static_cast<long long>(K) * ldb, BK);
    if (r) return r;
    p.M = rows; p.N = N; p.K = K; p.a_mn = 0; p.b_mn = b_mn;
  } else if (mode == 2) {
    if (expert_offset == nullptr) return -2;
    // A stored [rows, M] and B stored [rows, N]: both contraction-major over the sorted rows
    if ((r = make_tmap_bf16(&ta, A, rows, M, lda, BK))) return r;
    if ((r = make_tmap3_bf16(&tb, B, 1, rows, N, ldb, static_cast<long long>(rows) * ldb, BK))) return r;
    p.M = M; p.N = N; p.K = rows; p.a_mn = 1; p.b_mn = 1;
    p.g.c_expert_stride = static_cast<long long>(M) * ldc;
  } else {
    return -2;
  }
  p.C = C; p.ldc = ldc; p.c_f32 = c_f32; p.accumulate = accumulate; p.status = status; p.alpha = 1.f;
  p.e.src = C; p.e.ldsrc = ldc;
  p.g.mode = mode; p.g.tile_expert = tile_expert; p.g.expert_offset = expert_offset;
  p.g.expert_rows = expert_rows;
  p.g.n_experts = n_experts;
  return dispatch(ta, tb, p, bn, sm_count(), reinterpret_cast<cudaStream_t>(stream));
}

// Row-grouped expert GEMM whose output rows are scattered: row r of A x B[expert]^T
// (bf16) is written to the byte address row_dst[r] (16-byte aligned; 0 = dropped),
// which may lie in a peer GPU's mapped memory.
int ss_gemm_grouped_scatter_bf16(const void* A, const void* B, const long long* row_dst, int rows,
                                 int N, int K, int n_experts, long long lda, long long ldb, int b_mn,
                                 const int* tile_expert, int bn, int* status, void* stream) {
  using namespace ss;
  if (rows <= 0 || n_experts <= 0) return 0;
  if ((lda % 8) || (ldb % 8) || (N % 8) || (rows % BM) || !tile_expert || !row_dst) return -2;
  if (bn != 128 && bn != 256) bn = (N <= 128) ? 128 : 256;
  CUtensorMap ta, tb;
  GemmParams p{};
  int r;
  if ((r = make_tmap_bf16(&ta, A, rows, K, lda, BM))) return r;
  if (!b_mn) r = make_tmap3_bf16(&tb, B, n_experts, N, K, ldb, static_cast<long long>(N) * ldb, bn);
  else       r = make_tmap3_bf16(&tb, B, n_experts, K, N, ldb, static_cast<long long>(K) * ldb, BK);
  if (r) return r;
  p.M = rows; p.N = N; p.K = K; p.a_mn = 0; p.b_mn = b_mn;
  p.C = nullptr; p.ldc = 0; p.c_f32 = 0; p.accumulate = 0; p.status = status; p.alpha = 1.f;
  p.g.mode = 1; p.g.tile_expert = tile_expert; p.g.n_experts = n_experts; p.g.row_dst = row_dst;
  return dispatch(ta, tb, p, bn, sm_count(), reinterpret_cast<cudaStream_t>(stream));
}

// h[M, F] = silu(A gate^T) * (A up^T) for B = [gate; up], [2F, K]; unless gu is null the two products go there, [M, 2F].
// The single-CTA form; ss_gemm2_swiglu_bf16 hands it the outputs whose 128 x 128 tiles of gate and up fit one wave.
int ss_gemm_swiglu_bf16(const void* A, const void* B, void* gu, void* h, int M, int F, int K, long long lda,
                        long long ldb, long long ldgu, long long ldh, int bn, int* status, void* stream) {
  using namespace ss;
  if (M <= 0 || F <= 0 || K <= 0) return 0;
  if ((lda % 8) || (ldb % 8) || (ldgu % 8) || (ldh % 8) || (F % 8) || (reinterpret_cast<uintptr_t>(A) & 15) ||
      (reinterpret_cast<uintptr_t>(B) & 15) || (reinterpret_cast<uintptr_t>(gu) & 15) ||
      (reinterpret_cast<uintptr_t>(h) & 15))
    return -2;
  const int num_sms = sm_count();
  if (bn != 128 && bn != 256) bn = gemm_fits_one_wave(M, 2 * F, num_sms) ? 128 : 256;
  CUtensorMap ta, tb;
  int r;
  if ((r = make_tmap_bf16(&ta, A, M, K, lda, BM))) return r;
  if ((r = make_tmap3_bf16(&tb, B, 1, 2LL * F, K, ldb, 2LL * F * ldb, bn / 2))) return r;
  GemmParams p{};
  p.C = gu; p.M = M; p.N = F; p.K = K; p.ldc = ldgu; p.status = status; p.alpha = 1.f;
  p.e.h = reinterpret_cast<__nv_bfloat16*>(h); p.e.ldh = ldh;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (bn == 256) return launch<256, false, false, EPI_SWIGLU>(ta, tb, p, num_sms, s);
  return launch<128, false, false, EPI_SWIGLU>(ta, tb, p, num_sms, s);
}

// dgu[M, 2F] = the gradient of [gate, up] in gu [M, 2F] for dh = A[M, K] @ B[K, F], the gradient of silu(gate) * up.
int ss_gemm_swiglu_bwd_bf16(const void* A, const void* B, const void* gu, void* dgu, int M, int F, int K, long long lda,
                            long long ldb, long long ldgu, long long lddgu, int bn, int* status, void* stream) {
  using namespace ss;
  if (M <= 0 || F <= 0 || K <= 0) return 0;
  if ((lda % 8) || (ldb % 8) || (ldgu % 8) || (lddgu % 8) || (F % 8) || (reinterpret_cast<uintptr_t>(A) & 15) ||
      (reinterpret_cast<uintptr_t>(B) & 15) || (reinterpret_cast<uintptr_t>(gu) & 15) ||
      (reinterpret_cast<uintptr_t>(dgu) & 15))
    return -2;
  const int num_sms = sm_count();
  if (bn != 128 && bn != 256) bn = gemm_fits_one_wave(M, F, num_sms) ? 128 : 256;
  CUtensorMap ta, tb;
  int r;
  if ((r = make_tmap_bf16(&ta, A, M, K, lda, BM))) return r;
  if ((r = make_tmap3_bf16(&tb, B, 1, K, F, ldb, static_cast<long long>(K) * ldb, BK))) return r;
  GemmParams p{};
  p.C = dgu; p.M = M; p.N = F; p.K = K; p.ldc = lddgu; p.b_mn = 1; p.status = status; p.alpha = 1.f;
  p.e.src = gu; p.e.ldsrc = ldgu;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (bn == 256) return launch<256, false, true, EPI_SWIGLU_BWD>(ta, tb, p, num_sms, s);
  return launch<128, false, true, EPI_SWIGLU_BWD>(ta, tb, p, num_sms, s);
}

// The forward form over expert-sorted rows (segments as in mode 1 above): bank [E, 2F, K], gu [rows, 2F], h [rows, F].
int ss_gemm_grouped_swiglu_bf16(const void* A, const void* B, void* gu, void* h, int rows, int F, int K, int n_experts,
                                long long lda, long long ldb, long long ldgu, long long ldh, const int* tile_expert,
                                int* status, void* stream) {
  using namespace ss;
  if (rows <= 0 || n_experts <= 0) return 0;
  if ((lda % 8) || (ldb % 8) || (ldgu % 8) || (ldh % 8) || (F % 8) || (rows % BM) || tile_expert == nullptr ||
      (reinterpret_cast<uintptr_t>(gu) & 15) || (reinterpret_cast<uintptr_t>(h) & 15))
    return -2;
  const int bn = 2 * F <= 128 ? 128 : 256;
  CUtensorMap ta, tb;
  int r;
  if ((r = make_tmap_bf16(&ta, A, rows, K, lda, BM))) return r;
  if ((r = make_tmap3_bf16(&tb, B, n_experts, 2LL * F, K, ldb, 2LL * F * ldb, bn / 2))) return r;
  GemmParams p{};
  p.C = gu; p.M = rows; p.N = F; p.K = K; p.ldc = ldgu; p.status = status; p.alpha = 1.f;
  p.e.h = reinterpret_cast<__nv_bfloat16*>(h); p.e.ldh = ldh;
  p.g.mode = 1; p.g.tile_expert = tile_expert; p.g.n_experts = n_experts;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (bn == 256) return launch<256, false, false, EPI_SWIGLU>(ta, tb, p, sm_count(), s);
  return launch<128, false, false, EPI_SWIGLU>(ta, tb, p, sm_count(), s);
}

}  // extern "C"
