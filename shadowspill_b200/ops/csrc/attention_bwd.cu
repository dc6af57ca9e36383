// Packed variable-length causal GQA attention, backward, for sm_100a.
//
// Two tcgen05 kernels, neither of which needs atomics, so every gradient is the same each time:
//
//   dQ kernel   one CTA per (128-query tile, query head); streams K/V tiles.
//               S = Q K^T and dP = dO V^T land in TMEM, the softmax warps form
//               dS = P o (dP - delta) and dQ += dS K accumulates in TMEM.
//   dKV kernel  one CTA per (128-key tile, KV head); streams the query tiles
//               of every query head of the group. S^T = K Q^T and dP^T = V dO^T
//               (keys on TMEM lanes); dV += P^T dO and dK += dS^T Q accumulate in
//               TMEM across tiles and across the heads of the GQA group.
//
// P^T, dS^T and dS go back to TMEM and are the A operand of their products there. A 128-row product
// reads A and B from shared memory at the full rate of that memory when both are there, and the 64-row
// tiles of K, V, Q or dO that an operand in shared memory left room for need 1.5 times that rate; with
// these operands in TMEM the tiles have 128 rows (64 for head width 256) and half of the products read
// only B.
//
// For head width 256 the dK and dV accumulators do not fit TMEM together with
// the score buffers, so the dKV kernel runs twice (dV only, then dK only).
// delta[h,t] = sum_d dO*O comes from a small preprocess kernel into caller
// scratch (fp32 [Hq, T]).
//
// Measured, 16,384 tokens in two sequences, 32/8 heads of 128: dQ 2.42 -> 1.19 ms, dKV 3.15 -> 1.58 ms
// against P^T and dS through shared memory in 64-row tiles.
//
// warps 0..7 softmax: warp w owns TMEM lanes 32*(w%4)..+31 and the left or right half (w/4) of
// every score tile; warp 8 TMA producer, warp 9 MMA, warp 10 row statistics (dKV kernel).
#include "sm100_ptx.cuh"
#include "attention_tiles.cuh"

#include <cudaTypedefs.h>
#include <math.h>

namespace ss {

int make_tmap_bf16(CUtensorMap* map, const void* base, long long rows, long long cols,
                   long long ld, int box_rows);

constexpr int BW_THREADS = 352;
constexpr int BW_TMA_WARP = 8, BW_MMA_WARP = 9, BW_STAT_WARP = 10;
constexpr float LOG2E = 1.4426950408889634f;

struct AttnBwdParams {
  void* dq; void* dk; void* dv;
  const float* lse;      // [Hq, T] natural log
  const float* delta;    // [Hq, T]
  const int* cu_seqlens;
  int nseq, T, Hq, Hkv;
  int split;                 // CTAs that share a key tile of the dKV kernel: a divisor of Hq / Hkv
  long long ldq, ldk, ldv;   // row pitches of dq / dk / dv (elements)
  float scale;
  int* status;
};

// ============================================================================ preprocess
// A row of DH values per DH / 8 lanes, 16 bytes a lane (four-byte loads by a whole warp moved 3 TB/s:
// 8,192 x 32 heads of 128, 44 -> 26 us). `out` may lie on any 4-byte boundary; off 16 bytes (WIDE = false) it is
// read four bytes at a time. dout is a TMA operand of the kernels behind this one and always on 16.
template <int DH, bool WIDE>
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __nv_bfloat16* out, const __nv_bfloat16* dout, float* delta, int T, int Hq,
                  long long ld_out, long long ld_dout) {
  chain_wait();
  chain_release();
  constexpr int LANES = DH / 8;
  const long long row = (blockIdx.x * 256ll + threadIdx.x) / LANES;
  const int lane = threadIdx.x % LANES;
  const bool in = row < static_cast<long long>(T) * Hq;
  // heads fastest: neighbouring lane groups read neighbouring bytes
  const int t = in ? static_cast<int>(row / Hq) : 0, h = in ? static_cast<int>(row % Hq) : 0;
  uint4 o;
  const __nv_bfloat16* at = out + t * ld_out + h * DH + lane * 8;
  if constexpr (WIDE) {
    o = *reinterpret_cast<const uint4*>(at);
  } else {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(at);
    o = make_uint4(w[0], w[1], w[2], w[3]);
  }
  const uint4 d = *reinterpret_cast<const uint4*>(dout + t * ld_dout + h * DH + lane * 8);
  float acc = 0.f;
  const uint32_t ow[4] = {o.x, o.y, o.z, o.w}, dw[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 a = unpack_bf16(ow[e]), b = unpack_bf16(dw[e]);
    acc += a.x * b.x + a.y * b.y;
  }
#pragma unroll
  for (int s = LANES / 2; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if (in && lane == 0) delta[static_cast<long long>(h) * T + t] = acc;
}

// ============================================================================ TMEM operands
// P^T, dS^T and dS go back into the TMEM columns of the scores they come from: the two warps of a
// lane quarter own the left and the right half of a score tile, and each packs its half into the
// first half of its own columns, so neither overwrites columns that the other still has to read.
// Column offset of the 16-element step kk of such an operand whose score tile has BN columns:
template <int BN>
__device__ __forceinline__ constexpr uint32_t packed_col(int kk) {
  return (kk * 16) / (BN / 2) * (BN / 2) + ((kk * 16) % (BN / 2)) / 2;
}

// Two pairs of fp32 in one 16-byte load, in the registers that the packed arithmetic takes.
__device__ __forceinline__ void ld_shared_2x2(uint32_t addr, f32x2& a, f32x2& b) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}

__device__ __forceinline__ void st_shared_f32(uint32_t addr, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

template <int HN>   // HN score columns per warp: 64 or 32
__device__ __forceinline__ void tmem_ld_half(uint32_t addr, uint32_t (&r)[HN]) {
#pragma unroll
  for (int c = 0; c < HN; c += 32) tmem_ld_32x32(addr + c, reinterpret_cast<uint32_t (&)[32]>(r[c]));
  tmem_ld_wait();
}
template <int HN>
__device__ __forceinline__ void tmem_st_half(uint32_t addr, const uint32_t (&pk)[HN / 2]) {
  if constexpr (HN == 64) tmem_st_32x32(addr, pk);
  else tmem_st_32x16(addr, pk);
  tmem_st_wait();
}

template <int PN>   // PN packed pairs' columns: 32 or 16 score columns
__device__ __forceinline__ void tmem_st_quarter(uint32_t addr, const uint32_t (&pk)[PN / 2]) {
  if constexpr (PN == 32) tmem_st_32x16(addr, pk);
  else tmem_st_32x8(addr, pk);
  tmem_st_wait();
}

// ============================================================================ dQ kernel
// S is double-buffered and dP single: S of the next tile is formed under this tile's
// exponentials, dP of the next tile under this tile's dS. K is released by the dQ product and has
// KS stages, V already by the dP product and has VS.
// Both are issued before dS of this tile is waited for, so two warps may be a tile apart: dS has a barrier
// for even and one for odd tiles, or a warp a tile ahead would count for one that has yet to write. dP of the
// next tile waits until all warps have read this one's, so one barrier is enough there.
template <int DH, int BKV, int KS, int VS, int CTAS>
struct DqCfg {
  static constexpr int Q_BYTES = 128 * DH * 2;
  static constexpr int KV_BYTES = BKV * DH * 2;
  static constexpr int OFF_DO = Q_BYTES;
  static constexpr int OFF_K = 2 * Q_BYTES;
  static constexpr int OFF_V = OFF_K + KS * KV_BYTES;
  static constexpr int OFF_BAR = OFF_V + VS * KV_BYTES;
  static constexpr int SMEM = OFF_BAR + 256 + 1024;
  static constexpr int TM_S = 0, TM_DP = 2 * BKV, TM_DQ = 3 * BKV;
  static constexpr int TM_COLS = TM_DQ + DH <= 256 ? 256 : 512;
  static_assert(TM_DQ + DH <= TM_COLS && CTAS * TM_COLS <= 512, "TMEM budget");
  static_assert(CTAS * (SMEM + 1024) <= 233472, "shared memory budget");
};

template <int DH, int BKV, int KS, int VS, int CTAS>
__global__ void __launch_bounds__(BW_THREADS, CTAS)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
                   const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                   const AttnBwdParams p) {
  using Cfg = DqCfg<DH, BKV, KS, VS, CTAS>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_smem_1024(smem_raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* qdo_full = bars;            // 1
  uint64_t* k_full = bars + 1;          // 3
  uint64_t* k_empty = bars + 4;         // 3
  uint64_t* v_full = bars + 7;          // 2
  uint64_t* v_empty = bars + 9;         // 2
  uint64_t* s_full = bars + 11;         // 2
  uint64_t* dp_full = bars + 13;        // 1
  uint64_t* dp_free = bars + 14;        // 1
  uint64_t* ds_full = bars + 15;        // 2
  uint64_t* dq_done = bars + 17;        // 1
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
  TileSlot* slot = reinterpret_cast<TileSlot*>(bars + 19);

  const int warp = static_cast<int>(warp_uniform(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const int head = blockIdx.x % p.Hq, rank = blockIdx.x / p.Hq;
  const int kv_head = head / (p.Hq / p.Hkv);

  if (threadIdx.x == 0) {
    mbar_init(qdo_full, 1);
    for (int i = 0; i < KS; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); }
    for (int i = 0; i < VS; ++i) { mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&ds_full[i], 8); }
    mbar_init(dp_full, 1);
    mbar_init(dp_free, 8);
    mbar_init(dq_done, 1);
    mbar_fence_init();
  }
  if (warp == BW_MMA_WARP) { tmem_alloc(tmem_slot, Cfg::TM_COLS); tmem_relinquish(); }
  chain_wait();
  if (warp == BW_TMA_WARP) find_tile_by_work(p.cu_seqlens, p.nseq, 128, rank, slot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  chain_release();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  const int seq_start = slot->seq_start, seq_end = slot->seq_end;
  const int q0 = seq_start + (slot->work - 1) * 128;
  const int q_hi = min(q0 + 128, seq_end);
  const int n_kv = slot->work > 0 ? (q_hi - seq_start + BKV - 1) / BKV : 0;

  if (warp == BW_TMA_WARP) {
    if (n_kv > 0 && elect_one()) {
      mbar_expect_tx(qdo_full, 2 * Cfg::Q_BYTES);
#pragma unroll
      for (int c = 0; c < DH / 64; ++c) {
        tma_load_2d(smem + c * (128 * 128), &tmQ, qdo_full, head * DH + c * 64, q0);
        tma_load_2d(smem + Cfg::OFF_DO + c * (128 * 128), &tmDO, qdo_full, head * DH + c * 64, q0);
      }
      for (int j = 0; j < n_kv; ++j) {
        const int ks = j % KS, vs = j % VS;
        const int k0 = seq_start + j * BKV;
        if (j >= KS && !mbar_wait(&k_empty[ks], ((j / KS) - 1) & 1, p.status, KS_TIMEOUT_EMPTY)) break;
        uint8_t* sk = smem + Cfg::OFF_K + ks * Cfg::KV_BYTES;
        mbar_expect_tx(&k_full[ks], Cfg::KV_BYTES);
#pragma unroll
        for (int c = 0; c < DH / 64; ++c)
          tma_load_2d(sk + c * (BKV * 128), &tmK, &k_full[ks], kv_head * DH + c * 64, k0);
        if (j >= VS && !mbar_wait(&v_empty[vs], ((j / VS) - 1) & 1, p.status, KS_TIMEOUT_EMPTY)) break;
        uint8_t* sv = smem + Cfg::OFF_V + vs * Cfg::KV_BYTES;
        mbar_expect_tx(&v_full[vs], Cfg::KV_BYTES);
#pragma unroll
        for (int c = 0; c < DH / 64; ++c)
          tma_load_2d(sv + c * (BKV * 128), &tmV, &v_full[vs], kv_head * DH + c * 64, k0);
      }
    }
  } else if (warp == BW_MMA_WARP) {
    if (n_kv > 0) {
      const uint32_t leader = elect_one();
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, BKV, false, false);
      constexpr uint32_t idesc_dq = umma_idesc_bf16(128, DH, false, true);
      const uint32_t sq = smem_u32(smem), sdo = smem_u32(smem + Cfg::OFF_DO);
      const uint32_t sk0 = smem_u32(smem + Cfg::OFF_K), sv0 = smem_u32(smem + Cfg::OFF_V);
      auto scores = [&](uint32_t d, uint32_t a, uint32_t b) {
#pragma unroll
        for (int kk = 0; kk < DH / 16; ++kk)
          umma_bf16_if(leader, d, umma_smem_desc(a + (kk >> 2) * (128 * 128) + (kk & 3) * 32, 16, 1024),
                    umma_smem_desc(b + (kk >> 2) * (BKV * 128) + (kk & 3) * 32, 16, 1024), idesc_s, kk != 0);
      };
      auto issue_s = [&](int j) -> bool {
        if (!mbar_wait(&k_full[j % KS], (j / KS) & 1, p.status, KS_TIMEOUT_FULL)) return false;
        tc_fence_after();
        scores(tmem_base + Cfg::TM_S + (j & 1) * BKV, sq, sk0 + (j % KS) * Cfg::KV_BYTES);
        umma_commit_if(leader, &s_full[j & 1]);
        return true;
      };
      auto issue_dp = [&](int j) -> bool {
        if (!mbar_wait(&v_full[j % VS], (j / VS) & 1, p.status, KS_TIMEOUT_FULL)) return false;
        if (j > 0 && !mbar_wait(dp_free, (j - 1) & 1, p.status, KS_TIMEOUT_TMEM_EMPTY)) return false;
        tc_fence_after();
        scores(tmem_base + Cfg::TM_DP, sdo, sv0 + (j % VS) * Cfg::KV_BYTES);
        umma_commit_if(leader, dp_full);
        umma_commit_if(leader, &v_empty[j % VS]);
        return true;
      };
      bool ok = mbar_wait(qdo_full, 0, p.status, KS_TIMEOUT_FULL) && issue_s(0) && issue_dp(0);
      for (int j = 0; j < n_kv && ok; ++j) {
        // S of the next tile goes to the buffer whose dS the dQ product before this point reads:
        // products of one issuing thread run in order
        if (j + 1 < n_kv) ok = issue_s(j + 1) && issue_dp(j + 1);
        if (!ok || !mbar_wait(&ds_full[j & 1], (j >> 1) & 1, p.status, KS_TIMEOUT_FULL)) break;
        tc_fence_after();
        const uint32_t sk = sk0 + (j % KS) * Cfg::KV_BYTES;
        const uint32_t ds = tmem_base + Cfg::TM_S + (j & 1) * BKV;
#pragma unroll
        for (int kk = 0; kk < BKV / 16; ++kk)
          umma_bf16_ts_if(leader, tmem_base + Cfg::TM_DQ, ds + packed_col<BKV>(kk),
                       umma_smem_desc(sk + kk * (16 * 128), BKV * 128, 1024), idesc_dq, (j | kk) != 0);
        umma_commit_if(leader, &k_empty[j % KS]);
        if (j + 1 == n_kv) umma_commit_if(leader, dq_done);
      }
    }
  } else if (warp < 8) {
    constexpr int HN = BKV / 2;
    const int quarter = warp & 3, half = warp >> 2;
    const int row = quarter * 32 + lane;
    const int gq = q0 + row;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t dp_addr = lane_addr + Cfg::TM_DP + half * HN;
    const long long li = static_cast<long long>(head) * p.T + max(0, min(gq, p.T - 1));
    const float nlse1 = -p.lse[li] * LOG2E, ndl1 = -p.delta[li], c21 = p.scale * LOG2E;
    const f32x2 nlse = pack_x2(nlse1, nlse1), ndl = pack_x2(ndl1, ndl1), c2 = pack_x2(c21, c21);
    bool ok = true;
    for (int j = 0; j < n_kv; ++j) {
      const int b = j & 1;
      const uint32_t s_addr = lane_addr + Cfg::TM_S + b * BKV + half * HN;
      if (!mbar_wait(&s_full[b], (j >> 1) & 1, p.status, KS_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      uint32_t s[HN];
      tmem_ld_half<HN>(s_addr, s);
      const int k0 = seq_start + j * BKV + half * HN;
#pragma unroll
      for (int e = 0; e < HN; e += 2) {
        const float2 t = unpack_x2(fma_x2(pack_x2(__uint_as_float(s[e]), __uint_as_float(s[e + 1])), c2, nlse));
        s[e] = __float_as_uint(fast_exp2(t.x));
        s[e + 1] = __float_as_uint(fast_exp2(t.y));
      }
      if (k0 + HN - 1 > q0) {                      // some key of this half is hidden from some row
#pragma unroll
        for (int e = 0; e < HN; ++e)
          if (k0 + e > gq) s[e] = 0u;
      }
      if (!mbar_wait(dp_full, j & 1, p.status, KS_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      uint32_t d[HN];
      tmem_ld_half<HN>(dp_addr, d);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(dp_free);
      uint32_t pk[HN / 2];
#pragma unroll
      for (int e = 0; e < HN; e += 2) {           // the softmax scale is applied to dQ once, at the end
        const float2 ds = unpack_x2(mul_x2(pack_x2(__uint_as_float(s[e]), __uint_as_float(s[e + 1])),
                                           add_x2(pack_x2(__uint_as_float(d[e]), __uint_as_float(d[e + 1])), ndl)));
        pk[e >> 1] = pack_bf16(ds.x, ds.y);
      }
      tmem_st_half<HN>(s_addr, pk);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ds_full[b]);
    }
    if (ok && n_kv > 0 && mbar_wait(dq_done, 0, p.status, KS_TIMEOUT_TMEM_FULL)) {
      tc_fence_after();
      __nv_bfloat16* orow = reinterpret_cast<__nv_bfloat16*>(p.dq) +
                            static_cast<long long>(gq) * p.ldq + head * DH;
#pragma unroll 1
      for (int c = half; c < DH / 32; c += 2) {
        uint32_t r[32];
        tmem_ld_32x32(lane_addr + Cfg::TM_DQ + c * 32, r);
        tmem_ld_wait();
        if (gq < q_hi) {
          const float sc = p.scale;
#pragma unroll
          for (int e = 0; e < 32; e += 8) {
            uint4 v;
            v.x = pack_bf16(__uint_as_float(r[e]) * sc, __uint_as_float(r[e + 1]) * sc);
            v.y = pack_bf16(__uint_as_float(r[e + 2]) * sc, __uint_as_float(r[e + 3]) * sc);
            v.z = pack_bf16(__uint_as_float(r[e + 4]) * sc, __uint_as_float(r[e + 5]) * sc);
            v.w = pack_bf16(__uint_as_float(r[e + 6]) * sc, __uint_as_float(r[e + 7]) * sc);
            *reinterpret_cast<uint4*>(orow + c * 32 + e) = v;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == BW_MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem_base, Cfg::TM_COLS); }
}

// ============================================================================ dKV kernel
// dV and dK together: one buffer each for S^T and dP^T; the products of a tile are ordered so that the tensor pipe
// always has work while the softmax warps do theirs:
//   softmax warps   P^T of tile i                 dS^T of tile i
//   tensor pipe     dK of tile i-1, dP^T of i     dV of tile i, S^T of tile i+1
// dK alone follows the same order without P^T; dV alone has no second phase to hide S^T under and
// keeps two buffers of it instead: S^T of tile i+1 is then issued before P^T of tile i is waited for, so
// P^T has barriers for even and for odd tiles, as S^T has. With one buffer, every warp has arrived for a tile
// before any can start on the next, and one barrier is enough; the same holds for dP^T and dS^T.
enum { MODE_BOTH = 0, MODE_DV = 1, MODE_DK = 2 };

// Short batches: a key tile's queries are those of every head of its group, one CTA after another, and a
// few long tiles outlast the rest of the grid. With `split` > 1 a cluster of that many CTAs shares the
// tile, each with its part of the group's heads; their fp32 sums are added through distributed shared
// memory in the order of the CTAs, each CTA finishing its share of the rows.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t local, uint32_t rank) {
  float4 v;
  asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %4, %5;\n\t"
               "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n\t}"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(local), "r"(rank) : "memory");
  return v;
}
// Byte offset of four consecutive sums of a row; rows are a multiple of 128 bytes, so without the swizzle
// the lanes of a warp (a row each) would share banks.
__device__ __forceinline__ uint32_t sum_offset(int row, int cols, int c4) {
  return row * cols * 4 + (((c4 & ~7) | ((c4 ^ row) & 7)) << 4);
}

template <int DH, int BQ, int QS, int DOS, int MODE, int CTAS>
struct DkvCfg {
  static constexpr bool DO_DV = MODE != MODE_DK;
  static constexpr bool DO_DK = MODE != MODE_DV;
  static constexpr int SB = MODE == MODE_DV ? 2 : 1;       // buffers of S^T
  static constexpr int STS = DH == 256 ? 2 : 4;           // stages of the row statistics
  static constexpr int K_BYTES = 128 * DH * 2;
  static constexpr int QT_BYTES = BQ * DH * 2;
  static constexpr int OFF_V = K_BYTES;
  static constexpr int OFF_Q = OFF_V + (DO_DK ? K_BYTES : 0);
  static constexpr int OFF_DO = OFF_Q + QS * QT_BYTES;
  static constexpr int OFF_STAT = OFF_DO + DOS * QT_BYTES;
  static constexpr int OFF_BAR = OFF_STAT + STS * 2 * BQ * 4;
  static constexpr int SMEM = OFF_BAR + 256 + 1024;
  static constexpr int TM_ST = 0, TM_DPT = SB * BQ;
  static constexpr int TM_DV = 2 * BQ;
  static constexpr int TM_DK = TM_DV + (DO_DV ? DH : 0);
  static constexpr int SUMS = (DO_DV ? DH : 0) + (DO_DK ? DH : 0);
  static constexpr int TM_COLS = TM_DK + (DO_DK ? DH : 0) <= 256 ? 256 : 512;
  static_assert(TM_DK + (DO_DK ? DH : 0) <= TM_COLS && CTAS * TM_COLS <= 512, "TMEM budget");
  static_assert(128 * SUMS * 4 <= OFF_STAT, "the sums of a tile reuse the operands' space");
  static_assert(CTAS * (SMEM + 1024) <= 233472, "shared memory budget");
};

template <int DH, int BQ, int QS, int DOS, int MODE, int CTAS>
__global__ void __launch_bounds__(BW_THREADS, CTAS)
attn_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
                    const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                    const AttnBwdParams p) {
  using Cfg = DkvCfg<DH, BQ, QS, DOS, MODE, CTAS>;
  constexpr int STS = Cfg::STS, SB = Cfg::SB;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_smem_1024(smem_raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* kv_full = bars;             // 1
  uint64_t* q_full = bars + 1;          // 2
  uint64_t* q_empty = bars + 3;         // 2
  uint64_t* do_full = bars + 5;         // 2
  uint64_t* do_empty = bars + 7;        // 2
  uint64_t* stat_full = bars + 9;       // 4
  uint64_t* stat_empty = bars + 13;     // 4
  uint64_t* s_full = bars + 17;         // 2
  uint64_t* p_full = bars + 19;         // [buffer of S^T][first and second half of every warp's columns]
  uint64_t* dp_full = bars + 23;        // 1
  uint64_t* ds_full = bars + 24;        // 1
  uint64_t* s_free = bars + 25;         // 1 (only without a P^T to wait for)
  uint64_t* acc_done = bars + 26;       // 1
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 27);
  TileSlot* slot = reinterpret_cast<TileSlot*>(bars + 28);
  static_assert(28 * 8 + sizeof(TileSlot) <= 256, "barrier space");
  float* s_stat = reinterpret_cast<float*>(smem + Cfg::OFF_STAT);   // [STS][2][BQ]: -lse log2(e), -delta

  const int warp = static_cast<int>(warp_uniform(threadIdx.x >> 5)), lane = threadIdx.x & 31;
  const int shared = p.Hkv * p.split, rank = blockIdx.x / shared;      // tile; the CTAs of a cluster are neighbours
  const int kv_head = blockIdx.x % shared / p.split, part = blockIdx.x % p.split;
  const int rep = p.Hq / p.Hkv / p.split;                  // query heads of this CTA
  const int head0 = kv_head * (p.Hq / p.Hkv) + part * rep;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int i = 0; i < QS; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1); }
    for (int i = 0; i < DOS; ++i) { mbar_init(&do_full[i], 1); mbar_init(&do_empty[i], 1); }
    for (int i = 0; i < STS; ++i) { mbar_init(&stat_full[i], 1); mbar_init(&stat_empty[i], 8); }
    for (int i = 0; i < SB; ++i) mbar_init(&s_full[i], 1);
    for (int i = 0; i < 2 * SB; ++i) mbar_init(&p_full[i], 8);
    mbar_init(dp_full, 1);
    mbar_init(ds_full, 8);
    mbar_init(s_free, 8);
    mbar_init(acc_done, 1);
    mbar_fence_init();
  }
  if (warp == BW_MMA_WARP) { tmem_alloc(tmem_slot, Cfg::TM_COLS); tmem_relinquish(); }
  chain_wait();
  if (warp == BW_TMA_WARP) find_tile_by_work(p.cu_seqlens, p.nseq, 128, rank, slot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  chain_release();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  const int seq_start = slot->seq_start, seq_end = slot->seq_end;
  const int k0 = seq_start + ((seq_end - seq_start + 127) / 128 - slot->work) * 128;
  const int n_q = slot->work > 0 ? (seq_end - k0 + BQ - 1) / BQ : 0;   // query tiles at or after the key tile
  const int n_it = rep * n_q;

  if (warp == BW_TMA_WARP) {
    if (n_it > 0 && elect_one()) {
      mbar_expect_tx(kv_full, Cfg::DO_DK ? 2 * Cfg::K_BYTES : Cfg::K_BYTES);
#pragma unroll
      for (int c = 0; c < DH / 64; ++c) {
        tma_load_2d(smem + c * (128 * 128), &tmK, kv_full, kv_head * DH + c * 64, k0);
        if (Cfg::DO_DK)
          tma_load_2d(smem + Cfg::OFF_V + c * (128 * 128), &tmV, kv_full, kv_head * DH + c * 64, k0);
      }
      for (int it = 0; it < n_it; ++it) {
        const int qs = it % QS, ds = it % DOS;
        const int head = head0 + it / n_q;
        const int qt0 = k0 + (it % n_q) * BQ;
        if (it >= QS && !mbar_wait(&q_empty[qs], ((it / QS) - 1) & 1, p.status, KS_TIMEOUT_EMPTY)) break;
        uint8_t* sq = smem + Cfg::OFF_Q + qs * Cfg::QT_BYTES;
        mbar_expect_tx(&q_full[qs], Cfg::QT_BYTES);
#pragma unroll
        for (int c = 0; c < DH / 64; ++c)
          tma_load_2d(sq + c * (BQ * 128), &tmQ, &q_full[qs], head * DH + c * 64, qt0);
        if (it >= DOS && !mbar_wait(&do_empty[ds], ((it / DOS) - 1) & 1, p.status, KS_TIMEOUT_EMPTY)) break;
        uint8_t* sdo = smem + Cfg::OFF_DO + ds * Cfg::QT_BYTES;
        mbar_expect_tx(&do_full[ds], Cfg::QT_BYTES);
#pragma unroll
        for (int c = 0; c < DH / 64; ++c)
          tma_load_2d(sdo + c * (BQ * 128), &tmDO, &do_full[ds], head * DH + c * 64, qt0);
      }
    }
  } else if (warp == BW_MMA_WARP) {
    if (n_it > 0) {
      const uint32_t leader = elect_one();
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, BQ, false, false);
      constexpr uint32_t idesc_acc = umma_idesc_bf16(128, DH, false, true);
      const uint32_t sk = smem_u32(smem), sv = smem_u32(smem + Cfg::OFF_V);
      const uint32_t sq0 = smem_u32(smem + Cfg::OFF_Q), sdo0 = smem_u32(smem + Cfg::OFF_DO);
      auto scores = [&](uint32_t d, uint32_t a, uint32_t b) {
#pragma unroll
        for (int kk = 0; kk < DH / 16; ++kk)
          umma_bf16_if(leader, d, umma_smem_desc(a + (kk >> 2) * (128 * 128) + (kk & 3) * 32, 16, 1024),
                    umma_smem_desc(b + (kk >> 2) * (BQ * 128) + (kk & 3) * 32, 16, 1024), idesc_s, kk != 0);
      };
      // part 0 / 1: the steps over the first / second half of each warp's columns; -1: all
      auto accumulate = [&](uint32_t d, uint32_t a, uint32_t b, bool fresh, int part) {
#pragma unroll
        for (int kk = 0; kk < BQ / 16; ++kk)
          if (part < 0 || (kk * 16) % (BQ / 2) / (BQ / 4) == part)
            umma_bf16_ts_if(leader, d, a + packed_col<BQ>(kk), umma_smem_desc(b + kk * (16 * 128), BQ * 128, 1024),
                       idesc_acc, !(fresh && kk == 0));
      };
      auto issue_s = [&](int it) -> bool {
        if (!mbar_wait(&q_full[it % QS], (it / QS) & 1, p.status, KS_TIMEOUT_FULL)) return false;
        tc_fence_after();
        scores(tmem_base + Cfg::TM_ST + (it % SB) * BQ, sk, sq0 + (it % QS) * Cfg::QT_BYTES);
        umma_commit_if(leader, &s_full[it % SB]);
        return true;
      };
      bool ok = mbar_wait(kv_full, 0, p.status, KS_TIMEOUT_FULL) && issue_s(0);
      for (int it = 0; it < n_it && ok; ++it) {
        const uint32_t sq = sq0 + (it % QS) * Cfg::QT_BYTES, sdo = sdo0 + (it % DOS) * Cfg::QT_BYTES;
        ok = mbar_wait(&do_full[it % DOS], (it / DOS) & 1, p.status, KS_TIMEOUT_FULL);
        if (!ok) break;
        tc_fence_after();
        if (Cfg::DO_DK) {
          // dP^T overwrites the dS^T that the dK product before it reads: products of one issuing
          // thread run in order (the same holds for S^T and P^T below)
          scores(tmem_base + Cfg::TM_DPT, sv, sdo);
          umma_commit_if(leader, dp_full);
        }
        if (SB == 2 && it + 1 < n_it) { ok = issue_s(it + 1); if (!ok) break; }
        if (Cfg::DO_DV) {
          // S^T of the next tile waits behind this product, and P^T of the next tile for that: its first half
          // starts under the exponentials of the second
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            ok = mbar_wait(&p_full[it % SB * 2 + x], (it / SB) & 1, p.status, KS_TIMEOUT_FULL);
            if (!ok) break;
            tc_fence_after();
            accumulate(tmem_base + Cfg::TM_DV, tmem_base + Cfg::TM_ST + (it % SB) * BQ, sdo, it == 0, x);
          }
          if (!ok) break;
          if (!Cfg::DO_DK) umma_commit_if(leader, &q_empty[it % QS]);
        } else {
          ok = mbar_wait(s_free, it & 1, p.status, KS_TIMEOUT_TMEM_EMPTY);
          if (!ok) break;
          tc_fence_after();
        }
        umma_commit_if(leader, &do_empty[it % DOS]);
        if (SB == 1 && it + 1 < n_it) { ok = issue_s(it + 1); if (!ok) break; }
        if (Cfg::DO_DK) {
          ok = mbar_wait(ds_full, it & 1, p.status, KS_TIMEOUT_FULL);
          if (!ok) break;
          tc_fence_after();
          accumulate(tmem_base + Cfg::TM_DK, tmem_base + Cfg::TM_DPT, sq, it == 0, -1);
          umma_commit_if(leader, &q_empty[it % QS]);
        }
        if (it + 1 == n_it) umma_commit_if(leader, acc_done);
      }
    }
  } else if (warp == BW_STAT_WARP) {
    // log-sum-exp and delta of each tile's queries, fetched ahead of the softmax warps. A query past
    // the end of the sequence gets a probability of zero. All loads of a tile are issued before its
    // first store: with a store between them, each waits for the one before it (a full memory
    // latency per load, which held the whole kernel back).
    constexpr int NU = BQ / 32;
    for (int it = 0; it < n_it; ++it) {
      const int st = it % STS;
      const int qt0 = k0 + (it % n_q) * BQ;
      const long long base = static_cast<long long>(head0 + it / n_q) * p.T;
      float nl[NU], dl[NU];
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        const int gq = qt0 + lane + u * 32;
        const bool in = gq < seq_end;
        nl[u] = in ? -p.lse[base + gq] * LOG2E : -INFINITY;
        dl[u] = in ? -p.delta[base + gq] : 0.f;
      }
      if (it >= STS && !mbar_wait(&stat_empty[st], ((it / STS) - 1) & 1, p.status, KS_TIMEOUT_EMPTY)) break;
      const uint32_t dst = smem_u32(s_stat + st * (2 * BQ) + lane);
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        st_shared_f32(dst + u * 128, nl[u]);
        st_shared_f32(dst + BQ * 4 + u * 128, dl[u]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&stat_full[st]);
    }
  } else {
    constexpr int HN = BQ / 2;
    const int quarter = warp & 3, half = warp >> 2;
    const int row = quarter * 32 + lane;     // key row within the tile
    const int gk = k0 + row;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const uint32_t dp_addr = lane_addr + Cfg::TM_DPT + half * HN;
    const f32x2 c2 = pack_x2(p.scale * LOG2E, p.scale * LOG2E);
    const uint32_t stat = smem_u32(s_stat);
    bool ok = true;
    for (int it = 0; it < n_it; ++it) {
      const int st = it % STS;
      const int qt0 = k0 + (it % n_q) * BQ;
      const uint32_t nlse = stat + (st * (2 * BQ) + half * HN) * 4, ndelta = nlse + BQ * 4;
      if (!mbar_wait(&stat_full[st], (it / STS) & 1, p.status, KS_TIMEOUT_FULL)) { ok = false; break; }
      const uint32_t s_addr = lane_addr + Cfg::TM_ST + (it % SB) * BQ + half * HN;
      if (!mbar_wait(&s_full[it % SB], (it / SB) & 1, p.status, KS_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      uint32_t s[HN];
      tmem_ld_half<HN>(s_addr, s);
      if (!Cfg::DO_DV) {                      // nothing goes back into these columns
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_free);
      }
      // whole tile visible: every query of the tile is at or after every key, none past the end
      const bool all_valid = qt0 >= k0 + 127 && qt0 + BQ <= seq_end;
      const int first = gk - (qt0 + half * HN), last = seq_end - (qt0 + half * HN);   // visible: [first, last)
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        constexpr int PN = HN / 2;
        uint32_t pk[PN / 2];
#pragma unroll
        for (int e = x * PN; e < (x + 1) * PN; e += 4) {
          f32x2 l[2];
          ld_shared_2x2(nlse + e * 4, l[0], l[1]);
#pragma unroll
          for (int u = 0; u < 4; u += 2) {
            const float2 t = unpack_x2(fma_x2(pack_x2(__uint_as_float(s[e + u]), __uint_as_float(s[e + u + 1])), c2,
                                              l[u >> 1]));
            s[e + u] = __float_as_uint(fast_exp2(t.x));
            s[e + u + 1] = __float_as_uint(fast_exp2(t.y));
          }
        }
        if (!all_valid) {
#pragma unroll
          for (int e = x * PN; e < (x + 1) * PN; ++e)
            if (e < first || e >= last) s[e] = 0u;
        }
        if (Cfg::DO_DV) {
#pragma unroll
          for (int e = 0; e < PN; e += 2)
            pk[e >> 1] = pack_bf16(__uint_as_float(s[x * PN + e]), __uint_as_float(s[x * PN + e + 1]));
          tmem_st_quarter<PN>(s_addr + x * (PN / 2), pk);
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&p_full[it % SB * 2 + x]);
        }
      }
      if (Cfg::DO_DK) {
        if (!mbar_wait(dp_full, it & 1, p.status, KS_TIMEOUT_TMEM_FULL)) { ok = false; break; }
        tc_fence_after();
        uint32_t d[HN], pk[HN / 2];
        tmem_ld_half<HN>(dp_addr, d);
#pragma unroll
        for (int e = 0; e < HN; e += 4) {     // the softmax scale is applied to dK once, at the end
          f32x2 ndl[2];
          ld_shared_2x2(ndelta + e * 4, ndl[0], ndl[1]);
#pragma unroll
          for (int u = 0; u < 4; u += 2) {
            const float2 ds =
                unpack_x2(mul_x2(pack_x2(__uint_as_float(s[e + u]), __uint_as_float(s[e + u + 1])),
                                 add_x2(pack_x2(__uint_as_float(d[e + u]), __uint_as_float(d[e + u + 1])), ndl[u >> 1])));
            pk[(e + u) >> 1] = pack_bf16(ds.x, ds.y);
          }
        }
        tmem_st_half<HN>(dp_addr, pk);
        tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) {
        if (Cfg::DO_DK) mbar_arrive(ds_full);
        mbar_arrive(&stat_empty[st]);
      }
    }
    if (ok && n_it > 0 && mbar_wait(acc_done, 0, p.status, KS_TIMEOUT_TMEM_FULL)) {
      tc_fence_after();
      const bool valid = gk < seq_end;
      auto leave_sums = [&](uint32_t tm_col, int col0) {
#pragma unroll 1
        for (int c = half; c < DH / 32; c += 2) {
          uint32_t r[32];
          tmem_ld_32x32(lane_addr + tm_col + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; e += 4)
            *reinterpret_cast<uint4*>(smem + sum_offset(row, Cfg::SUMS, (col0 + c * 32 + e) >> 2)) =
                make_uint4(r[e], r[e + 1], r[e + 2], r[e + 3]);
        }
      };
      auto store_acc = [&](uint32_t tm_col, void* base, long long ld, float sc) {
        __nv_bfloat16* orow = reinterpret_cast<__nv_bfloat16*>(base) +
                              static_cast<long long>(gk) * ld + kv_head * DH;
#pragma unroll 1
        for (int c = half; c < DH / 32; c += 2) {
          uint32_t r[32];
          tmem_ld_32x32(lane_addr + tm_col + c * 32, r);
          tmem_ld_wait();
          if (valid) {
#pragma unroll
            for (int e = 0; e < 32; e += 8) {
              uint4 v;
              v.x = pack_bf16(__uint_as_float(r[e]) * sc, __uint_as_float(r[e + 1]) * sc);
              v.y = pack_bf16(__uint_as_float(r[e + 2]) * sc, __uint_as_float(r[e + 3]) * sc);
              v.z = pack_bf16(__uint_as_float(r[e + 4]) * sc, __uint_as_float(r[e + 5]) * sc);
              v.w = pack_bf16(__uint_as_float(r[e + 6]) * sc, __uint_as_float(r[e + 7]) * sc);
              *reinterpret_cast<uint4*>(orow + c * 32 + e) = v;
            }
          }
        }
      };
      if (p.split > 1) {
        if (Cfg::DO_DV) leave_sums(Cfg::TM_DV, 0);
        if (Cfg::DO_DK) leave_sums(Cfg::TM_DK, Cfg::DO_DV ? DH : 0);
      } else {
        if (Cfg::DO_DK) store_acc(Cfg::TM_DK, p.dk, p.ldk, p.scale);
        if (Cfg::DO_DV) store_acc(Cfg::TM_DV, p.dv, p.ldv, 1.f);
      }
    }
  }
  if (p.split > 1) {
    __syncwarp();
    cluster_sync();                                        // every CTA's sums are in its shared memory
    if (warp < 8 && n_it > 0) {
      const int rows = 128 / p.split, per_row = Cfg::SUMS / 4;
      for (int x = threadIdx.x; x < rows * per_row; x += 256) {
        const int row = part * rows + x / per_row, c4 = x % per_row, gk = k0 + row;
        const uint32_t at = smem_u32(smem) + sum_offset(row, Cfg::SUMS, c4);
        float4 v = ld_cluster_f4(at, 0);
        for (int r = 1; r < p.split; ++r) {
          const float4 o = ld_cluster_f4(at, r);
          v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
        }
        if (gk >= seq_end) continue;
        const bool is_dk = !Cfg::DO_DV || (Cfg::DO_DK && c4 * 4 >= DH);
        const int col = c4 * 4 - (is_dk && Cfg::DO_DV ? DH : 0);
        const float sc = is_dk ? p.scale : 1.f;
        __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(is_dk ? p.dk : p.dv) +
                             static_cast<long long>(gk) * (is_dk ? p.ldk : p.ldv) + kv_head * DH + col;
        *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16(v.x * sc, v.y * sc), pack_bf16(v.z * sc, v.w * sc));
      }
    }
    cluster_sync();                                        // no CTA leaves while another reads its sums
  }
  tc_fence_before();
  __syncthreads();
  if (warp == BW_MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem_base, Cfg::TM_COLS); }
}

template <int DH, int BKV, int KS, int VS, int CTAS>
static int launch_dq(const CUtensorMap& tq, const CUtensorMap& tdo, const CUtensorMap& tk,
                     const CUtensorMap& tv, const AttnBwdParams& p, int tiles, cudaStream_t s) {
  using Cfg = DqCfg<DH, BKV, KS, VS, CTAS>;
  auto kern = attn_bwd_dq_kernel<DH, BKV, KS, VS, CTAS>;
  static SmemOptIn opt_in;
  if (int e = opt_in.ensure(kern, Cfg::SMEM)) return e;
  const long long grid = static_cast<long long>(p.Hq) * tiles;       // see attention_fwd.cu
  if (grid > 0x7fffffffLL) return -2;
  launch_chained(kern, static_cast<unsigned>(grid), BW_THREADS, Cfg::SMEM, s, tq, tdo, tk, tv, p);
  return static_cast<int>(cudaGetLastError());
}

template <int DH, int BQ, int QS, int DOS, int MODE, int CTAS>
static int launch_dkv(const CUtensorMap& tq, const CUtensorMap& tdo, const CUtensorMap& tk,
                      const CUtensorMap& tv, const AttnBwdParams& p, int tiles, cudaStream_t s) {
  using Cfg = DkvCfg<DH, BQ, QS, DOS, MODE, CTAS>;
  auto kern = attn_bwd_dkv_kernel<DH, BQ, QS, DOS, MODE, CTAS>;
  static SmemOptIn opt_in;
  if (int e = opt_in.ensure(kern, Cfg::SMEM)) return e;
  cudaLaunchConfig_t cfg = {};
  const long long grid = static_cast<long long>(p.Hkv) * p.split * tiles;
  if (grid > 0x7fffffffLL) return -2;
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(BW_THREADS);
  cfg.dynamicSmemBytes = Cfg::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attrs[2];
  attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // as launch_chained
  attrs[0].val.programmaticStreamSerializationAllowed = 1;
  attrs[1].id = cudaLaunchAttributeClusterDimension;
  attrs[1].val.clusterDim.x = p.split;
  attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
  cfg.attrs = attrs;
  cfg.numAttrs = p.split > 1 ? 2 : 1;
  if (cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tq, tdo, tk, tv, p)) return static_cast<int>(e);
  return static_cast<int>(cudaGetLastError());
}

// CTAs per key tile of the dKV kernel, from the number of key tiles (all KV heads) and the heads of a group.
// A split halves the longest tile and costs each CTA its own K, V and the exchange of its sums. Measured
// (dKV kernels, us at split 1 / 2 / 4):
//   16 tiles   256 x 32/8 heads of 128      23.5 / 18.7 / 15.2      48   3000 x 8/2 of 256    539 / 293 / 159
//   64         1000 x 32/8 of 128             48 / 32 / 47         128   2048 x 32/8 of 64     66 / 51 / 80
//  188         6001 x 16/4 of 256            723 / 444 / 603       256   4096 x 32/8 of 128   166 / 180 / 234
//  256         8192 x 16/4 of 256            564 / 580 / 743       512   8192 x 32/8 of 128   326 / 378 / 498
static int key_tile_split(long long tiles, int group) {
  if (group % 4 == 0 && tiles * 8 <= 3 * 148) return 4;
  if (group % 2 == 0 && tiles * 3 <= 4 * 148) return 2;
  return 1;
}

}  // namespace ss

// delta_scratch: fp32 [Hq, T] caller-provided scratch.
// lddq / lddk / lddv: row pitches of the gradient buffers, which need not be those of q, k, v
// (a fused q/k/v projection read through views, gradients written to tensors of their own).
extern "C" int ss_attn_bwd_g(const void* q, const void* k, const void* v, const void* out,
                             const float* lse, const void* dout, void* dq, void* dk, void* dv,
                             const int* cu_seqlens, float* delta_scratch, int nseq, int T, int Hq,
                             int Hkv, int dh, long long ldq, long long ldk, long long ldv,
                             long long ldo, long long lddq, long long lddk, long long lddv,
                             float scale, int* status, void* stream) {
  using namespace ss;
  if (T <= 0 || nseq <= 0) return 0;
  if (delta_scratch == nullptr) return -2;
  if ((ldq % 8) || (ldk % 8) || (ldv % 8) || (ldo % 8) || Hq % Hkv) return -2;
  if ((lddq % 8) || (lddk % 8) || (lddv % 8)) return -2;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (dh != 64 && dh != 128 && dh != 256) return -2;
  if ((reinterpret_cast<uintptr_t>(out) & 3) || (reinterpret_cast<uintptr_t>(dout) & 15)) return -2;
  {
    const long long blocks = (static_cast<long long>(T) * Hq * (dh / 8) + 255) / 256;
    auto run = [&](auto kern) {
      launch_chained(kern, static_cast<unsigned>(blocks), 256, 0, s,
          reinterpret_cast<const __nv_bfloat16*>(out), reinterpret_cast<const __nv_bfloat16*>(dout), delta_scratch, T,
          Hq, static_cast<long long>(Hq) * dh, ldo);
    };
    const bool wide = (reinterpret_cast<uintptr_t>(out) & 15) == 0;
    if (dh == 64) run(wide ? attn_delta_kernel<64, true> : attn_delta_kernel<64, false>);
    else if (dh == 128) run(wide ? attn_delta_kernel<128, true> : attn_delta_kernel<128, false>);
    else run(wide ? attn_delta_kernel<256, true> : attn_delta_kernel<256, false>);
  }
  AttnBwdParams p;
  p.dq = dq; p.dk = dk; p.dv = dv; p.lse = lse; p.delta = delta_scratch; p.cu_seqlens = cu_seqlens;
  p.nseq = nseq; p.T = T; p.Hq = Hq; p.Hkv = Hkv; p.ldq = lddq; p.ldk = lddk; p.ldv = lddv;
  p.scale = scale; p.status = status;
  const int tiles = (T + 127) / 128 + nseq;
  p.split = key_tile_split(static_cast<long long>((T + 127) / 128) * Hkv, Hq / Hkv);
  const long long qc = static_cast<long long>(Hq) * dh, kc = static_cast<long long>(Hkv) * dh;
  const int stream_rows = dh == 128 ? 128 : 64;     // rows of the streamed tiles
  CUtensorMap tq128, tdo128, tk128, tv128, tqs, tdos, tks, tvs;
  int r;
  if ((r = make_tmap_bf16(&tq128, q, T, qc, ldq, 128))) return r;
  if ((r = make_tmap_bf16(&tdo128, dout, T, qc, ldo, 128))) return r;
  if ((r = make_tmap_bf16(&tk128, k, T, kc, ldk, 128))) return r;
  if ((r = make_tmap_bf16(&tv128, v, T, kc, ldv, 128))) return r;
  if ((r = make_tmap_bf16(&tqs, q, T, qc, ldq, stream_rows))) return r;
  if ((r = make_tmap_bf16(&tdos, dout, T, qc, ldo, stream_rows))) return r;
  if ((r = make_tmap_bf16(&tks, k, T, kc, ldk, stream_rows))) return r;
  if ((r = make_tmap_bf16(&tvs, v, T, kc, ldv, stream_rows))) return r;
  if (dh == 128) {
    if ((r = launch_dq<128, 128, 3, 2, 1>(tq128, tdo128, tks, tvs, p, tiles, s))) return r;
    return launch_dkv<128, 128, 2, 2, MODE_BOTH, 1>(tqs, tdos, tk128, tv128, p, tiles, s);
  }
  if (dh == 64) {
    if ((r = launch_dq<64, 64, 3, 2, 2>(tq128, tdo128, tks, tvs, p, tiles, s))) return r;
    return launch_dkv<64, 64, 2, 2, MODE_BOTH, 2>(tqs, tdos, tk128, tv128, p, tiles, s);
  }
  if (dh == 256) {
    if ((r = launch_dq<256, 64, 2, 1, 1>(tq128, tdo128, tks, tvs, p, tiles, s))) return r;
    if ((r = launch_dkv<256, 64, 2, 2, MODE_DV, 1>(tqs, tdos, tk128, tv128, p, tiles, s))) return r;
    return launch_dkv<256, 64, 2, 1, MODE_DK, 1>(tqs, tdos, tk128, tv128, p, tiles, s);
  }
  return -2;
}

// delta_scratch: fp32 [Hq, T] caller-provided scratch. Gradients have the pitches of their operands.
extern "C" int ss_attn_bwd(const void* q, const void* k, const void* v, const void* out,
                           const float* lse, const void* dout, void* dq, void* dk, void* dv,
                           const int* cu_seqlens, float* delta_scratch, int nseq, int T, int Hq,
                           int Hkv, int dh, long long ldq, long long ldk, long long ldv,
                           long long ldo, float scale, int* status, void* stream) {
  return ss_attn_bwd_g(q, k, v, out, lse, dout, dq, dk, dv, cu_seqlens, delta_scratch, nseq, T, Hq, Hkv,
                       dh, ldq, ldk, ldv, ldo, ldq, ldk, ldv, scale, status, stream);
}

// ============================================================================ no-allocation entry
// See attention_noalloc.h. The scratch that ss_attn_bwd takes from its caller
// (delta, fp32 [Hq, T]) lives here in a fixed device array instead, so the call
// performs no allocation of any kind.
#include "attention_noalloc.h"
#include "launchers.h"

#include <mutex>

namespace ss {

// Every GPU that loads this library holds this array until the process exits.
static __device__ __align__(256) float g_attn_delta_scratch[SS_ATTN_NOALLOC_MAX_ELEMENTS];

constexpr int kMaxDevices = 64;
static float* g_scratch_address[kMaxDevices];   // device address of the array, per device
static std::mutex g_scratch_mutex;

// In host code `g_attn_delta_scratch` is only a stand-in symbol, not an address a
// kernel can use; the device address has to be asked for, once per device, with
// that device current.
static int scratch_for_current_device(float** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return static_cast<int>(e);
  if (dev < 0 || dev >= kMaxDevices) return SS_ATTN_NOALLOC_BAD_DEVICE;
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (g_scratch_address[dev] == nullptr) {
    float* ptr = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_attn_delta_scratch);
    if (e != cudaSuccess) return static_cast<int>(e);
    g_scratch_address[dev] = ptr;
  }
  *out = g_scratch_address[dev];
  return 0;
}

}  // namespace ss

extern "C" long long ss_attn_bwd_noalloc_max_elements(void) { return SS_ATTN_NOALLOC_MAX_ELEMENTS; }

extern "C" int ss_attn_bwd_noalloc(const void* q, const void* k, const void* v, const void* out,
                                   const float* lse, const void* dout, void* dq, void* dk, void* dv,
                                   const int* cu_seqlens, int nseq, int T, int Hq, int Hkv, int dh,
                                   long long ldq, long long ldk, long long ldv, long long ldo,
                                   float scale, int* status, void* stream) {
  if (T <= 0 || nseq <= 0) return 0;
  if (Hq <= 0 || Hkv <= 0) return -2;          // the same answer ss_attn_bwd gives
  if (static_cast<long long>(Hq) * T > SS_ATTN_NOALLOC_MAX_ELEMENTS)
    return SS_ATTN_NOALLOC_TOO_LARGE;
  // The scratch array handed to the kernels is the CURRENT device's copy. If the operands
  // live on another GPU the kernels would run there (the tensor-map set-up binds the
  // operands' device) with this GPU's array: refuse instead.
  {
    int current = -1;
    if (cudaGetDevice(&current) != cudaSuccess) return SS_ATTN_NOALLOC_BAD_DEVICE;
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, dq) != cudaSuccess) {
      cudaGetLastError();
      return SS_ATTN_NOALLOC_BAD_DEVICE;
    }
    if (attr.type != cudaMemoryTypeDevice || attr.device != current)
      return SS_ATTN_NOALLOC_BAD_DEVICE;
  }
  float* scratch = nullptr;
  if (int rc = ss::scratch_for_current_device(&scratch)) return rc;
  return ss_attn_bwd(q, k, v, out, lse, dout, dq, dk, dv, cu_seqlens, scratch, nseq, T, Hq, Hkv,
                     dh, ldq, ldk, ldv, ldo, scale, status, stream);
}
