// Packed variable-length causal GQA attention, forward, for sm_100a.
//
// One CTA per (128-query tile of a sequence, query head). Head widths 64 and 128 take half of TMEM (two 64-key score
// buffers and O) and half of an SM's shared memory, so two CTAs share an SM: one's set-up, waits and epilogue run under
// the other's steps, and neither waits for the other's probabilities. Two tiles in one CTA shared K and V, but their
// products were issued by one warp in one order. Head width 256: O takes half of TMEM, one CTA per SM.
// S = Q K^T of the next 64 keys is always issued before O += P V of these, so the softmax warps never
// wait for a product.
// P goes back to TMEM over the scores it comes from and is the A operand of P V from there: it never
// passes through shared memory, whose bandwidth the two products need for K, V and Q.
// Measured (two tiles in a CTA -> two CTAs, both kernels in turn, the forward kernel alone): 8,192 packed tokens, 32/8 heads
// of 128: 208 -> 192.5 us; 16,384 tokens in two sequences: 1,013 -> 968; 2,048 tokens in five sequences: 47 -> 39; heads of
// 64, 2,048 tokens: 39 -> 32.7, 16,384: 810 -> 784. 6,001 tokens, 16/4 heads of 256 (one CTA): 158 us. What is left is the
// softmax warps' chain (read, maximum, exponentials, write). Replacing a quarter of the exponentials by polynomials of ten
// instructions made it slower (1.08 against 0.97 ms), and so did scores two steps ahead (1.04).
//
//   warps 0..3  softmax, rescaling of O, epilogue: one query row per thread
//   then one TMA producer warp and one MMA warp
//
// The scores of step j + 1 are issued before P of step j is waited for, so two steps are in flight and the
// warps of a tile may be a step apart. Whatever is arrived on or waited for once per step therefore has a
// barrier for even and one for odd steps: with one for both, a warp a step ahead completes the phase that a
// slower one has yet to arrive on, or a phase that is waited for passes twice and its parity turns back.
// Scores of step j + 2 are only issued once P of step j has been taken, so no barrier is arrived on twice
// before it has been waited for.
//
// Semantics: the reference's packed attention contract
// (packages/workloads/src/shadowspill_workloads/models/shared/decoder.py:251):
// each [cu_seqlens[i], cu_seqlens[i+1]) is an independent causal sequence.
#include "sm100_ptx.cuh"
#include "attention_tiles.cuh"
#include "launchers.h"

#include <cudaTypedefs.h>
#include <math.h>

namespace ss {

int make_tmap_bf16(CUtensorMap* map, const void* base, long long rows, long long cols,
                   long long ld, int box_rows);  // gemm_tcgen05.cu

// BKV keys per step, KS / VS stages of K and V (K is released by its score products, V one step later by P V), CTAS to
// an SM.
template <int DH, int BKV, int KS, int VS, int CTAS>
struct AttnCfg {
  static constexpr int THREADS = 4 * 32 + 64;
  static constexpr int TMA_WARP = 4, MMA_WARP = 5;
  static constexpr int QT_BYTES = 128 * DH * 2;
  static constexpr int KV_BYTES = BKV * DH * 2;        // one of K or V
  static constexpr int OFF_K = QT_BYTES;
  static constexpr int OFF_V = OFF_K + KS * KV_BYTES;
  static constexpr int OFF_BAR = OFF_V + VS * KV_BYTES;
  static constexpr int SMEM = OFF_BAR + 256 + 1024;
  static constexpr int TM_O = 2 * BKV;                 // behind the two score buffers
  static constexpr int TM_COLS = TM_O + DH <= 256 ? 256 : 512;
  static_assert(TM_O + DH <= TM_COLS && CTAS * TM_COLS <= 512, "TMEM budget");
  static_assert(CTAS * (SMEM + 1024) <= 233472, "shared memory budget");
};

struct AttnParams {
  void* out;
  float* lse;
  const int* cu_seqlens;
  int nseq, T, Hq, Hkv;
  long long ldo;
  float scale_log2;   // softmax scale * log2(e)
  int* status;
};

template <int DH, int BKV, int KS, int VS, int CTAS>
__global__ void __launch_bounds__(192, CTAS)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const AttnParams p) {
  using Cfg = AttnCfg<DH, BKV, KS, VS, CTAS>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_smem_1024(smem_raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* q_full = bars;                // 1
  uint64_t* k_full = bars + 1;            // KS
  uint64_t* k_empty = k_full + KS;        // KS
  uint64_t* v_full = k_empty + KS;        // VS
  uint64_t* v_empty = v_full + VS;        // VS
  uint64_t* s_full = v_empty + VS;        // [buffer]
  uint64_t* p_full = s_full + 2;          // [step & 1]
  uint64_t* o_done = p_full + 2;          // [step & 1]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_done + 2);
  TileSlot* slot = reinterpret_cast<TileSlot*>(o_done + 3);
  static_assert((1 + 2 * KS + 2 * VS + 7) * 8 + sizeof(TileSlot) <= 256, "barrier space");

  const int warp = static_cast<int>(warp_uniform(threadIdx.x >> 5));
  const int lane = threadIdx.x & 31;
  const int head = blockIdx.x % p.Hq, rank = blockIdx.x / p.Hq;
  const int kv_head = head / (p.Hq / p.Hkv);

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < KS; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); }
    for (int i = 0; i < VS; ++i) { mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 4);
      mbar_init(&o_done[i], 1);
    }
    mbar_fence_init();
  }
  if (warp == Cfg::MMA_WARP) {
    tmem_alloc(tmem_slot, Cfg::TM_COLS);
    tmem_relinquish();
  }
  chain_wait();
  if (warp == Cfg::TMA_WARP) find_tile_by_work(p.cu_seqlens, p.nseq, 128, rank, slot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  chain_release();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  const int seq_start = slot->seq_start, seq_end = slot->seq_end;
  const int q0 = seq_start + (slot->work - 1) * 128;
  // key steps of the tile, up to its diagonal
  const int n = slot->work > 0 ? (min(q0 + 128, seq_end) - seq_start + BKV - 1) / BKV : 0;

  if (warp == Cfg::TMA_WARP) {
    // ---------------------------------------------------------------- producer
    if (n > 0 && elect_one()) {
      tma_prefetch_desc(&tmQ);
      tma_prefetch_desc(&tmK);
      tma_prefetch_desc(&tmV);
      mbar_expect_tx(q_full, Cfg::QT_BYTES);
#pragma unroll
      for (int c = 0; c < DH / 64; ++c) tma_load_2d(smem + c * (128 * 128), &tmQ, q_full, head * DH + c * 64, q0);
      for (int j = 0; j < n; ++j) {
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
  } else if (warp == Cfg::MMA_WARP) {
    // ---------------------------------------------------------------- MMA issuer
    if (n > 0) {
      const uint32_t leader = elect_one();
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, BKV, false, false);
      constexpr uint32_t idesc_o = umma_idesc_bf16(128, DH, false, true);
      const uint32_t sq = smem_u32(smem);
      const uint32_t sk0 = smem_u32(smem + Cfg::OFF_K), sv0 = smem_u32(smem + Cfg::OFF_V);
      // products of one issuing thread run in order: S may be issued over the P that the P V product
      // before it reads
      auto issue_s = [&](int j) -> bool {
        if (!mbar_wait(&k_full[j % KS], (j / KS) & 1, p.status, KS_TIMEOUT_FULL)) return false;
        tc_fence_after();
        const uint32_t k = sk0 + (j % KS) * Cfg::KV_BYTES;
#pragma unroll
        for (int kk = 0; kk < DH / 16; ++kk)
          umma_bf16_if(leader, tmem_base + (j & 1) * BKV, umma_smem_desc(sq + (kk >> 2) * (128 * 128) + (kk & 3) * 32, 16, 1024),
                    umma_smem_desc(k + (kk >> 2) * (BKV * 128) + (kk & 3) * 32, 16, 1024), idesc_s, kk != 0);
        umma_commit_if(leader, &s_full[j & 1]);
        umma_commit_if(leader, &k_empty[j % KS]);
        return true;
      };
      bool ok = mbar_wait(q_full, 0, p.status, KS_TIMEOUT_FULL) && issue_s(0);
      for (int j = 0; j < n && ok; ++j) {
        // V ahead of the next scores where a CTA has the SM to itself: 160.4 -> 157.9 us at 6,001 tokens of width 256 (two
        // to an SM: 192.5 -> 193.3 for the packed case above)
        if constexpr (CTAS == 1) {
          if (!mbar_wait(&v_full[j % VS], (j / VS) & 1, p.status, KS_TIMEOUT_FULL)) break;
          if (j + 1 < n) ok = issue_s(j + 1);
        } else {
          if (j + 1 < n) ok = issue_s(j + 1);
          if (ok) ok = mbar_wait(&v_full[j % VS], (j / VS) & 1, p.status, KS_TIMEOUT_FULL);
        }
        if (!ok || !mbar_wait(&p_full[j & 1], (j >> 1) & 1, p.status, KS_TIMEOUT_FULL)) break;
        tc_fence_after();
        const uint32_t v = sv0 + (j % VS) * Cfg::KV_BYTES, pa = tmem_base + (j & 1) * BKV;
#pragma unroll
        for (int kk = 0; kk < BKV / 16; ++kk)
          umma_bf16_ts_if(leader, tmem_base + Cfg::TM_O, pa + kk * 8, umma_smem_desc(v + kk * (16 * 128), BKV * 128, 1024),
                       idesc_o, (j | kk) != 0);
        umma_commit_if(leader, &o_done[j & 1]);
        umma_commit_if(leader, &v_empty[j % VS]);
      }
    }
  } else {
    // ---------------------------------------------------------------- softmax warps
    const int gq = q0 + warp * 32 + lane;        // global query index; its row is the TMEM lane
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);
    const uint32_t o_addr = lane_addr + Cfg::TM_O;
    const bool negative = p.scale_log2 < 0.f;    // the row maximum is taken before the scale
    const float c = fabsf(p.scale_log2);
    float m_used = -INFINITY;                    // reference max (log2 domain, scaled)
    float l = 0.f;
    bool ok = true;
    for (int j = 0; j < n; ++j) {
      const int b = j & 1;
      const uint32_t s_addr = lane_addr + b * BKV;
      if (!mbar_wait(&s_full[b], (j >> 1) & 1, p.status, KS_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      tc_fence_after();
      float s[BKV];
#pragma unroll
      for (int x = 0; x < BKV; x += 32)
        tmem_ld_32x32(s_addr + x, reinterpret_cast<uint32_t (&)[32]>(s[x]));
      tmem_ld_wait();
      if (negative) {
#pragma unroll
        for (int e = 0; e < BKV; ++e) s[e] = -s[e];
      }
      const int k0 = seq_start + j * BKV;
      const bool diag = k0 + BKV - 1 > q0;      // some key of this step may exceed some query
      if (diag) {
#pragma unroll
        for (int e = 0; e < BKV; ++e)
          if (k0 + e > gq) s[e] = -INFINITY;
      }
      float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
      for (int e = 4; e + 8 <= BKV; e += 8) {
#pragma unroll
        for (int u = 0; u < 4; ++u) mx[u] = max3(mx[u], s[e + u], s[e + 4 + u]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) mx[u] = fmaxf(mx[u], s[BKV - 4 + u]);
      const float m_t = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * c;
      // lazy rescale: move the reference max only when it would grow by > 8 (2^8 headroom)
      const bool want = m_t > m_used + 8.f;
      if (j == 0) {
        m_used = fmaxf(m_used, m_t);
      } else if (__ballot_sync(0xffffffffu, want) != 0u) {
        const float m_new = fmaxf(m_used, m_t);
        const float alpha = m_used == -INFINITY ? 0.f : fast_exp2(m_used - m_new);
        m_used = m_new;
        l *= alpha;
        if (!mbar_wait(&o_done[b ^ 1], ((j - 1) >> 1) & 1, p.status, KS_TIMEOUT_TMEM_FULL)) { ok = false; break; }
        tc_fence_after();
#pragma unroll 1
        for (int x = 0; x < DH; x += 32) {
          uint32_t r[32];
          tmem_ld_32x32(o_addr + x, r);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(__uint_as_float(r[e]) * alpha);
          tmem_st_32x32(o_addr + x, r);
        }
      }
      const f32x2 nm = pack_x2(-m_used, -m_used), cc = pack_x2(c, c);
      f32x2 sum[2] = {0ull, 0ull};
#pragma unroll
      for (int x = 0; x < BKV; x += 32) {
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          const float2 t = unpack_x2(fma_x2(pack_x2(s[x + e], s[x + e + 1]), cc, nm));
          float p0 = fast_exp2(t.x);
          float p1 = fast_exp2(t.y);
          if (diag) {
            if (k0 + x + e > gq) p0 = 0.f;
            if (k0 + x + e + 1 > gq) p1 = 0.f;
          }
          sum[(e & 2) >> 1] = add_x2(sum[(e & 2) >> 1], pack_x2(p0, p1));
          pk[e >> 1] = pack_bf16(p0, p1);
        }
        tmem_st_32x16(s_addr + (x >> 1), pk);
      }
      const float2 sa = unpack_x2(sum[0]), sb = unpack_x2(sum[1]);
      l += (sa.x + sa.y) + (sb.x + sb.y);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[b]);
    }
    // ---------------------------------------------------------------- epilogue
    if (ok && n > 0 && mbar_wait(&o_done[(n - 1) & 1], ((n - 1) >> 1) & 1, p.status, KS_TIMEOUT_TMEM_FULL)) {
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      const bool valid = gq < seq_end;
      __nv_bfloat16* orow = reinterpret_cast<__nv_bfloat16*>(p.out) +
                            static_cast<long long>(gq) * p.ldo + head * DH;
#pragma unroll 1
      for (int x = 0; x < DH; x += 32) {
        uint32_t r[32];
        tmem_ld_32x32(o_addr + x, r);
        tmem_ld_wait();
        if (valid) {
#pragma unroll
          for (int e = 0; e < 32; e += 8) {
            uint4 v;
            v.x = pack_bf16(__uint_as_float(r[e]) * inv, __uint_as_float(r[e + 1]) * inv);
            v.y = pack_bf16(__uint_as_float(r[e + 2]) * inv, __uint_as_float(r[e + 3]) * inv);
            v.z = pack_bf16(__uint_as_float(r[e + 4]) * inv, __uint_as_float(r[e + 5]) * inv);
            v.w = pack_bf16(__uint_as_float(r[e + 6]) * inv, __uint_as_float(r[e + 7]) * inv);
            *reinterpret_cast<uint4*>(orow + x + e) = v;
          }
        }
      }
      if (valid)
        p.lse[static_cast<long long>(head) * p.T + gq] =
            (m_used + log2f(l)) * 0.6931471805599453f;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == Cfg::MMA_WARP) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TM_COLS);
  }
}

template <int DH, int BKV, int KS, int VS, int CTAS>
static int launch_fwd(const void* q, const void* k, const void* v, AttnParams p, long long ldq,
                      long long ldk, long long ldv, cudaStream_t stream) {
  using Cfg = AttnCfg<DH, BKV, KS, VS, CTAS>;
  CUtensorMap tq, tk, tv;
  int r;
  if ((r = make_tmap_bf16(&tq, q, p.T, static_cast<long long>(p.Hq) * DH, ldq, 128))) return r;
  if ((r = make_tmap_bf16(&tk, k, p.T, static_cast<long long>(p.Hkv) * DH, ldk, BKV))) return r;
  if ((r = make_tmap_bf16(&tv, v, p.T, static_cast<long long>(p.Hkv) * DH, ldv, BKV))) return r;
  auto kern = attn_fwd_kernel<DH, BKV, KS, VS, CTAS>;
  static SmemOptIn opt_in;
  if (int e = opt_in.ensure(kern, Cfg::SMEM)) return e;
  // every sequence adds at most one partial tile; heads and tiles share x, whose limit many short sequences
  // do not reach (y ends at 65,535)
  const long long grid = ((p.T + 127) / 128 + static_cast<long long>(p.nseq)) * p.Hq;
  if (grid > 0x7fffffffLL) return -2;
  launch_chained(kern, static_cast<unsigned>(grid), Cfg::THREADS, Cfg::SMEM, stream, tq, tk, tv, p);
  return static_cast<int>(cudaGetLastError());
}

}  // namespace ss

extern "C" int ss_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse,
                           const int* cu_seqlens, int nseq, int T, int Hq, int Hkv, int dh,
                           long long ldq, long long ldk, long long ldv, long long ldo, float scale,
                           int* status, void* stream) {
  using namespace ss;
  if (T <= 0 || nseq <= 0) return 0;
  if ((ldq % 8) || (ldk % 8) || (ldv % 8) || (ldo % 8) || Hq % Hkv) return -2;
  AttnParams p;
  p.out = out; p.lse = lse; p.cu_seqlens = cu_seqlens; p.nseq = nseq; p.T = T; p.Hq = Hq;
  p.Hkv = Hkv; p.ldo = ldo; p.scale_log2 = scale * 1.4426950408889634f; p.status = status;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (dh == 128) return launch_fwd<128, 64, 2, 2, 2>(q, k, v, p, ldq, ldk, ldv, s);
  if (dh == 64) return launch_fwd<64, 64, 4, 4, 2>(q, k, v, p, ldq, ldk, ldv, s);
  if (dh == 256) return launch_fwd<256, 64, 3, 2, 1>(q, k, v, p, ldq, ldk, ldv, s);
  return -2;
}
