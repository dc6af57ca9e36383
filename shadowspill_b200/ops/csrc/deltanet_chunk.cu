// Gated DeltaNet, chunked form, forward and backward, on tcgen05 (sm_100a).
//
// The packed token stream is cut into chunks of 64 tokens. With g the log decay, gam its running
// sum inside the chunk, R[t,i] = exp(gam_t - gam_i) for i <= t inside one sequence (0 otherwise):
//
//     A  = diag(beta) (R o K K^T), strictly lower           Tm = (I + A)^-1
//     W  = Tm diag(beta Gt) K        U0 = Tm diag(beta) V    Gt_t = exp(gam_t) [t continues the
//     U  = U0 - W S                                                 sequence of the previous chunk]
//     O  = diag(s Gt) Q S + (s R o Q K^T) U                  s = dk^-1/2
//     S' = Gc S + (diag(d) K)^T U                            d_t = exp(gam_63 - gam_t) [same
//                                                                   sequence as the chunk's end]
//
// which equals the token recurrence S <- a S; u = beta (v - k S); S <- S + k u^T; o = s q S
// (reference definition: packages/workloads/src/shadowspill_workloads/models/qwen35/
// implementations/pytorch/delta_rule/reference.py:8-41, backward :43-132; call site
// models/shared/delta_net.py:76). Sequence boundaries act only through the masks, so a packed
// batch needs no loop over sequences and no padding to chunk multiples.
//
// Kernels (dk = dv = 128; QK heads are shared by `rep` V heads, handled two V heads at a time):
//   dn_prep_kernel   per (chunk, pair of V heads): K K^T and Q K^T on the tensor cores, the
//                    64x64 triangular inverse in blocks, then W^T and U0^T as MMAs; writes every per-chunk operand.
//   dn_fwd_kernel    per V head and run of chunks between two that hold a sequence's start, sequential over its chunks:
//                    the state S^T lives in registers (fp32);
//                    U^T = U0^T - S^T W^T, O^T = S^T Qg^T + U^T Mq^T, S'^T = Gc S^T + U^T Kd.
//   dn_bwd_state_kernel   the same walk in reverse for dS and dU.
//   dn_bwd_chunk_kernel   per (chunk, V head): the products that need S or dS' of one chunk.
//   dn_bwd_prep_kernel    per (chunk, pair): gradients of the chunk-local algebra -> dq dk dv
//                         dbeta dg.
// All matrices are kept transposed where that makes the M dimension 128 (features), so every MMA
// is 128 x {64,128} x 16 with operands either loaded by TMA or written one row per thread.
// No operand ever comes from another GPU; every wait is bounded.
#include "sm100_ptx.cuh"

#include <cudaTypedefs.h>
#include <math.h>

namespace ss {
int make_tmap_bf16(CUtensorMap* map, const void* base, long long rows, long long cols,
                   long long ld, int box_rows);  // gemm_tcgen05.cu
}

namespace ss_dnc {
using namespace ss;

constexpr int CH = 64;         // tokens per chunk
constexpr int D = 128;         // dk = dv
constexpr int THREADS = 160;   // 4 row warps + 1 control warp
constexpr int CTRL = 128;      // the thread that issues TMA loads and MMAs

struct Geo {
  int T, n, H, Hk, rep, P, NP;   // P pairs of V heads per QK head, NP = Hk * P pairs per chunk
};

__device__ __forceinline__ void head_slot(const Geo& g, int h, int& pr, int& hh) {
  const int kh = h / g.rep, r = h % g.rep;
  pr = kh * g.P + (r >> 1);
  hh = r & 1;
}

// Byte offset of the 16-byte chunk holding columns [8*col8, 8*col8+8) of `row` in a tile made of
// 64-column blocks of `rows_per_blk` rows each (128-byte rows, 128B swizzle).
__device__ __forceinline__ uint32_t sw_off(int rows_per_blk, int row, int col8) {
  return static_cast<uint32_t>((col8 >> 3) * rows_per_blk * 128 + row * 128 +
                               (((col8 & 7) ^ (row & 7)) << 4));
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  return make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]),
                    pack_bf16(f[6], f[7]));
}
__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  const float2 a = unpack_bf16(u.x), b = unpack_bf16(u.y), c = unpack_bf16(u.z), d = unpack_bf16(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ float bf16_at(const uint8_t* p) {
  return __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(p));
}
// 32 fp32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_row32(uint32_t addr, float* out) {
  uint32_t r[32];
  tmem_ld_32x32(addr, r);
  tmem_ld_wait();
#pragma unroll
  for (int e = 0; e < 32; ++e) out[e] = __uint_as_float(r[e]);
}
// Operands written by threads (shared memory, TMEM) become visible to the MMA issuer.
__device__ __forceinline__ void publish() {
  tc_fence_before();
  fence_async_proxy();
  __syncthreads();
  tc_fence_after();
}
// Sums of N values per lane over the warp's lanes (each step hands half of the remaining columns to the
// partner lane; through shared memory it was N stores and a chain of dependent loads per sum), written to
// out[0..N). The values are consumed.
template <int N>
__device__ __forceinline__ void warp_col_sums(float (&v)[N], float* out) {
  const int lane = threadIdx.x & 31;
  __syncwarp();                                 // lanes that a branch has left apart take each shuffle one by one
#pragma unroll
  for (int o = 16, n = N / 2; o > 0; o >>= 1, n >>= 1) {
    if (n == 0) {                               // one column left, in both partners
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
      continue;
    }
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  if constexpr (N == 64) reinterpret_cast<float2*>(out)[lane] = make_float2(v[0], v[1]);
  else if constexpr (N == 32) out[lane] = v[0];
  else if ((lane & 1) == 0) out[lane >> 1] = v[0];
}
__device__ __forceinline__ void all_rows_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
// exp(x) where `on`, else 0, without a branch: a choice between an exponential and 0 became one per element, which
// diverged in every warp that holds a diagonal.
__device__ __forceinline__ float decay_if(bool on, float x) { return __expf(on ? x : -INFINITY); }
// The first chunk position of each token's sequence: `starts` has a bit where a sequence begins.
__device__ __forceinline__ int seq_begin(const unsigned* starts, int t) {
  const unsigned long long m = (static_cast<unsigned long long>(starts[1]) << 32) | starts[0];
  return 63 - __clzll(static_cast<long long>(m & (~0ull >> (63 - t))));
}
// Bits lo..hi of the 32 columns from c0 on: what a thread's tests of 32 columns come to.
__device__ __forceinline__ uint32_t span_bits(int lo, int hi, int c0) {
  const int b0 = max(lo - c0, 0), b1 = min(hi - c0, 31);
  return b0 <= b1 ? (0xffffffffu >> (31 - b1)) & (0xffffffffu << b0) : 0u;
}
// ============================================================================ sequence ids
__global__ void dn_seq_ids_kernel(const int* __restrict__ cu, int nseq, int T, int Tp,
                                  int* __restrict__ sid) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= Tp) return;
  if (t >= T) { sid[t] = 0x7fffffff; return; }       // padding is a sequence of its own
  int lo = 0, hi = nseq;                              // boundaries cu[1..nseq] that are <= t
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (cu[mid + 1] <= t) lo = mid + 1; else hi = mid;
  }
  sid[t] = lo;
}

// ============================================================================ prep (forward)
struct PrepParams {
  const float* beta; const float* g; const int* sid;
  __nv_bfloat16* TMT;              // null unless a backward follows
  int save;                        // a backward follows: keep the inverse and its two scaled forms
  float *gam, *gc;
  Geo geo; float scale; int* status;
};
namespace prep {
constexpr int ROW_THREADS = 256, PTHREADS = ROW_THREADS + 32, PCTRL = ROW_THREADS, MQ_THREAD = 64;
// A (fp32) and, once the inverse has been formed from it, the two operands share one region: two CTAs
// fit an SM, and one's substitution runs under the other's loads and stores.
constexpr int AP = 68;                                  // pitch of A: rows 16-byte aligned for float4 reads
constexpr int OFF_KQ = 0, OFF_V = 32768, OFF_XW = 65536, OFF_XU = 81920, OFF_AF = 65536;
constexpr int OFF_MQ = OFF_AF + 36864;                  // 8 KiB: Mq of a head on its way out
constexpr int OFF_MISC = OFF_MQ + 8192;
static_assert(2 * 64 * AP * 4 <= 36864, "A runs into the next tile");
constexpr int OFF_BAR = OFF_MISC + 2048;
constexpr int SMEM = OFF_BAR + 64 + 1024;
static_assert(2 * (SMEM + 1024) <= 233472, "two CTAs per SM");
}

// (I + A)^-1 over A, 64 x 64 strictly lower triangular (fp32, pitch AP), by the 128 row threads of one head (four warps:
// j = 0..63 in two parts); what lies above the diagonal 16 x 16 blocks is scratch. The diagonal blocks by forward
// substitution, a column per thread of part 0, then twice [[P, 0], [-Q B P, Q]] from the inverses P and Q of two
// neighbouring blocks and the block B between them. Substitution in one piece was a chain of 64 steps in 2,000
// straight-line multiplications, and fetching those took as long as running them.
__device__ __forceinline__ void head_sync(int hh) {
  if (hh == 0) asm volatile("bar.sync 2, 128;" ::: "memory");
  else asm volatile("bar.sync 3, 128;" ::: "memory");
}

__device__ __forceinline__ void fma_row(float (&acc)[4], float a, const float4& b) {
  acc[0] += a * b.x; acc[1] += a * b.y; acc[2] += a * b.z; acc[3] += a * b.w;
}
// acc[R][4] = rows r0.. of L (columns k0..k1 of it) times columns c0..c0+3 of M
template <int R>
__device__ __forceinline__ void block_product(float (&acc)[R][4], const float* L, const float* M, int k0, int k1) {
  using prep::AP;
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;
#pragma unroll 1
  for (int k = k0; k < k1; k += 4) {
    float4 l[R], m[4];
#pragma unroll
    for (int r = 0; r < R; ++r) l[r] = *reinterpret_cast<const float4*>(L + r * AP + k);
#pragma unroll
    for (int x = 0; x < 4; ++x) m[x] = *reinterpret_cast<const float4*>(M + (k + x) * AP);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      fma_row(acc[r], l[r].x, m[0]);
      fma_row(acc[r], l[r].y, m[1]);
      fma_row(acc[r], l[r].z, m[2]);
      fma_row(acc[r], l[r].w, m[3]);
    }
  }
}

__device__ __forceinline__ void unit_lower_inverse(float* A, int hh, int j, int part) {
  using prep::AP;
  if (part == 0) {
    float* D = A + (j & ~15) * (AP + 1);
    const int jj = j & 15;
    float x[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      float a[4] = {t == jj ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < t; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(D + t * AP + i);
        a[0] -= v.x * x[i];
        if (i + 1 < t) a[1] -= v.y * x[i + 1];
        if (i + 2 < t) a[2] -= v.z * x[i + 2];
        if (i + 3 < t) a[3] -= v.w * x[i + 3];
      }
      x[t] = (a[0] + a[1]) + (a[2] + a[3]);
    }
    __syncwarp();                                  // a warp holds both blocks whose columns it has read
#pragma unroll
    for (int t = 0; t < 16; ++t) D[t * AP + jj] = x[t];
  }
  head_sync(hh);
  {                                                // 16 -> 32: two pairs of blocks, 1 x 4 values per thread
    float* B0 = A + (j & 32) * (AP + 1);
    const int r0 = part * 8 + ((j & 31) >> 2), c0 = (j & 3) * 4;
    float v[1][4];
    block_product<1>(v, B0 + (16 + r0) * AP, B0 + c0, 0, 16);                     // B P
    *reinterpret_cast<float4*>(B0 + r0 * AP + 16 + c0) = make_float4(v[0][0], v[0][1], v[0][2], v[0][3]);
    head_sync(hh);
    block_product<1>(v, B0 + (16 + r0) * AP + 16, B0 + 16 + c0, 0, 16);           // Q (B P)
    *reinterpret_cast<float4*>(B0 + (16 + r0) * AP + c0) = make_float4(-v[0][0], -v[0][1], -v[0][2], -v[0][3]);
  }
  head_sync(hh);
  {                                                // 32 -> 64: 2 x 4 values per thread, zero blocks left out
    const int r0 = part * 16 + (j >> 3) * 2, c0 = (j & 7) * 4;
    float v[2][4];
    block_product<2>(v, A + (32 + r0) * AP, A + c0, c0 & 16, 32);
#pragma unroll
    for (int r = 0; r < 2; ++r)
      *reinterpret_cast<float4*>(A + (r0 + r) * AP + 32 + c0) = make_float4(v[r][0], v[r][1], v[r][2], v[r][3]);
    head_sync(hh);
    block_product<2>(v, A + (32 + r0) * AP + 32, A + 32 + c0, 0, (r0 & 16) + 16);
#pragma unroll
    for (int r = 0; r < 2; ++r)
      *reinterpret_cast<float4*>(A + (32 + r0 + r) * AP + c0) = make_float4(-v[r][0], -v[r][1], -v[r][2], -v[r][3]);
  }
}

// Bound by latency: two CTAs an SM, each with two row warps to a scheduler (one: 0.146 ms). 8,192 tokens, 16 / 32 heads:
// 0.199 -> 0.132 ms (436 MB, 0.067 ms at the copy bandwidth) with the inverse in blocks, the scalars' loads ahead of the
// set-up, no branch around an exponential and Mq through a tile.
__global__ void __launch_bounds__(prep::PTHREADS, 2)
dn_prep_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
               const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmWT,
               const __grid_constant__ CUtensorMap tmU0T, const __grid_constant__ CUtensorMap tmQG,
               const __grid_constant__ CUtensorMap tmKD, const __grid_constant__ CUtensorMap tmMQ,
               const __grid_constant__ CUtensorMap tmXW, const __grid_constant__ CUtensorMap tmXU, const PrepParams p) {
  using namespace prep;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_smem_1024(smem_raw);
  float* Af = reinterpret_cast<float*>(smem + OFF_AF);
  float* gam_s = reinterpret_cast<float*>(smem + OFF_MISC);        // [2][64]
  float* beta_s = gam_s + 128;
  float* g_s = beta_s + 128;
  int* sid_s = reinterpret_cast<int*>(g_s + 128);                  // [65]; [64] = previous chunk's last
  unsigned* starts_s = reinterpret_cast<unsigned*>(sid_s + 68);    // [2]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint64_t* tma_bar = bars; uint64_t* mma_bar = bars + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2);

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = static_cast<int>(warp_uniform(tid >> 5));
  const Geo G = p.geo;
  const int c = blockIdx.x, pr = blockIdx.y;
  const int kh = pr / G.P, z = pr % G.P, h0 = kh * G.rep + 2 * z;
  const int nh = (2 * z + 1 < G.rep) ? 2 : 1;
  const int t0 = c * CH;

  // the chunk's scalars, asked for ahead of all else: a memory latency that the set-up runs under
  float gam = 0.f, beta = 0.f;                           // log decay of the token, later its running sum
  int sid = -1;
  if (tid < 128 && (tid >> 6) < nh && t0 + (tid & 63) < G.T) {
    const long long at = static_cast<long long>(t0 + (tid & 63)) * G.H + h0 + (tid >> 6);
    gam = p.g[at];
    beta = p.beta[at];
  }
  if (tid < 64 || (tid == 64 && c > 0)) sid = p.sid[tid < 64 ? t0 + tid : t0 - 1];

  if (tid == PCTRL) {
    mbar_init(tma_bar, 1); mbar_init(mma_bar, 1); mbar_fence_init();
    mbar_expect_tx(tma_bar, 32768 + nh * 16384);
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      tma_load_2d(smem + OFF_KQ + b * 16384, &tmK, tma_bar, kh * D + b * 64, t0);
      tma_load_2d(smem + OFF_KQ + b * 16384 + 64 * 128, &tmQ, tma_bar, kh * D + b * 64, t0);
    }
    for (int hh = 0; hh < nh; ++hh)
#pragma unroll
      for (int b = 0; b < 2; ++b)
        tma_load_2d(smem + OFF_V + hh * 16384 + b * 8192, &tmV, tma_bar, (h0 + hh) * D + b * 64, t0);
  }
  if (warp == 8) { __syncwarp(); tmem_alloc(tmem_slot, 256); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);

  if (tid < 128) beta_s[tid] = beta;
  if (tid < 65) sid_s[tid] = sid;
  if (tid < 128) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float before = __shfl_up_sync(0xffffffffu, gam, o);
      if (lane >= o) gam += before;
    }
    if (lane == 31) g_s[warp] = gam;
  }
  __syncthreads();
  if (tid < 64) {
    const unsigned m = __ballot_sync(0xffffffffu, tid == 0 || sid_s[tid] != sid_s[tid - 1]);
    if (lane == 0) starts_s[warp] = m;
  }
  if (tid < 128) {
    const int hh = tid >> 6, j = tid & 63;
    if (j >= 32) gam += g_s[warp - 1];
    gam_s[tid] = gam;
    if (hh < nh) p.gam[(static_cast<long long>(c) * G.H + h0 + hh) * 64 + j] = gam;
  }
  __syncthreads();

  // ---- [K; Q] K^T
  if (warp == 8) {
    const uint32_t leader = elect_one();
    mbar_wait(tma_bar, 0, p.status, KS_TIMEOUT_FULL);
    tc_fence_after();
    constexpr uint32_t idesc = umma_idesc_bf16(128, 64, false, false);
    const uint32_t s = smem_u32(smem + OFF_KQ);
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      const uint64_t d = umma_smem_desc(s + (kk >> 2) * 16384 + (kk & 3) * 32, 16, 1024);
      umma_bf16_if(leader, tmem_base, d, d, idesc, kk != 0);
    }
    umma_commit_if(leader, mma_bar);
  }
  mbar_wait(tma_bar, 0, p.status, KS_TIMEOUT_FULL);
  mbar_wait(mma_bar, 0, p.status, KS_TIMEOUT_TMEM_FULL);
  tc_fence_after();

  // ---- A (fp32; only below the diagonal) and Mq, eight columns at a time
  const int row = tid & 127, part = (tid >> 7) & 1;      // of the row threads: a lane of TMEM and the half of its columns
  if (tid < ROW_THREADS) {
    const int t = row & 63, last = t | 31;               // the warp's last row
    const int lo = seq_begin(starts_s, t);
    const bool is_q = row >= 64;
    const uint32_t span = span_bits(lo, is_q ? t : t - 1, part * 32);    // Mq includes the diagonal, A does not
#pragma unroll 1
    for (int hh = 0; hh < nh; ++hh) {
      const float gt = gam_s[hh * 64 + t], f = is_q ? p.scale : beta_s[hh * 64 + t];
      float* a = Af + (hh * 64 + t) * AP;
      if (is_q && hh > 0) {                              // the head before has left the tile
        if (tid == MQ_THREAD) tma_store_wait_read<0>();
        head_sync(1);
      }
#pragma unroll 1
      for (int i0 = part * 32; i0 < part * 32 + 32; i0 += 16) {
        float m[16];
        if (i0 > last) {
#pragma unroll
          for (int e = 0; e < 16; ++e) m[e] = 0.f;
        } else {
          uint32_t r[16];
          tmem_ld_32x16(lane_addr + i0, r);
#pragma unroll
          for (int e = 0; e < 16; e += 4)
            *reinterpret_cast<float4*>(m + e) = *reinterpret_cast<const float4*>(gam_s + hh * 64 + i0 + e);
          const uint32_t seen = span >> (i0 & 31);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const bool on = seen & (1u << e);
            const float v = f * decay_if(on, gt - m[e]) * __uint_as_float(r[e]);
            m[e] = on ? v : 0.f;
          }
        }
        if (is_q) {
#pragma unroll
          for (int q = 0; q < 2; ++q)
            *reinterpret_cast<uint4*>(smem + OFF_MQ + sw_off(64, t, (i0 >> 3) + q)) = pack8(m + q * 8);
        } else {
#pragma unroll
          for (int e = 0; e < 16; e += 4)
            *reinterpret_cast<float4*>(a + i0 + e) = *reinterpret_cast<const float4*>(m + e);
        }
      }
      if (is_q) {
        fence_async_proxy();
        head_sync(1);
        if (tid == MQ_THREAD) {
          tma_store_2d(&tmMQ, smem + OFF_MQ, 0, (c * G.NP + pr) * 128 + hh * 64);
          tma_store_commit();
        }
      }
    }
  }
  __syncthreads();

  // ---- Tm = (I + A)^-1; thread (hh, j) takes half of its column j
  if (tid < ROW_THREADS) {
    const int hh = row >> 6, j = row & 63;
    float col[32];
    if (hh < nh) {
      unit_lower_inverse(Af + hh * 64 * AP, hh, j, part);
      head_sync(hh);
      const float* at = Af + hh * 64 * AP + j;
#pragma unroll
      for (int e = 0; e < 32; ++e) col[e] = part * 32 + e >= j ? at[(part * 32 + e) * AP] : 0.f;
    }
    all_rows_sync();                                    // A has been read: its region takes the operands
    if (hh < nh) {
      const float bj = beta_s[row];
      const float gtj = (sid_s[j] == sid_s[64]) ? __expf(gam_s[row]) : 0.f;
      float w[32];
#pragma unroll
      for (int e = 0; e < 32; ++e) w[e] = col[e] * bj * gtj;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<uint4*>(smem + OFF_XW + sw_off(128, row, part * 4 + q)) = pack8(w + q * 8);
#pragma unroll
      for (int e = 0; e < 32; ++e) w[e] = col[e] * bj;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<uint4*>(smem + OFF_XU + sw_off(128, row, part * 4 + q)) = pack8(w + q * 8);
      if (p.TMT) {
        uint4* dst = reinterpret_cast<uint4*>(p.TMT + ((static_cast<long long>(c) * G.NP + pr) * 128 + row) * 64 + part * 32);
#pragma unroll
        for (int q = 0; q < 4; ++q) dst[q] = pack8(col + q * 8);
      }
    }
  }
  publish();

  // ---- W^T = K^T (Tm diag(beta Gt))^T, U0^T = V^T (Tm diag(beta))^T
  if (warp == 8) {
    const uint32_t leader = elect_one();
    constexpr uint32_t idesc = umma_idesc_bf16(128, 64, true, true);
    const uint32_t sk = smem_u32(smem + OFF_KQ), sv = smem_u32(smem + OFF_V);
    const uint32_t sxw = smem_u32(smem + OFF_XW), sxu = smem_u32(smem + OFF_XU);
    for (int hh = 0; hh < nh; ++hh) {
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        umma_bf16_if(leader, tmem_base + hh * 64, umma_smem_desc(sk + kk * 2048, 16384, 1024),
                  umma_smem_desc(sxw + hh * 8192 + kk * 2048, 8192, 1024), idesc, kk != 0);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        umma_bf16_if(leader, tmem_base + 128 + hh * 64, umma_smem_desc(sv + hh * 16384 + kk * 2048, 8192, 1024),
                  umma_smem_desc(sxu + hh * 8192 + kk * 2048, 8192, 1024), idesc, kk != 0);
    }
    umma_commit_if(leader, mma_bar);
    if (p.save && tid == PCTRL) {                // the operands are saved from the tiles the products read
      for (int hh = 0; hh < nh; ++hh) {
        tma_store_2d(&tmXW, smem + OFF_XW + hh * 8192, 0, (c * G.NP + pr) * 128 + hh * 64);
        tma_store_2d(&tmXU, smem + OFF_XU + hh * 8192, 0, (c * G.NP + pr) * 128 + hh * 64);
      }
      tma_store_commit();
      tma_store_wait_read<0>();
    }
  }
  mbar_wait(mma_bar, 1, p.status, KS_TIMEOUT_TMEM_FULL);
  tc_fence_after();
  __syncthreads();                               // V and the operands have been read: their tiles are free

  // ---- every result leaves by TMA from a tile laid out like its operands (a row per thread straight to
  // memory is 16 bytes to each of 32 lines per store, half of this kernel's time): W^T over V, U0^T over
  // the operands, then the scaled K and Q rows of the last head in place and those of the first over W^T.
  uint4 kq[8];
  const int t = row & 63;
  const bool is_q = row >= 64;
  auto factor = [&](int hh) {                    // Kd (rows 0..63, of K) and Qg (rows 64..127, of Q)
    const float gt = gam_s[hh * 64 + t];
    if (is_q) return (sid_s[t] == sid_s[64]) ? p.scale * __expf(gt) : 0.f;
    return (sid_s[t] == sid_s[63]) ? __expf(gam_s[hh * 64 + 63] - gt) : 0.f;
  };
  auto write_kq = [&](uint8_t* tile, int hh) {
    const float f = factor(hh);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      float v[8];
      unpack8(kq[q], v);
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] *= f;
      *reinterpret_cast<uint4*>(tile + sw_off(128, row, part * 8 + q)) = pack8(v);
    }
  };
  auto store_kq = [&](const uint8_t* tile, int hh) {
    const int hrow = (c * G.H + h0 + hh) * 64;
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      tma_store_2d(&tmKD, tile + b * 16384, b * 64, hrow);
      tma_store_2d(&tmQG, tile + b * 16384 + 8192, b * 64, hrow);
    }
    tma_store_commit();
  };
  if (tid < ROW_THREADS) {
#pragma unroll 1
    for (int hh = 0; hh < nh; ++hh) {
      float v[32];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        tmem_row32(lane_addr + x * 128 + hh * 64 + part * 32, v);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          *reinterpret_cast<uint4*>(smem + (x == 0 ? OFF_V : OFF_XW) + hh * 16384 + sw_off(128, row, part * 4 + q)) =
              pack8(v + q * 8);
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q)
      kq[q] = *reinterpret_cast<const uint4*>(smem + OFF_KQ + sw_off(128, row, part * 8 + q));
    write_kq(smem + OFF_KQ, nh - 1);
    if (tid < nh) {
      const float g63 = gam_s[tid * 64 + 63];
      p.gc[static_cast<long long>(c) * G.H + h0 + tid] = (sid_s[63] == sid_s[64]) ? __expf(g63) : 0.f;
    }
  }
  publish();
  if (tid == PCTRL) {
    for (int hh = 0; hh < nh; ++hh) {
      tma_store_2d(&tmWT, smem + OFF_V + hh * 16384, hh * 64, (c * G.NP + pr) * 128);
      tma_store_2d(&tmU0T, smem + OFF_XW + hh * 16384, hh * 64, (c * G.NP + pr) * 128);
    }
    tma_store_commit();
    store_kq(smem + OFF_KQ, nh - 1);
    if (nh == 2) tma_store_wait_read<1>();       // W^T has left its tile
  }
  if (nh == 2) {
    __syncthreads();
    if (tid < ROW_THREADS) write_kq(smem + OFF_V, 0);
    publish();
    if (tid == PCTRL) store_kq(smem + OFF_V, 0);
  }
  if (tid == PCTRL || tid == MQ_THREAD) tma_store_wait<0>();
  tc_fence_before();
  __syncthreads();
  if (warp == 8) { tc_fence_after(); tmem_dealloc(tmem_base, 256); }
}

// ============================================================================ state walks
// A CTA walks a run of chunks of one V head; nothing but the chain state -> (W S) -> U -> state has to be
// serial, so that chain is all the state warps wait for:
//   * the state lives in their registers (fp32, STATE_COLS of the 128 columns per warp),
//     S <- Gc S + dS with dS fresh from the tensor cores, so it is never scaled in TMEM;
//   * its bf16 form and U go back to the products as A operands in TMEM; the copies that are saved are written
//     to shared memory behind them, off the chain, and leave by TMA;
//   * products that do not need the chain's next value (S^T Qg^T; dO^T Mq, dO^T Qg) are issued while
//     the state warps work, and the forward output has its own accumulators, warps and barrier.
// A chunk in which a sequence ends passes nothing on (its Gc is 0, and its rows of Kd belong to the sequence it
// ends with, whose rows of W are 0), so the chunks behind it are a run of their own, which takes that chunk first,
// from a zero state and without results ("warm"). The same holds in reverse, where the chunk belongs to the later
// run. Runs are taken by position: bucket r of a head has the chunks between the first run start at or behind
// chunk r * bucket and the next bucket's; most buckets of long sequences are empty and leave at once.
// Measured, 8,192 tokens in four sequences (the longest 47 chunks of 128), 32 V heads: forward 0.237 -> 0.095 ms,
// backward 0.206 -> 0.094 ms; the chain takes 1.9 us a chunk either way, 32 heads alone on 148 SMs were the loss.
struct WalkParams {
  const float* gc;
  const int* sid;
  int bucket;                               // chunks
  Geo geo; int* status;
};
namespace walk {
// 128 walks at once move 4 to 5 TB/s, and a chunk's operands then take longer than the chunk before: the loads have to
// be further ahead. A walk without an output leaves Qg and Mq out, and one without saves writes O over the Qg it has
// used, which makes room for a third stage. Saves leave from a warp of their own, or the next loads would wait for them.
// 8,192 tokens of four sequences, 32 V heads: 95 us for either walk with two stages, 76 us (0.37 GB) for the one without
// saves and 81 us (0.40 GB) for the one without an output now; of one sequence 183 us, and now 138 and 172 us.
// U0 in registers, loaded a chunk ahead for a fourth stage: 117 us, since an mbarrier's arrival waits for the loads.
template <bool OUT, bool SAVE>
struct Fwd {
  static constexpr int OFF_U0 = 16384, OFF_KD = 32768, OFF_QG = 49152, OFF_MQ = 65536;    // of a stage; W^T comes first
  static constexpr int STAGE = OUT ? 73728 : 49152, STAGES = OUT && SAVE ? 2 : 3;
  static constexpr int OFF_SOP = STAGES * STAGE;                                  // [128 x 128] saved copy of the state
  static constexpr int OFF_UOP = OFF_SOP + (SAVE ? 32768 : 0);                    // [128 x 64] saved copy of U
  static constexpr bool O_IN_STAGE = OUT && !SAVE;
  static constexpr int OFF_O = OFF_UOP + (SAVE ? 16384 : 0);                      // O of a chunk
  static constexpr int OFF_BAR = OFF_O + (OUT && !O_IN_STAGE ? 16384 : 0);
  static constexpr int SMEM = OFF_BAR + 256 + 1024;
  static constexpr int MMA_WARP = 8 + (OUT ? 4 : 0), LOAD_WARP = MMA_WARP + 1, SAVE_WARP = MMA_WARP + 2;
  static constexpr int THREADS = (MMA_WARP + (SAVE ? 3 : 2)) * 32;
  static_assert(SMEM <= 232448, "exceeds the shared memory of one CTA");
};
// backward
constexpr int STAGE = 73728;
constexpr int OFF_SOP = 2 * STAGE;          // [128 x 128] saved copy of the state
constexpr int OFF_UOP = OFF_SOP + 32768;    // [128 x 64] saved copy of dU
constexpr int OFF_BAR = OFF_UOP + 16384;
constexpr int SMEM = OFF_BAR + 256 + 1024;
constexpr int STATE_WARPS = 8, STATE_COLS = 512 / STATE_WARPS, TOKEN_COLS = STATE_COLS / 2;
constexpr int TM_DS = 0, TM_WS = 128, TM_O = 192, TM_SOP = 320, TM_UOP = 384;   // TMEM columns: 128, 64, 2 x 64, 64, 32
constexpr int BWD_THREADS = (STATE_WARPS + 3) * 32;
static_assert(SMEM <= 232448, "exceeds the shared memory of one CTA");
}

// The first chunk at or behind `c` that a run may start at: 0, the number of chunks, or one with a sequence begun
// in it or in the chunk before behind its first token. Sequence ids rise with the tokens. Executed by a full warp.
__device__ __forceinline__ int run_start(const int* sid, int n, int c) {
  if (c <= 0) return 0;
  if (c >= n) return n;
  const int lane = threadIdx.x & 31, before = sid[(c - 1) * CH];
  int lo = c, hi = n;
  while (lo < hi) {
    const int step = (hi - lo + 31) >> 5, s = lo + lane * step;
    const unsigned past = __ballot_sync(0xffffffffu, s >= hi || sid[s * CH] != before);
    if (past == 0) { lo += 31 * step + 1; continue; }
    const int first = __ffs(static_cast<int>(past)) - 1;
    hi = min(hi, lo + first * step);
    lo = first ? lo + (first - 1) * step + 1 : hi;
  }
  return lo;
}
// Does the sequence of chunk s begin before it, so that a run that starts there needs the chunk before?
__device__ __forceinline__ bool run_warm(const int* sid, int n, int s) {
  return s > 0 && s < n && sid[s * CH - 1] == sid[s * CH];
}

// N fp32 columns of this thread's lane, one wait for all of them.
template <int N>
__device__ __forceinline__ void tmem_cols(uint32_t addr, float (&out)[N]) {
  if constexpr (N == 16) {
    tmem_ld_32x16(addr, reinterpret_cast<uint32_t (&)[16]>(out));
  } else {
#pragma unroll
    for (int c = 0; c < N; c += 32) tmem_ld_32x32(addr + c, reinterpret_cast<uint32_t (&)[32]>(out[c]));
  }
  tmem_ld_wait();
}
// N fp32 values -> N / 2 columns of bf16 pairs of this thread's lane: the A operand of a product.
template <int N>
__device__ __forceinline__ void tmem_put_bf16(uint32_t addr, const float (&v)[N], uint32_t (&pk)[N / 2]) {
#pragma unroll
  for (int e = 0; e < N / 2; ++e) pk[e] = pack_bf16(v[2 * e], v[2 * e + 1]);
  if constexpr (N == 64) tmem_st_32x32(addr, pk);
  else if constexpr (N == 32) tmem_st_32x16(addr, pk);
  else tmem_st_32x8(addr, pk);
  tmem_st_wait();
}
// The same values as columns [N * part, N * part + N) of `row` of a swizzled tile of 128 rows.
template <int N>
__device__ __forceinline__ void smem_put_bf16(uint8_t* tile, int row, int part, const uint32_t (&pk)[N / 2]) {
#pragma unroll
  for (int q = 0; q < N / 8; ++q)
    *reinterpret_cast<uint4*>(tile + sw_off(128, row, part * (N / 8) + q)) =
        make_uint4(pk[4 * q], pk[4 * q + 1], pk[4 * q + 2], pk[4 * q + 3]);
}
// The state warps' part of a row: S <- gc S + dS (dS in TMEM, none before the first chunk).
template <int N>
__device__ __forceinline__ void state_step(float (&S)[N], float gc, uint32_t ds_addr) {
  constexpr int M = N < 32 ? N : 32;           // all of a row's dS at once does not fit the registers beside S
#pragma unroll
  for (int c = 0; c < N; c += M) {
    float d[M];
    tmem_cols(ds_addr + c, d);
#pragma unroll
    for (int e = 0; e < M; ++e) S[c + e] = fmaf(gc, S[c + e], d[e]);
  }
}
// What this warp wrote to TMEM is visible to the products that wait for `bar`.
__device__ __forceinline__ void warp_publish(uint64_t* bar) {
  tc_fence_before();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}
// What this warp wrote to shared memory is visible to the TMA stores that wait for `bar`.
__device__ __forceinline__ void warp_publish_copy(uint64_t* bar) {
  fence_async_proxy();
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}

// OUT: the rule's output; SAVE: S and U are kept for a backward pass.
template <bool OUT, bool SAVE>
__global__ void __launch_bounds__(walk::Fwd<OUT, SAVE>::THREADS, 1)
dn_fwd_kernel(const __grid_constant__ CUtensorMap tmWT, const __grid_constant__ CUtensorMap tmU0T,
              const __grid_constant__ CUtensorMap tmQG, const __grid_constant__ CUtensorMap tmKD,
              const __grid_constant__ CUtensorMap tmMQ, const __grid_constant__ CUtensorMap tmST,
              const __grid_constant__ CUtensorMap tmUT, const __grid_constant__ CUtensorMap tmO, const WalkParams p) {
  using namespace walk;
  using W = Fwd<OUT, SAVE>;
  constexpr int NST = W::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_smem_1024(smem_raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + W::OFF_BAR);
  uint64_t* full = bars;               // [STAGES] a stage has arrived
  uint64_t* stage_free = bars + 4;     // [STAGES] its products are done, and O has left it
  uint64_t* sop_ready = bars + 8;      // S^T operand written
  uint64_t* ws_done = bars + 9;
  uint64_t* u_ready = bars + 10;       // U^T operand written
  uint64_t* s_done = bars + 11;
  uint64_t* o_full = bars + 12;        // [2]
  uint64_t* o_free = bars + 14;        // [2]
  uint64_t* s_copied = bars + 16;      // the copies to be saved have been written
  uint64_t* u_copied = bars + 17;
  uint64_t* saved = bars + 18;         // both have been read by their stores
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 19);
  int* run = reinterpret_cast<int*>(bars + 20);          // first chunk, one behind the last, warm
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = static_cast<int>(warp_uniform(tid >> 5));
  const Geo G = p.geo;
  const int h = blockIdx.x;
  int pr, hh;
  head_slot(G, h, pr, hh);

  if (warp == 0) {
    const int first = run_start(p.sid, G.n, blockIdx.y * p.bucket);
    const int end = run_start(p.sid, G.n, (blockIdx.y + 1) * p.bucket);
    if (lane == 0) { run[0] = first; run[1] = end; run[2] = run_warm(p.sid, G.n, first); }
  }
  if (tid == 0) {
    for (int i = 0; i < NST; ++i) { mbar_init(&full[i], 1); mbar_init(&stage_free[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&o_full[i], 1); mbar_init(&o_free[i], 4); }
    mbar_init(sop_ready, STATE_WARPS); mbar_init(ws_done, 1);
    mbar_init(u_ready, STATE_WARPS); mbar_init(s_done, 1);
    mbar_init(s_copied, STATE_WARPS); mbar_init(u_copied, STATE_WARPS); mbar_init(saved, 1);
    mbar_fence_init();
  }
  __syncthreads();
  if (run[0] >= run[1]) return;
  const int skip = run[2], c0 = run[0] - skip, steps = run[1] - c0;    // the first `skip` steps leave no results
  if (warp == W::MMA_WARP) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
  const int row = (warp & 3) * 32 + lane;      // V feature

  if (warp < STATE_WARPS) {
    const int part = warp >> 2;
    float S[STATE_COLS];
#pragma unroll
    for (int e = 0; e < STATE_COLS; ++e) S[e] = 0.f;
    float gc = 0.f;
    for (int it = 0; it < steps; ++it) {
      const int st = it % NST;
      const bool keep = SAVE && it >= skip;
      const float gc_next = p.gc[static_cast<long long>(c0 + it) * G.H + h];
      if (it > 0) {
        if (!mbar_wait(s_done, (it - 1) & 1, p.status, KS_TIMEOUT_TMEM_FULL)) break;
        tc_fence_after();
        state_step(S, gc, lane_addr + TM_DS + part * STATE_COLS);
      }
      uint32_t sk[STATE_COLS / 2];
      tmem_put_bf16(lane_addr + TM_SOP + part * (STATE_COLS / 2), S, sk);
      warp_publish(sop_ready);
      gc = gc_next;
      if (keep) {
        if (it > skip && !mbar_wait(saved, (it - skip - 1) & 1, p.status, KS_TIMEOUT_EMPTY)) break;
        smem_put_bf16<STATE_COLS>(smem + W::OFF_SOP, row, part, sk);
        warp_publish_copy(s_copied);
      }
      if (!mbar_wait(&full[st], (it / NST) & 1, p.status, KS_TIMEOUT_FULL)) break;
      uint4 u0[TOKEN_COLS / 8];
#pragma unroll
      for (int q = 0; q < TOKEN_COLS / 8; ++q)
        u0[q] = *reinterpret_cast<const uint4*>(smem + st * W::STAGE + W::OFF_U0 +
                                                sw_off(128, row, part * (TOKEN_COLS / 8) + q));
      if (!mbar_wait(ws_done, it & 1, p.status, KS_TIMEOUT_TMEM_FULL)) break;
      tc_fence_after();
      float u[TOKEN_COLS];
      tmem_cols(lane_addr + TM_WS + part * TOKEN_COLS, u);
#pragma unroll
      for (int q = 0; q < TOKEN_COLS / 8; ++q) {
        float f[8];
        unpack8(u0[q], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) u[q * 8 + e] = f[e] - u[q * 8 + e];
      }
      uint32_t uk[TOKEN_COLS / 2];
      tmem_put_bf16(lane_addr + TM_UOP + part * (TOKEN_COLS / 2), u, uk);
      warp_publish(u_ready);
      if (keep) {
        smem_put_bf16<TOKEN_COLS>(smem + W::OFF_UOP, row, part, uk);
        warp_publish_copy(u_copied);
      }
    }
  } else if (OUT && warp < STATE_WARPS + 4) {
    // O^T is transposed through shared memory and leaves by TMA, which also clips the last chunk's
    // rows: 64 two-byte stores per thread straight to memory took longer than the rest of the chunk
    const int col = (row & 63) * 2;
    const bool issuer = tid == STATE_WARPS * 32;
    for (int it = 0; it < steps; ++it) {
      const int b = it & 1, st = it % NST;
      uint8_t* o_tile = smem + (W::O_IN_STAGE ? st * W::STAGE + W::OFF_QG : W::OFF_O);
      const bool ok = mbar_wait(&o_full[b], (it >> 1) & 1, p.status, KS_TIMEOUT_TMEM_FULL);
      tc_fence_after();
      float o[64];
      if (ok) tmem_cols(lane_addr + TM_O + b * 64, o);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&o_free[b]);
      if (!W::O_IN_STAGE && issuer) tma_store_wait_read<0>();
      // the chunk before has left the tile; the four warps also agree on whether to go on, so that none
      // waits at a barrier for one that gave up
      uint32_t all_ok;
      asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, 1, 128, p;\n\t"
                   "selp.u32 %0, 1, 0, q;\n\t}" : "=r"(all_ok) : "r"(static_cast<uint32_t>(ok)) : "memory");
      if (!all_ok) break;
      if (it >= skip) {
        uint8_t* so = o_tile + (row >> 6) * 8192;
#pragma unroll
        for (int t = 0; t < 64; ++t)
          *reinterpret_cast<__nv_bfloat16*>(so + t * 128 + (col ^ ((t & 7) << 4))) = __float2bfloat16_rn(o[t]);
        fence_async_proxy();
        asm volatile("bar.sync 2, 128;" ::: "memory");
        if (issuer) {
#pragma unroll
          for (int x = 0; x < 2; ++x) tma_store_2d(&tmO, o_tile + x * 8192, h * D + x * 64, (c0 + it) * CH);
          tma_store_commit();
        }
      }
      if (W::O_IN_STAGE && issuer) {
        tma_store_wait_read<0>();
        mbar_arrive(&stage_free[st]);
      }
    }
    if (issuer) tma_store_wait<0>();
  } else if (warp == W::MMA_WARP) {
    const uint32_t leader = elect_one();
    const uint32_t sop = tmem_base + TM_SOP, uop = tmem_base + TM_UOP;
    constexpr uint32_t idesc_w = umma_idesc_bf16(128, 64, false, true);
    constexpr uint32_t idesc_o = umma_idesc_bf16(128, 64, false, false);
    constexpr uint32_t idesc_s = umma_idesc_bf16(128, 128, false, true);
    for (int it = 0; it < steps; ++it) {
      const int st = it % NST, ob = it & 1;
      const uint32_t sst = smem_u32(smem + st * W::STAGE), to = tmem_base + TM_O + ob * 64;
      if (!mbar_wait(&full[st], (it / NST) & 1, p.status, KS_TIMEOUT_FULL)) break;
      if (!mbar_wait(sop_ready, it & 1, p.status, KS_TIMEOUT_TMEM_EMPTY)) break;
      tc_fence_after();
      // (W S)^T = S^T W^T
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma_bf16_ts_if(leader, tmem_base + TM_WS, sop + kk * 8, umma_smem_desc(sst + kk * 2048, 16384, 1024), idesc_w,
                        kk != 0);
      umma_commit_if(leader, ws_done);
      if constexpr (OUT) {
        // O^T = S^T Qg^T, while the state warps form U
        if (it >= 2 && !mbar_wait(&o_free[ob], ((it >> 1) - 1) & 1, p.status, KS_TIMEOUT_TMEM_EMPTY)) break;
        tc_fence_after();
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
          umma_bf16_ts_if(leader, to, sop + kk * 8,
                          umma_smem_desc(sst + W::OFF_QG + (kk >> 2) * 8192 + (kk & 3) * 32, 16, 1024), idesc_o, kk != 0);
      }
      if (!mbar_wait(u_ready, it & 1, p.status, KS_TIMEOUT_TMEM_EMPTY)) break;
      tc_fence_after();
      // dS^T = U^T Kd, then O^T += U^T Mq^T behind it
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        umma_bf16_ts_if(leader, tmem_base + TM_DS, uop + kk * 8, umma_smem_desc(sst + W::OFF_KD + kk * 2048, 8192, 1024),
                        idesc_s, kk != 0);
      umma_commit_if(leader, s_done);
      if constexpr (OUT) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
          umma_bf16_ts_if(leader, to, uop + kk * 8, umma_smem_desc(sst + W::OFF_MQ + kk * 32, 16, 1024), idesc_o, 1);
        umma_commit_if(leader, &o_full[ob]);
      }
      if (!W::O_IN_STAGE) umma_commit_if(leader, &stage_free[st]);
    }
  } else if (warp == W::LOAD_WARP) {
    if (elect_one()) {
      for (int it = 0; it < steps; ++it) {
        const int c = c0 + it, st = it % NST;
        if (it >= NST && !mbar_wait(&stage_free[st], (it / NST - 1) & 1, p.status, KS_TIMEOUT_EMPTY)) break;
        uint8_t* s = smem + st * W::STAGE;
        const int prow = (c * G.NP + pr) * 128, hrow = (c * G.H + h) * 64;
        mbar_expect_tx(&full[st], W::STAGE);
        tma_load_2d(s, &tmWT, &full[st], hh * 64, prow);
        tma_load_2d(s + W::OFF_U0, &tmU0T, &full[st], hh * 64, prow);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          tma_load_2d(s + W::OFF_KD + b * 8192, &tmKD, &full[st], b * 64, hrow);
          if (OUT) tma_load_2d(s + W::OFF_QG + b * 8192, &tmQG, &full[st], b * 64, hrow);
        }
        if (OUT) tma_load_2d(s + W::OFF_MQ, &tmMQ, &full[st], 0, prow + hh * 64);
      }
    }
  } else if (SAVE && elect_one()) {
    for (int it = skip; it < steps; ++it) {
      const int c = c0 + it;
      if (!mbar_wait(s_copied, (it - skip) & 1, p.status, KS_TIMEOUT_FULL)) break;
#pragma unroll
      for (int b = 0; b < 2; ++b)
        tma_store_2d(&tmST, smem + W::OFF_SOP + b * 16384, b * 64, (c * G.H + h) * 128);
      tma_store_commit();
      if (!mbar_wait(u_copied, (it - skip) & 1, p.status, KS_TIMEOUT_FULL)) break;
      tma_store_2d(&tmUT, smem + W::OFF_UOP, hh * 64, (c * G.NP + pr) * 128);
      tma_store_commit();
      tma_store_wait_read<0>();
      mbar_arrive(saved);
    }
    tma_store_wait<0>();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == W::MMA_WARP) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// ============================================================================ backward state walk
// The same walk in reverse: dU^T = dO^T Mq + dS'^T Kd^T, then dS^T = Gc dS'^T + dO^T Qg - dU^T W.
// Stage layout: dO @0 (64 x 128), MQ @16384, KD @24576, QG @40960, WT @57344.
__global__ void __launch_bounds__(walk::BWD_THREADS, 1)
dn_bwd_state_kernel(const __grid_constant__ CUtensorMap tmDO, const __grid_constant__ CUtensorMap tmMQ,
                    const __grid_constant__ CUtensorMap tmKD, const __grid_constant__ CUtensorMap tmQG,
                    const __grid_constant__ CUtensorMap tmWT, const __grid_constant__ CUtensorMap tmDSP,
                    const __grid_constant__ CUtensorMap tmDUT, const WalkParams p) {
  using namespace walk;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_smem_1024(smem_raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint64_t* full = bars;               // [2]
  uint64_t* stage_free = bars + 2;     // [2]
  uint64_t* sop_ready = bars + 4;      // dS'^T operand written
  uint64_t* du_done = bars + 5;
  uint64_t* u_ready = bars + 6;        // -dU^T operand written
  uint64_t* s_done = bars + 7;
  uint64_t* s_copied = bars + 8;       // the copies to be saved have been written
  uint64_t* u_copied = bars + 9;
  uint64_t* saved = bars + 10;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 11);
  int* run = reinterpret_cast<int*>(bars + 12);          // lowest chunk with results, one behind the highest, warm
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = static_cast<int>(warp_uniform(tid >> 5));
  const Geo G = p.geo;
  const int h = blockIdx.x;
  int pr, hh;
  head_slot(G, h, pr, hh);

  if (warp == 0) {
    // a chunk in which a run's sequence begins belongs to that run here; the run before takes it first, as its warm
    const int first = run_start(p.sid, G.n, blockIdx.y * p.bucket);
    const int end = run_start(p.sid, G.n, (blockIdx.y + 1) * p.bucket);
    const int warm = run_warm(p.sid, G.n, end);
    if (lane == 0) { run[0] = first - run_warm(p.sid, G.n, first); run[1] = first < end ? end - warm : 0; run[2] = warm; }
  }
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(&full[i], 1); mbar_init(&stage_free[i], 1); }
    mbar_init(sop_ready, STATE_WARPS); mbar_init(du_done, 1);
    mbar_init(u_ready, STATE_WARPS); mbar_init(s_done, 1);
    mbar_init(s_copied, STATE_WARPS); mbar_init(u_copied, STATE_WARPS); mbar_init(saved, 1);
    mbar_fence_init();
  }
  __syncthreads();
  if (run[0] >= run[1]) return;
  const int skip = run[2], c_top = run[1] - 1 + skip, steps = c_top - run[0] + 1;
  if (warp == STATE_WARPS) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);

  if (warp < STATE_WARPS) {
    const int part = warp >> 2, row = (warp & 3) * 32 + lane;
    float S[STATE_COLS];
#pragma unroll
    for (int e = 0; e < STATE_COLS; ++e) S[e] = 0.f;
    float gc = 0.f;
    for (int it = 0; it < steps; ++it) {
      const bool keep = it >= skip;
      const float gc_next = p.gc[static_cast<long long>(c_top - it) * G.H + h];
      if (it > 0) {
        if (!mbar_wait(s_done, (it - 1) & 1, p.status, KS_TIMEOUT_TMEM_FULL)) break;
        tc_fence_after();
        state_step(S, gc, lane_addr + TM_DS + part * STATE_COLS);
      }
      uint32_t sk[STATE_COLS / 2];
      tmem_put_bf16(lane_addr + TM_SOP + part * (STATE_COLS / 2), S, sk);
      warp_publish(sop_ready);
      gc = gc_next;
      if (keep) {
        if (it > skip && !mbar_wait(saved, (it - skip - 1) & 1, p.status, KS_TIMEOUT_EMPTY)) break;
        smem_put_bf16<STATE_COLS>(smem + OFF_SOP, row, part, sk);
        warp_publish_copy(s_copied);
      }
      if (!mbar_wait(du_done, it & 1, p.status, KS_TIMEOUT_TMEM_FULL)) break;
      tc_fence_after();
      float du[TOKEN_COLS];
      tmem_cols(lane_addr + TM_WS + part * TOKEN_COLS, du);
#pragma unroll
      for (int e = 0; e < TOKEN_COLS; ++e) du[e] = -du[e];
      uint32_t uk[TOKEN_COLS / 2];
      tmem_put_bf16(lane_addr + TM_UOP + part * (TOKEN_COLS / 2), du, uk);
      warp_publish(u_ready);
      if (keep) {
#pragma unroll
        for (int e = 0; e < TOKEN_COLS / 2; ++e) uk[e] ^= 0x80008000u;   // saved is dU, the operand -dU
        smem_put_bf16<TOKEN_COLS>(smem + OFF_UOP, row, part, uk);
        warp_publish_copy(u_copied);
      }
    }
  } else if (warp == STATE_WARPS) {
    const uint32_t leader = elect_one();
    const uint32_t sop = tmem_base + TM_SOP, uop = tmem_base + TM_UOP;
    constexpr uint32_t i_mn64 = umma_idesc_bf16(128, 64, true, true), i_k64 = umma_idesc_bf16(128, 64, false, false);
    constexpr uint32_t i_mn128 = umma_idesc_bf16(128, 128, true, true), i_k128 = umma_idesc_bf16(128, 128, false, false);
    for (int it = 0; it < steps; ++it) {
      const int st = it & 1;
      const uint32_t sst = smem_u32(smem + st * STAGE);
      if (!mbar_wait(&full[st], (it >> 1) & 1, p.status, KS_TIMEOUT_FULL)) break;
      tc_fence_after();
      // dU^T = dO^T Mq (the state warps have read the dU before it: they published -dU since)
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        umma_bf16_if(leader, tmem_base + TM_WS, umma_smem_desc(sst + kk * 2048, 8192, 1024),
                     umma_smem_desc(sst + 16384 + kk * 2048, 8192, 1024), i_mn64, kk != 0);
      if (!mbar_wait(sop_ready, it & 1, p.status, KS_TIMEOUT_TMEM_EMPTY)) break;
      tc_fence_after();
      //      + dS'^T Kd^T
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma_bf16_ts_if(leader, tmem_base + TM_WS, sop + kk * 8,
                        umma_smem_desc(sst + 24576 + (kk >> 2) * 8192 + (kk & 3) * 32, 16, 1024), i_k64, 1);
      umma_commit_if(leader, du_done);
      // dO^T Qg while the state warps form -dU (they have taken dS before they published dS')
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        umma_bf16_if(leader, tmem_base + TM_DS, umma_smem_desc(sst + kk * 2048, 8192, 1024),
                     umma_smem_desc(sst + 40960 + kk * 2048, 8192, 1024), i_mn128, kk != 0);
      if (!mbar_wait(u_ready, it & 1, p.status, KS_TIMEOUT_TMEM_EMPTY)) break;
      tc_fence_after();
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        umma_bf16_ts_if(leader, tmem_base + TM_DS, uop + kk * 8, umma_smem_desc(sst + 57344 + kk * 32, 16, 1024), i_k128,
                        1);
      umma_commit_if(leader, s_done);
      umma_commit_if(leader, &stage_free[st]);
    }
  } else if (warp == STATE_WARPS + 1) {
    if (elect_one()) {
      for (int it = 0; it < steps; ++it) {
        const int c = c_top - it, st = it & 1;
        if (it >= 2 && !mbar_wait(&stage_free[st], ((it >> 1) - 1) & 1, p.status, KS_TIMEOUT_EMPTY)) break;
        uint8_t* s = smem + st * STAGE;
        const int prow = (c * G.NP + pr) * 128, hrow = (c * G.H + h) * 64;
        mbar_expect_tx(&full[st], STAGE);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          tma_load_2d(s + b * 8192, &tmDO, &full[st], h * D + b * 64, c * CH);
          tma_load_2d(s + 24576 + b * 8192, &tmKD, &full[st], b * 64, hrow);
          tma_load_2d(s + 40960 + b * 8192, &tmQG, &full[st], b * 64, hrow);
        }
        tma_load_2d(s + 16384, &tmMQ, &full[st], 0, prow + hh * 64);
        tma_load_2d(s + 57344, &tmWT, &full[st], hh * 64, prow);
      }
    }
  } else if (elect_one()) {
    for (int it = skip; it < steps; ++it) {
      const int c = c_top - it;
      if (!mbar_wait(s_copied, (it - skip) & 1, p.status, KS_TIMEOUT_FULL)) break;
#pragma unroll
      for (int b = 0; b < 2; ++b)
        tma_store_2d(&tmDSP, smem + OFF_SOP + b * 16384, b * 64, (c * G.H + h) * 128);
      tma_store_commit();
      if (!mbar_wait(u_copied, (it - skip) & 1, p.status, KS_TIMEOUT_FULL)) break;
      tma_store_2d(&tmDUT, smem + OFF_UOP, hh * 64, (c * G.NP + pr) * 128);
      tma_store_commit();
      tma_store_wait_read<0>();
      mbar_arrive(saved);
    }
    tma_store_wait<0>();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == STATE_WARPS) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
}

// ============================================================================ backward, per chunk and head
struct ChunkParams {
  float* dgc;
  Geo geo; int* status;
};
namespace chunkk {
// dO comes first: as the A operand of dMq it has 64 of 128 rows, and the products read what lies behind it as the
// others, whose results nothing takes. The operands fill half of an SM's shared memory to within 1 KiB, so that two
// CTAs fit and one's products and stores run under the other's loads (alone: 10,000 cycles a CTA, 6,200 of them
// waiting for its operands; 0.177 -> 0.114 ms at 8,192 tokens, 32 V heads: 0.70 GB, 0.107 ms at the copy bandwidth).
constexpr int OFF_DO = 0, OFF_DSP = 16384, OFF_ST = 49152, OFF_UT = 81920, OFF_DUT = 98304;
constexpr int OFF_RED = 114688, OFF_BAR = OFF_RED + 64, ALIGN_SLACK = 768;
constexpr int SMEM = OFF_BAR + 64 + ALIGN_SLACK;
static_assert(2 * (SMEM + 1024) <= 233472, "two CTAs per SM");
}

__global__ void __launch_bounds__(THREADS, 2)
dn_bwd_chunk_kernel(const __grid_constant__ CUtensorMap tmDSP, const __grid_constant__ CUtensorMap tmST,
                    const __grid_constant__ CUtensorMap tmUT, const __grid_constant__ CUtensorMap tmDUT,
                    const __grid_constant__ CUtensorMap tmDO, const __grid_constant__ CUtensorMap tmDKD,
                    const __grid_constant__ CUtensorMap tmDQG, const __grid_constant__ CUtensorMap tmDWT,
                    const __grid_constant__ CUtensorMap tmDMQ, const ChunkParams p) {
  using namespace chunkk;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_smem_1024(smem_raw);
  if (smem - smem_raw > ALIGN_SLACK) {             // dynamic shared memory starts on 1 KiB: there is no room if it did not
    report(p.status, KS_BAD_ARGUMENT);
    return;
  }
  float* red = reinterpret_cast<float*>(smem + OFF_RED);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint64_t* tma_bar = bars; uint64_t* mma_bar = bars + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2);
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = static_cast<int>(warp_uniform(tid >> 5));
  const Geo G = p.geo;
  const int c = blockIdx.x, h = blockIdx.y;
  int pr, hh;
  head_slot(G, h, pr, hh);

  if (tid == 0) { mbar_init(tma_bar, 1); mbar_init(mma_bar, 1); mbar_fence_init(); }
  if (warp == 4) { tmem_alloc(tmem_slot, 256); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);

  if (warp == 4) {
    const uint32_t leader = elect_one();
    if (leader) {
      const int prow = (c * G.NP + pr) * 128, hrow = (c * G.H + h) * 128;
      mbar_expect_tx(tma_bar, 114688);
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        tma_load_2d(smem + OFF_DSP + b * 16384, &tmDSP, tma_bar, b * 64, hrow);
        tma_load_2d(smem + OFF_ST + b * 16384, &tmST, tma_bar, b * 64, hrow);
        tma_load_2d(smem + OFF_DO + b * 8192, &tmDO, tma_bar, h * D + b * 64, c * CH);
      }
      tma_load_2d(smem + OFF_UT, &tmUT, tma_bar, hh * 64, prow);
      tma_load_2d(smem + OFF_DUT, &tmDUT, tma_bar, hh * 64, prow);
    }
    mbar_wait(tma_bar, 0, p.status, KS_TIMEOUT_FULL);
    tc_fence_after();
    const uint32_t sdsp = smem_u32(smem + OFF_DSP), sst = smem_u32(smem + OFF_ST);
    const uint32_t sut = smem_u32(smem + OFF_UT), sdut = smem_u32(smem + OFF_DUT);
    const uint32_t sdo = smem_u32(smem + OFF_DO);
    constexpr uint32_t i_mm = umma_idesc_bf16(128, 64, true, true);
    constexpr uint32_t i_mk = umma_idesc_bf16(128, 64, true, false);
    constexpr uint32_t i_km = umma_idesc_bf16(128, 64, false, true);
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
      const uint64_t a_dsp = umma_smem_desc(sdsp + kk * 2048, 16384, 1024);
      const uint64_t a_st = umma_smem_desc(sst + kk * 2048, 16384, 1024);
      const uint64_t b_ut = umma_smem_desc(sut + kk * 2048, 16384, 1024);
      const uint64_t b_dut = umma_smem_desc(sdut + kk * 2048, 16384, 1024);
      const uint64_t k_do = umma_smem_desc(sdo + (kk >> 2) * 8192 + (kk & 3) * 32, 16, 1024);
      umma_bf16_if(leader, tmem_base, a_dsp, b_ut, i_mm, kk != 0);          // dKd^T = dS' U^T
      umma_bf16_if(leader, tmem_base + 64, a_st, k_do, i_mk, kk != 0);      // dQg^T = S dO^T
      umma_bf16_if(leader, tmem_base + 128, a_st, b_dut, i_mm, kk != 0);    // (S dU^T), negated below
      umma_bf16_if(leader, tmem_base + 192, k_do, b_ut, i_km, kk != 0);     // dMq = dO U^T (rows 0..63; the tile has no others)
    }
    umma_commit_if(leader, mma_bar);
  }
  mbar_wait(tma_bar, 0, p.status, KS_TIMEOUT_FULL);
  // dGc = <S, dS'> while the MMAs run (both tiles share one layout, so no unswizzling)
  if (tid < 128) {
    float acc = 0.f;
    for (int idx = tid; idx < 2048; idx += 128) {
      float a[8], b[8];
      unpack8(reinterpret_cast<const uint4*>(smem + OFF_ST)[idx], a);
      unpack8(reinterpret_cast<const uint4*>(smem + OFF_DSP)[idx], b);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc += a[e] * b[e];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) red[warp] = acc;
  }
  __syncthreads();
  if (tid == 0) p.dgc[static_cast<long long>(c) * G.H + h] = (red[0] + red[1]) + (red[2] + red[3]);
  mbar_wait(mma_bar, 0, p.status, KS_TIMEOUT_TMEM_FULL);
  tc_fence_after();
  // The results leave by TMA from tiles over the operands (all of them have been read): rows stored by their own
  // threads touch 32 lines a store.
  if (tid < 128) {
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      float kd[32], qg[32], w[32], mq[32];
      tmem_row32(lane_addr + half * 32, kd);
      tmem_row32(lane_addr + 64 + half * 32, qg);
      tmem_row32(lane_addr + 128 + half * 32, w);
      tmem_row32(lane_addr + 192 + half * 32, mq);
#pragma unroll
      for (int e = 0; e < 32; ++e) w[e] = -w[e];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t at = sw_off(128, tid, half * 4 + q);
        *reinterpret_cast<uint4*>(smem + OFF_DSP + at) = pack8(kd + q * 8);
        *reinterpret_cast<uint4*>(smem + OFF_DSP + 16384 + at) = pack8(qg + q * 8);
        *reinterpret_cast<uint4*>(smem + OFF_ST + at) = pack8(w + q * 8);
        if (tid < 64)
          *reinterpret_cast<uint4*>(smem + OFF_ST + 16384 + sw_off(64, tid, half * 4 + q)) = pack8(mq + q * 8);
      }
    }
  }
  publish();
  if (tid == CTRL) {
    const int prow = (c * G.NP + pr) * 128;
    tma_store_2d(&tmDKD, smem + OFF_DSP, hh * 64, prow);
    tma_store_2d(&tmDQG, smem + OFF_DSP + 16384, hh * 64, prow);
    tma_store_2d(&tmDWT, smem + OFF_ST, hh * 64, prow);
    tma_store_2d(&tmDMQ, smem + OFF_ST + 16384, 0, prow + hh * 64);
    tma_store_commit();
    tma_store_wait<0>();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 4) { tc_fence_after(); tmem_dealloc(tmem_base, 256); }
}

// ============================================================================ backward of the chunk-local algebra
struct BwdPrepParams {
  const float* beta; const int* sid; const float* gam; const float* gc; const float* dgc;
  const __nv_bfloat16* dMQ;
  float *dbeta, *dg;               // [T, H]
  Geo geo; float scale; int* status;
};
// Eight row warps, two to each quarter of the TMEM lanes: a thread has half the columns of its row. One CTA an SM, so its
// chain of loads, products and row work is all there is: 44,000 -> 26,000 cycles, 0.373 -> 0.209 ms at 8,192 tokens
// and 16 / 32 heads, with the tokens' dot products on the tensor cores, all operands and results by TMA, twice the warps,
// products as their operands arrive (0.026 ms) and a warp in step that issues them from uniform registers (0.021 ms).
namespace bprep {
constexpr int ROW_THREADS = 256, BTHREADS = ROW_THREADS + 32, BCTRL = ROW_THREADS;
constexpr int OFF_KQ = 0, OFF_TMT = 32768, OFF_V = 49152, OFF_DWT = 81920, OFF_DUT = 114688;
constexpr int OFF_XW = 147456, OFF_XU = 163840;
// after the first group of MMAs the range [OFF_V, OFF_XU + 16384) is reused:
constexpr int OFF_KKF = 49152, OFF_QKF = OFF_KKF + 16640;          // fp32 [64][65] each
constexpr int OFF_DTM = 82944, OFF_XOP = OFF_DTM + 16384;          // operands
constexpr int OFF_SYM = OFF_XOP + 16384, OFF_DQK = OFF_SYM + 8192;
constexpr int OFF_KKA = OFF_DQK + 8192, OFF_QKA = OFF_KKA + 16640;  // fp32 accumulators over heads
constexpr int OFF_OUT = OFF_KKF;                                   // two 16 KiB tiles of the output transposes
constexpr int OFF_DKD = OFF_XU + 16384, OFF_DQG = OFF_DTM;         // dKd^T and dQg^T of both heads, 32 KiB each
constexpr int OFF_MISC = OFF_DKD + 32768;
constexpr int OFF_BAR = OFF_MISC + 10240;
static_assert(OFF_OUT + 32768 <= OFF_DTM, "output tiles overlap dQg");
static_assert(OFF_QKA + 16640 <= OFF_MISC, "scratch overlaps the per-token values");
constexpr int SMEM = OFF_BAR + 64 + 1024;
static_assert(OFF_KKF >= OFF_TMT + 16384, "scratch overlaps a tile that stays live");
static_assert(SMEM <= 232448, "exceeds the shared memory of one CTA");
}

__global__ void __launch_bounds__(bprep::BTHREADS, 1)
dn_bwd_prep_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDWT,
                   const __grid_constant__ CUtensorMap tmDUT, const __grid_constant__ CUtensorMap tmTMT,
                   const __grid_constant__ CUtensorMap tmXW, const __grid_constant__ CUtensorMap tmXU,
                   const __grid_constant__ CUtensorMap tmDKD, const __grid_constant__ CUtensorMap tmDQG,
                   const __grid_constant__ CUtensorMap tmOK, const __grid_constant__ CUtensorMap tmOQ,
                   const __grid_constant__ CUtensorMap tmOV, const BwdPrepParams p) {
  using namespace bprep;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = align_smem_1024(smem_raw);
  float* KKf = reinterpret_cast<float*>(smem + OFF_KKF);
  float* QKf = reinterpret_cast<float*>(smem + OFF_QKF);
  float* KKa = reinterpret_cast<float*>(smem + OFF_KKA);
  float* QKa = reinterpret_cast<float*>(smem + OFF_QKA);
  float* misc = reinterpret_cast<float*>(smem + OFF_MISC);
  float* gam_s = misc;            // [2][64] each from here on
  float* beta_s = misc + 128;
  float* gt_s = misc + 256;       // exp(gam) [continues the previous chunk's sequence]
  float* d_s = misc + 384;        // exp(gam_63 - gam) [same sequence as the chunk's end]
  // column sums, one part per row warp: [4][64]
  float* cs1 = misc + 512;
  float* cs2 = misc + 768;
  float* colG = misc + 1024;
  float* dotq = misc + 1280;      // [2][64] a token's <dQg, Q> and <dKd, K>
  float* dotk = misc + 1408;
  float* sums_s = misc + 1536;    // [2][4] warp sums of the last step
  float* rows_s = misc + 1552;    // [2][128] the right halves' parts of two row sums
  int* sid_s = reinterpret_cast<int*>(misc + 2432);     // [65]
  unsigned* starts_s = reinterpret_cast<unsigned*>(misc + 2500);   // [2]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
  uint64_t* kq_bar = bars; uint64_t* u_bar = bars + 1; uint64_t* w_bar = bars + 2;   // groups of operands, as loaded
  uint64_t* dkd_bar = bars + 3; uint64_t* dqg_bar = bars + 4;
  uint64_t* mma_bar = bars + 5;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 6);

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = static_cast<int>(warp_uniform(tid >> 5));
  const Geo G = p.geo;
  const int c = blockIdx.x, pr = blockIdx.y;
  const int kh = pr / G.P, z = pr % G.P, h0 = kh * G.rep + 2 * z;
  const int nh = (2 * z + 1 < G.rep) ? 2 : 1;
  const int t0 = c * CH;
  const long long prow0 = (static_cast<long long>(c) * G.NP + pr) * 128;

  // the chunk's scalars, asked for ahead of all else: a memory latency that the set-up runs under
  float gam = 0.f, beta = 0.f, dgc = 0.f;
  int sid = -1;
  if (tid < 128 && (tid >> 6) < nh) {
    const int hh = tid >> 6, j = tid & 63;
    const long long hi = static_cast<long long>(c) * G.H + h0 + hh;
    dgc = p.dgc[hi] * p.gc[hi];
    gam = p.gam[(static_cast<long long>(c) * G.H + h0 + hh) * 64 + j];
    if (t0 + j < G.T) beta = p.beta[static_cast<long long>(t0 + j) * G.H + h0 + hh];
  }
  if (tid < 64 || (tid == 64 && c > 0)) sid = p.sid[tid < 64 ? t0 + tid : t0 - 1];

  if (tid == BCTRL) {
    for (int i = 0; i < 6; ++i) mbar_init(&bars[i], 1);
    mbar_fence_init();
    mbar_expect_tx(kq_bar, 32768);
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      tma_load_2d(smem + OFF_KQ + b * 16384, &tmK, kq_bar, kh * D + b * 64, t0);
      tma_load_2d(smem + OFF_KQ + b * 16384 + 64 * 128, &tmQ, kq_bar, kh * D + b * 64, t0);
    }
    mbar_expect_tx(u_bar, 32768 + nh * 16384 + 16384);
#pragma unroll
    for (int b = 0; b < 2; ++b)
      tma_load_2d(smem + OFF_DUT + b * 16384, &tmDUT, u_bar, b * 64, static_cast<int>(prow0));
    for (int hh = 0; hh < nh; ++hh)
#pragma unroll
      for (int b = 0; b < 2; ++b)
        tma_load_2d(smem + OFF_V + hh * 16384 + b * 8192, &tmV, u_bar, (h0 + hh) * D + b * 64, t0);
    tma_load_2d(smem + OFF_XU, &tmXU, u_bar, 0, static_cast<int>(prow0));
    mbar_expect_tx(w_bar, 32768 + 2 * 16384);
#pragma unroll
    for (int b = 0; b < 2; ++b)
      tma_load_2d(smem + OFF_DWT + b * 16384, &tmDWT, w_bar, b * 64, static_cast<int>(prow0));
    tma_load_2d(smem + OFF_XW, &tmXW, w_bar, 0, static_cast<int>(prow0));
    tma_load_2d(smem + OFF_TMT, &tmTMT, w_bar, 0, static_cast<int>(prow0));
    mbar_expect_tx(dkd_bar, nh * 16384);
    for (int hh = 0; hh < nh; ++hh)
      tma_load_2d(smem + OFF_DKD + hh * 16384, &tmDKD, dkd_bar, hh * 64, static_cast<int>(prow0));
  }
  if (warp == 8) { __syncwarp(); tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_slot);
  const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
  uint32_t mma_phase = 0;

  if (tid < 65) sid_s[tid] = sid;
  if (tid < 128) { gam_s[tid] = gam; beta_s[tid] = beta; }
  __syncthreads();
  if (tid < 64) {
    const unsigned m = __ballot_sync(0xffffffffu, tid == 0 || sid_s[tid] != sid_s[tid - 1]);
    if ((tid & 31) == 0) starts_s[warp] = m;
  }
  if (tid < 128) {
    const int hh = tid >> 6, j = tid & 63;
    gt_s[tid] = (sid_s[j] == sid_s[64]) ? __expf(gam_s[tid]) : 0.f;
    d_s[tid] = (sid_s[j] == sid_s[63]) ? __expf(gam_s[hh * 64 + 63] - gam_s[tid]) : 0.f;
  }

  // ---- first group of products, each as soon as its operands are there: the loads take longer than the products
  if (warp == 8) {
    const uint32_t leader = elect_one();
    const uint32_t skq = smem_u32(smem + OFF_KQ), sv = smem_u32(smem + OFF_V);
    const uint32_t sdw = smem_u32(smem + OFF_DWT), sdu = smem_u32(smem + OFF_DUT);
    const uint32_t sxw = smem_u32(smem + OFF_XW), sxu = smem_u32(smem + OFF_XU);
    constexpr uint32_t i_kk = umma_idesc_bf16(128, 64, false, false);
    constexpr uint32_t i_mk = umma_idesc_bf16(128, 64, true, false);
    auto kq = [&](int kk) { return umma_smem_desc(skq + (kk >> 2) * 16384 + (kk & 3) * 32, 16, 1024); };
    mbar_wait(kq_bar, 0, p.status, KS_TIMEOUT_FULL);
    tc_fence_after();
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) umma_bf16_if(leader, tmem_base, kq(kk), kq(kk), i_kk, kk != 0);       // [K;Q] K^T
    mbar_wait(u_bar, 0, p.status, KS_TIMEOUT_FULL);
    tc_fence_after();
    for (int hh = 0; hh < nh; ++hh) {
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)                                                   // P2 = dU V^T
        umma_bf16_if(leader, tmem_base + 128 + hh * 64, umma_smem_desc(sdu + kk * 2048, 16384, 1024),
                  umma_smem_desc(sv + hh * 16384 + (kk >> 2) * 8192 + (kk & 3) * 32, 16, 1024), i_mk, kk != 0);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)                                                   // dV^T
        umma_bf16_if(leader, tmem_base + 320 + hh * 64, umma_smem_desc(sdu + hh * 16384 + kk * 32, 16, 1024),
                  umma_smem_desc(sxu + hh * 8192 + kk * 32, 16, 1024), i_kk, kk != 0);
    }
    mbar_wait(w_bar, 0, p.status, KS_TIMEOUT_FULL);
    tc_fence_after();
#pragma unroll
    for (int kk = 0; kk < 8; ++kk)                                                     // P1 = dW K^T
      umma_bf16_if(leader, tmem_base + 64, umma_smem_desc(sdw + kk * 2048, 16384, 1024), kq(kk), i_mk, kk != 0);
    for (int hh = 0; hh < nh; ++hh)
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)                                                   // dK^T
        umma_bf16_if(leader, tmem_base + 256, umma_smem_desc(sdw + hh * 16384 + kk * 32, 16, 1024),
                  umma_smem_desc(sxw + hh * 8192 + kk * 32, 16, 1024), i_kk, (hh | kk) != 0);
    umma_commit_if(leader, mma_bar);
  }
  const int row = tid & 127, part = (tid >> 7) & 1;      // of the row threads: a lane of TMEM and the half of its columns
  const int hh_me = row >> 6, t_me = row & 63;
  const bool live = tid < ROW_THREADS && hh_me < nh;
  uint4 m[4] = {};                                       // dMq, ahead of the wait for the products
  if (live) {
    const uint4* mq = reinterpret_cast<const uint4*>(p.dMQ + (prow0 + row) * 64 + part * 32);
#pragma unroll
    for (int x = 0; x < 4; ++x) m[x] = mq[x];
  }
  mbar_wait(w_bar, 0, p.status, KS_TIMEOUT_FULL);
  mbar_wait(mma_bar, mma_phase, p.status, KS_TIMEOUT_TMEM_FULL);
  mma_phase ^= 1;
  tc_fence_after();

  // ---- K K^T and Q K^T to shared memory (both heads need both)
  if (tid < ROW_THREADS) {
    float v[32];
    tmem_row32(lane_addr + part * 32, v);
    float* dst = (row < 64 ? KKf : QKf) + (row & 63) * 65 + part * 32;
#pragma unroll
    for (int i = 0; i < 32; ++i) dst[i] = v[i];
  }
  __syncthreads();

  // ---- dTm = (P1, P2) scaled per column; column sums of Tm o P1 and Tm o P2
  if (tid < ROW_THREADS) {
    float p1[32], p2[32], dtm[32];
    tmem_row32(lane_addr + 64 + part * 32, p1);
    tmem_row32(lane_addr + 128 + (hh_me < nh ? hh_me : 0) * 64 + part * 32, p2);
#pragma unroll
    for (int e = 0; e < 32; ++e) {
      const int i = part * 32 + e;
      const float tm = bf16_at(smem + OFF_TMT + (hh_me * 64 + i) * 128 +
                               (((t_me >> 3) ^ (i & 7)) << 4) + (t_me & 7) * 2);
      dtm[e] = live ? beta_s[hh_me * 64 + i] * (gt_s[hh_me * 64 + i] * p1[e] + p2[e]) : 0.f;
      p1[e] = live ? tm * p1[e] : 0.f;
      p2[e] = live ? tm * p2[e] : 0.f;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *reinterpret_cast<uint4*>(smem + OFF_DTM + sw_off(128, row, part * 4 + q)) = pack8(dtm + q * 8);
    warp_col_sums(p1, cs1 + (warp & 3) * 64 + part * 32);
    warp_col_sums(p2, cs2 + (warp & 3) * 64 + part * 32);
  }
  publish();

  // ---- X = dTm Tm^T
  if (warp == 8) {
    const uint32_t leader = elect_one();
    constexpr uint32_t i_km = umma_idesc_bf16(128, 64, false, true);
    const uint32_t sd = smem_u32(smem + OFF_DTM), st = smem_u32(smem + OFF_TMT);
    for (int h2 = 0; h2 < nh; ++h2)
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        umma_bf16_if(leader, tmem_base + 64 + h2 * 64, umma_smem_desc(sd + kk * 32, 16, 1024),
                  umma_smem_desc(st + h2 * 8192 + kk * 2048, 8192, 1024), i_km, kk != 0);
    umma_commit_if(leader, mma_bar);
  }
  mbar_wait(mma_bar, mma_phase, p.status, KS_TIMEOUT_TMEM_FULL);
  mma_phase ^= 1;
  tc_fence_after();
  if (live) {
    float x[32];
    tmem_row32(lane_addr + 64 + hh_me * 64 + part * 32, x);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      *reinterpret_cast<uint4*>(smem + OFF_XOP + hh_me * 8192 + sw_off(64, t_me, part * 4 + q)) = pack8(x + q * 8);
  }
  publish();

  // ---- dA = -Tm^T X
  if (warp == 8) {
    const uint32_t leader = elect_one();
    constexpr uint32_t i_km = umma_idesc_bf16(128, 64, false, true);
    const uint32_t st = smem_u32(smem + OFF_TMT), sx = smem_u32(smem + OFF_XOP);
    for (int h2 = 0; h2 < nh; ++h2)
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        umma_bf16_if(leader, tmem_base + (h2 == 0 ? 192 : 0), umma_smem_desc(st + kk * 32, 16, 1024),
                  umma_smem_desc(sx + h2 * 8192 + kk * 2048, 8192, 1024), i_km, kk != 0);
    umma_commit_if(leader, mma_bar);
  }
  mbar_wait(mma_bar, mma_phase, p.status, KS_TIMEOUT_TMEM_FULL);
  mma_phase ^= 1;
  tc_fence_after();
  if (tid == BCTRL) {                                    // dTm and X have been read: dQg^T takes their place
    mbar_expect_tx(dqg_bar, nh * 16384);
    for (int hh = 0; hh < nh; ++hh)
      tma_load_2d(smem + OFF_DQG + hh * 16384, &tmDQG, dqg_bar, hh * 64, static_cast<int>(prow0));
  }

  // ---- gradients through A and Mq, 16 columns at a time: everything a step reads is in registers before
  // it writes, head 0 writes its dKK and dQK to KKa / QKa and head 1 over the scores both have just read.
  // The loops of this kernel stay rolled where registers allow: it runs each line once per block with two
  // warps per scheduler, and fetching straight-line code was its largest stall.
  float rowG = 0.f, rowdb = 0.f;
  if (tid < ROW_THREADS) {
    const uint32_t span = live ? span_bits(seq_begin(starts_s, t_me), t_me, part * 32) : 0u;
    const uint32_t below = t_me >> 5 == part ? span & ~(1u << (t_me & 31)) : span;       // without the diagonal
    const float gt = gam_s[row], bt = beta_s[row];
#pragma unroll 1
    for (int i0 = part * 32; i0 < part * 32 + 32; i0 += 16) {
      float w[16];
      uint32_t acc[16];
      tmem_ld_32x16(lane_addr + (hh_me == 0 ? 192 : 0) + i0, acc);
      float gi[16], kk[16], qk[16], dmq[16];
#pragma unroll
      for (int x = 0; x < 4; ++x)
        *reinterpret_cast<float4*>(gi + 4 * x) = *reinterpret_cast<const float4*>(gam_s + hh_me * 64 + i0 + 4 * x);
#pragma unroll
      for (int e = 0; e < 16; ++e) { kk[e] = KKf[t_me * 65 + i0 + e]; qk[e] = QKf[t_me * 65 + i0 + e]; }
      unpack8(m[0], dmq);
      unpack8(m[1], dmq + 8);
      m[0] = m[2]; m[1] = m[3];
      const uint32_t on = span >> (i0 & 31), under = below >> (i0 & 31);
      tmem_ld_wait();
      all_rows_sync();
      float* ko = (hh_me == 0 ? KKa : KKf) + t_me * 65 + i0;
      float* qo = (hh_me == 0 ? QKa : QKf) + t_me * 65 + i0;
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const bool seen = on & (1u << e);
        const float R = decay_if(seen, gt - gi[e]);
        const float da = under & (1u << e) ? -__uint_as_float(acc[e]) : 0.f;
        rowdb += da * R * kk[e];
        const float dkk = da * bt * R, dqk = dmq[e] * p.scale * R;
        w[e] = seen ? dkk * kk[e] + dqk * qk[e] : 0.f;           // dR o R
        rowG += w[e];
        ko[e] = dkk;
        qo[e] = seen ? dqk : 0.f;
      }
      warp_col_sums(w, colG + (warp & 3) * 64 + i0);
    }
    if (part) { rows_s[row] = rowG; rows_s[128 + row] = rowdb; }
    all_rows_sync();
#pragma unroll 1
    for (int q = part * 4; q < part * 4 + 4; ++q) {
      float o[8];
      if (row < 64) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int i = q * 8 + e;
          o[e] = (KKa[t_me * 65 + i] + KKa[i * 65 + t_me]) + (KKf[t_me * 65 + i] + KKf[i * 65 + t_me]);
        }
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = QKa[t_me * 65 + q * 8 + e] + QKf[t_me * 65 + q * 8 + e];
      }
      *reinterpret_cast<uint4*>(smem + (row < 64 ? OFF_SYM : OFF_DQK) + sw_off(64, t_me, q)) = pack8(o);
    }
  }
  publish();

  // ---- dK^T += K^T (dKK + dKK^T) + Q^T dQK;  dQ^T = K^T dQK^T;  and [K; Q] dKd^T, [K; Q] dQg^T, whose diagonals are
  // the tokens' <dKd, K> and <dQg, Q> (as sums over the row threads they were 260 shuffles and two-byte loads each)
  if (warp == 8) {
    const uint32_t leader = elect_one();
    constexpr uint32_t i_mm = umma_idesc_bf16(128, 64, true, true);
    constexpr uint32_t i_mk = umma_idesc_bf16(128, 64, true, false);
    constexpr uint32_t i_km = umma_idesc_bf16(128, 64, false, true);
    const uint32_t skq = smem_u32(smem + OFF_KQ), ssym = smem_u32(smem + OFF_SYM);
    const uint32_t sdqk = smem_u32(smem + OFF_DQK);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const uint64_t ak = umma_smem_desc(skq + kk * 2048, 16384, 1024);
      const uint64_t aq = umma_smem_desc(skq + 8192 + kk * 2048, 16384, 1024);
      umma_bf16_if(leader, tmem_base + 256, ak, umma_smem_desc(ssym + kk * 2048, 8192, 1024), i_mm, 1);
      umma_bf16_if(leader, tmem_base + 256, aq, umma_smem_desc(sdqk + kk * 2048, 8192, 1024), i_mm, 1);
      umma_bf16_if(leader, tmem_base + 448, ak, umma_smem_desc(sdqk + kk * 32, 16, 1024), i_mk, kk != 0);
    }
    mbar_wait(dkd_bar, 0, p.status, KS_TIMEOUT_FULL);
    mbar_wait(dqg_bar, 0, p.status, KS_TIMEOUT_FULL);
    tc_fence_after();
#pragma unroll 1
    for (int x = 0; x < 4; ++x) {                       // columns 0, 64: dKd of the heads, 128, 192: dQg
      if ((x & 1) >= nh) continue;
      const uint32_t sb = smem_u32(smem + (x < 2 ? OFF_DKD : OFF_DQG) + (x & 1) * 16384);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        umma_bf16_if(leader, tmem_base + x * 64, umma_smem_desc(skq + (kk >> 2) * 16384 + (kk & 3) * 32, 16, 1024),
                  umma_smem_desc(sb + kk * 2048, 16384, 1024), i_km, kk != 0);
    }
    umma_commit_if(leader, mma_bar);
  }

  // ---- the feature rows, 16 tokens at a time, through tiles that turn them into token rows, which leave by TMA (the last
  // chunk's rows clipped): dv of the heads while those products run, then dk and dq
  const int lim = min(CH, G.T - t0);
  if (tid < ROW_THREADS) {
#pragma unroll 1
    for (int y = 0; y < nh + 2; ++y) {
      const int x = y < nh ? 2 + y : y - nh;           // dk (with Kd), dq (with Qg), dv of the heads
      const uint32_t col = x == 0 ? 256 : x == 1 ? 448 : 320 + (x - 2) * 64;
      uint8_t* out = smem + OFF_OUT + (y & 1) * 16384; // has left: see below
      if (y == nh) {
        mbar_wait(dkd_bar, 0, p.status, KS_TIMEOUT_FULL);
        mbar_wait(dqg_bar, 0, p.status, KS_TIMEOUT_FULL);
        mbar_wait(mma_bar, mma_phase, p.status, KS_TIMEOUT_TMEM_FULL);
        tc_fence_after();
        // the diagonals: K rows on the first two warps' lanes, Q rows on the other two's
        if (part < nh) {                               // the left halves' threads take head 0, the right's head 1
          uint32_t r[32];
          tmem_ld_32x32(lane_addr + (row < 64 ? 0 : 128) + part * 64 + (warp & 1) * 32, r);
          tmem_ld_wait();
          float v = 0.f;
#pragma unroll
          for (int e = 0; e < 32; ++e) v = lane == e ? __uint_as_float(r[e]) : v;
          (row < 64 ? dotk : dotq)[part * 64 + t_me] = v;
        }
      }
#pragma unroll 1
      for (int i0 = part * 32; i0 < part * 32 + 32; i0 += 16) {
        uint32_t r[16];
        tmem_ld_32x16(lane_addr + col + i0, r);
        tmem_ld_wait();
        float acc[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[e] = __uint_as_float(r[e]);
        if (x < 2) {
          const float fmul = x == 0 ? 1.f : p.scale;
#pragma unroll 1
          for (int hh = 0; hh < nh; ++hh) {
            const uint8_t* tile = smem + (x == 0 ? OFF_DKD : OFF_DQG) + hh * 16384;
            const float* fs = (x == 0 ? d_s : gt_s) + hh * 64 + i0;
            float a[16];
            unpack8(*reinterpret_cast<const uint4*>(tile + sw_off(128, row, i0 >> 3)), a);
            unpack8(*reinterpret_cast<const uint4*>(tile + sw_off(128, row, (i0 >> 3) + 1)), a + 8);
#pragma unroll
            for (int e = 0; e < 16; e += 4) {
              const float4 f = *reinterpret_cast<const float4*>(fs + e);
              acc[e] += f.x * fmul * a[e];
              acc[e + 1] += f.y * fmul * a[e + 1];
              acc[e + 2] += f.z * fmul * a[e + 2];
              acc[e + 3] += f.w * fmul * a[e + 3];
            }
          }
        }
#pragma unroll
        for (int e = 0; e < 16; ++e)
          *reinterpret_cast<__nv_bfloat16*>(out + (row >> 6) * 8192 + (i0 + e) * 128 + (((row & 63) * 2) ^ ((e & 7) << 4))) =
              __float2bfloat16_rn(acc[e]);
      }
      fence_async_proxy();
      if (tid == 0) tma_store_wait_read<0>();          // the tile before has left when all have passed the barrier
      all_rows_sync();
      if (tid == 0) {
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          if (x >= 2) tma_store_2d(&tmOV, out + b * 8192, (h0 + x - 2) * D + b * 64, t0);
          else tma_store_2d(x == 0 ? &tmOK : &tmOQ, out + b * 8192, pr * D + b * 64, t0);
        }
        tma_store_commit();
      }
    }
  }
  __syncthreads();

  // ---- per-token scalars: dgam -> dg (suffix sum over the chunk), dbeta
  // sums of a column's parts over one head's two row warps
  auto two = [&](const float* part, int i) { return part[(hh_me * 2) * 64 + i] + part[(hh_me * 2 + 1) * 64 + i]; };
  float s = 0.f;
  if (tid < 128) {
    rowG += rows_s[row];
    rowdb += rows_s[128 + row];
    float tail = 0.f;                                   // of the chunk's last token alone
    if (live) {
      tail = d_s[tid] * dotk[tid];
      s = rowG - two(colG, t_me) + beta_s[tid] * gt_s[tid] * two(cs1, t_me) + p.scale * gt_s[tid] * dotq[tid] - tail;
    }
    __syncwarp();                                       // see warp_col_sums: here 3,100 -> 900 cycles
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tail += __shfl_xor_sync(0xffffffffu, tail, o);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float after = __shfl_down_sync(0xffffffffu, s, o);
      if (lane + o < 32) s += after;
    }
    if (lane == 0) { sums_s[warp] = tail; sums_s[4 + warp] = s; }
  }
  __syncthreads();
  if (live && tid < 128 && t_me < lim) {
    s += (sums_s[hh_me * 2] + sums_s[hh_me * 2 + 1]) + dgc;
    if (t_me < 32) s += sums_s[4 + hh_me * 2 + 1];
    const long long o = static_cast<long long>(t0 + t_me) * G.H + h0 + hh_me;
    p.dg[o] = s;
    p.dbeta[o] = rowdb + gt_s[tid] * two(cs1, t_me) + two(cs2, t_me);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) { tc_fence_after(); tmem_dealloc(tmem_base, 512); }
  if (tid == 0) tma_store_wait<0>();
}

static Geo make_geo(int T, int H, int Hk) {
  Geo g;
  g.T = T; g.n = (T + CH - 1) / CH; g.H = H; g.Hk = Hk; g.rep = H / Hk;
  g.P = (g.rep + 1) / 2; g.NP = Hk * g.P;
  return g;
}

// Chunks per bucket of the walks. Four buckets per SM, so that runs of sequences as long as a head's share of the SMs
// seldom fall into one bucket and are walked one after the other; a bucket without a run start costs about 2 us.
static int walk_bucket(const Geo& g) {
  const long long chunks = static_cast<long long>(g.n) * g.H, buckets = 4 * 148;
  const long long b = (chunks + buckets - 1) / buckets;
  return b < 1 ? 1 : static_cast<int>(b);
}

}  // namespace ss_dnc

// ---------------------------------------------------------------------------- launchers
// ss_dn_fwd: `out` may be null where ST and UTp are given, which may be null where `out` is.
// Shapes: q, k [T, Hk, 128] bf16; v, out, dout, dv [T, H, 128] bf16; beta, g, dbeta, dg [T, H] fp32;
// sid int32 [n*64]; n = ceil(T/64); P = ceil((H/Hk)/2); NP = Hk*P.
// Pair arrays [n, NP, 128, 128] bf16: WTp U0Tp UTp dUTp dWTp dKdTp dQgTp (columns = (head of pair, token)).
// Row-stacked arrays [n, NP, 128, 64] bf16: MQ TMT XW XU dMQ (rows = (head of pair, token)).
// Per-head arrays: QG KD [n, H, 64, 128]; ST dSpT [n, H, 128, 128] bf16; gam [n, H, 64], gc dgc [n, H] fp32.
extern "C" {
using namespace ss_dnc;

int ss_dn_seq_ids(const int* cu_seqlens, int nseq, int T, int* sid, void* stream) {
  if (T <= 0) return 0;
  const int Tp = (T + CH - 1) / CH * CH;
  dn_seq_ids_kernel<<<(Tp + 255) / 256, 256, 0, (cudaStream_t)stream>>>(cu_seqlens, nseq, T, Tp, sid);
  return (int)cudaGetLastError();
}

int ss_dn_prep(const void* q, const void* k, const void* v, const float* beta, const float* g,
               const int* sid, void* WTp, void* U0Tp, void* QG, void* KD, void* MQ, void* TMT, void* XW,
               void* XU, float* gam, float* gc, int T, int H, int Hk, float scale, int* status,
               void* stream) {
  if (T <= 0) return 0;
  if (H <= 0 || Hk <= 0 || H % Hk) return -2;
  const Geo geo = make_geo(T, H, Hk);
  CUtensorMap tq, tk, tv, twt, tu0, tqg, tkd, tmq, txw, txu;
  int r;
  const bool save = TMT != nullptr;
  if ((XW != nullptr) != save || (XU != nullptr) != save) return -2;
  const long long prow = (long long)geo.n * geo.NP * 128, hrow = (long long)geo.n * H * 64;
  if ((r = ss::make_tmap_bf16(&tq, q, T, (long long)Hk * D, (long long)Hk * D, 64))) return r;
  if ((r = ss::make_tmap_bf16(&tk, k, T, (long long)Hk * D, (long long)Hk * D, 64))) return r;
  if ((r = ss::make_tmap_bf16(&tv, v, T, (long long)H * D, (long long)H * D, 64))) return r;
  if ((r = ss::make_tmap_bf16(&twt, WTp, prow, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tu0, U0Tp, prow, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tqg, QG, hrow, 128, 128, 64))) return r;
  if ((r = ss::make_tmap_bf16(&tkd, KD, hrow, 128, 128, 64))) return r;
  if ((r = ss::make_tmap_bf16(&tmq, MQ, prow, 64, 64, 64))) return r;
  if ((r = ss::make_tmap_bf16(&txw, save ? XW : MQ, prow, 64, 64, 64))) return r;
  if ((r = ss::make_tmap_bf16(&txu, save ? XU : MQ, prow, 64, 64, 64))) return r;
  PrepParams p;
  p.beta = beta; p.g = g; p.sid = sid;
  p.TMT = (__nv_bfloat16*)TMT; p.save = save; p.gam = gam; p.gc = gc;
  p.geo = geo; p.scale = scale; p.status = status;
  static ss::SmemOptIn opt_in;
  if (int e = opt_in.ensure(dn_prep_kernel, prep::SMEM)) return e;
  dn_prep_kernel<<<dim3(geo.n, geo.NP), prep::PTHREADS, prep::SMEM, (cudaStream_t)stream>>>(tq, tk, tv, twt, tu0, tqg, tkd, tmq,
                                                                                     txw, txu, p);
  return (int)cudaGetLastError();
}

int ss_dn_fwd(const void* WTp, const void* U0Tp, const void* QG, const void* KD, const void* MQ,
              const float* gc, const int* sid, void* out, void* ST, void* UTp, int T, int H, int Hk, int* status,
              void* stream) {
  if (T <= 0) return 0;
  if (H <= 0 || Hk <= 0 || H % Hk) return -2;
  const Geo geo = make_geo(T, H, Hk);
  const long long prow = (long long)geo.n * geo.NP * 128, hrow = (long long)geo.n * H * 64;
  const bool save = ST != nullptr;
  if (save != (UTp != nullptr) || (out == nullptr && !save)) return -2;
  CUtensorMap twt, tu0, tqg, tkd, tmq, tst, tut, to;
  int r;
  if ((r = ss::make_tmap_bf16(&twt, WTp, prow, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tu0, U0Tp, prow, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tqg, QG, hrow, 128, 128, 64))) return r;
  if ((r = ss::make_tmap_bf16(&tkd, KD, hrow, 128, 128, 64))) return r;
  if ((r = ss::make_tmap_bf16(&tmq, MQ, prow, 64, 64, 64))) return r;
  tst = tut = to = twt;                            // maps of what this walk does not write are not used
  if (save) {
    if ((r = ss::make_tmap_bf16(&tst, ST, (long long)geo.n * H * 128, 128, 128, 128))) return r;
    if ((r = ss::make_tmap_bf16(&tut, UTp, prow, 128, 128, 128))) return r;
  }
  if (out != nullptr && (r = ss::make_tmap_bf16(&to, out, T, (long long)H * D, (long long)H * D, 64))) return r;
  WalkParams p;
  p.gc = gc; p.sid = sid; p.bucket = walk_bucket(geo); p.geo = geo; p.status = status;
  auto go = [&](auto kern, auto w, ss::SmemOptIn& opt_in) -> int {
    using W = decltype(w);
    if (int e = opt_in.ensure(kern, W::SMEM)) return e;
    kern<<<dim3(H, (geo.n + p.bucket - 1) / p.bucket), W::THREADS, W::SMEM, (cudaStream_t)stream>>>(twt, tu0, tqg, tkd,
                                                                                                    tmq, tst, tut, to, p);
    return (int)cudaGetLastError();
  };
  static ss::SmemOptIn o1, o2, o3;
  if (!save) return go(dn_fwd_kernel<true, false>, walk::Fwd<true, false>{}, o1);
  return out != nullptr ? go(dn_fwd_kernel<true, true>, walk::Fwd<true, true>{}, o2)
                        : go(dn_fwd_kernel<false, true>, walk::Fwd<false, true>{}, o3);
}

int ss_dn_bwd_state(const void* dout, const void* MQ, const void* KD, const void* QG, const void* WTp,
                    const float* gc, const int* sid, void* dSpT, void* dUTp, int T, int H, int Hk, int* status,
                    void* stream) {
  if (T <= 0) return 0;
  if (H <= 0 || Hk <= 0 || H % Hk) return -2;
  const Geo geo = make_geo(T, H, Hk);
  const long long prow = (long long)geo.n * geo.NP * 128, hrow = (long long)geo.n * H * 64;
  CUtensorMap tdo, tmq, tkd, tqg, twt, tdsp, tdut;
  int r;
  if ((r = ss::make_tmap_bf16(&tdo, dout, T, (long long)H * D, (long long)H * D, 64))) return r;
  if ((r = ss::make_tmap_bf16(&tmq, MQ, prow, 64, 64, 64))) return r;
  if ((r = ss::make_tmap_bf16(&tkd, KD, hrow, 128, 128, 64))) return r;
  if ((r = ss::make_tmap_bf16(&tqg, QG, hrow, 128, 128, 64))) return r;
  if ((r = ss::make_tmap_bf16(&twt, WTp, prow, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tdsp, dSpT, (long long)geo.n * H * 128, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tdut, dUTp, prow, 128, 128, 128))) return r;
  WalkParams p;
  p.gc = gc; p.sid = sid; p.bucket = walk_bucket(geo); p.geo = geo; p.status = status;
  static ss::SmemOptIn opt_in;
  if (int e = opt_in.ensure(dn_bwd_state_kernel, walk::SMEM)) return e;
  dn_bwd_state_kernel<<<dim3(H, (geo.n + p.bucket - 1) / p.bucket), walk::BWD_THREADS, walk::SMEM,
                        (cudaStream_t)stream>>>(tdo, tmq, tkd, tqg, twt, tdsp, tdut, p);
  return (int)cudaGetLastError();
}

int ss_dn_bwd_chunk(const void* dSpT, const void* ST, const void* UTp, const void* dUTp, const void* dout,
                    void* dKdTp, void* dQgTp, void* dWTp, void* dMQ, float* dgc, int T, int H, int Hk,
                    int* status, void* stream) {
  if (T <= 0) return 0;
  if (H <= 0 || Hk <= 0 || H % Hk) return -2;
  const Geo geo = make_geo(T, H, Hk);
  const long long prow = (long long)geo.n * geo.NP * 128, srow = (long long)geo.n * H * 128;
  CUtensorMap tdsp, tst, tut, tdut, tdo, tkd, tqg, tdw, tmq;
  int r;
  if ((r = ss::make_tmap_bf16(&tdsp, dSpT, srow, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tst, ST, srow, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tut, UTp, prow, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tdut, dUTp, prow, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tdo, dout, T, (long long)H * D, (long long)H * D, 64))) return r;
  if ((r = ss::make_tmap_bf16(&tkd, dKdTp, prow, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tqg, dQgTp, prow, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tdw, dWTp, prow, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tmq, dMQ, prow, 64, 64, 64))) return r;
  ChunkParams p;
  p.dgc = dgc; p.geo = geo; p.status = status;
  static ss::SmemOptIn opt_in;
  if (int e = opt_in.ensure(dn_bwd_chunk_kernel, chunkk::SMEM)) return e;
  dn_bwd_chunk_kernel<<<dim3(geo.n, H), THREADS, chunkk::SMEM, (cudaStream_t)stream>>>(tdsp, tst, tut, tdut,
                                                                                      tdo, tkd, tqg, tdw, tmq, p);
  return (int)cudaGetLastError();
}

int ss_dn_bwd_prep(const void* q, const void* k, const void* v, const float* beta, const int* sid,
                   const float* gam, const float* gc, const float* dgc, const void* dWTp,
                   const void* dUTp, const void* TMT, const void* XW, const void* XU, const void* dKdTp,
                   const void* dQgTp, const void* dMQ, void* dq, void* dk, void* dv, float* dbeta,
                   float* dg, int T, int H, int Hk, float scale, int* status, void* stream) {
  if (T <= 0) return 0;
  if (H <= 0 || Hk <= 0 || H % Hk) return -2;
  const Geo geo = make_geo(T, H, Hk);
  const long long prow = (long long)geo.n * geo.NP * 128;
  CUtensorMap tq, tk, tv, tdw, tdu, ttm, txw, txu, tkd, tqg, tok, toq, tov;
  int r;
  if ((r = ss::make_tmap_bf16(&tq, q, T, (long long)Hk * D, (long long)Hk * D, 64))) return r;
  if ((r = ss::make_tmap_bf16(&tk, k, T, (long long)Hk * D, (long long)Hk * D, 64))) return r;
  if ((r = ss::make_tmap_bf16(&tv, v, T, (long long)H * D, (long long)H * D, 64))) return r;
  if ((r = ss::make_tmap_bf16(&tdw, dWTp, prow, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tdu, dUTp, prow, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&ttm, TMT, prow, 64, 64, 128))) return r;
  if ((r = ss::make_tmap_bf16(&txw, XW, prow, 64, 64, 128))) return r;
  if ((r = ss::make_tmap_bf16(&txu, XU, prow, 64, 64, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tkd, dKdTp, prow, 128, 128, 128))) return r;
  if ((r = ss::make_tmap_bf16(&tqg, dQgTp, prow, 128, 128, 128))) return r;
  const long long owidth = (long long)geo.NP * D;        // dq, dk: [T, NP, D], summed over pairs by the caller
  if ((r = ss::make_tmap_bf16(&tok, dk, T, owidth, owidth, 64))) return r;
  if ((r = ss::make_tmap_bf16(&toq, dq, T, owidth, owidth, 64))) return r;
  if ((r = ss::make_tmap_bf16(&tov, dv, T, (long long)H * D, (long long)H * D, 64))) return r;
  BwdPrepParams p;
  p.beta = beta; p.sid = sid; p.gam = gam; p.gc = gc; p.dgc = dgc;
  p.dMQ = (const __nv_bfloat16*)dMQ; p.dbeta = dbeta; p.dg = dg; p.geo = geo; p.scale = scale; p.status = status;
  static ss::SmemOptIn opt_in;
  if (int e = opt_in.ensure(dn_bwd_prep_kernel, bprep::SMEM)) return e;
  dn_bwd_prep_kernel<<<dim3(geo.n, geo.NP), bprep::BTHREADS, bprep::SMEM, (cudaStream_t)stream>>>(
      tq, tk, tv, tdw, tdu, ttm, txw, txu, tkd, tqg, tok, toq, tov, p);
  return (int)cudaGetLastError();
}
}  // extern "C"
