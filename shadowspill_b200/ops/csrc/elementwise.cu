// Bandwidth-bound model ops for sm_100a: rotary embedding, SwiGLU, embedding gather / scatter-add, masked weighted cross-entropy
// over a logits block, AdamW with bf16 stochastic rounding, sum-of-squares.
//
// All kernels move 16-byte vectors, keep reductions in fp32 and take explicit
// extents. The math follows the reference's pure-PyTorch definitions in
// packages/workloads/src/shadowspill_workloads/models/shared/decoder.py
// (apply_rotary :232, swiglu :292, language_model_loss :320).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "chained_launch.cuh"
#include "swiglu_math.cuh"
#include "launchers.h"

namespace ss {

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ float2 up2(uint32_t u) {
  __nv_bfloat162 v = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(v);
}
__device__ __forceinline__ uint32_t pk2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  float2 a = up2(u.x), b = up2(u.y), c = up2(u.z), d = up2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  u.x = pk2(f[0], f[1]); u.y = pk2(f[2], f[3]); u.z = pk2(f[4], f[5]); u.w = pk2(f[6], f[7]);
  return u;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Block-wide sum; `red` is >= 33 floats of shared memory.
__device__ __forceinline__ float block_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    float t = lane < nw ? red[lane] : 0.f;
    t = warp_sum(t);
    if (lane == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}
__device__ __forceinline__ float block_max(float v, float* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    float t = lane < nw ? red[lane] : -INFINITY;
    t = warp_max(t);
    if (lane == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}

// =============================================================== rotary embedding
// In place on a [T, row_stride] buffer holding `heads` heads of width dh starting
// at column col0; rotates the first `rot` channels of each head with the
// half-split convention: (a, b) = (x[i], x[i + rot/2]) ->
// (a cos - b sin, b cos + a sin). inverse != 0 applies the transposed rotation,
// which is the backward pass.
__global__ void rope_kernel(bf16* buf, const int* positions, int T,
                            long long row_stride, int col0, int heads, int dh, int rot,
                            float log2_theta, int inverse) {
  chain_wait();
  chain_release();
  const int half = rot >> 1;
  const int pairs_per_head = half >> 1;  // two pairs per thread (bf16x2)
  const long long total = static_cast<long long>(T) * heads * pairs_per_head;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int pp = static_cast<int>(idx % pairs_per_head);
    const long long rest = idx / pairs_per_head;
    const int h = static_cast<int>(rest % heads);
    const int t = static_cast<int>(rest / heads);
    const float pos = static_cast<float>(positions[t]);
    bf16* base = buf + static_cast<long long>(t) * row_stride + col0 + h * dh;
    const int i = pp * 2;
    __nv_bfloat162 a2 = *reinterpret_cast<__nv_bfloat162*>(base + i);
    __nv_bfloat162 b2 = *reinterpret_cast<__nv_bfloat162*>(base + i + half);
    float2 a = __bfloat1622float2(a2), b = __bfloat1622float2(b2);
    float s0, c0, s1, c1;
    // inv_freq_i = theta^(-2i/rot)
    const float f0 = exp2f(-log2_theta * (2.f * i) / rot);
    const float f1 = exp2f(-log2_theta * (2.f * (i + 1)) / rot);
    sincosf(pos * f0, &s0, &c0);
    sincosf(pos * f1, &s1, &c1);
    if (inverse) { s0 = -s0; s1 = -s1; }
    float2 oa, ob;
    oa.x = a.x * c0 - b.x * s0; ob.x = b.x * c0 + a.x * s0;
    oa.y = a.y * c1 - b.y * s1; ob.y = b.y * c1 + a.y * s1;
    *reinterpret_cast<__nv_bfloat162*>(base + i) = __float22bfloat162_rn(oa);
    *reinterpret_cast<__nv_bfloat162*>(base + i + half) = __float22bfloat162_rn(ob);
  }
}

// Vector form: a thread owns eight adjacent frequencies of one token (its sines and
// cosines are computed once) and walks `heads_per_thread` heads with 16-byte loads, so
// the transcendental work is amortised over the heads and the kernel runs at memory
// speed. Needs rot % 16 == 0 and 16-byte aligned heads.
__global__ void rope_vec_kernel(bf16* buf, const int* positions, int T,
                                long long row_stride, int col0, int heads, int dh, int rot,
                                float log2_theta, int inverse, int slots) {
  chain_wait();
  chain_release();
  const int half = rot >> 1;
  const int vph = half >> 3;
  const int per_token = vph * slots;
  const long long total = static_cast<long long>(T) * per_token;
  for (long long gid = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; gid < total;
       gid += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int t = static_cast<int>(gid / per_token);
    const int r = static_cast<int>(gid % per_token);
    const int slot = r / vph;
    const int i0 = (r % vph) * 8;
    const float pos = static_cast<float>(positions[t]);
    float sn[8], cs[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float f = exp2f(-log2_theta * (2.f * (i0 + e)) / rot);
      // sin/cos of pi*(angle/pi): the argument reduction of sincospif is exact and short
      sincospif(pos * f * 0.31830988618379067f, &sn[e], &cs[e]);
      if (inverse) sn[e] = -sn[e];
    }
    bf16* row = buf + static_cast<long long>(t) * row_stride + col0 + i0;
    // up to four heads per pass with every load issued before the first use
    for (int h0 = slot; h0 < heads; h0 += 4 * slots) {
      uint4 av[4], bv[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int h = h0 + k * slots;
        if (h < heads) {
          av[k] = *reinterpret_cast<const uint4*>(row + h * dh);
          bv[k] = *reinterpret_cast<const uint4*>(row + h * dh + half);
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int h = h0 + k * slots;
        if (h >= heads) continue;
        __nv_bfloat162* a2 = reinterpret_cast<__nv_bfloat162*>(&av[k]);
        __nv_bfloat162* b2 = reinterpret_cast<__nv_bfloat162*>(&bv[k]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 a = __bfloat1622float2(a2[e]), b = __bfloat1622float2(b2[e]);
          float2 oa, ob;
          oa.x = a.x * cs[2 * e] - b.x * sn[2 * e];
          ob.x = b.x * cs[2 * e] + a.x * sn[2 * e];
          oa.y = a.y * cs[2 * e + 1] - b.y * sn[2 * e + 1];
          ob.y = b.y * cs[2 * e + 1] + a.y * sn[2 * e + 1];
          a2[e] = __float22bfloat162_rn(oa);
          b2[e] = __float22bfloat162_rn(ob);
        }
        *reinterpret_cast<uint4*>(row + h * dh) = av[k];
        *reinterpret_cast<uint4*>(row + h * dh + half) = bv[k];
      }
    }
  }
}

// idx = t * nv + c with 32-bit arithmetic whenever idx fits (a 64-bit division costs ~100 instructions)
__device__ __forceinline__ void split_index(long long idx, int nv, long long& t, int& c) {
  if (idx < (1LL << 31)) {
    const unsigned i = static_cast<unsigned>(idx), q = i / static_cast<unsigned>(nv);
    t = q; c = static_cast<int>(i - q * static_cast<unsigned>(nv));
  } else {
    t = idx / nv; c = static_cast<int>(idx - t * nv);
  }
}

// =============================================================== SwiGLU
// gu is [T, 2F] with gate in columns [0,F) and up in [F,2F) (one fused GEMM
// output). h = bf16(silu(float(gate))) * up.
// `used` (optional, device memory): rows at and past *used are left alone.
__global__ void swiglu_fwd_kernel(const bf16* gu, bf16* h, int T, int F, const int* used) {
  chain_wait();
  chain_release();
  const int nv = F >> 3;
  if (used) T = min(T, *used);
  const long long total = static_cast<long long>(T) * nv;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    long long t; int c;
    split_index(idx, nv, t, c);
    const uint4* row = reinterpret_cast<const uint4*>(gu + t * 2 * F);
    float g[8], u[8], o[8];
    unpack8(row[c], g);
    unpack8(row[nv + c], u);
#pragma unroll
    for (int e = 0; e < 8; ++e) o[e] = swiglu_value(g[e], u[e]);
    reinterpret_cast<uint4*>(h + t * F)[c] = pack8(o);
  }
}
// dgu[T,2F] from dh[T,F] and the saved gu.
__global__ void swiglu_bwd_kernel(const bf16* gu, const bf16* dh, bf16* dgu, int T, int F) {
  chain_wait();
  chain_release();
  const int nv = F >> 3;
  const long long total = static_cast<long long>(T) * nv;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    long long t; int c;
    split_index(idx, nv, t, c);
    const uint4* row = reinterpret_cast<const uint4*>(gu + t * 2 * F);
    float g[8], u[8], d[8], og[8], ou[8];
    unpack8(row[c], g);
    unpack8(row[nv + c], u);
    unpack8(reinterpret_cast<const uint4*>(dh + t * F)[c], d);
#pragma unroll
    for (int e = 0; e < 8; ++e) swiglu_grad(g[e], u[e], d[e], og[e], ou[e]);
    uint4* orow = reinterpret_cast<uint4*>(dgu + t * 2 * F);
    orow[c] = pack8(og);
    orow[nv + c] = pack8(ou);
  }
}

// =============================================================== embedding
__global__ void embedding_fwd_kernel(const long long* __restrict__ ids, const bf16* __restrict__ W,
                                     bf16* __restrict__ out, int T, int D, int V) {
  const int nv = D >> 3;
  for (int row = blockIdx.x; row < T; row += gridDim.x) {
    long long id = ids[row];
    if (id < 0 || id >= V) id = 0;
    const uint4* src = reinterpret_cast<const uint4*>(W + id * D);
    uint4* dst = reinterpret_cast<uint4*>(out + static_cast<size_t>(row) * D);
    for (int c = threadIdx.x; c < nv; c += blockDim.x) dst[c] = src[c];
  }
}
// dW[id] += g[row] (fp32 accumulator table, one atomic per element).
__global__ void embedding_bwd_kernel(const long long* __restrict__ ids, const bf16* __restrict__ g,
                                     float* __restrict__ dW, int T, int D, int V) {
  for (int row = blockIdx.x; row < T; row += gridDim.x) {
    long long id = ids[row];
    if (id < 0 || id >= V) continue;
    const bf16* src = g + static_cast<size_t>(row) * D;
    float* dst = dW + id * D;
    for (int c = threadIdx.x; c < D; c += blockDim.x) atomicAdd(dst + c, __bfloat162float(src[c]));
  }
}
// bf16 gradient table variant (packed bf16x2 atomics).
__global__ void embedding_bwd_bf16_kernel(const long long* __restrict__ ids,
                                          const bf16* __restrict__ g, bf16* __restrict__ dW, int T,
                                          int D, int V) {
  for (int row = blockIdx.x; row < T; row += gridDim.x) {
    long long id = ids[row];
    if (id < 0 || id >= V) continue;
    const __nv_bfloat162* src = reinterpret_cast<const __nv_bfloat162*>(g + static_cast<size_t>(row) * D);
    __nv_bfloat162* dst = reinterpret_cast<__nv_bfloat162*>(dW + id * D);
    for (int c = threadIdx.x; c < (D >> 1); c += blockDim.x) atomicAdd(dst + c, src[c]);
  }
}

// =============================================================== cross-entropy on a logits block
// logits [R, V] bf16 (row pitch ld). For each row: lse, loss contribution
// weight * (lse - logit[target]); then the row is REWRITTEN IN PLACE with its
// gradient weight * grad_scale * (softmax - onehot). Rows with weight 0 (masked)
// produce a zero gradient row. loss_sum / weight_sum accumulate with atomics.
//
// mode 1 is the clipped policy objective on the same block: with
// logp = logit[target] - lse, r = exp(logp - old_logp), A = advantage,
//   L = -min(r A, clamp(r, 1-clip, 1+clip) A)  [+ beta * (exp(ref-logp) - (ref-logp) - 1)]
// and the row becomes weight * grad_scale * dL/dlogp * (onehot - softmax).
struct PolicyArgs {
  int mode;                 // 0 cross-entropy, 1 clipped policy
  const float* old_logp;
  const float* advantage;
  const float* ref_logp;    // optional
  float clip, ref_beta;
  float* logp_out;          // optional: per-row log-probability of the target
};
// A block of logits of listed rows: its row i is token rows[from + i] where from + i < *used. What lies behind them is
// not a token's, and zeroed up to the next multiple of 64 rows of the block, the depth to which the weight gradient's
// products read it.
struct RowList {
  const int* rows;          // null: row i is token i
  const int* used;
  int from;
};
constexpr int CE_THREADS = 512;
__global__ void __launch_bounds__(CE_THREADS)
cross_entropy_kernel(bf16* __restrict__ logits, const long long* __restrict__ targets,
                     const float* __restrict__ weights, float* __restrict__ loss_sum,
                     float* __restrict__ lse_out, int R, int V, long long ld, float grad_scale,
                     int write_grad, PolicyArgs pa, RowList list) {
  __shared__ float red[33];
  int row = blockIdx.x;
  if (row >= R) return;
  bf16* lr = logits + static_cast<long long>(row) * ld;
  const int nv = V >> 3;
  auto clear = [&] {
    for (int c = threadIdx.x; c < nv; c += CE_THREADS) reinterpret_cast<uint4*>(lr)[c] = make_uint4(0, 0, 0, 0);
    for (int c = nv * 8 + threadIdx.x; c < V; c += CE_THREADS) lr[c] = __float2bfloat16_rn(0.f);
  };
  if (list.rows != nullptr) {
    const int at = list.from + row, used = *list.used;
    if (at >= used) {
      if (write_grad && row < (used - list.from + 63) / 64 * 64) clear();
      return;
    }
    row = list.rows[at];
  }
  // Nothing is asked of a masked row but its gradient, so a row longer than one load per thread is looked at first; its
  // start is on its way meanwhile. Shorter ones would only wait for their target (300 rows of 1,000: 4.7 -> 5.5 us).
  if (V > 8 * CE_THREADS && lse_out == nullptr && pa.logp_out == nullptr) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint4*>(lr) + threadIdx.x));
    const long long t = targets[row];
    if (t < 0 || t >= V || (weights != nullptr && weights[row] == 0.f)) {
      if (write_grad) clear();
      return;
    }
  }
  const uint4* lv = reinterpret_cast<const uint4*>(lr);
  float m = -INFINITY, s = 0.f;
  for (int c = threadIdx.x; c < nv; c += CE_THREADS) {
    float f[8];
    unpack8(lv[c], f);
    float lm = f[0];
#pragma unroll
    for (int e = 1; e < 8; ++e) lm = fmaxf(lm, f[e]);
    if (lm > m) {
      s *= __expf(m - lm);
      m = lm;
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) s += __expf(f[e] - m);
  }
  for (int c = nv * 8 + threadIdx.x; c < V; c += CE_THREADS) {
    const float f = __bfloat162float(lr[c]);
    if (f > m) { s *= __expf(m - f); m = f; }
    s += __expf(f - m);
  }
  // read again rather than kept: with two registers less for the pass above, 2,048 rows of 128,256 took 271 us, not 255
  asm volatile("" : "+r"(row));
  const float wgt = weights ? weights[row] : 1.f;
  const long long tgt = targets[row];
  const bool in_vocab = tgt >= 0 && tgt < V;
  const bool valid = in_vocab && wgt != 0.f;
  const float gm = block_max(m, red);
  s = (m == -INFINITY) ? 0.f : s * __expf(m - gm);
  const float gs = block_sum(s, red);
  const float lse = gm + __logf(gs);
  const float logp = in_vocab ? __bfloat162float(lr[tgt]) - lse : 0.f;
  float row_loss = -logp, dl_dlogp = -1.f;
  if (pa.mode == 1 && valid) {
    const float r = __expf(logp - pa.old_logp[row]);
    const float A = pa.advantage[row];
    const float unclipped = r * A;
    const float clipped = fminf(fmaxf(r, 1.f - pa.clip), 1.f + pa.clip) * A;
    row_loss = -fminf(unclipped, clipped);
    dl_dlogp = (unclipped <= clipped) ? -unclipped : 0.f;
    if (pa.ref_logp != nullptr) {
      const float d = pa.ref_logp[row] - logp;
      row_loss += pa.ref_beta * (__expf(d) - d - 1.f);
      dl_dlogp += pa.ref_beta * (1.f - __expf(d));
    }
  }
  if (threadIdx.x == 0) {
    if (lse_out) lse_out[row] = lse;
    if (pa.logp_out) pa.logp_out[row] = logp;
    if (valid) atomicAdd(loss_sum, wgt * row_loss);
  }
  if (!write_grad) return;
  __syncthreads();
  if (!valid) {
    clear();
    return;
  }
  const float scale = -wgt * grad_scale * dl_dlogp;
  uint4* gv = reinterpret_cast<uint4*>(lr);
  for (int c = threadIdx.x; c < nv; c += CE_THREADS) {
    float f[8];
    unpack8(lv[c], f);
    const int base = c * 8;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float p = __expf(f[e] - lse);
      if (base + e == tgt) p -= 1.f;
      f[e] = p * scale;
    }
    gv[c] = pack8(f);
  }
  for (int c = nv * 8 + threadIdx.x; c < V; c += CE_THREADS) {
    float p = __expf(__bfloat162float(lr[c]) - lse);
    if (c == tgt) p -= 1.f;
    lr[c] = __float2bfloat16_rn(p * scale);
  }
}

// =============================================================== rows that the loss scores
__global__ void __launch_bounds__(1024)
scored_rows_kernel(const long long* __restrict__ targets, const float* __restrict__ weights, int T, int V,
                   int* __restrict__ rows, int* __restrict__ slot, int* __restrict__ count) {
  __shared__ int per_warp[32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int base = 0;
  for (int t0 = 0; t0 < T; t0 += 1024) {
    const int t = t0 + threadIdx.x;
    const long long tgt = t < T ? targets[t] : -1;
    const bool scored = tgt >= 0 && tgt < V && (weights == nullptr || weights[t] != 0.f);
    const unsigned vote = __ballot_sync(0xffffffffu, scored);
    if (lane == 0) per_warp[warp] = __popc(vote);
    __syncthreads();
    const int mine = per_warp[lane];
    const int before = __reduce_add_sync(0xffffffffu, lane < warp ? mine : 0);
    const int at = base + before + __popc(vote & ((1u << lane) - 1));
    base += __reduce_add_sync(0xffffffffu, mine);
    if (t < T) slot[t] = scored ? at : -1;
    if (scored) rows[at] = t;
    __syncthreads();
  }
  for (int i = base + threadIdx.x; i < T; i += 1024) rows[i] = -1;
  if (threadIdx.x == 0) *count = base;
}
__global__ void __launch_bounds__(256)
take_rows_kernel(const bf16* x, long long ldx, const int* index, bf16* out, long long ldo, int n, int D) {
  chain_wait();
  chain_release();
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const int from = index[i];
    const uint4* src = reinterpret_cast<const uint4*>(x + from * ldx);
    uint4* dst = reinterpret_cast<uint4*>(out + i * ldo);
    for (int c = threadIdx.x; c < D / 8; c += 256) dst[c] = from < 0 ? make_uint4(0, 0, 0, 0) : src[c];
  }
}

// =============================================================== AdamW with stochastic rounding
// Philox4x32-10 counter RNG: (seed, step) key, element index counter.
__device__ __forceinline__ uint4 philox4x32(uint4 ctr, uint2 key) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(M0, ctr.x), lo0 = M0 * ctr.x;
    const uint32_t hi1 = __umulhi(M1, ctr.z), lo1 = M1 * ctr.z;
    ctr = make_uint4(hi1 ^ ctr.y ^ key.x, lo1, hi0 ^ ctr.w ^ key.y, lo0);
    key.x += W0;
    key.y += W1;
  }
  return ctr;
}
struct AdamWArgs {
  float lr, beta1, beta2, eps, weight_decay, bias1, bias2, grad_scale;
  unsigned long long seed;
  unsigned long long offset;  // global element offset of this flat range (sharding-invariant RNG)
};

// Eight updated values in fp32 -> bf16 in the upper halves of `u`: stochastic rounding adds 16 random
// bits below the kept mantissa and truncates (inf and nan are only truncated), else round to nearest.
template <bool SR>
__device__ __forceinline__ void round8(const float (&f)[8], const uint32_t* rnd, uint32_t (&u)[8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e)
    u[e] = SR ? __float_as_uint(f[e]) + ((e & 1) ? rnd[e >> 1] >> 16 : rnd[e >> 1] & 0xffffu)
              : static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(f[e]))) << 16;
  if (SR) {
    // x * 0 is nan for inf and nan and zero otherwise: one test for the eight values, on the pipe that
    // has room (the integer pipe is what bounds this kernel)
    float z = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) z = fmaf(f[e], 0.f, z);
    if (z != 0.f) {
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if ((__float_as_uint(f[e]) & 0x7f800000u) == 0x7f800000u) u[e] = __float_as_uint(f[e]);
    }
  }
}
__device__ __forceinline__ uint4 upper_halves(const uint32_t (&u)[8]) {
  return make_uint4(__byte_perm(u[0], u[1], 0x7632), __byte_perm(u[2], u[3], 0x7632),
                    __byte_perm(u[4], u[5], 0x7632), __byte_perm(u[6], u[7], 0x7632));
}

// Eight elements from global index `gidx` (a multiple of 8): new values as bf16 in the upper halves.
template <bool SR_PARAM, bool SR_STATE>
__device__ __forceinline__ void adamw_update8(const AdamWArgs& a, unsigned long long gidx, const float (&pf)[8],
                                              const float (&gf)[8], const float (&mf)[8], const float (&vf)[8],
                                              uint32_t (&po)[8], uint32_t (&mo)[8], uint32_t (&vo)[8]) {
  const float c1 = 1.f - a.beta1, c2 = 1.f - a.beta2, keep = 1.f - a.lr * a.weight_decay;
  const uint2 key = make_uint2(static_cast<uint32_t>(a.seed), static_cast<uint32_t>(a.seed >> 32));
  uint32_t rw[12];
  if (SR_PARAM || SR_STATE) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const uint4 r = philox4x32(make_uint4(static_cast<uint32_t>(gidx >> 3), static_cast<uint32_t>(gidx >> 35),
                                            static_cast<uint32_t>(k), 0x5353u), key);
      rw[4 * k] = r.x; rw[4 * k + 1] = r.y; rw[4 * k + 2] = r.z; rw[4 * k + 3] = r.w;
    }
  }
  float pn[8], mn[8], vn[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float gg = gf[e] * a.grad_scale;
    mn[e] = fmaf(a.beta1, mf[e], c1 * gg);
    vn[e] = fmaf(a.beta2, vf[e], c2 * gg * gg);
    // bias1/bias2 hold the reciprocals of the bias corrections (set by the launcher)
    const float mhat = mn[e] * a.bias1;
    const float vhat = vn[e] * a.bias2;
    pn[e] = pf[e] * keep;
    pn[e] -= a.lr * __fdividef(mhat, __fsqrt_rn(vhat) + a.eps);
  }
  round8<SR_PARAM>(pn, rw, po);
  round8<SR_STATE>(mn, rw + 4, mo);
  round8<SR_STATE>(vn, rw + 8, vo);
}
// The last one to seven elements of a tensor, from element e0.
template <bool SR_PARAM, bool SR_STATE, bool G_F32>
__device__ __forceinline__ void adamw_tail(bf16* p, const void* g, bf16* m, bf16* v, const AdamWArgs& a,
                                           unsigned long long offset, long long e0, int tail) {
  float pf[8], gf[8], mf[8], vf[8];
  uint32_t po[8], mo[8], vo[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const bool in = e < tail;
    pf[e] = in ? __bfloat162float(p[e0 + e]) : 0.f;
    mf[e] = in ? __bfloat162float(m[e0 + e]) : 0.f;
    vf[e] = in ? __bfloat162float(v[e0 + e]) : 0.f;
    gf[e] = in ? (G_F32 ? static_cast<const float*>(g)[e0 + e]
                        : __bfloat162float(static_cast<const bf16*>(g)[e0 + e]))
               : 0.f;
  }
  adamw_update8<SR_PARAM, SR_STATE>(a, offset + static_cast<unsigned long long>(e0), pf, gf, mf, vf, po, mo, vo);
#pragma unroll
  for (int e = 0; e < 8; ++e) {              // static indices keep po/mo/vo in registers
    if (e < tail) {
      p[e0 + e] = __ushort_as_bfloat16(static_cast<unsigned short>(po[e] >> 16));
      m[e0 + e] = __ushort_as_bfloat16(static_cast<unsigned short>(mo[e] >> 16));
      v[e0 + e] = __ushort_as_bfloat16(static_cast<unsigned short>(vo[e] >> 16));
    }
  }
}

// p, m, v bf16; g bf16 or fp32. Eight elements per thread. Bound by the integer pipe (three Philox calls
// and 24 roundings per eight elements), not by memory: the rounding and gradient-type choices are
// template parameters, halves are packed by byte permutes and the inf / nan test is shared by eight
// values. One vector per thread is always in flight behind the arithmetic, in two persistent blocks per SM
// (three at 80 registers spill: 667 against 594 us for a 218 M element layer). 58.7 M elements: 647 -> 525
// instructions per eight, 192 -> 153 us (kernel durations, L2 flushed before each launch); the results keep
// their bits.
constexpr int ADAMW_THREADS = 256;
template <bool SR_PARAM, bool SR_STATE, bool G_F32>
__global__ void __launch_bounds__(ADAMW_THREADS, 2)
adamw_sr_kernel(bf16* __restrict__ p, const void* __restrict__ g, bf16* __restrict__ m, bf16* __restrict__ v,
                long long n, AdamWArgs a) {
  float pf[8], gf[8], mf[8], vf[8];
  uint32_t po[8], mo[8], vo[8];
  const long long nvec = n >> 3, first = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  // the next vector's loads are in flight under this one's arithmetic
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  uint4 q[5] = {};
  auto fetch = [&](long long i) {
    q[0] = *reinterpret_cast<const uint4*>(p + (i << 3));
    q[1] = *reinterpret_cast<const uint4*>(m + (i << 3));
    q[2] = *reinterpret_cast<const uint4*>(v + (i << 3));
    if (G_F32) {
      const uint4* gv = reinterpret_cast<const uint4*>(static_cast<const float*>(g) + (i << 3));
      q[3] = gv[0];
      q[4] = gv[1];
    } else {
      q[3] = *reinterpret_cast<const uint4*>(static_cast<const bf16*>(g) + (i << 3));
    }
  };
  if (first < nvec) fetch(first);
  for (long long i = first; i < nvec; i += step) {
    const long long e0 = i << 3;
    unpack8(q[0], pf);
    unpack8(q[1], mf);
    unpack8(q[2], vf);
    if (G_F32) {
      gf[0] = __uint_as_float(q[3].x); gf[1] = __uint_as_float(q[3].y);
      gf[2] = __uint_as_float(q[3].z); gf[3] = __uint_as_float(q[3].w);
      gf[4] = __uint_as_float(q[4].x); gf[5] = __uint_as_float(q[4].y);
      gf[6] = __uint_as_float(q[4].z); gf[7] = __uint_as_float(q[4].w);
    } else {
      unpack8(q[3], gf);
    }
    if (i + step < nvec) fetch(i + step);
    adamw_update8<SR_PARAM, SR_STATE>(a, a.offset + static_cast<unsigned long long>(e0), pf, gf, mf, vf, po, mo, vo);
    *reinterpret_cast<uint4*>(p + e0) = upper_halves(po);
    *reinterpret_cast<uint4*>(m + e0) = upper_halves(mo);
    *reinterpret_cast<uint4*>(v + e0) = upper_halves(vo);
  }
  const int tail = static_cast<int>(n & 7);
  if (tail && first == nvec % (static_cast<long long>(gridDim.x) * blockDim.x))
    adamw_tail<SR_PARAM, SR_STATE, G_F32>(p, g, m, v, a, a.offset, nvec << 3, tail);
}

// Many small tensors in one launch: a block of 256 vectors belongs to one tensor, found in the launch's own
// table. Bound by launches: 27 tensors of a 256-wide model took 80 us on the device one by one, 23 us with
// the 25 small ones in one launch, and the host's part of 24 launches is gone (whole step 2.27 -> 2.11 ms).
constexpr int ADAMW_MANY = 40;
struct AdamWTensor {
  bf16 *p, *m, *v;
  const void* g;
  unsigned long long offset;
  int n, g_f32;
};
struct AdamWTable {
  AdamWTensor t[ADAMW_MANY];
  int first_block[ADAMW_MANY];
  int count;
};
template <bool SR_PARAM, bool SR_STATE>
__global__ void __launch_bounds__(ADAMW_THREADS, 2)
adamw_sr_many_kernel(const __grid_constant__ AdamWTable tab, AdamWArgs a) {
  const int blk = blockIdx.x;
  int lo = 0, hi = tab.count - 1;                     // the last tensor that starts at or before this block
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (tab.first_block[mid] <= blk) lo = mid; else hi = mid - 1;
  }
  const AdamWTensor& t = tab.t[lo];
  const int e0 = ((blk - tab.first_block[lo]) * ADAMW_THREADS + static_cast<int>(threadIdx.x)) * 8;
  if (e0 >= t.n) return;
  if (t.n - e0 < 8) {
    if (t.g_f32) adamw_tail<SR_PARAM, SR_STATE, true>(t.p, t.g, t.m, t.v, a, t.offset, e0, t.n - e0);
    else         adamw_tail<SR_PARAM, SR_STATE, false>(t.p, t.g, t.m, t.v, a, t.offset, e0, t.n - e0);
    return;
  }
  float pf[8], gf[8], mf[8], vf[8];
  uint32_t po[8], mo[8], vo[8];
  const uint4 qp = *reinterpret_cast<const uint4*>(t.p + e0), qm = *reinterpret_cast<const uint4*>(t.m + e0),
              qv = *reinterpret_cast<const uint4*>(t.v + e0);
  if (t.g_f32) {
    const float4* gv = reinterpret_cast<const float4*>(static_cast<const float*>(t.g) + e0);
    const float4 g0 = gv[0], g1 = gv[1];
    gf[0] = g0.x; gf[1] = g0.y; gf[2] = g0.z; gf[3] = g0.w;
    gf[4] = g1.x; gf[5] = g1.y; gf[6] = g1.z; gf[7] = g1.w;
  } else {
    unpack8(*reinterpret_cast<const uint4*>(static_cast<const bf16*>(t.g) + e0), gf);
  }
  unpack8(qp, pf);
  unpack8(qm, mf);
  unpack8(qv, vf);
  adamw_update8<SR_PARAM, SR_STATE>(a, t.offset + static_cast<unsigned long long>(e0), pf, gf, mf, vf, po, mo, vo);
  *reinterpret_cast<uint4*>(t.p + e0) = upper_halves(po);
  *reinterpret_cast<uint4*>(t.m + e0) = upper_halves(mo);
  *reinterpret_cast<uint4*>(t.v + e0) = upper_halves(vo);
}

// fp32 state variant (master-free fp32 parameters, e.g. A_log / dt_bias exceptions).
__global__ void adamw_f32_kernel(float* __restrict__ p, const float* __restrict__ g,
                                 float* __restrict__ m, float* __restrict__ v, long long n,
                                 AdamWArgs a) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const float gg = g[i] * a.grad_scale;
    const float mn = a.beta1 * m[i] + (1.f - a.beta1) * gg;
    const float vn = a.beta2 * v[i] + (1.f - a.beta2) * gg * gg;
    float pn = p[i] * (1.f - a.lr * a.weight_decay);
    pn -= a.lr * (mn / a.bias1) / (sqrtf(vn / a.bias2) + a.eps);
    p[i] = pn; m[i] = mn; v[i] = vn;
  }
}

// =============================================================== sum of squares (parameter norms)
// <=256 partials then one scalar; allocation-free, mirrors the reference's two
// diagnostic kernels (packages/engine/src/shadowspill/execution/observations/kernels.py:18,40).
__global__ void sumsq_partials_kernel(const bf16* __restrict__ x, long long n,
                                      float* __restrict__ partials) {
  __shared__ float red[33];
  float acc = 0.f;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const float f = __bfloat162float(x[i]);
    acc += f * f;
  }
  const float t = block_sum(acc, red);
  if (threadIdx.x == 0) partials[blockIdx.x] = t;
}
__global__ void sumsq_final_kernel(const float* __restrict__ partials, int n, float* __restrict__ out,
                                   int accumulate) {
  __shared__ float red[33];
  float acc = 0.f;
  for (int i = threadIdx.x; i < n; i += blockDim.x) acc += partials[i];
  const float t = block_sum(acc, red);
  if (threadIdx.x == 0) out[0] = accumulate ? out[0] + t : t;
}

// fp32 -> bf16 cast with optional scale (used to publish fp32 accumulators).
__global__ void cast_f32_bf16_kernel(const float* __restrict__ src, bf16* __restrict__ dst,
                                     long long n, float scale) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    dst[i] = __float2bfloat16_rn(src[i] * scale);
}

static inline int grid_for(long long work, int threads, int cap = 148 * 8) {
  long long g = (work + threads - 1) / threads;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return static_cast<int>(g);
}

static AdamWArgs adamw_args(float lr, float beta1, float beta2, float eps, float weight_decay, int step,
                            float grad_scale, unsigned long long seed, unsigned long long offset) {
  AdamWArgs a;
  a.lr = lr; a.beta1 = beta1; a.beta2 = beta2; a.eps = eps; a.weight_decay = weight_decay;
  a.bias1 = 1.f / (1.f - powf(beta1, (float)step));     // reciprocals: the kernel multiplies
  a.bias2 = 1.f / (1.f - powf(beta2, (float)step));
  a.grad_scale = grad_scale;
  a.seed = seed ^ (0x9E3779B97F4A7C15ull * (unsigned long long)(step + 1));
  a.offset = offset;
  return a;
}
// One vector per thread of the persistent form's grid: a larger tensor fills the GPU by itself, and its next
// vector's loads run under the arithmetic there. The caller of the shared form has the same number.
constexpr long long ADAMW_MANY_ELEMENTS = 148ll * 2 * ADAMW_THREADS * 8;

}  // namespace ss

extern "C" {
using namespace ss;

int ss_rope(void* buf, const int* positions, int T, long long row_stride, int col0, int heads,
            int dh, int rot, float theta, int inverse, void* stream) {
  if (rot % 4 || rot > dh || row_stride % 2 || col0 % 2) return -2;
  if (T <= 0) return 0;
  if (rot % 16 == 0 && dh % 8 == 0 && col0 % 8 == 0 && row_stride % 8 == 0 &&
      (reinterpret_cast<uintptr_t>(buf) & 15) == 0) {
    const int hpt = heads >= 8 ? 4 : 1;              // heads walked by one thread
    const int slots = (heads + hpt - 1) / hpt;
    const long long threads = (long long)T * (rot >> 4) * slots;
    launch_chained(rope_vec_kernel, grid_for(threads, 256), 256, 0, (cudaStream_t)stream,
                   (bf16*)buf, positions, T, row_stride, col0, heads, dh, rot, log2f(theta), inverse, slots);
    return (int)cudaGetLastError();
  }
  const long long total = (long long)T * heads * (rot >> 2);
  launch_chained(rope_kernel, grid_for(total, 256), 256, 0, (cudaStream_t)stream,
                 (bf16*)buf, positions, T, row_stride, col0, heads, dh, rot, log2f(theta), inverse);
  return (int)cudaGetLastError();
}
int ss_swiglu_fwd(const void* gu, void* h, int T, int F, void* stream) {
  if (F % 8) return -2;
  if (T <= 0) return 0;
  launch_chained(swiglu_fwd_kernel, grid_for((long long)T * (F >> 3), 256, 148 * 16), 256, 0, (cudaStream_t)stream,
                 (const bf16*)gu, (bf16*)h, T, F, nullptr);
  return (int)cudaGetLastError();
}
// The first *used rows only (`used` in device memory): sorted expert rows, whose count the host does not know.
int ss_swiglu_fwd_used(const void* gu, void* h, int T, int F, const int* used, void* stream) {
  if (F % 8) return -2;
  if (T <= 0) return 0;
  swiglu_fwd_kernel<<<grid_for((long long)T * (F >> 3), 256, 148 * 16), 256, 0, (cudaStream_t)stream>>>(
      (const bf16*)gu, (bf16*)h, T, F, used);
  return (int)cudaGetLastError();
}
int ss_swiglu_bwd(const void* gu, const void* dh, void* dgu, int T, int F, void* stream) {
  if (F % 8) return -2;
  if (T <= 0) return 0;
  launch_chained(swiglu_bwd_kernel, grid_for((long long)T * (F >> 3), 256, 148 * 16), 256, 0, (cudaStream_t)stream,
                 (const bf16*)gu, (const bf16*)dh, (bf16*)dgu, T, F);
  return (int)cudaGetLastError();
}
int ss_embedding_fwd(const long long* ids, const void* W, void* out, int T, int D, int V,
                     void* stream) {
  if (D % 8) return -2;
  if (T <= 0) return 0;
  embedding_fwd_kernel<<<T < 148 * 8 ? T : 148 * 8, 256, 0, (cudaStream_t)stream>>>(
      ids, (const bf16*)W, (bf16*)out, T, D, V);
  return (int)cudaGetLastError();
}
int ss_embedding_bwd(const long long* ids, const void* g, void* dW, int T, int D, int V,
                     int dw_f32, void* stream) {
  if (D % 2) return -2;
  if (T <= 0) return 0;
  if (dw_f32)
    embedding_bwd_kernel<<<T < 148 * 8 ? T : 148 * 8, 256, 0, (cudaStream_t)stream>>>(
        ids, (const bf16*)g, (float*)dW, T, D, V);
  else
    embedding_bwd_bf16_kernel<<<T < 148 * 8 ? T : 148 * 8, 256, 0, (cudaStream_t)stream>>>(
        ids, (const bf16*)g, (bf16*)dW, T, D, V);
  return (int)cudaGetLastError();
}
int ss_cross_entropy(void* logits, const long long* targets, const float* weights, float* loss_sum,
                     float* lse, int R, int V, long long ld, float grad_scale, int write_grad,
                     void* stream) {
  if (ld % 8) return -2;
  if (R <= 0) return 0;
  cross_entropy_kernel<<<R, CE_THREADS, 0, (cudaStream_t)stream>>>(
      (bf16*)logits, targets, weights, loss_sum, lse, R, V, ld, grad_scale, write_grad, PolicyArgs{}, RowList{});
  return (int)cudaGetLastError();
}
// Token objectives on a logits block: mode 0 cross-entropy, mode 1 clipped policy
// (old_logp and advantage required; ref_logp optional). logp_out, when given,
// receives log p(target) per row.
int ss_token_objective(void* logits, const long long* targets, const float* weights, float* loss_sum,
                       float* logp_out, int R, int V, long long ld, float grad_scale, int write_grad,
                       int mode, const float* old_logp, const float* advantage, float clip,
                       const float* ref_logp, float ref_beta, void* stream) {
  if (ld % 8 || mode < 0 || mode > 1) return -2;
  if (mode == 1 && (!old_logp || !advantage)) return -2;
  if (R <= 0) return 0;
  PolicyArgs pa{mode, old_logp, advantage, ref_logp, clip, ref_beta, logp_out};
  cross_entropy_kernel<<<R, CE_THREADS, 0, (cudaStream_t)stream>>>(
      (bf16*)logits, targets, weights, loss_sum, nullptr, R, V, ld, grad_scale, write_grad, pa, RowList{});
  return (int)cudaGetLastError();
}
// The same on a block of listed rows (see RowList): targets, weights and the policy's inputs are indexed by token.
int ss_token_objective_rows(void* logits, const long long* targets, const float* weights, const int* rows,
                            const int* used, int from, float* loss_sum, int R, int V, long long ld, float grad_scale,
                            int write_grad, int mode, const float* old_logp, const float* advantage, float clip,
                            const float* ref_logp, float ref_beta, void* stream) {
  if (ld % 8 || mode < 0 || mode > 1 || rows == nullptr || used == nullptr) return -2;
  if (mode == 1 && (!old_logp || !advantage)) return -2;
  if (R <= 0) return 0;
  cross_entropy_kernel<<<R, CE_THREADS, 0, (cudaStream_t)stream>>>(
      (bf16*)logits, targets, weights, loss_sum, nullptr, R, V, ld, grad_scale, write_grad,
      PolicyArgs{mode, old_logp, advantage, ref_logp, clip, ref_beta, nullptr}, RowList{rows, used, from});
  return (int)cudaGetLastError();
}
// rows: the tokens whose loss counts (a target in [0, V) and a weight that is not zero), in order, then -1 up to T;
// slot: each token's place in that list or -1; count: their number.
int ss_scored_rows(const long long* targets, const float* weights, int T, int V, int* rows, int* slot, int* count,
                   void* stream) {
  if (T <= 0) return 0;
  scored_rows_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(targets, weights, T, V, rows, slot, count);
  return (int)cudaGetLastError();
}
// out[i] = x[index[i]], or a row of zeros where index[i] < 0.
int ss_take_rows(const void* x, long long ldx, const int* index, void* out, long long ldo, int n, int D, void* stream) {
  if (D % 8 || ldx % 8 || ldo % 8) return -2;
  if (n <= 0) return 0;
  launch_chained(take_rows_kernel, n < 148 * 16 ? n : 148 * 16, 256, 0, (cudaStream_t)stream, (const bf16*)x, ldx, index,
                 (bf16*)out, ldo, n, D);
  return (int)cudaGetLastError();
}
int ss_adamw_sr(void* p, const void* g, void* m, void* v, long long n, int g_f32, float lr,
                float beta1, float beta2, float eps, float weight_decay, int step, float grad_scale,
                unsigned long long seed, unsigned long long offset, int sr_param, int sr_state,
                void* stream) {
  if (n <= 0) return 0;
  if (offset % 8) return -2;
  const AdamWArgs a = adamw_args(lr, beta1, beta2, eps, weight_decay, step, grad_scale, seed, offset);
  auto go = [&](auto kern) {
    kern<<<grid_for((n + 7) >> 3, ADAMW_THREADS, 148 * 2), ADAMW_THREADS, 0, (cudaStream_t)stream>>>((bf16*)p, g, (bf16*)m, (bf16*)v, n, a);
    return (int)cudaGetLastError();
  };
  if (sr_param)
    return sr_state ? (g_f32 ? go(adamw_sr_kernel<true, true, true>) : go(adamw_sr_kernel<true, true, false>))
                    : (g_f32 ? go(adamw_sr_kernel<true, false, true>) : go(adamw_sr_kernel<true, false, false>));
  return sr_state ? (g_f32 ? go(adamw_sr_kernel<false, true, true>) : go(adamw_sr_kernel<false, true, false>))
                  : (g_f32 ? go(adamw_sr_kernel<false, false, true>) : go(adamw_sr_kernel<false, false, false>));
}
// `tensors`: seven values per tensor, {p, g, m, v, elements, offset, gradient is fp32}, in host memory, read
// before the call returns. Distinct tensors of up to ADAMW_MANY_ELEMENTS elements.
int ss_adamw_sr_many(const long long* tensors, int count, float lr, float beta1, float beta2, float eps,
                     float weight_decay, int step, float grad_scale, unsigned long long seed, int sr_param,
                     int sr_state, void* stream) {
  for (int i = 0; i < count; ++i) {
    const long long* t = tensors + 7 * i;
    if (t[4] < 0 || t[4] > ADAMW_MANY_ELEMENTS || t[5] % 8) return -2;
  }
  const AdamWArgs a = adamw_args(lr, beta1, beta2, eps, weight_decay, step, grad_scale, seed, 0);
  for (int done = 0; done < count;) {
    AdamWTable tab;
    tab.count = 0;
    int blocks = 0;
    for (; done < count && tab.count < ADAMW_MANY; ++done) {
      const long long* t = tensors + 7 * done;
      if (t[4] == 0) continue;
      tab.first_block[tab.count] = blocks;
      tab.t[tab.count++] = {reinterpret_cast<bf16*>(t[0]), reinterpret_cast<bf16*>(t[2]), reinterpret_cast<bf16*>(t[3]),
                            reinterpret_cast<const void*>(t[1]), static_cast<unsigned long long>(t[5]),
                            static_cast<int>(t[4]), static_cast<int>(t[6])};
      blocks += static_cast<int>((t[4] + 8 * ADAMW_THREADS - 1) / (8 * ADAMW_THREADS));
    }
    if (tab.count == 0) break;
    auto go = [&](auto kern) {
      kern<<<blocks, ADAMW_THREADS, 0, (cudaStream_t)stream>>>(tab, a);
      return (int)cudaGetLastError();
    };
    const int e = sr_param ? (sr_state ? go(adamw_sr_many_kernel<true, true>) : go(adamw_sr_many_kernel<true, false>))
                           : (sr_state ? go(adamw_sr_many_kernel<false, true>) : go(adamw_sr_many_kernel<false, false>));
    if (e) return e;
  }
  return 0;
}
int ss_adamw_f32(float* p, const float* g, float* m, float* v, long long n, float lr, float beta1,
                 float beta2, float eps, float weight_decay, int step, float grad_scale,
                 void* stream) {
  if (n <= 0) return 0;
  AdamWArgs a;
  a.lr = lr; a.beta1 = beta1; a.beta2 = beta2; a.eps = eps; a.weight_decay = weight_decay;
  a.bias1 = 1.f - powf(beta1, (float)step);
  a.bias2 = 1.f - powf(beta2, (float)step);
  a.grad_scale = grad_scale; a.seed = 0; a.offset = 0;
  adamw_f32_kernel<<<grid_for(n, 256), 256, 0, (cudaStream_t)stream>>>(p, g, m, v, n, a);
  return (int)cudaGetLastError();
}
// partials: caller-provided float[256]; out: float[1].
int ss_sumsq(const void* x, long long n, float* partials, float* out, int accumulate,
             void* stream) {
  const int blocks = grid_for(n, 256 * 16, 256);
  sumsq_partials_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>((const bf16*)x, n, partials);
  sumsq_final_kernel<<<1, 256, 0, (cudaStream_t)stream>>>(partials, blocks, out, accumulate);
  return (int)cudaGetLastError();
}
int ss_cast_f32_bf16(const float* src, void* dst, long long n, float scale, void* stream) {
  if (n <= 0) return 0;
  cast_f32_bf16_kernel<<<grid_for(n, 256, 148 * 16), 256, 0, (cudaStream_t)stream>>>(
      src, (bf16*)dst, n, scale);
  return (int)cudaGetLastError();
}
}  // extern "C"
