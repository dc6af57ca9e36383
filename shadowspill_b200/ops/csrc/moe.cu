// Mixture-of-experts routing and token movement for sm_100a.
//
//   ss_moe_route      per token: top-k over the router logits, softmax over the
//                     selected logits (renormalised) or over all experts, and a
//                     per-expert histogram -- one warp per token, no sorting pass
//   ss_moe_layout     expert segments padded to 128 rows (so a GEMM tile never
//                     straddles two experts), the expert of every 128-row tile,
//                     and a destination row for every (token, slot) assignment
//   ss_moe_gather     token rows -> expert-sorted rows, padding rows zero (optionally
//                     scaled by the routing weights)
//   ss_moe_act_bwd    backward of the weighted expert activation on sorted rows
//   ss_moe_route_bwd  gradient of the routing weights -> gradient of the logits
//   ss_moe_combine    expert-sorted rows -> token rows: out[t] (+)= sum_j w[t,j] *
//                     y[dest[t,j]], deterministic (a gather, no atomics); can also
//                     emit <dout[t], y[dest[t,j]]> for the router-weight gradient
//
// The same kernels serve expert parallelism: `dest` rows may live in a peer GPU's
// staging buffer (plain P2P stores / loads through the symmetric pool), which is
// how dispatch and combine cross NVLink without a separate all-to-all.
//
// Semantics: the reference's routed-expert layer (top-k then softmax for Qwen,
// softmax then top-k for OLMoE; packages/workloads/src/shadowspill_workloads/
// models/shared/qwen_moe/experts.py:31-72, router_statistics.py:9-32).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

namespace ss {

constexpr int MOE_MAX_E = 512;
constexpr int MOE_MAX_K = 32;

__device__ __forceinline__ float wmax(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float wsum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One warp per token, PER experts per lane in registers, the j-th pick kept by lane j. The histogram is
// summed per block in shared memory: one atomic per token and pick on a few dozen global counters was
// most of the kernel (8,192 tokens, top 8 of 64: 51 -> 14 us).
constexpr int ROUTE_THREADS = 256;
template <int PER>
__global__ void __launch_bounds__(ROUTE_THREADS)
moe_route_kernel(const float* __restrict__ logits, long long ld, int T, int E, int k, int renormalize,
                 int* __restrict__ ids, float* __restrict__ weights, int* __restrict__ counts) {
  __shared__ int hist[PER * 32];
  for (int e = threadIdx.x; e < PER * 32; e += ROUTE_THREADS) hist[e] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warps = gridDim.x * (ROUTE_THREADS / 32);
  for (int t = (blockIdx.x * ROUTE_THREADS + threadIdx.x) >> 5; t < T; t += warps) {
    const float* row = logits + static_cast<long long>(t) * ld;
    float v[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = lane + i * 32;
      v[i] = e < E ? row[e] : -INFINITY;
    }
    float lmax = -INFINITY;
#pragma unroll
    for (int i = 0; i < PER; ++i) lmax = fmaxf(lmax, v[i]);
    const float gmax = wmax(lmax);
    float denom = 0.f;
    if (!renormalize) {
#pragma unroll
      for (int i = 0; i < PER; ++i) denom += (v[i] == -INFINITY) ? 0.f : __expf(v[i] - gmax);
      denom = wsum(denom);
    }
    float my_v = -INFINITY;
    int my_e = 0;
    unsigned taken = 0;                        // this lane's experts that have been picked, by i
    for (int j = 0; j < k; ++j) {
      float best = -INFINITY;
      int bi = 0x7fffffff;
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int e = lane + i * 32;
        if (v[i] > best || (v[i] == best && e < bi && v[i] != -INFINITY)) { best = v[i]; bi = e; }
      }
      // warp arg-max; ties go to the lower expert index (matches a stable top-k)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
      }
      if (bi >= E) {                           // fewer than k comparable scores: the first experts not yet picked,
        int left = 0x7fffffff;                 // each once, as the gradient of a pick is stored by its own lane
#pragma unroll
        for (int i = PER - 1; i >= 0; --i)
          if (lane + i * 32 < E && !((taken >> i) & 1)) left = lane + i * 32;
        bi = __reduce_min_sync(0xffffffffu, left);
      }
      if (lane == j) { my_v = best; my_e = bi; }
      if ((bi & 31) == lane) {                 // remove the winner
        taken |= 1u << (bi >> 5);
#pragma unroll
        for (int i = 0; i < PER; ++i)
          if (i == (bi >> 5)) v[i] = -INFINITY;
      }
    }
    const float top = renormalize ? __shfl_sync(0xffffffffu, my_v, 0) : gmax;
    const float x = lane < k ? __expf(my_v - top) : 0.f;
    const float total = renormalize ? wsum(x) : denom;
    if (lane < k) {
      ids[static_cast<long long>(t) * k + lane] = my_e;
      weights[static_cast<long long>(t) * k + lane] = x / total;
      atomicAdd(&hist[my_e], 1);
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += ROUTE_THREADS)
    if (hist[e]) atomicAdd(counts + e, hist[e]);
}

// Gradient of the routing weights with respect to the scores; one warp per token.
//   renormalised   w = softmax over the picks:  dl[pick j] = w_j (dw_j - sum_i w_i dw_i), 0 elsewhere
//   otherwise      w_j = p[pick j], p = softmax over all: dl_e = p_e ([e picked] dw_e - sum_i w_i dw_i)
__global__ void __launch_bounds__(ROUTE_THREADS)
moe_route_bwd_kernel(const float* __restrict__ logits, long long ld, const int* __restrict__ ids,
                     const float* __restrict__ weights, const float* __restrict__ dweights,
                     float* __restrict__ dlogits, int T, int E, int k, int renormalize) {
  const int lane = threadIdx.x & 31;
  const int t = (blockIdx.x * ROUTE_THREADS + threadIdx.x) >> 5;
  if (t >= T) return;
  const long long a = static_cast<long long>(t) * k + lane;
  const float w = lane < k ? weights[a] : 0.f, dw = lane < k ? dweights[a] : 0.f;
  const int id = lane < k ? ids[a] : 0;
  const float inner = wsum(w * dw);
  float* out = dlogits + static_cast<long long>(t) * E;
  if (renormalize) {
    for (int e = lane; e < E; e += 32) out[e] = 0.f;
  } else {
    const float* row = logits + static_cast<long long>(t) * ld;
    float m = -INFINITY, s = 0.f;
    for (int e = lane; e < E; e += 32) m = fmaxf(m, row[e]);
    m = wmax(m);
    for (int e = lane; e < E; e += 32) s += expf(row[e] - m);
    s = wsum(s);
    for (int e = lane; e < E; e += 32) out[e] = -(expf(row[e] - m) / s) * inner;
  }
  __syncwarp();                                // the picks overwrite what another lane wrote above
  if (lane < k) out[id] = w * (dw - inner);
}

// One block. offsets[E+1] (padded to 128), tile_expert[max_tiles], cursor[E] = first row of each expert.
__global__ void __launch_bounds__(MOE_MAX_E)
moe_layout_kernel(const int* __restrict__ counts, int E, int* __restrict__ offsets,
                  int* __restrict__ tile_expert, int max_tiles, int* __restrict__ cursor) {
  __shared__ int s_off[MOE_MAX_E + 1];
  __shared__ int s_warp[MOE_MAX_E / 32];
  const int e = threadIdx.x, lane = e & 31, warp = e >> 5;
  int incl = e < E ? (counts[e] + 127) / 128 * 128 : 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  for (int w = 0; w < warp; ++w) incl += s_warp[w];
  if (e < E) s_off[e + 1] = incl;
  if (e == 0) s_off[0] = 0;
  __syncthreads();
  if (e < E) { offsets[e + 1] = s_off[e + 1]; cursor[e] = s_off[e]; }
  if (e == 0) offsets[0] = 0;
  for (int t = threadIdx.x; t < max_tiles; t += blockDim.x) {
    const int row = t * 128;
    int found = -1;
    if (row < s_off[E]) {
      int lo = 0, hi = E;            // largest e with s_off[e] <= row
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (s_off[mid] <= row) lo = mid; else hi = mid;
      }
      found = lo;
    }
    tile_expert[t] = found;
  }
}

// dest[i] = the sorted row of assignment i, src[row] = i. A block counts its assignments per expert in
// shared memory and takes its share of every expert's rows with one atomic each (65,536 assignments to
// 64 experts: 19.5 -> 3.2 us against an atomic per assignment).
constexpr int ASSIGN_THREADS = 256;
constexpr int ASSIGN_PER_THREAD = 4;
__global__ void __launch_bounds__(ASSIGN_THREADS)
moe_assign_kernel(const int* __restrict__ ids, long long n, int E, int* __restrict__ cursor,
                  int* __restrict__ dest, int* __restrict__ src) {
  __shared__ int count[MOE_MAX_E];
  for (int e = threadIdx.x; e < E; e += ASSIGN_THREADS) count[e] = 0;
  __syncthreads();
  const long long i0 = blockIdx.x * static_cast<long long>(ASSIGN_THREADS * ASSIGN_PER_THREAD) + threadIdx.x;
  int id[ASSIGN_PER_THREAD], at[ASSIGN_PER_THREAD];
#pragma unroll
  for (int u = 0; u < ASSIGN_PER_THREAD; ++u) {
    const long long i = i0 + u * ASSIGN_THREADS;
    id[u] = i < n ? ids[i] : -1;
  }
#pragma unroll
  for (int u = 0; u < ASSIGN_PER_THREAD; ++u)
    if (id[u] >= 0) at[u] = atomicAdd(&count[id[u]], 1);
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += ASSIGN_THREADS)
    if (count[e]) count[e] = atomicAdd(cursor + e, count[e]);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < ASSIGN_PER_THREAD; ++u) {
    if (id[u] < 0) continue;
    const long long i = i0 + u * ASSIGN_THREADS;
    const int row = count[id[u]] + at[u];
    dest[i] = row;
    src[row] = static_cast<int>(i);
  }
}

// sorted[r, :] = scale * x[src[r] / k, :]   (scale = weights[src[r]] or 1), zero where src[r] < 0, for the
// rows below *used. Row-driven, so the padding of the segments is written here and nothing else has to
// clear the buffer.
__global__ void moe_gather_kernel(const __nv_bfloat16* __restrict__ x, long long ldx,
                                  const int* __restrict__ src, const int* __restrict__ used,
                                  const float* __restrict__ weights, __nv_bfloat16* __restrict__ sorted,
                                  long long lds, int max_rows, int k, int D) {
  const int nv = D >> 3, rows = min(*used, max_rows);
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const int a = src[r];
    uint4* dst = reinterpret_cast<uint4*>(sorted + static_cast<long long>(r) * lds);
    if (a < 0) {
      for (int c = threadIdx.x; c < nv; c += blockDim.x) dst[c] = make_uint4(0, 0, 0, 0);
      continue;
    }
    const uint4* row = reinterpret_cast<const uint4*>(x + static_cast<long long>(a / k) * ldx);
    if (weights == nullptr) {
#pragma unroll 2
      for (int c = threadIdx.x; c < nv; c += blockDim.x) dst[c] = row[c];
    } else {
      const float w = weights[a];
#pragma unroll 2
      for (int c = threadIdx.x; c < nv; c += blockDim.x) {
        uint4 u = row[c];
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float2 f = __bfloat1622float2(h[e]);
          f.x *= w; f.y *= w;
          h[e] = __float22bfloat162_rn(f);
        }
        dst[c] = u;
      }
    }
  }
}

// Backward of the weighted expert activation, one warp per sorted row below *used. With h = silu(g) * u,
// d = the gradient of h's row before the routing weight w is applied (dout w2) and a = src[row]:
//   dots[a] = <d, h>   dgu = gradient of (g, u) for w * d   hw = w * h
// so neither the expert outputs nor w * dout are needed: <dout, h w2^T> = <dout w2, h>, and the bank's
// gradient takes the weight on its other operand, dout^T (w h) = (w dout)^T h. That saves one bank product,
// a pass over the expert outputs and one over the activations: backward kernels of olmoe-7b-a1b's experts on
// 8,192 tokens 2.4 -> 1.8 ms. Padding rows (a < 0) hold
// zeros in gu and d and get zeros.
__global__ void __launch_bounds__(256)
moe_act_bwd_kernel(const __nv_bfloat16* __restrict__ gu, const __nv_bfloat16* __restrict__ d,
                   const int* __restrict__ src, const int* __restrict__ used, const float* __restrict__ weights,
                   __nv_bfloat16* __restrict__ dgu, __nv_bfloat16* __restrict__ hw, float* __restrict__ dots, int max_rows,
                   int F) {
  const int nv = F >> 3, rows = min(*used, max_rows), lane = threadIdx.x & 31;
  const int warps = gridDim.x * 8;
  for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += warps) {
    const int a = src[r];
    const float w = a >= 0 ? weights[a] : 0.f;
    const uint4* gr = reinterpret_cast<const uint4*>(gu + static_cast<long long>(r) * 2 * F);
    const uint4* dr = reinterpret_cast<const uint4*>(d + static_cast<long long>(r) * F);
    uint4* og = reinterpret_cast<uint4*>(dgu + static_cast<long long>(r) * 2 * F);
    uint4* oh = reinterpret_cast<uint4*>(hw + static_cast<long long>(r) * F);
    float dot = 0.f;
#pragma unroll 2
    for (int c = lane; c < nv; c += 32) {
      const uint4 gq = gr[c], uq = gr[nv + c], dq = dr[c];
      const __nv_bfloat162* g2 = reinterpret_cast<const __nv_bfloat162*>(&gq);
      const __nv_bfloat162* u2 = reinterpret_cast<const __nv_bfloat162*>(&uq);
      const __nv_bfloat162* d2 = reinterpret_cast<const __nv_bfloat162*>(&dq);
      uint4 qg, qu, qh;
      __nv_bfloat162* xg = reinterpret_cast<__nv_bfloat162*>(&qg);
      __nv_bfloat162* xu = reinterpret_cast<__nv_bfloat162*>(&qu);
      __nv_bfloat162* xh = reinterpret_cast<__nv_bfloat162*>(&qh);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 g = __bfloat1622float2(g2[e]), u = __bfloat1622float2(u2[e]), q = __bfloat1622float2(d2[e]);
        const float gv[2] = {g.x, g.y}, uv[2] = {u.x, u.y}, dv[2] = {q.x, q.y};
        float ag[2], au[2], ah[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const float sig = __fdividef(1.f, 1.f + __expf(-gv[x]));
          const float s = gv[x] * sig;
          // the forward pass rounds silu(g) and h to bf16
          const float h = __bfloat162float(__float2bfloat16_rn(__bfloat162float(__float2bfloat16_rn(s)) * uv[x]));
          dot += dv[x] * h;
          const float wd = w * dv[x];
          au[x] = wd * s;
          ag[x] = wd * uv[x] * (sig * (1.f + gv[x] * (1.f - sig)));
          ah[x] = w * h;
        }
        xg[e] = __floats2bfloat162_rn(ag[0], ag[1]);
        xu[e] = __floats2bfloat162_rn(au[0], au[1]);
        xh[e] = __floats2bfloat162_rn(ah[0], ah[1]);
      }
      og[c] = qg;
      og[nv + c] = qu;
      oh[c] = qh;
    }
    dot = wsum(dot);
    if (lane == 0 && a >= 0) dots[a] = dot;
  }
}

// out[t,:] (+)= sum_j w[t,j] * y[dest[t,j], :];  optionally dots[t,j] = <g[t,:], y[dest[t,j],:]>
__global__ void moe_combine_kernel(const __nv_bfloat16* __restrict__ y, long long ldy,
                                   const int* __restrict__ dest, const float* __restrict__ weights,
                                   __nv_bfloat16* __restrict__ out, long long ldo, int T, int k, int D,
                                   int accumulate, const __nv_bfloat16* __restrict__ g, long long ldg,
                                   float* __restrict__ dots) {
  const int nv = D >> 3;
  for (int t = blockIdx.x; t < T; t += gridDim.x) {
    if (out != nullptr) {
      for (int c = threadIdx.x; c < nv; c += blockDim.x) {
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (accumulate) {
          const uint4 u = reinterpret_cast<const uint4*>(out + static_cast<long long>(t) * ldo)[c];
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
          for (int e = 0; e < 4; ++e) { const float2 f = __bfloat1622float2(h[e]); acc[2 * e] = f.x; acc[2 * e + 1] = f.y; }
        }
        // eight rows' loads are in flight before the first is used (8,192 x 8 rows of 2048: 73 -> 57 us)
        for (int j0 = 0; j0 < k; j0 += 8) {
          uint4 u[8];
          float w[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (j0 + j >= k) break;
            const long long a = static_cast<long long>(t) * k + j0 + j;
            w[j] = weights ? weights[a] : 1.f;
            u[j] = reinterpret_cast<const uint4*>(y + static_cast<long long>(dest[a]) * ldy)[c];
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            if (j0 + j >= k) break;
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u[j]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 f = __bfloat1622float2(h[e]);
              acc[2 * e] += w[j] * f.x; acc[2 * e + 1] += w[j] * f.y;
            }
          }
        }
        uint4 o;
        __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int e = 0; e < 4; ++e) oh[e] = __floats2bfloat162_rn(acc[2 * e], acc[2 * e + 1]);
        reinterpret_cast<uint4*>(out + static_cast<long long>(t) * ldo)[c] = o;
      }
    }
    if (dots != nullptr) {
      // one warp per slot: 16-byte loads, a shuffle reduction, no block barrier
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
      const uint4* gv = reinterpret_cast<const uint4*>(g + static_cast<long long>(t) * ldg);
      for (int j = warp; j < k; j += nwarps) {
        const long long a = static_cast<long long>(t) * k + j;
        const uint4* yv = reinterpret_cast<const uint4*>(y + static_cast<long long>(dest[a]) * ldy);
        float part = 0.f;
        for (int c = lane; c < nv; c += 32) {
          const uint4 u = yv[c], w = gv[c];
          const __nv_bfloat162* uh = reinterpret_cast<const __nv_bfloat162*>(&u);
          const __nv_bfloat162* wh = reinterpret_cast<const __nv_bfloat162*>(&w);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 fu = __bfloat1622float2(uh[e]), fw = __bfloat1622float2(wh[e]);
            part += fu.x * fw.x + fu.y * fw.y;
          }
        }
        part = wsum(part);
        if (lane == 0) dots[a] = part;
      }
    }
  }
}

}  // namespace ss

extern "C" {
using namespace ss;

int ss_moe_route(const float* logits, long long ld, int T, int E, int k, int renormalize, int* ids,
                 float* weights, int* counts, void* stream) {
  if (T > 0 && (E > MOE_MAX_E || k > MOE_MAX_K || k > E)) return -2;
  cudaStream_t s = (cudaStream_t)stream;
  cudaMemsetAsync(counts, 0, sizeof(int) * E, s);
  if (T <= 0) return (int)cudaGetLastError();
  const int blocks = (T + 7) / 8, grid = blocks < 148 * 4 ? blocks : 148 * 4;
  auto go = [&](auto kern) {
    kern<<<grid, ROUTE_THREADS, 0, s>>>(logits, ld, T, E, k, renormalize, ids, weights, counts);
    return (int)cudaGetLastError();
  };
  if (E <= 64) return go(moe_route_kernel<2>);
  if (E <= 128) return go(moe_route_kernel<4>);
  if (E <= 256) return go(moe_route_kernel<8>);
  return go(moe_route_kernel<MOE_MAX_E / 32>);
}

// dlogits fp32 [T, E] contiguous, every element written.
int ss_moe_route_bwd(const float* logits, long long ld, const int* ids, const float* weights, const float* dweights,
                     float* dlogits, int T, int E, int k, int renormalize, void* stream) {
  if (E > MOE_MAX_E || k > MOE_MAX_K || k > E) return -2;
  if (T <= 0) return 0;
  moe_route_bwd_kernel<<<(T + 7) / 8, ROUTE_THREADS, 0, (cudaStream_t)stream>>>(logits, ld, ids, weights, dweights,
                                                                                dlogits, T, E, k, renormalize);
  return (int)cudaGetLastError();
}

// src: int32 [rows], the inverse of dest (-1 for padding rows).
int ss_moe_layout(const int* counts, const int* ids, int T, int E, int k, int* offsets,
                  int* tile_expert, int max_tiles, int* cursor, int* dest, int* src, int rows, void* stream) {
  if (E > MOE_MAX_E) return -2;
  cudaStream_t s = (cudaStream_t)stream;
  cudaMemsetAsync(src, 0xff, sizeof(int) * (size_t)rows, s);
  moe_layout_kernel<<<1, MOE_MAX_E, 0, s>>>(counts, E, offsets, tile_expert, max_tiles, cursor);
  const long long n = (long long)T * k, per = ASSIGN_THREADS * ASSIGN_PER_THREAD;
  if (n > 0)
    moe_assign_kernel<<<(int)((n + per - 1) / per), ASSIGN_THREADS, 0, s>>>(ids, n, E, cursor, dest, src);
  return (int)cudaGetLastError();
}

// `used`: device pointer to the number of rows in use (the last of the layout's offsets); `rows` bounds it.
int ss_moe_gather(const void* x, long long ldx, const int* src, const int* used, const float* weights, void* sorted,
                  long long lds, int rows, int k, int D, void* stream) {
  if (D % 8 || ldx % 8 || lds % 8) return -2;
  if (rows <= 0 || k <= 0) return 0;
  moe_gather_kernel<<<rows > 148 * 16 ? 148 * 16 : rows, 128, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)x, ldx, src, used, weights, (__nv_bfloat16*)sorted, lds, rows, k, D);
  return (int)cudaGetLastError();
}

int ss_moe_act_bwd(const void* gu, const void* d, const int* src, const int* used, const float* weights, void* dgu,
                   void* hw, float* dots, int rows, int F, void* stream) {
  if (F % 8) return -2;
  if (rows <= 0) return 0;
  const int blocks = (rows + 7) / 8;
  moe_act_bwd_kernel<<<blocks < 148 * 8 ? blocks : 148 * 8, 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)gu, (const __nv_bfloat16*)d, src, used, weights, (__nv_bfloat16*)dgu, (__nv_bfloat16*)hw,
      dots, rows, F);
  return (int)cudaGetLastError();
}

int ss_moe_combine(const void* y, long long ldy, const int* dest, const float* weights, void* out,
                   long long ldo, int T, int k, int D, int accumulate, const void* g, long long ldg,
                   float* dots, void* stream) {
  if (D % 8 || ldy % 8 || (out && ldo % 8) || (dots && ldg % 8)) return -2;
  if (T <= 0) return 0;
  moe_combine_kernel<<<T > 148 * 8 ? 148 * 8 : T, 256, 0, (cudaStream_t)stream>>>(
      (const __nv_bfloat16*)y, ldy, dest, weights, (__nv_bfloat16*)out, ldo, T, k, D, accumulate,
      (const __nv_bfloat16*)g, ldg, dots);
  return (int)cudaGetLastError();
}
}  // extern "C"
