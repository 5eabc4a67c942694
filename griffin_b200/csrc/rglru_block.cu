// Small kernels of the recurrent block around the conv and the scan: what its masks mean for every token, and the
// product with its GeLU branch.  Reference behaviour: griffin/griffin.py:309-358 (positions), :464 and :520 (branch).

#include "rglru_internal.h"
#include "rglru_vec.cuh"

namespace rglru {

// ---------------------------------------------------------------- token plan
// One CTA per batch row: positions, flag bytes and the position of the row's last real token from whatever masks the
// call has.  As tensor operations this is about fifteen launches (running count, comparisons, shifts, a maximum, a
// gather), which at the sizes of a prompt are all launch cost: a prompt of 6 x 1200 tokens, padded, took 421 us a block
// call and takes 292 with this kernel (2.5 us) and the one below.
constexpr int PLAN_THREADS = 512;
constexpr int PLAN_TOKENS = 4;      // per thread and tile

// Whether any byte of the mask is zero; the CTA stops looking at the first one it finds.
__device__ __forceinline__ bool any_zero_byte(const uint8_t* m, long long n) {
  const long long lead = min(static_cast<long long>((16 - (reinterpret_cast<uintptr_t>(m) & 15u)) & 15u), n);   // up to a 16-byte boundary
  const uint4* mw = reinterpret_cast<const uint4*>(m + lead);
  const long long nw = (n - lead) / 16;
  constexpr int FLIGHT = 4;
  for (long long w0 = 0; w0 < nw; w0 += PLAN_THREADS * FLIGHT) {
    uint4 v[FLIGHT];
#pragma unroll
    for (int j = 0; j < FLIGHT; ++j) {
      const long long w = w0 + j * PLAN_THREADS + threadIdx.x;
      v[j] = w < nw ? mw[w] : make_uint4(0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u);
    }
    uint32_t least = 0x01010101u;
#pragma unroll
    for (int j = 0; j < FLIGHT; ++j) least = __vminu4(least, __vminu4(__vminu4(v[j].x, v[j].y), __vminu4(v[j].z, v[j].w)));
    if (__syncthreads_or(least != 0x01010101u)) return true;
  }
  int zero = threadIdx.x < lead && m[threadIdx.x] == 0;
  for (long long i = lead + nw * 16 + threadIdx.x; i < n; i += PLAN_THREADS) zero |= m[i] == 0;
  return __syncthreads_or(zero) != 0;
}

// One pass over the mask of the whole batch: block i notes whether its stretch of PLAN_STRETCH bytes, and every
// gridDim.x-th one after it, has a zero.
constexpr long long PLAN_STRETCH = 32768;
constexpr long long PLAN_BLOCKS = 4 * 148;
constexpr long long PLAN_LOOK = 65536;
__global__ void __launch_bounds__(PLAN_THREADS) token_padding_kernel(const uint8_t* mask, long long n, uint8_t* part) {
  bool zero = false;
  for (long long i = blockIdx.x * PLAN_STRETCH; i < n && !zero; i += gridDim.x * PLAN_STRETCH)
    zero = any_zero_byte(mask + i, min(PLAN_STRETCH, n - i));
  if (threadIdx.x == 0) part[blockIdx.x] = zero;
}

__global__ void __launch_bounds__(PLAN_THREADS) token_plan_kernel(const TokenPlanArgs p) {
  __shared__ int s_warp[PLAN_THREADS / 32];
  __shared__ int s_last;
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint8_t* active = p.active ? p.active + static_cast<size_t>(b) * p.T : nullptr;
  const uint8_t* reset = p.reset ? p.reset + static_cast<size_t>(b) * p.T : nullptr;
  const long long* seg = p.seg ? p.seg + static_cast<size_t>(b) * p.T : nullptr;
  uint8_t* flags = p.flags + static_cast<size_t>(b) * p.T;
  const long long prev = p.prev ? p.prev[b] : -1;
  // Padding anywhere in the batch: the first token of a document then wipes the history it would leave behind.
  bool padded = false;
  if (p.positions && p.active) {
    if (p.parts) {
      int zero = 0;
      for (int i = tid; i < p.nparts; i += PLAN_THREADS) zero |= p.parts[i];
      padded = __syncthreads_or(zero) != 0;
    } else {
      padded = any_zero_byte(active, p.T) || (p.B > 1 && any_zero_byte(p.active, static_cast<long long>(p.B) * p.T));
    }
  }
  if (tid == 0) s_last = -1;
  const bool counted = p.positions && p.active && !p.seg;      // positions are the running count of real tokens
  int carry = 0;
  int last_t = -1;
  long long last_pos = prev;
  for (int t0 = 0; t0 < p.T; t0 += PLAN_THREADS * PLAN_TOKENS) {
    const int tb = t0 + tid * PLAN_TOKENS;
    bool act[PLAN_TOKENS];
    int count = 0;
#pragma unroll
    for (int j = 0; j < PLAN_TOKENS; ++j) {
      act[j] = tb + j < p.T && (!active || active[tb + j] != 0);
      count += act[j];
    }
    int before = 0;
    if (counted) {
      int inc = count;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, s);
        if (lane >= s) inc += v;
      }
      __syncthreads();                   // the previous tile's totals have been read
      if (lane == 31) s_warp[warp] = inc;
      __syncthreads();
      int total = 0;
#pragma unroll
      for (int w = 0; w < PLAN_THREADS / 32; ++w) {
        if (w == warp) before = total;
        total += s_warp[w];
      }
      before += carry + inc - count;     // real tokens in front of this thread's
      carry += total;
    }
#pragma unroll
    for (int j = 0; j < PLAN_TOKENS; ++j) {
      const int t = tb + j;
      if (t >= p.T) break;
      before += act[j];
      uint32_t f = act[j] ? 0u : TOK_INACTIVE;
      if (p.positions) {
        const long long pos = seg ? seg[t] : prev + (p.active ? before : t + 1);
        f |= 3u - static_cast<uint32_t>(pos < 0 ? 0 : (pos > 3 ? 3 : pos));
        if (pos == 0) f |= TOK_RESET | (act[j] && padded ? TOK_ZERO_HISTORY : 0u);
        if (act[j]) { last_t = t; last_pos = pos; }
      } else if (reset && reset[t]) {
        f |= TOK_RESET;
      }
      flags[t] = static_cast<uint8_t>(f);
    }
  }
  if (!p.last) return;
  __syncthreads();
  atomicMax(&s_last, last_t);
  __syncthreads();
  if (last_t == s_last && (last_t >= 0 || tid == 0)) p.last[b] = last_pos;
}

// A mask of up to 64 KB is looked through by every row's CTA, which costs less than the launch of token_padding_kernel;
// beyond, that is the batch's rows times the mask (an all-true 1024 x 2048 mask: 254 us, 13 in two launches; 256 x 2048: 25 and 7; 64 x 2048: 6.5 and 5.9).
int token_plan_parts(int B, int T) {
  const long long n = static_cast<long long>(B) * T;
  if (B == 1 || n <= PLAN_LOOK) return 0;
  const long long want = (n + PLAN_STRETCH - 1) / PLAN_STRETCH;
  return static_cast<int>(want < PLAN_BLOCKS ? want : PLAN_BLOCKS);
}
cudaError_t launch_token_plan(const TokenPlanArgs& a, cudaStream_t s) {
  if (a.parts) token_padding_kernel<<<a.nparts, PLAN_THREADS, 0, s>>>(a.active, static_cast<long long>(a.B) * a.T, a.parts);
  token_plan_kernel<<<a.B, PLAN_THREADS, 0, s>>>(a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- product with the GeLU branch
// out = y * gelu_tanh(g) and its gradient, one streaming pass each way (3 and 5 tensors) instead of two and three
// passes (5 and 11 tensors).  fp32 inside, so the result is rounded once.  Bound by HBM.  7200 x 1024 bf16, forward: 6.6 us
// against 8.4 + 6.8.
template <typename IO, int VEC, bool BWD>
__global__ void __launch_bounds__(256) gelu_mul_kernel(const GeluMulArgs p) {
  using V = Vec<IO, VEC>;
  const long long i = (static_cast<long long>(blockIdx.x) * 256 + threadIdx.x) * VEC;
  if (i >= p.n) return;
  constexpr int N = VEC == 1 ? 2 : VEC;      // the helpers work on pairs
  float y[N], g[N], d[N], a[N], c[N];
  if constexpr (VEC == 1) y[1] = g[1] = d[1] = 0.0f;
  V::load(static_cast<const IO*>(p.y) + i, reinterpret_cast<float (&)[VEC]>(y));
  V::load(static_cast<const IO*>(p.g) + i, reinterpret_cast<float (&)[VEC]>(g));
  if constexpr (BWD) V::load(static_cast<const IO*>(p.dout) + i, reinterpret_cast<float (&)[VEC]>(d));
#pragma unroll
  for (int v = 0; v < N; v += 2) {
    const float2 gv = make_float2(g[v], g[v + 1]), yv = make_float2(y[v], y[v + 1]);
    const float2 s = gelu_sigmoid2<false>(gv);
    const float2 gelu = mul2(gv, s);
    if constexpr (BWD) {
      const float2 dv = make_float2(d[v], d[v + 1]);
      const float2 dy = mul2(dv, gelu), dg = mul2(mul2(dv, yv), gelu_slope2(gv, s));
      a[v] = dy.x; a[v + 1] = dy.y; c[v] = dg.x; c[v + 1] = dg.y;
    } else {
      const float2 o = mul2(yv, gelu);
      a[v] = o.x; a[v + 1] = o.y;
    }
  }
  V::store(static_cast<IO*>(p.out) + i, reinterpret_cast<float (&)[VEC]>(a));
  if constexpr (BWD) V::store(static_cast<IO*>(p.dg) + i, reinterpret_cast<float (&)[VEC]>(c));
}

// ---------------------------------------------------------------- padding rows of the output
// The block's output is zero at padding tokens (griffin/griffin.py:488-510).  In place, a warp per row, only the padding rows
// are written and only the mask is read; a select over the whole tensor takes 13.5 us for 6 x 1200 rows of 768 bf16, this 3.0.
__global__ void __launch_bounds__(256) zero_rows_kernel(uint4* __restrict__ x, const uint8_t* __restrict__ keep, long long rows, int pieces) {
  const long long row = static_cast<long long>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (row >= rows || keep[row]) return;
  for (int i = threadIdx.x & 31; i < pieces; i += 32) x[row * pieces + i] = make_uint4(0u, 0u, 0u, 0u);
}
cudaError_t launch_zero_rows(void* x, const uint8_t* keep, long long rows, int pieces, cudaStream_t s) {
  zero_rows_kernel<<<static_cast<unsigned>((rows + 7) / 8), 256, 0, s>>>(static_cast<uint4*>(x), keep, rows, pieces);
  return cudaGetLastError();
}

template <typename IO, bool BWD>
static cudaError_t gelu_mul_t(const GeluMulArgs& a, bool vector_ok, cudaStream_t s) {
  constexpr int V = vec_width<IO>();
  const long long threads = vector_ok ? a.n / V : a.n;
  const unsigned blocks = static_cast<unsigned>((threads + 255) / 256);
  if (vector_ok) gelu_mul_kernel<IO, V, BWD><<<blocks, 256, 0, s>>>(a);
  else gelu_mul_kernel<IO, 1, BWD><<<blocks, 256, 0, s>>>(a);
  return cudaGetLastError();
}
cudaError_t launch_gelu_mul(bool bf16, const GeluMulArgs& a, bool vector_ok, cudaStream_t s) {
  if (a.dout) return bf16 ? gelu_mul_t<__nv_bfloat16, true>(a, vector_ok, s) : gelu_mul_t<float, true>(a, vector_ok, s);
  return bf16 ? gelu_mul_t<__nv_bfloat16, false>(a, vector_ok, s) : gelu_mul_t<float, false>(a, vector_ok, s);
}

}  // namespace rglru
