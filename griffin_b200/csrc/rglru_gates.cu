// The gate parameters on their way into and out of the interleaved gate layout.
//
// Both gate projections of a head run as one GEMM whose output columns alternate between the two gates in groups of
// `unit` channels, [r (unit) | i (unit)] [r | i] ..., with `unit` the largest power of two up to 64 that divides the head
// width: column (d / unit) * 2 unit + d % unit of the [B, T, 2 D] gate tensor is channel d's recurrence gate, `unit`
// columns further its input gate, whatever head d is in.  A 64-channel scan tile may therefore straddle heads, and heads of any
// width go through one GEMM without a re-layout.  bf16, B = 8, T = 8192, D = 5632, 16 heads of 352 channels, forward and
// backward of the layer: 9.0 ms with the projections as modules (4.7 of it re-layouts), 3.4 ms this way.  Narrow groups
// cost the scan little: B = 8, T = 4096, D = 5632 bf16 forward / backward 306 / 530 us in groups of 8, 263 / 562 of 16,
// 271 / 564 of 32, 256 / 537 of 64.
//
//   gate_pack_kernel     the two [G, bw, bw] weights as the GEMM's one [G, 2 bw, bw] operand in the activation type, and
//                        the biases and Lambda in fp32: one launch instead of two concatenations and three casts;
//   gate_dw_kernel       fp32 weight gradient, split over the tokens;
//   gate_unpack_kernel   the gradients of all five parameters in their own types and shapes: one launch instead of four
//                        slices with a cast or a copy each and the cast of Lambda's.
//
// Reference: BlockDiagonalLinear, griffin/griffin.py:129-154, called twice at :237-238.

#include "rglru_internal.h"
#include "rglru_vec.cuh"

namespace rglru {

__device__ __forceinline__ float load_as(const void* p, size_t i, bool f32) {
  return f32 ? static_cast<const float*>(p)[i] : __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
}
__device__ __forceinline__ void store_as(void* p, size_t i, bool f32, float v) {
  if (f32) static_cast<float*>(p)[i] = v;
  else static_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(v);
}

// Row R of a head's stacked operand: unit group R / (2 unit), gate (R / unit) % 2, channel within the head.
struct GateRow {
  int gate, channel;
};
__device__ __forceinline__ GateRow gate_row(int R, int unit) {
  return {(R / unit) & 1, (R / (2 * unit)) * unit + R % unit};
}

constexpr int GATE_WARPS = 8;

// A warp per row of the operand: bw elements in groups of four (bw is a multiple of 4).
template <typename P, typename IO>
__global__ void __launch_bounds__(32 * GATE_WARPS) gate_pack_kernel(const GatePackArgs p) {
  const int row = blockIdx.x * GATE_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= 2 * p.D) return;
  const int head = row / (2 * p.bw);
  const GateRow r = gate_row(row % (2 * p.bw), p.unit);
  const int d = head * p.bw + r.channel;
  const P* src = static_cast<const P*>(r.gate ? p.w_i : p.w_r) + static_cast<size_t>(d) * p.bw;
  IO* dst = static_cast<IO*>(p.wcat) + static_cast<size_t>(row) * p.bw;
  for (int k = lane * 4; k < p.bw; k += 128) {
    float v[4];
    Pack<P>::unpack(Pack<P>::load(src + k), v);
    Pack<IO>::store(dst + k, v);
  }
  if (lane == 0) {
    p.params[row] = load_as(r.gate ? p.b_i : p.b_r, d, p.f32_bias);
    if (r.gate == 0) p.params[2 * p.D + d] = load_as(p.lambda, d, p.f32_lambda);
  }
}

// The way back.  `dw` is one [G, 2 bw, bw] gradient, or `splits` fp32 ones that are added in index order.
template <typename S, typename P>
__global__ void __launch_bounds__(32 * GATE_WARPS) gate_unpack_kernel(const GateUnpackArgs p) {
  const int row = blockIdx.x * GATE_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= 2 * p.D) return;
  const int head = row / (2 * p.bw);
  const GateRow r = gate_row(row % (2 * p.bw), p.unit);
  const int d = head * p.bw + r.channel;
  const S* src = static_cast<const S*>(p.dw) + static_cast<size_t>(row) * p.bw;
  const size_t split_stride = static_cast<size_t>(2) * p.D * p.bw;
  P* dst = static_cast<P*>(r.gate ? p.dw_i : p.dw_r) + static_cast<size_t>(d) * p.bw;
  for (int k = lane * 4; k < p.bw; k += 128) {
    float v[4];
    Pack<S>::unpack(Pack<S>::load(src + k), v);
    for (int s0 = 1; s0 < p.splits; s0 += 8) {            // eight loads in flight
      float t[8][4];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (s0 + j < p.splits) Pack<S>::unpack(Pack<S>::load(src + (s0 + j) * split_stride + k), t[j]);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (s0 + j < p.splits) { v[0] += t[j][0]; v[1] += t[j][1]; v[2] += t[j][2]; v[3] += t[j][3]; }
    }
    Pack<P>::store(dst + k, v);
  }
  if (lane == 0) {
    store_as(r.gate ? p.db_i : p.db_r, d, p.f32_bias, p.dbias[row]);
    if (r.gate == 0) store_as(p.dlambda, d, p.f32_lambda, p.dlam[d]);
  }
}

// ---------------------------------------------------------------- fp32 weight gradient
// dw[g][o][i] = sum over tokens n of du[n, 2 bw g + o] x[n, bw g + i].  The output is small (2 bw x bw per head) and the
// contraction long, so a CTA takes a 64 x TI tile of one head and one stretch of the tokens, 32 of them per stage, and
// leaves a partial sum for gate_unpack_kernel.  A thread owns 4 x 4 outputs; both operands lie with the contracted axis
// outermost, so it reads two float4 per token.
// A library's batched GEMM walks all tokens with the few CTAs the output has: at 7685 tokens and 16 heads of 48 channels
// two calls took 359 us, this kernel takes 51.
constexpr int DW_TO = 64, DW_TK = 32;

__device__ __forceinline__ void dw_copy16(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

template <int TI>
__global__ void __launch_bounds__(16 * (TI / 4)) gate_dw_kernel(const GateDwArgs p) {
  constexpr int NT = 16 * (TI / 4);
  __shared__ __align__(16) float sa[2][DW_TK][DW_TO];
  __shared__ __align__(16) float sb[2][DW_TK][TI];
  const int tid = threadIdx.x, to = (tid / (TI / 4)) * 4, ti = (tid % (TI / 4)) * 4;
  const int tiles_i = (p.bw + TI - 1) / TI;
  const int o0 = (blockIdx.x / tiles_i) * DW_TO, i0 = (blockIdx.x % tiles_i) * TI, head = blockIdx.y;
  const long long n0 = blockIdx.z * p.per_split, n1 = n0 + p.per_split < p.rows ? n0 + p.per_split : p.rows;
  const float* du = p.du + static_cast<size_t>(head) * 2 * p.bw;
  const float* x = p.x + static_cast<size_t>(head) * p.bw;

  auto load = [&](int st, long long n) {
    for (int i = tid; i < DW_TK * DW_TO / 4; i += NT) {
      const int k = i / (DW_TO / 4), c = (i % (DW_TO / 4)) * 4;
      const bool ok = n + k < n1 && o0 + c < 2 * p.bw;
      dw_copy16(&sa[st][k][c], ok ? du + (n + k) * 2 * p.D + o0 + c : p.du, ok);
    }
    for (int i = tid; i < DW_TK * TI / 4; i += NT) {
      const int k = i / (TI / 4), c = (i % (TI / 4)) * 4;
      const bool ok = n + k < n1 && i0 + c < p.bw;
      dw_copy16(&sb[st][k][c], ok ? x + (n + k) * p.D + i0 + c : p.x, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.0f;
  load(0, n0);
  int st = 0;
  for (long long n = n0; n < n1; n += DW_TK, st ^= 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                       // this stage is there for all, and all are done with the other one
    if (n + DW_TK < n1) load(st ^ 1, n + DW_TK);
#pragma unroll 8
    for (int k = 0; k < DW_TK; ++k) {
      const float4 a4 = *reinterpret_cast<const float4*>(&sa[st][k][to]);
      const float4 b4 = *reinterpret_cast<const float4*>(&sb[st][k][ti]);
      const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = fmaf(a[u], b[v], acc[u][v]);
    }
  }
  if (i0 + ti >= p.bw) return;             // bw is a multiple of 4
  float* out = p.part + (static_cast<size_t>(blockIdx.z) * 2 * p.D + static_cast<size_t>(head) * 2 * p.bw) * p.bw;
#pragma unroll
  for (int u = 0; u < 4; ++u)
    if (o0 + to + u < 2 * p.bw)
      *reinterpret_cast<float4*>(out + static_cast<size_t>(o0 + to + u) * p.bw + i0 + ti) =
          make_float4(acc[u][0], acc[u][1], acc[u][2], acc[u][3]);
}

// ---------------------------------------------------------------- launchers
cudaError_t launch_gate_pack(bool f32_w, bool bf16, const GatePackArgs& a, cudaStream_t s) {
  const unsigned blocks = static_cast<unsigned>((2 * a.D + GATE_WARPS - 1) / GATE_WARPS);
  using H = __nv_bfloat16;
  if (f32_w) {
    if (bf16) gate_pack_kernel<float, H><<<blocks, 32 * GATE_WARPS, 0, s>>>(a);
    else gate_pack_kernel<float, float><<<blocks, 32 * GATE_WARPS, 0, s>>>(a);
  } else {
    if (bf16) gate_pack_kernel<H, H><<<blocks, 32 * GATE_WARPS, 0, s>>>(a);
    else gate_pack_kernel<H, float><<<blocks, 32 * GATE_WARPS, 0, s>>>(a);
  }
  return cudaGetLastError();
}
cudaError_t launch_gate_unpack(bool bf16, bool f32_w, const GateUnpackArgs& a, cudaStream_t s) {
  const unsigned blocks = static_cast<unsigned>((2 * a.D + GATE_WARPS - 1) / GATE_WARPS);
  using H = __nv_bfloat16;
  if (bf16) {
    if (f32_w) gate_unpack_kernel<H, float><<<blocks, 32 * GATE_WARPS, 0, s>>>(a);
    else gate_unpack_kernel<H, H><<<blocks, 32 * GATE_WARPS, 0, s>>>(a);
  } else {
    if (f32_w) gate_unpack_kernel<float, float><<<blocks, 32 * GATE_WARPS, 0, s>>>(a);
    else gate_unpack_kernel<float, H><<<blocks, 32 * GATE_WARPS, 0, s>>>(a);
  }
  return cudaGetLastError();
}

// Tile width in i: 32, 48 or 64, whichever leaves the least of the last tile empty (the wider of equals).
static int dw_tile(int bw) {
  int best = 64, waste = (bw + 63) / 64 * 64;
  const int other[2] = {48, 32};
  for (int t : other)
    if ((bw + t - 1) / t * t < waste) { best = t; waste = (bw + t - 1) / t * t; }
  return best;
}
// Stretches of tokens: enough CTAs for six on every SM, at least 128 tokens each.
int gate_dw_splits(long long rows, int D, int bw) {
  const int ti = dw_tile(bw);
  const long long tiles = static_cast<long long>(D / bw) * ((2 * bw + DW_TO - 1) / DW_TO) * ((bw + ti - 1) / ti);
  long long want = (6 * 148 + tiles - 1) / tiles;
  const long long most = (rows + 127) / 128;
  if (want > most) want = most;
  return static_cast<int>(want < 1 ? 1 : want);
}
cudaError_t launch_gate_dw(const GateDwArgs& args, int splits, cudaStream_t s) {
  GateDwArgs a = args;
  a.per_split = ((a.rows + splits - 1) / splits + DW_TK - 1) / DW_TK * DW_TK;
  const int ti = dw_tile(a.bw);
  const dim3 grid(static_cast<unsigned>(((2 * a.bw + DW_TO - 1) / DW_TO) * ((a.bw + ti - 1) / ti)),
                  static_cast<unsigned>(a.D / a.bw), static_cast<unsigned>(splits));
  if (ti == 64) gate_dw_kernel<64><<<grid, 256, 0, s>>>(a);
  else if (ti == 48) gate_dw_kernel<48><<<grid, 192, 0, s>>>(a);
  else gate_dw_kernel<32><<<grid, 128, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace rglru
