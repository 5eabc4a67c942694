// The gate parameters on their way into and out of the interleaved gate layout.
//
// Both gate projections of a head run as one GEMM whose output columns alternate between the two gates in groups of
// `unit` channels, [r (unit) | i (unit)] [r | i] ..., with `unit` the largest power of two up to 64 that divides the head
// width: column (d / unit) * 2 unit + d % unit of the [B, T, 2 D] gate tensor is channel d's recurrence gate, `unit`
// columns further its input gate, whatever head d is in.  A 64-channel scan tile may therefore straddle heads, and heads of any
// width go through one GEMM without a re-layout.  bf16, B = 8, T = 8192, D = 5632, 16 heads of 352 channels, forward and
// backward of the layer: 9.0 ms with the projections as modules (4.7 of it re-layouts), 3.7 ms this way (3.3 of kernels).  Narrow groups
// cost the scan little: B = 8, T = 4096, D = 5632 bf16 forward / backward 306 / 530 us in groups of 8, 263 / 562 of 16,
// 271 / 564 of 32, 256 / 537 of 64.
//
//   gate_pack_kernel     the two [G, bw, bw] weights as the GEMM's one [G, 2 bw, bw] operand in the activation type, and
//                        the biases and Lambda in fp32: one launch instead of two concatenations and three casts;
//   gate_project_*       the projections, and the gates' share of the input gradient;
//   gate_dw_*            the weight gradient, split over the tokens;
//   gate_unpack_kernel   the gradients of all five parameters in their own types and shapes: one launch instead of four
//                        slices with a cast or a copy each and the cast of Lambda's.
//
// Reference: BlockDiagonalLinear, griffin/griffin.py:129-154, called twice at :237-238.

#include <atomic>

#include "rglru_internal.h"
#include "rglru_mma.cuh"
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
// leaves a partial sum for gate_unpack_kernel.  Both operands lie with the contracted axis outermost; a thread owns 8 x 4
// outputs as pairs along o, which the eight values it reads come in, and so issues 16 packed FMAs per three 16-byte loads.
// A library's batched GEMM walks all tokens with the few CTAs the output has: at 7685 tokens and 16 heads of 48 channels
// two calls took 359 us, this kernel takes 47 (55 with 4 x 4 outputs and single FMAs).
constexpr int DW_TO = 64, DW_TK = 32;

template <int TI>
__global__ void __launch_bounds__(8 * (TI / 4)) gate_dw_kernel(const GateDwArgs p) {
  const float* du_all = static_cast<const float*>(p.du);
  const float* x_all = static_cast<const float*>(p.x);
  constexpr int NT = 8 * (TI / 4);
  __shared__ __align__(16) float sa[2][DW_TK][DW_TO];
  __shared__ __align__(16) float sb[2][DW_TK][TI];
  // (a thread's eight rows of o lie in two groups of four 32 apart, so that the threads of a warp read adjacent pieces)
  const int tid = threadIdx.x, to = (tid / (TI / 4)) * 4, ti = (tid % (TI / 4)) * 4;
  const int tiles_i = (p.bw + TI - 1) / TI;
  const int o0 = (blockIdx.x / tiles_i) * DW_TO, i0 = (blockIdx.x % tiles_i) * TI, head = blockIdx.y;
  const long long n0 = blockIdx.z * p.per_split, n1 = n0 + p.per_split < p.rows ? n0 + p.per_split : p.rows;
  const float* du = du_all + static_cast<size_t>(head) * 2 * p.bw;
  const float* x = x_all + static_cast<size_t>(head) * p.bw;

  auto load = [&](int st, long long n) {
#pragma unroll
    for (int i = tid; i < DW_TK * DW_TO / 4; i += NT) {
      const int k = i / (DW_TO / 4), c = (i % (DW_TO / 4)) * 4;
      const bool ok = n + k < n1 && o0 + c < 2 * p.bw;
      cp_async16(smem_u32(&sa[st][k][c]), ok ? du + (n + k) * 2 * p.D + o0 + c : du_all, ok);
    }
#pragma unroll
    for (int i = tid; i < DW_TK * TI / 4; i += NT) {
      const int k = i / (TI / 4), c = (i % (TI / 4)) * 4;
      const bool ok = n + k < n1 && i0 + c < p.bw;
      cp_async16(smem_u32(&sb[st][k][c]), ok ? x + (n + k) * p.D + i0 + c : x_all, ok);
    }
    cp_async_commit();
  };
  float2 acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = f2(0.0f);
  load(0, n0);
  int st = 0;
  for (long long n = n0; n < n1; n += DW_TK, st ^= 1) {
    cp_async_wait<0>();
    __syncthreads();                       // this stage is there for all, and all are done with the other one
    if (n + DW_TK < n1) load(st ^ 1, n + DW_TK);
#pragma unroll 8
    for (int k = 0; k < DW_TK; ++k) {
      const float4 l4 = *reinterpret_cast<const float4*>(&sa[st][k][to]);
      const float4 h4 = *reinterpret_cast<const float4*>(&sa[st][k][to + 32]);
      const float4 b4 = *reinterpret_cast<const float4*>(&sb[st][k][ti]);
      const float2 a[4] = {make_float2(l4.x, l4.y), make_float2(l4.z, l4.w), make_float2(h4.x, h4.y), make_float2(h4.z, h4.w)};
      const float b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
      for (int v = 0; v < 4; ++v)
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u][v] = fma2(a[u], f2(b[v]), acc[u][v]);
    }
  }
  if (i0 + ti >= p.bw) return;             // bw is a multiple of 4
  float* out = p.part + (static_cast<size_t>(blockIdx.z) * 2 * p.D + static_cast<size_t>(head) * 2 * p.bw) * p.bw;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int o = o0 + to + (u >> 2) * 32 + (u & 3);
    const float2(&r)[4] = acc[u >> 1];
    if (o < 2 * p.bw)
      *reinterpret_cast<float4*>(out + static_cast<size_t>(o) * p.bw + i0 + ti) =
          (u & 1) ? make_float4(r[0].y, r[1].y, r[2].y, r[3].y) : make_float4(r[0].x, r[1].x, r[2].x, r[3].x);
  }
}

// ---------------------------------------------------------------- fp32 projections
// NN = false: u[n][g][o] = sum_k x[n][g][k] w[g][o][k]              (k: the head's channels, o: its 2 bw gate columns)
// NN = true:  dx[n][g][i] += sum_o du[n][g][o] w[g][o][i]           (the gates' share of the input gradient)
// in full fp32.  A CTA takes 128 tokens x TN columns of one head and 16 of the contracted axis per stage; a thread owns
// 8 x 4 outputs, reads its rows and (NN = false) columns in float4 along the contracted axis from rows 80 bytes apart
// (no bank conflicts), and so does 128 FMAs per twelve 16-byte loads.
constexpr int GP_TM = 128, GP_TK = 16, GP_PITCH = GP_TK + 4;

template <int TN, bool NN>
__global__ void __launch_bounds__(16 * (TN / 4)) gate_project_kernel(const GateProjectArgs p) {
  constexpr int NT = 16 * (TN / 4), CG = TN / 4;
  constexpr int WROWS = NN ? GP_TK : TN, WCOLS = NN ? TN : GP_TK, WPITCH = NN ? TN : GP_PITCH;
  __shared__ __align__(16) float sa[2][GP_TM][GP_PITCH];
  __shared__ __align__(16) float sw[2][WROWS][WPITCH];
  const int tid = threadIdx.x, cg = tid % CG, rg = tid / CG;
  const int K = NN ? 2 * p.bw : p.bw, N = NN ? p.bw : 2 * p.bw;
  const int lda = NN ? 2 * p.D : p.D, ldo = NN ? p.D : 2 * p.D;
  const int tiles_n = (N + TN - 1) / TN, head = blockIdx.y;
  const long long m0 = static_cast<long long>(blockIdx.x / tiles_n) * GP_TM;
  const int n0 = (blockIdx.x % tiles_n) * TN;
  const float* a_all = static_cast<const float*>(p.a);
  const float* w_all = static_cast<const float*>(p.w);
  const float* a = a_all + static_cast<size_t>(head) * K;
  const float* w = w_all + static_cast<size_t>(head) * 2 * p.bw * p.bw;

  auto load = [&](int st, int k0) {
    for (int i = tid; i < GP_TM * (GP_TK / 4); i += NT) {
      const int r = i / (GP_TK / 4), c = (i % (GP_TK / 4)) * 4;
      const bool ok = m0 + r < p.rows && k0 + c < K;
      cp_async16(smem_u32(&sa[st][r][c]), ok ? a + (m0 + r) * lda + k0 + c : a_all, ok);
    }
    for (int i = tid; i < WROWS * (WCOLS / 4); i += NT) {
      const int r = i / (WCOLS / 4), c = (i % (WCOLS / 4)) * 4;
      const int o = NN ? k0 + r : n0 + r, k = NN ? n0 + c : k0 + c;        // row and column of the head's [2 bw, bw] weights
      const bool ok = o < 2 * p.bw && k < p.bw;
      cp_async16(smem_u32(&sw[st][r][c]), ok ? w + static_cast<size_t>(o) * p.bw + k : w_all, ok);
    }
    cp_async_commit();
  };
  float acc[8][4];
#pragma unroll
  for (int q = 0; q < 8; ++q)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[q][j] = 0.0f;
  load(0, 0);
  int st = 0;
  for (int k0 = 0; k0 < K; k0 += GP_TK, st ^= 1) {
    cp_async_wait<0>();
    __syncthreads();                       // this stage is there for all, and all are done with the other one
    if (k0 + GP_TK < K) load(st ^ 1, k0 + GP_TK);
#pragma unroll
    for (int k = 0; k < GP_TK; k += 4) {
      float4 wv[4];                        // NN: row k + j, the thread's four columns; else column j, contracted k .. k + 3
#pragma unroll
      for (int j = 0; j < 4; ++j)
        wv[j] = NN ? *reinterpret_cast<const float4*>(&sw[st][(k + j) % WROWS][(cg * 4) % WPITCH])
                   : *reinterpret_cast<const float4*>(&sw[st][(cg + CG * j) % WROWS][k]);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 av = *reinterpret_cast<const float4*>(&sa[st][rg + 16 * q][k]);
        if (NN) {
          acc[q][0] = fmaf(av.w, wv[3].x, fmaf(av.z, wv[2].x, fmaf(av.y, wv[1].x, fmaf(av.x, wv[0].x, acc[q][0]))));
          acc[q][1] = fmaf(av.w, wv[3].y, fmaf(av.z, wv[2].y, fmaf(av.y, wv[1].y, fmaf(av.x, wv[0].y, acc[q][1]))));
          acc[q][2] = fmaf(av.w, wv[3].z, fmaf(av.z, wv[2].z, fmaf(av.y, wv[1].z, fmaf(av.x, wv[0].z, acc[q][2]))));
          acc[q][3] = fmaf(av.w, wv[3].w, fmaf(av.z, wv[2].w, fmaf(av.y, wv[1].w, fmaf(av.x, wv[0].w, acc[q][3]))));
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            acc[q][j] = fmaf(av.w, wv[j].w, fmaf(av.z, wv[j].z, fmaf(av.y, wv[j].y, fmaf(av.x, wv[j].x, acc[q][j]))));
        }
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const long long m = m0 + rg + 16 * q;
    if (m >= p.rows) break;
    float* out = static_cast<float*>(p.out) + m * ldo + static_cast<size_t>(head) * N;
    if (NN) {
      const int n = n0 + cg * 4;
      if (n < N) {                         // N is a multiple of 4
        float4 v = *reinterpret_cast<const float4*>(out + n);
        v.x += acc[q][0]; v.y += acc[q][1]; v.z += acc[q][2]; v.w += acc[q][3];
        *reinterpret_cast<float4*>(out + n) = v;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (n0 + cg + CG * j < N) out[n0 + cg + CG * j] = acc[q][j];
    }
  }
}

// ---------------------------------------------------------------- bf16 projections and weight gradient
// The same two contractions on mma.sync, fp32 accumulators, for layers whose call is bound by its launches and streams, 64
// of the contracted axis per stage, rows 144 bytes apart in shared memory (conflict-free for ldmatrix).  Operands that
// lie with the contracted axis outermost are transposed by ldmatrix.  A projection CTA keeps 64 columns of one head and
// walks tiles of 128 tokens, the next stage -- the next tile's first, at the end of one -- in flight while it contracts
// and stores; heads are at most a few stages deep, so a CTA per tile would spend its time waiting.  A weight-gradient CTA
// takes 64 x 64 outputs of one head over a stretch of the tokens.
// Projection / input gradient / weight gradient, us, against the library's batched GEMMs: 512 tokens, 4 heads of 64: 5 / 6 / 5
// against 10 / 9 / 11; 7685 tokens, 16 heads of 24: 12 / 17 / 10 against 10 / 10 / 19; 16384 tokens, 16 heads of 64: 33 / 42 / 26
// against 18 / 15 / 25; 8192 tokens, 16 heads of 176: 122 / 127 / 87 against 33 / 39 / 42.  (fp32, the kernels above: 7685 tokens,
// 16 heads of 48: 48 / 43 / 56 against 50 / 48 / 118; 16384 tokens, 8 heads of 128: 234 / 230 / 255 against 185 / 217 / 384.)
constexpr int HP_TM = 128, HP_TN = 64, HP_TK = 64, HP_ROW = 144;
constexpr int HP_A = HP_TM * HP_ROW, HP_STAGE = HP_A + HP_TK * HP_ROW, HP_BYTES = 2 * HP_STAGE + HP_TM * HP_ROW;
constexpr int HP_CTAS = 3 * 148;            // three on every SM
constexpr int HW_STAGES = 3, HW_STAGE = 2 * HP_TK * HP_ROW;

template <bool NN>
__global__ void __launch_bounds__(256, 3) gate_project_bf16_kernel(const GateProjectArgs p) {
  using H = __nv_bfloat16;
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;     // the warp's 32 x 32 of the tile
  const int K = NN ? 2 * p.bw : p.bw, N = NN ? p.bw : 2 * p.bw;
  const int lda = NN ? 2 * p.D : p.D, ldo = NN ? p.D : 2 * p.D;
  const int tiles_n = (N + HP_TN - 1) / HP_TN, head = blockIdx.y, nk = (K + HP_TK - 1) / HP_TK;
  const int n0 = (blockIdx.x % tiles_n) * HP_TN;
  const int slot = blockIdx.x / tiles_n, slots = gridDim.x / tiles_n;
  const int tiles_m = static_cast<int>((p.rows + HP_TM - 1) / HP_TM);
  const int total = slot < tiles_m ? ((tiles_m - slot + slots - 1) / slots) * nk : 0;
  const H* a_all = static_cast<const H*>(p.a);
  const H* w_all = static_cast<const H*>(p.w);
  const H* a = a_all + static_cast<size_t>(head) * K;
  const H* w = w_all + static_cast<size_t>(head) * 2 * p.bw * p.bw;
  H* out = static_cast<H*>(p.out) + static_cast<size_t>(head) * N;

  auto load = [&](int step) {
    const uint32_t da = sbase + (step & 1) * HP_STAGE, dw = da + HP_A;
    const long long m0 = static_cast<long long>(slot + step / nk * slots) * HP_TM;
    const int k0 = step % nk * HP_TK;
#pragma unroll
    for (int i = 0; i < HP_TM * 8 / 256; ++i) {
      const int idx = tid + i * 256, r = idx >> 3, c = (idx & 7) * 8;
      const bool ok = m0 + r < p.rows && k0 + c < K;
      cp_async16(da + r * HP_ROW + c * 2, ok ? a + (m0 + r) * lda + k0 + c : a_all, ok);
    }
#pragma unroll
    for (int i = 0; i < HP_TK * 8 / 256; ++i) {
      const int idx = tid + i * 256, r = idx >> 3, c = (idx & 7) * 8;
      const int o = NN ? k0 + r : n0 + r, k = NN ? n0 + c : k0 + c;        // row and column of the head's [2 bw, bw] weights
      const bool ok = o < 2 * p.bw && k < p.bw;
      cp_async16(dw + r * HP_ROW + c * 2, ok ? w + static_cast<size_t>(o) * p.bw + k : w_all, ok);
    }
    cp_async_commit();
  };
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0f;
  if (total > 0) load(0);
  for (int step = 0; step < total; ++step) {
    cp_async_wait<0>();
    __syncthreads();                       // this stage is there for all, and all are done with the other one
    if (step + 1 < total) load(step + 1);
    const uint32_t sa = sbase + (step & 1) * HP_STAGE + (wm + (lane & 15)) * HP_ROW + (lane >> 4) * 16;
    const uint32_t sw = sbase + (step & 1) * HP_STAGE + HP_A;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t af[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) ldmatrix4(sa + i * 16 * HP_ROW + kk * 32, af[i]);
#pragma unroll
      for (int j = 0; j < 4; j += 2) {     // two 8-column tiles per load
        uint32_t bf[4];
        if (NN) ldmatrix4_trans(sw + (kk * 16 + (lane & 15)) * HP_ROW + (wn + j * 8 + (lane >> 4) * 8) * 2, bf);
        else ldmatrix4(sw + (wn + j * 8 + (lane >> 4) * 8 + (lane & 7)) * HP_ROW + kk * 32 + ((lane >> 3) & 1) * 16, bf);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          mma_bf16(acc[i][j], af[i], bf[0], bf[1]);
          mma_bf16(acc[i][j + 1], af[i], bf[2], bf[3]);
        }
      }
    }
    if (step % nk != nk - 1) continue;
    // The tile leaves through shared memory of its own, in 16-byte pieces; the input gradient is added to before it is
    // rounded.  (The barrier at the head of the loop keeps the next tile's results from overtaking this one's stores.)
    const long long m0 = static_cast<long long>(slot + step / nk * slots) * HP_TM;
    uint8_t* so = smem + 2 * HP_STAGE;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = wm + i * 16 + (lane >> 2) + h * 8, c = wn + j * 8 + (lane & 3) * 2;
          float2 v = make_float2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
          if (NN && m0 + r < p.rows && n0 + c < N) {
            const float2 d = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(out + (m0 + r) * ldo + n0 + c));
            v.x += d.x; v.y += d.y;
          }
          *reinterpret_cast<__nv_bfloat162*>(so + r * HP_ROW + c * 2) = __floats2bfloat162_rn(v.x, v.y);
          acc[i][j][2 * h] = acc[i][j][2 * h + 1] = 0.0f;
        }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < HP_TM * 8 / 256; ++i) {
      const int idx = tid + i * 256, r = idx >> 3, c = (idx & 7) * 8;
      if (m0 + r < p.rows && n0 + c < N)                 // N is a multiple of 8
        *reinterpret_cast<uint4*>(out + (m0 + r) * ldo + n0 + c) = *reinterpret_cast<const uint4*>(so + r * HP_ROW + c * 2);
    }
  }
}

__global__ void __launch_bounds__(128) gate_dw_bf16_kernel(const GateDwArgs p) {
  using H = __nv_bfloat16;
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wo = (warp >> 1) * 32, wi = (warp & 1) * 32;
  const int tiles_i = (p.bw + 63) / 64;
  const int o0 = (blockIdx.x / tiles_i) * 64, i0 = (blockIdx.x % tiles_i) * 64, head = blockIdx.y;
  const long long n0 = blockIdx.z * p.per_split, n1 = n0 + p.per_split < p.rows ? n0 + p.per_split : p.rows;
  const H* du_all = static_cast<const H*>(p.du);
  const H* x_all = static_cast<const H*>(p.x);
  const H* du = du_all + static_cast<size_t>(head) * 2 * p.bw;
  const H* x = x_all + static_cast<size_t>(head) * p.bw;
  const int steps = n1 > n0 ? static_cast<int>((n1 - n0 + HP_TK - 1) / HP_TK) : 0;

  auto load = [&](int it) {
    const uint32_t da = sbase + (it % HW_STAGES) * HW_STAGE, db = da + HP_TK * HP_ROW;
    const long long n = n0 + static_cast<long long>(it) * HP_TK;
#pragma unroll
    for (int i = 0; i < HP_TK * 8 / 128; ++i) {
      const int idx = tid + i * 128, r = idx >> 3, c = (idx & 7) * 8;
      const bool row = n + r < n1, oka = row && o0 + c < 2 * p.bw, okb = row && i0 + c < p.bw;
      cp_async16(da + r * HP_ROW + c * 2, oka ? du + (n + r) * 2 * p.D + o0 + c : du_all, oka);
      cp_async16(db + r * HP_ROW + c * 2, okb ? x + (n + r) * p.D + i0 + c : x_all, okb);
    }
  };
  float acc[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0f;
#pragma unroll
  for (int s = 0; s < HW_STAGES - 1; ++s) {
    if (s < steps) load(s);
    cp_async_commit();
  }
  for (int it = 0; it < steps; ++it) {
    cp_async_wait<HW_STAGES - 2>();
    __syncthreads();                       // stage `it` is there for all, and all are done with the one refilled next
    if (it + HW_STAGES - 1 < steps) load(it + HW_STAGES - 1);
    cp_async_commit();
    const uint32_t sa = sbase + (it % HW_STAGES) * HW_STAGE, sb = sa + HP_TK * HP_ROW;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t af[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
        ldmatrix4_trans(sa + (kk * 16 + (lane & 7) + ((lane >> 4) & 1) * 8) * HP_ROW + (wo + i * 16 + ((lane >> 3) & 1) * 8) * 2, af[i]);
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        uint32_t bf[4];
        ldmatrix4_trans(sb + (kk * 16 + (lane & 15)) * HP_ROW + (wi + j * 8 + (lane >> 4) * 8) * 2, bf);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          mma_bf16(acc[i][j], af[i], bf[0], bf[1]);
          mma_bf16(acc[i][j + 1], af[i], bf[2], bf[3]);
        }
      }
    }
  }
  float* out = p.part + (static_cast<size_t>(blockIdx.z) * 2 * p.D + static_cast<size_t>(head) * 2 * p.bw) * p.bw;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int o = o0 + wo + i * 16 + (lane >> 2), c = i0 + wi + j * 8 + (lane & 3) * 2;
      if (c >= p.bw) continue;
      if (o < 2 * p.bw) *reinterpret_cast<float2*>(out + static_cast<size_t>(o) * p.bw + c) = make_float2(acc[i][j][0], acc[i][j][1]);
      if (o + 8 < 2 * p.bw) *reinterpret_cast<float2*>(out + static_cast<size_t>(o + 8) * p.bw + c) = make_float2(acc[i][j][2], acc[i][j][3]);
    }
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

// Tile width of n columns: 32, 48 or 64, whichever leaves the least of the last tile empty (the wider of equals).
static int dw_tile(int n) {
  int best = 64, covered = (n + 63) / 64 * 64;
  const int other[2] = {48, 32};
  for (int t : other)
    if ((n + t - 1) / t * t < covered) { best = t; covered = (n + t - 1) / t * t; }
  return best;
}
// Stretches of tokens: enough CTAs for six on every SM, at least 128 tokens each.
int gate_dw_splits(bool bf16, long long rows, int D, int bw) {
  const int ti = bf16 ? 64 : dw_tile(bw);
  const long long tiles = static_cast<long long>(D / bw) * ((2 * bw + DW_TO - 1) / DW_TO) * ((bw + ti - 1) / ti);
  long long want = (6 * 148 + tiles - 1) / tiles;
  const long long most = (rows + 127) / 128;
  if (want > most) want = most;
  return static_cast<int>(want < 1 ? 1 : want);
}
// Dynamic shared memory above the default, once per device and kernel.
template <typename Kern>
static cudaError_t allow_smem(Kern kern, int bytes, std::atomic<unsigned long long>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = (dev >= 0 && dev < 64) ? (1ull << dev) : 0ull;
  if (bit && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && bit) done.fetch_or(bit, std::memory_order_release);
  return e;
}

cudaError_t launch_gate_dw(bool bf16, const GateDwArgs& args, int splits, cudaStream_t s) {
  GateDwArgs a = args;
  a.per_split = ((a.rows + splits - 1) / splits + HP_TK - 1) / HP_TK * HP_TK;
  if (bf16) {
    static std::atomic<unsigned long long> done{0ull};
    const cudaError_t e = allow_smem(gate_dw_bf16_kernel, HW_STAGES * HW_STAGE, done);
    if (e != cudaSuccess) return e;
    const dim3 g(static_cast<unsigned>(((2 * a.bw + 63) / 64) * ((a.bw + 63) / 64)), static_cast<unsigned>(a.D / a.bw),
                 static_cast<unsigned>(splits));
    gate_dw_bf16_kernel<<<g, 128, HW_STAGES * HW_STAGE, s>>>(a);
    return cudaGetLastError();
  }
  const int ti = dw_tile(a.bw);
  const dim3 grid(static_cast<unsigned>(((2 * a.bw + DW_TO - 1) / DW_TO) * ((a.bw + ti - 1) / ti)),
                  static_cast<unsigned>(a.D / a.bw), static_cast<unsigned>(splits));
  if (ti == 64) gate_dw_kernel<64><<<grid, 128, 0, s>>>(a);
  else if (ti == 48) gate_dw_kernel<48><<<grid, 96, 0, s>>>(a);
  else gate_dw_kernel<32><<<grid, 64, 0, s>>>(a);
  return cudaGetLastError();
}

template <bool NN>
static cudaError_t gate_project_t(const GateProjectArgs& a, cudaStream_t s) {
  const int n = NN ? a.bw : 2 * a.bw, t = dw_tile(n);
  const dim3 grid(static_cast<unsigned>((a.rows + GP_TM - 1) / GP_TM * ((n + t - 1) / t)), static_cast<unsigned>(a.D / a.bw));
  if (t == 64) gate_project_kernel<64, NN><<<grid, 256, 0, s>>>(a);
  else if (t == 48) gate_project_kernel<48, NN><<<grid, 192, 0, s>>>(a);
  else gate_project_kernel<32, NN><<<grid, 128, 0, s>>>(a);
  return cudaGetLastError();
}
template <bool NN>
static cudaError_t gate_project_bf16(const GateProjectArgs& a, cudaStream_t s) {
  static std::atomic<unsigned long long> done{0ull};
  const cudaError_t e = allow_smem(gate_project_bf16_kernel<NN>, HP_BYTES, done);
  if (e != cudaSuccess) return e;
  const long long tiles_m = (a.rows + HP_TM - 1) / HP_TM, heads = a.D / a.bw;
  const int n = NN ? a.bw : 2 * a.bw, tiles_n = (n + HP_TN - 1) / HP_TN;
  long long slots = HP_CTAS / (tiles_n * heads);
  if (slots > tiles_m) slots = tiles_m;
  if (slots < 1) slots = 1;
  const dim3 grid(static_cast<unsigned>(slots * tiles_n), static_cast<unsigned>(heads));
  gate_project_bf16_kernel<NN><<<grid, 256, HP_BYTES, s>>>(a);
  return cudaGetLastError();
}
cudaError_t launch_gate_project(bool bf16, bool backward, const GateProjectArgs& a, cudaStream_t s) {
  if (bf16) return backward ? gate_project_bf16<true>(a, s) : gate_project_bf16<false>(a, s);
  return backward ? gate_project_t<true>(a, s) : gate_project_t<false>(a, s);
}

}  // namespace rglru
