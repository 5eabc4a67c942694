// Device code of the scan that more than one kernel file uses -- row masks, the time split's exchange, the gate layout, the
// conv and gate arithmetic of a thread's steps in both directions -- and the launch helpers of those kernels.
#pragma once

#include <atomic>
#include <cfloat>
#include <cstddef>
#include <cstdlib>

#include "rglru_device.cuh"
#include "rglru_internal.h"

namespace rglru {


// Per-row multipliers that realise the reset / padding masks without branches.
struct RowMask {
  float keep;    // 0 at a reset, else 1          (a <- a * keep, gamma <- gamma * keep + (1 - keep))
  float live;    // 0 on padding, else 1          (a <- a * live + (1 - live), b <- b * live)
};

template <bool MASKED>
__device__ __forceinline__ RowMask row_mask(uint32_t packed, int st) {
  RowMask m{1.0f, 1.0f};
  if (MASKED) {
    const uint32_t byte = (packed >> (8 * (st & 3))) & 0xffu;
    m.keep = (byte & TOK_RESET) ? 0.0f : 1.0f;
    m.live = (byte & TOK_INACTIVE) ? 0.0f : 1.0f;
  }
  return m;
}

// Flag bytes of the TS steps a thread owns, packed four per word.  Steps at or
// beyond T are padding.
template <int TS>
__device__ __forceinline__ void load_flags(const uint8_t* tok, int b, int T, int t_first, uint32_t (&fl)[(TS + 3) / 4]) {
#pragma unroll
  for (int w = 0; w < (TS + 3) / 4; ++w) fl[w] = 0;
#pragma unroll
  for (int st = 0; st < TS; ++st) {
    const int t = t_first + st;
    uint32_t byte = TOK_INACTIVE;
    if (t < T) byte = tok ? tok[static_cast<size_t>(b) * T + t] : 0u;
    fl[st >> 2] |= byte << (8 * (st & 3));
  }
}

// Whether any of a thread's flag bytes is set.  Ordinary tokens have a zero byte, so a thread whose steps are
// all ordinary takes the mask-free arithmetic even when the caller passed a flag tensor.
template <int N>
__device__ __forceinline__ bool any_flag(const uint32_t (&fl)[N]) {
  uint32_t v = 0u;
#pragma unroll
  for (int i = 0; i < N; ++i) v |= fl[i];
  return v != 0u;
}

// The same for four steps, as one word when the four bytes are whole and 4-byte aligned (the byte of step st sits
// at bits 8 st).  Used by the conv kernels, whose per-element work is small enough for the byte loads to show;
// the scan kernels keep the byte loads (the word path perturbed their register allocation: +9 % backward time).
__device__ __forceinline__ void load_flags_word(const uint8_t* tok, int b, int T, int t_first, uint32_t (&fl)[1]) {
  if (tok && t_first + 4 <= T) {
    const uint8_t* p = tok + static_cast<size_t>(b) * T + t_first;
    if ((reinterpret_cast<uintptr_t>(p) & 3u) == 0) {
      fl[0] = *reinterpret_cast<const uint32_t*>(p);
      return;
    }
  }
  load_flags<4>(tok, b, T, t_first, fl);
}

// Plain-load staging of one [rows, CH] tile (zero-filled outside the tensor).
template <typename IO, int CH>
__device__ __forceinline__ void tile_load_plain(uint8_t* tile, const void* src, int b, int t0, int d0, int rows, int T, int D) {
  const IO* g = static_cast<const IO*>(src);
  IO* s = reinterpret_cast<IO*>(tile);
  for (int idx = threadIdx.x; idx < rows * CH; idx += blockDim.x) {
    const int row = idx / CH, col = idx % CH;
    const int t = t0 + row, d = d0 + col;
    IO v = Pack<IO>::from_float(0.0f);
    if (t >= 0 && t < T && d < D) v = g[(static_cast<size_t>(b) * T + t) * D + d];
    s[idx] = v;
  }
}
template <typename IO, int CH>
__device__ __forceinline__ void tile_store_plain(const uint8_t* tile, void* dst, int b, int t0, int d0, int rows, int T, int D) {
  IO* g = static_cast<IO*>(dst);
  const IO* s = reinterpret_cast<const IO*>(tile);
  for (int idx = threadIdx.x; idx < rows * CH; idx += blockDim.x) {
    const int row = idx / CH, col = idx % CH;
    const int t = t0 + row, d = d0 + col;
    if (t < T && d < D) g[(static_cast<size_t>(b) * T + t) * D + d] = s[idx];
  }
}

// Per-channel rate: -c * logsigmoid(Lambda) >= 0, and 0 for channels past D.
__device__ __forceinline__ float decay_rate(float lam, float c) {
  // softplus(-L) = -logsigmoid(L), evaluated without cancellation on either side.
  const float sp = lam >= 0.0f ? log1pf(expf(-lam)) : log1pf(expf(lam)) - lam;
  return c * sp;
}
__device__ __forceinline__ float decay_rate(const float* lambda, int d, int D, float c) {
  return d < D ? decay_rate(lambda[d], c) : 0.0f;
}

template <int LANES, int CH>
struct ChainSmem {
  static constexpr int AGG = LANES * CH * 8;  // float2 per (lane, channel)
  static constexpr int EIN = LANES * CH * 4;  // float per (lane, channel)
};

// Time split (SPLIT kernels).  A cluster of up to MAX_SPLIT CTAs shares one (batch row, channel tile): in round `it`
// the CTA of rank r takes chunk it * R + r.  Everything of a chunk but its entering state is worked out locally; then
// each CTA sends the affine map of its whole chunk, one (product, state) pair per channel, to every CTA of the
// cluster, and each folds the pairs of the ranks before it onto the carry of the rounds before (all CTAs keep
// identical copies of that carry, folded in rank order, so the result does not depend on timing).  Two buffers by
// round parity suffice: nobody can send round it + 2 before it has received everybody's round it + 1, which they
// send after they are done reading round it.
// What it buys: with fewer tiles than SMs a sequence is bound by one CTA walking it chunk by chunk.  B = 1, T = 16384,
// D = 1024 bf16 (16 tiles; eight CTAs each forward, six backward): forward 135 -> 67 us, backward 340 -> 80 us; B = 2, T = 2048: 25 -> 13 and
// 47 -> 21 us; fp32 B = 1, T = 16384: 310 -> 76 and 407 -> 93 us.
constexpr int MAX_SPLIT = 8;   // the portable cluster size
template <int CH>
struct SplitSmem {
  float2 pair[2][MAX_SPLIT][CH];
  uint64_t bar[2];
  float sums[MAX_SPLIT][3 * CH];   // rglru backward only: the per-channel sums of every rank, folded by rank 0
};
template <int CH>
struct SplitChain {
  SplitSmem<CH>* sm;
  uint32_t rank, size;
  __device__ __forceinline__ void init(SplitSmem<CH>* s) { sm = s; rank = cluster_rank(); size = cluster_size(); }
  __device__ __forceinline__ void arm(int it) { mbar_expect_tx(&sm->bar[it & 1], size * CH * 8); }   // one thread per round
  // Send this CTA's pair of one channel to the ranks first, first + step, ...
  __device__ __forceinline__ void send(int it, int ch, float2 v, uint32_t first, uint32_t step) {
    for (uint32_t r = first; r < size; r += step)
      st_async_pair(cluster_map(&sm->pair[it & 1][rank][ch], r), v, cluster_map(&sm->bar[it & 1], r));
  }
  // State entering this CTA's chunk of round `it`, and the carry behind the whole round.
  __device__ __forceinline__ float receive(int it, int ch, float& carry, float& prod, volatile int* dead, int* status) {
    mbar_wait_or_flag(&sm->bar[it & 1], (it >> 1) & 1, dead, status, DEV_TIMEOUT_SPLIT);
    return fold(it, ch, carry, prod);
  }
  // (`contractive`: no rank's product is above one, or NaN)
  __device__ __forceinline__ float receive(int it, int ch, float& carry, bool& contractive, bool& alive) {
    if (alive) alive = mbar_wait_bounded(&sm->bar[it & 1], (it >> 1) & 1);
    float unused = 1.0f;
    return fold(it, ch, carry, unused, &contractive);
  }
  __device__ __forceinline__ float fold(int it, int ch, float& carry, float& prod, bool* contractive = nullptr) {
    float2 v[MAX_SPLIT];
#pragma unroll
    for (int r = 0; r < MAX_SPLIT; ++r) v[r] = r < static_cast<int>(size) ? sm->pair[it & 1][r][ch] : make_float2(1.0f, 0.0f);
    if (contractive) {
      *contractive = true;
#pragma unroll
      for (int r = 0; r < MAX_SPLIT; ++r) *contractive = *contractive && fabsf(v[r].x) <= 1.0f;
    }
    float e = carry, enter = carry;
#pragma unroll
    for (int r = 0; r < MAX_SPLIT; ++r) {
      if (r == static_cast<int>(rank)) enter = e;
      e = fmaf(v[r].x, e, v[r].y);
      prod *= v[r].x;
    }
    carry = e;
    return enter;
  }
};

// Grouped gate layout: both gate pre-activations come from ONE tensor [B, T, 2 D] written by a single
// grouped GEMM with the two weight blocks of a gate head stacked.  Its columns alternate between the gates in groups of
// `bw` channels, [u_r (bw) | u_i (bw)] and so on: channel d's recurrence gate is column (d / bw) * 2 bw + d % bw, its
// input gate bw columns further.  A group is a multiple of the tile width -- a tile's columns of one gate are then
// adjacent -- or a power of two below it: a tile then takes every other group of 2 * 64 columns, which the copy engine
// gathers through a 5-D tensor map (channel in the group, gate, group, time, batch) into the same dense tile.  The
// gate biases (same column layout, fp32) are added in the kernel, pre-scaled for the sigmoid.
struct GateBias {
  float2 r[2], i[2];
};
__device__ __forceinline__ int grouped_col(int d, int bw) { return (d / bw) * 2 * bw + d % bw; }
template <bool HALF_IO>
__device__ __forceinline__ void load_gate_bias(const float* bias, int d, int D, int bw, GateBias& gb) {
  const float sc = gate_bias_scale<HALF_IO>();
  float4 br = make_float4(0.f, 0.f, 0.f, 0.f), bi = br;
  if (bias && d < D) {
    const int col = grouped_col(d, bw);
    br = *reinterpret_cast<const float4*>(bias + col);
    bi = *reinterpret_cast<const float4*>(bias + col + bw);
  }
  gb.r[0] = make_float2(br.x * sc, br.y * sc); gb.r[1] = make_float2(br.z * sc, br.w * sc);
  gb.i[0] = make_float2(bi.x * sc, bi.y * sc); gb.i[1] = make_float2(bi.z * sc, bi.w * sc);
}
// The tile of one gate (which: 0 recurrence, 1 input) of the channels from d0 on, at time t of batch row b.
template <bool GROUPED, int CH>
struct GateTile {
  int col, group, step;      // first column of a wide group, or first group of a narrow one (step 0)
  __device__ __forceinline__ GateTile(int d0, int bw)
      : col(GROUPED ? grouped_col(d0, bw) : d0), group(GROUPED ? d0 / bw : 0), step(GROUPED && bw >= CH ? bw : 0) {}
  __device__ __forceinline__ void load(void* dst, const void* map, int which, int t, int b, uint64_t* bar) const {
    if (!GROUPED || step) tma_load_3d(dst, map, col + which * step, t, b, bar);
    else tma_load_5d(dst, map, 0, which, group, t, b, bar);
  }
  __device__ __forceinline__ void prefetch(const void* map, int which, int t, int b) const {
    if (!GROUPED || step) tma_prefetch_3d(map, col + which * step, t, b);
    else tma_prefetch_5d(map, 0, which, group, t, b);
  }
  __device__ __forceinline__ void store(const void* map, const void* src, int which, int t, int b) const {
    if (!GROUPED || step) tma_store_3d(map, src, col + which * step, t, b);
    else tma_store_5d(map, src, 0, which, group, t, b);
  }
};

// Taps of the width-4 causal depthwise conv for the four channels a thread owns (column 3 of the
// [D, 4] weight multiplies the current token; griffin/griffin.py:474-486 of the reference).
struct ConvTaps {
  float2 w[4][2];
  float2 bias[2];
};

__device__ __forceinline__ void load_taps(const void* conv_w, const void* conv_b, int d, int D, ConvTaps& ct, bool half_w = false,
                                          bool half_b = false) {
  float w[4][4], bz[4];
#pragma unroll
  for (int ch = 0; ch < 4; ++ch) {
    const bool ok = d + ch < D;
    bz[ch] = (ok && conv_b) ? param_as_float(conv_b, d + ch, half_b) : 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k][ch] = ok ? param_as_float(conv_w, static_cast<size_t>(d + ch) * 4 + k, half_w) : 0.0f;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) { ct.w[k][0] = make_float2(w[k][0], w[k][1]); ct.w[k][1] = make_float2(w[k][2], w[k][3]); }
  ct.bias[0] = make_float2(bz[0], bz[1]);
  ct.bias[1] = make_float2(bz[2], bz[3]);
}

// Conv folded into the load stage: the x tile carries three extra rows in front (times t0-3 .. t0-1), a
// thread reads the TS+3 rows ending at its last step and forms the TS conv outputs in registers.
// `hist` (non-null only for the first lane of the first chunk when a conv state is carried) replaces
// the three rows before t = 0.  Tap l is dropped when the token's flag byte says fewer than l earlier
// tokens belong to its document.
template <typename IO, int TS, int CH, bool MASKED>
__device__ __forceinline__ void conv_front(const uint8_t* tx, int off0, const ConvTaps& ct,
                                           const uint32_t (&fl)[(TS + 3) / 4], const float2 (*hist)[2],
                                           float2 (&xc)[TS][2]) {
  constexpr int ROWB = CH * sizeof(IO);
  float2 raw[TS + 3][2];
#pragma unroll
  for (int r = 0; r < TS + 3; ++r) Pack<IO>::unpack2(Pack<IO>::load(tx + off0 + r * ROWB), raw[r]);
  if (hist) {
#pragma unroll
    for (int r = 0; r < 3; ++r) { raw[r][0] = hist[r][0]; raw[r][1] = hist[r][1]; }
  }
#pragma unroll
  for (int st = 0; st < TS; ++st) {
    float m1 = 1.0f, m2 = 1.0f, m3 = 1.0f;
    if (MASKED) {
      const int reach = 3 - static_cast<int>((fl[st >> 2] >> (8 * (st & 3))) & TOK_CUT_MASK);
      m1 = reach >= 1 ? 1.0f : 0.0f;
      m2 = reach >= 2 ? 1.0f : 0.0f;
      m3 = reach >= 3 ? 1.0f : 0.0f;
    }
#pragma unroll
    for (int cp = 0; cp < 2; ++cp) {
      float2 acc = fma2(ct.w[3][cp], raw[st + 3][cp], ct.bias[cp]);
      if (MASKED) {
        acc = fma2(mul2(ct.w[2][cp], f2(m1)), raw[st + 2][cp], acc);
        acc = fma2(mul2(ct.w[1][cp], f2(m2)), raw[st + 1][cp], acc);
        acc = fma2(mul2(ct.w[0][cp], f2(m3)), raw[st][cp], acc);
      } else {
        acc = fma2(ct.w[2][cp], raw[st + 2][cp], acc);
        acc = fma2(ct.w[1][cp], raw[st + 1][cp], acc);
        acc = fma2(ct.w[0][cp], raw[st][cp], acc);
      }
      xc[st][cp] = acc;
    }
  }
}

// The three inputs before t = 0 of one batch row, from the carried conv state [B, 3, D].
template <typename IO>
__device__ __forceinline__ void load_hist(const void* conv_state, int b, int d, int D, float2 (&hist)[3][2]) {
  const IO* st = static_cast<const IO*>(conv_state);
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    float v[4];
#pragma unroll
    for (int ch = 0; ch < 4; ++ch)
      v[ch] = (d + ch < D) ? Pack<IO>::to_float(st[(static_cast<size_t>(b) * 3 + r) * D + d + ch]) : 0.0f;
    hist[r][0] = make_float2(v[0], v[1]);
    hist[r][1] = make_float2(v[2], v[3]);
  }
}

// Where step `st` of a thread lies in a tile whose rows are `RSTEP` bytes apart, from the place `off0` of its first step.
// SWZ: 128-byte rows whose sixteen-byte pieces the copy engine has permuted, piece c of row r at c ^ (r % 8); a thread's
// steps are rows 4 q + st, so its pieces differ from the first one's in the two bits of st.
template <int RSTEP, bool SWZ>
__device__ __forceinline__ int step_at(int off0, int st) {
  return (SWZ ? off0 ^ (st << 4) : off0) + st * RSTEP;
}

template <typename IO, int TS, int CH, bool MASKED, bool POLY, bool CONV, bool GROUPED, int RSTEP = CH * sizeof(IO), bool SWZ = false>
__device__ __forceinline__ void fwd_local(const uint8_t* tx, const uint8_t* tr, const uint8_t* ti, int off0,
                                          const float2 (&K)[2], const uint32_t (&fl)[(TS + 3) / 4],
                                          const ConvTaps& ct, const float2 (*hist)[2], const GateBias& gb,
                                          float2 (&P)[TS][2], float2 (&S)[TS][2]) {
  float2 p[2] = {f2(1.0f), f2(1.0f)};
  float2 s[2] = {f2(0.0f), f2(0.0f)};
  float2 xc[CONV ? TS : 1][2];
  if (CONV) conv_front<IO, CONV ? TS : 1, CH, MASKED>(tx, off0, ct, fl, hist, xc);
#pragma unroll
  for (int st = 0; st < TS; ++st) {
    const int off = step_at<RSTEP, SWZ>(off0, st);
    float2 xv[2], rv[2], iv[2];
    if (CONV) { xv[0] = xc[CONV ? st : 0][0]; xv[1] = xc[CONV ? st : 0][1]; }
    else Pack<IO>::unpack2(Pack<IO>::load(tx + off), xv);
    Pack<IO>::unpack2(Pack<IO>::load(tr + off), rv);
    Pack<IO>::unpack2(Pack<IO>::load(ti + off), iv);
    const RowMask m = row_mask<MASKED>(fl[st >> 2], st);
#pragma unroll
    for (int cp = 0; cp < 2; ++cp) {
      float2 r, i;
      if (GROUPED) sigmoid_pair2_biased<sizeof(IO) == 2>(rv[cp], iv[cp], gb.r[cp], gb.i[cp], r, i);
      else sigmoid_pair2<sizeof(IO) == 2>(rv[cp], iv[cp], r, i);
      const float2 e = one_minus_exp_neg2<POLY, sizeof(IO) == 2>(mul2(r, K[cp]));   // 1 - a
      float2 a = fma2(e, f2(-1.0f), f2(1.0f));
      const float2 gsq = mul2(e, fma2(e, f2(-1.0f), f2(2.0f)));     // 1 - a^2
      // sqrt(gsq) as gsq * rsqrt(gsq): one MUFU operation; the offset keeps rsqrt finite (gamma error <= 1e-15)
      const float2 gq = add2(gsq, f2(1e-30f));
      float2 gam = mul2(gq, make_float2(rsqrt_approx(gq.x), rsqrt_approx(gq.y)));
      if (MASKED) {
        a = fma2(mul2(a, f2(m.keep)), f2(m.live), f2(1.0f - m.live));
        gam = mul2(fma2(gam, f2(m.keep), f2(1.0f - m.keep)), f2(m.live));
      }
      const float2 b = mul2(mul2(gam, i), xv[cp]);
      p[cp] = mul2(p[cp], a);
      s[cp] = fma2(a, s[cp], b);
      P[st][cp] = p[cp];
      S[st][cp] = s[cp];
    }
  }
}

template <typename IO, int TS>
struct BwdRegs {
  float2 am[TS][2];  // decay after masking
  float2 hb[TS][2];  // drive b, later the state entering the step
  float2 ar[TS][2];  // unmasked decay, zeroed where the decay receives no gradient
  float2 c1[TS][2];  // d x      = g * c1
  float2 c2[TS][2];  // d u_i    = g * c2
  float2 c3[TS][2];  // d log a  = g * (h_prev * ar + c3)   (c3 <= 0 side of the sqrt slope term)
  float2 rr[TS][2];  // recurrence gate r
  typename Pack<IO>::Raw dy[TS];
};

// Level one of the backward chunk: gate math, coefficients for the second pass, and the
// lane aggregates: prod a, the local state, and the local reverse carry,
// where the reverse carry is a_t g_t flowing from step t to step t-1.
// MERGE: the incoming gradient is that of h * gelu(branch).  This pass turns it into the gradient of h
// (kept, rounded to the I/O type, where the incoming gradient was) and leaves d_out * gelu'(branch) in the
// branch tile; the second pass multiplies that by h_t to get the branch gradient.
template <typename IO, int TS, int CH, bool MASKED, bool POLY, bool CONV, bool MERGE, bool GROUPED, bool SWZ = false>
__device__ __forceinline__ void bwd_local(uint8_t* tdy, uint8_t* tg, const uint8_t* tx, const uint8_t* tr, const uint8_t* ti,
                                          int off0, const float2 (&K)[2], const uint32_t (&fl)[(TS + 3) / 4],
                                          const ConvTaps& ct, const float2 (*hist)[2], const GateBias& gb,
                                          BwdRegs<IO, TS>& R, float2 (&prod)[2], float2 (&sfwd)[2],
                                          float2 (&crev)[2]) {
  constexpr int ROWB = CH * sizeof(IO);
  float2 p[2] = {f2(1.0f), f2(1.0f)};
  float2 s[2] = {f2(0.0f), f2(0.0f)};
  float2 xc[CONV ? TS : 1][2];
  if (CONV) conv_front<IO, CONV ? TS : 1, CH, MASKED>(tx, off0, ct, fl, hist, xc);
#pragma unroll
  for (int st = 0; st < TS; ++st) {
    const int off = step_at<ROWB, SWZ>(off0, st);
    float2 xv[2], rv[2], iv[2];
    if (CONV) { xv[0] = xc[CONV ? st : 0][0]; xv[1] = xc[CONV ? st : 0][1]; }
    else Pack<IO>::unpack2(Pack<IO>::load(tx + off), xv);
    Pack<IO>::unpack2(Pack<IO>::load(tr + off), rv);
    Pack<IO>::unpack2(Pack<IO>::load(ti + off), iv);
    R.dy[st] = Pack<IO>::load(tdy + off);
    if (MERGE) {
      float2 dm[2], gv[2], q[2];
      Pack<IO>::unpack2(R.dy[st], dm);
      Pack<IO>::unpack2(Pack<IO>::load(tg + off), gv);
#pragma unroll
      for (int cp = 0; cp < 2; ++cp) {
        const float2 sg = gelu_sigmoid2<sizeof(IO) == 2>(gv[cp]);
        q[cp] = mul2(dm[cp], gelu_slope2(gv[cp], sg));
        dm[cp] = mul2(dm[cp], mul2(gv[cp], sg));
      }
      R.dy[st] = Pack<IO>::pack2(dm);
      Pack<IO>::store2(tg + off, q);
    }
    const RowMask m = row_mask<MASKED>(fl[st >> 2], st);
#pragma unroll
    for (int cp = 0; cp < 2; ++cp) {
      float2 r, i;
      if (GROUPED) sigmoid_pair2_biased<sizeof(IO) == 2>(rv[cp], iv[cp], gb.r[cp], gb.i[cp], r, i);
      else sigmoid_pair2<sizeof(IO) == 2>(rv[cp], iv[cp], r, i);
      const float2 e = one_minus_exp_neg2<POLY, sizeof(IO) == 2>(mul2(r, K[cp]));       // 1 - a
      const float2 a = fma2(e, f2(-1.0f), f2(1.0f));
      float2 gsq = mul2(e, fma2(e, f2(-1.0f), f2(2.0f)));               // 1 - a^2
      // The offset keeps rsqrt finite; it changes gamma by at most 1e-15.
      gsq = add2(gsq, f2(1e-30f));
      const float2 rs = make_float2(rsqrt_approx(gsq.x), rsqrt_approx(gsq.y));
      float2 gam = mul2(gsq, rs);                                       // sqrt(gsq)
      // -2 * slope, slope = 1 / sqrt(max(4 gsq, 1e-6)) = min(rs / 2, 1000); the sign rides on the min for free
      const float2 nrs2 = make_float2(-fminf(rs.x, 2.0f * SLOPE_CAP), -fminf(rs.y, 2.0f * SLOPE_CAP));
      const float2 ix = mul2(i, xv[cp]);
      float2 am = a, ar = a;
      // slope term of d log a, stored negated: -2 a^2 slope i x.  Unmasked, one factor a is left to the second
      // pass, which has a g at hand as the reverse carry.
      float2 c3 = MASKED ? mul2(mul2(a, a), mul2(nrs2, ix)) : mul2(a, mul2(nrs2, ix));
      if (MASKED) {
        const float kl = m.keep * m.live;
        am = fma2(mul2(a, f2(m.keep)), f2(m.live), f2(1.0f - m.live));
        ar = mul2(a, f2(kl));
        c3 = mul2(c3, f2(kl));
        gam = mul2(fma2(gam, f2(m.keep), f2(1.0f - m.keep)), f2(m.live));
      }
      const float2 c1 = mul2(gam, i);
      const float2 bb = mul2(gam, ix);
      R.am[st][cp] = am;
      if (MASKED) R.ar[st][cp] = ar;
      R.c1[st][cp] = c1;
      R.c2[st][cp] = mul2(bb, fma2(i, f2(-1.0f), f2(1.0f)));
      R.c3[st][cp] = c3;
      R.rr[st][cp] = r;
      R.hb[st][cp] = bb;
      p[cp] = mul2(p[cp], am);
      s[cp] = fma2(am, s[cp], bb);
    }
  }
  float2 c[2] = {f2(0.0f), f2(0.0f)};
#pragma unroll
  for (int st = TS - 1; st >= 0; --st) {
    float2 dyv[2];
    Pack<IO>::unpack2(R.dy[st], dyv);
#pragma unroll
    for (int cp = 0; cp < 2; ++cp) c[cp] = mul2(R.am[st][cp], add2(dyv[cp], c[cp]));
  }
#pragma unroll
  for (int cp = 0; cp < 2; ++cp) { prod[cp] = p[cp]; sfwd[cp] = s[cp]; crev[cp] = c[cp]; }
}

// Second pass of the backward chunk: with the state `hin` entering the thread's first step and the reverse
// carry `cin` entering its last, rebuild the states, run the reverse recurrence and write dx, du_r, du_i (and,
// merged, the branch gradient) over the input tiles.  MASKED = false is the path of a thread whose tokens are
// all ordinary: the decay that takes the gradient is the decay itself, so R.ar is not read.  The incoming
// gradient is read back from its tile unless the merged variant replaced it in registers.
// SUMS: also accumulate the sums over time of du_r and du_i (the gate-bias gradient of the grouped layout).
template <typename IO, int TS, int CH, bool MASKED, bool CONV, bool MERGE, bool SUMS, bool SWZ = false>
__device__ __forceinline__ void bwd_apply(uint8_t* tiles, int off_dx, int off_dr, int off_di, int off_g, int off0,
                                          const float2 (&K)[2], const float2 (&hin)[2], const float2 (&cin)[2],
                                          BwdRegs<IO, TS>& R, float2 (&dlam)[2], float2 (&dsr)[2], float2 (&dsi)[2]) {
  constexpr int ROWB = CH * sizeof(IO);
  float2 h[2] = {hin[0], hin[1]};
  float2 c[2] = {cin[0], cin[1]};
  // States entering each step, rebuilt forward in time.
#pragma unroll
  for (int st = 0; st < TS; ++st) {
#pragma unroll
    for (int cp = 0; cp < 2; ++cp) {
      const float2 hprev = h[cp];
      h[cp] = fma2(R.am[st][cp], hprev, R.hb[st][cp]);
      R.hb[st][cp] = hprev;
    }
    if (MERGE) {   // d branch_t = d_out_t * gelu'(branch_t) * h_t, the first two factors left by the first pass
      uint8_t* tq = tiles + off_g + step_at<ROWB, SWZ>(off0, st);
      float2 q[2];
      Pack<IO>::unpack2(Pack<IO>::load(tq), q);
      q[0] = mul2(q[0], h[0]);
      q[1] = mul2(q[1], h[1]);
      Pack<IO>::store2(tq, q);
    }
  }
  uint8_t* tdx = tiles + off_dx;   // over x (past its halo rows)
  uint8_t* tdr = tiles + off_dr;   // over u_r
  uint8_t* tdi = tiles + off_di;   // over u_i
  const float2 nK[2] = {mul2(K[0], f2(-1.0f)), mul2(K[1], f2(-1.0f))};
#pragma unroll
  for (int st = TS - 1; st >= 0; --st) {
    const int off = step_at<ROWB, SWZ>(off0, st);
    float2 dyv[2], dxv[2], drv[2], div[2];
    if (MERGE) Pack<IO>::unpack2(R.dy[st], dyv);
    else Pack<IO>::unpack2(Pack<IO>::load(tiles + off), dyv);
#pragma unroll
    for (int cp = 0; cp < 2; ++cp) {
      const float2 g = add2(dyv[cp], c[cp]);
      c[cp] = mul2(R.am[st][cp], g);
      dxv[cp] = mul2(g, R.c1[st][cp]);
      div[cp] = mul2(g, R.c2[st][cp]);
      // d log a = g a (h_prev + c3 / a); unmasked, g a is the reverse carry just formed and c3 came divided by a
      const float2 dl = MASKED ? mul2(g, fma2(R.hb[st][cp], R.ar[st][cp], R.c3[st][cp]))
                               : mul2(c[cp], add2(R.hb[st][cp], R.c3[st][cp]));
      const float2 w = mul2(dl, R.rr[st][cp]);
      dlam[cp] = add2(dlam[cp], w);
      // d u_r = dl * d(log a)/d u_r = dl * (-K) r (1 - r) with K = -c logsigmoid(Lambda) >= 0
      drv[cp] = mul2(w, fma2(K[cp], R.rr[st][cp], nK[cp]));
      if (SUMS) {
        dsr[cp] = add2(dsr[cp], drv[cp]);
        dsi[cp] = add2(dsi[cp], div[cp]);
      }
    }
    Pack<IO>::store2(tdx + off, dxv);
    Pack<IO>::store2(tdr + off, drv);
    Pack<IO>::store2(tdi + off, div);
  }
}

// ---------------------------------------------------------------- launch helpers
// Launch with programmatic stream serialization, so that this kernel's launch and prologue may overlap
// the tail of the kernel before it on the stream (the kernels call pdl_wait before touching memory).
// `split` > 1 makes the grid's z axis the ranks of a cluster.
template <typename Kern, typename Maps, typename Args>
static cudaError_t launch_pdl(Kern kern, dim3 grid, int threads, int bytes, cudaStream_t s, const Maps& maps, const Args& a,
                              int split = 1) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = 1;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = static_cast<unsigned>(split);
  if (split > 1) cfg.gridDim.z = static_cast<unsigned>(split);
  cfg.attrs = attr;
  cfg.numAttrs = split > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, maps, a);
}

// Shared-memory attributes of one kernel: the largest carveout, so that occupancy is set by the kernel's own
// footprint and not by the default L1 / shared split, and the dynamic size.  They are per device and do not
// change, so each call site (one per kernel instantiation, told apart by TAG) sets them once per device.
template <typename TAG, typename Kern>
static cudaError_t set_smem(Kern kern, int bytes) {
  static std::atomic<unsigned long long> done{0ull};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = (dev >= 0 && dev < 64) ? (1ull << dev) : 0ull;
  if (bit && (done.load(std::memory_order_acquire) & bit)) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && bit) done.fetch_or(bit, std::memory_order_release);
  return e;
}
template <typename... Ts> struct KernelTag {};
template <int... Vs> struct IntTag {};

// Clusters of `size` CTAs of a kernel that fit on the device at once.  That depends on the chip's GPCs (a cluster
// lives inside one), so the runtime is asked once per device, kernel (K) and size.
template <typename K>
static int resident_clusters(int size) {
  static std::atomic<int> known[64][MAX_SPLIT + 1];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  std::atomic<int>& slot = known[dev][size];
  int n = slot.load(std::memory_order_relaxed);      // 0: not asked yet; else the count + 1
  if (n == 0) {
    cudaError_t e;
    auto kern = K::get(e);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, 1, size);
    cfg.blockDim = dim3(K::THREADS);
    cfg.dynamicSmemBytes = K::BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = static_cast<unsigned>(size);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int count = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&count, kern, &cfg);
    if (e != cudaSuccess) {
      cudaGetLastError();      // no split this time, and nothing remembered: the next call asks again
      return 0;
    }
    n = count + 1;
    slot.store(n, std::memory_order_relaxed);
  }
  return n - 1;
}
// Cluster size of the time split for `tiles` (batch row, channel tile) pairs: the largest that leaves every CTA a
// chunk and all clusters resident at once, 1 if not even pairs do.  A round costs about a third more than an unsplit
// chunk (the exchange through distributed shared memory), so a second wave of clusters gives the gain away again.
// Measured on B200, T = 2048, D = 1024, bf16, forward / backward us, 64-channel tiles: 16 tiles unsplit 19 / 47, pairs
// 23 / 32, six CTAs 11 / 16, eight (a second wave in the backward) 17 / 23; 64 tiles unsplit 26 / 48, pairs 24 / 34,
// three 34 / 47.
template <typename K>
static int pick_split(long long tiles, int nchunks) {
  for (int size = MAX_SPLIT; size > 1; --size)
    if (size <= nchunks && tiles <= resident_clusters<K>(size)) return size;
  return 1;
}

}  // namespace rglru
