// RG-LRU forward and backward kernels for sm_100a.
//
// Work decomposition.  A CTA owns CH (64 or 32) adjacent channels of one batch row and walks the whole
// sequence in chunks of LANES*TS time-steps.  Inside a chunk the time axis is split over LANES (16 or 32)
// time-lanes, each thread scanning TS = 4 steps of CV = 4 channels in registers (level one), after which a
// few threads per channel chain the lane aggregates and the carry from the previous chunk through shared
// memory (level two: one serial chain of 16 for the 64-channel shape, four segments of eight joined by a
// small exchange for the 32-lane shape) and every lane applies its incoming state.  Chunks are staged through
// shared memory by TMA (cp.async.bulk.tensor, 3-D tiles [1, rows, channels]) in a multi-stage mbarrier
// pipeline; results are written back into the stage in place and leave through TMA stores.  The bulk copies
// are issued either by a producer warp or, for the bf16 backward, by one compute thread (SELF_ISSUE: eight
// warps leave every thread the registers it wants).  The 64-byte rows of 32-channel bf16 tiles are staged two to a
// 128-byte line through 5-D tensor maps (PAIRED), which halves the forward's shared-memory bank conflicts.  A bounds-checked plain-load staging path with the same
// arithmetic covers shapes TMA cannot address (D * element size not a multiple of 16 bytes).
//
// What bounds them (ncu on B200, bf16, B = 8, T = 2048, D = 1024): DRAM traffic equals the algorithmic bytes;
// no pipe is more than 40 % busy and 0.4 instructions issue per scheduler and cycle: with one (backward) or two
// (forward) CTAs per SM the kernels are bound by dependent-instruction latency inside a warp and by what
// happens outside the chunk loop, so the channel arithmetic is written on float2 pairs (one issue slot per two
// fp32 operations), transcendental work is kept to three or four MUFU operations per element, and the
// prologue (first loads issued before the per-channel rates are worked out, the first chunk prefetched into
// L2 before the dependency wait) and the epilogue (row sums folded by the last CTA with all loads in flight
// at once) are kept short.  Sixteen-warp variants with two steps per thread measured 15 % slower.
//
// The gate epilogue follows griffin/griffin.py:237-258 of the reference, the scan :280-286, the backward is
// the closed form of autograd over those lines with the capped sqrt slope of :59-65.  All arithmetic is fp32.
//
// Template switches of the two kernels (each a separate instantiation, so the plain kernels pay nothing for
// them):
//   CONV    the width-4 causal conv in front of the layer (:474-486) is applied while a chunk is loaded, from
//           an x tile with a three-row halo;
//   MERGE   the block's GeLU-branch product (:464, :520) is formed in the store stage and differentiated in
//           the backward's load stage;
//   GROUPED both gate pre-activations come from one [B, T, 2 D] tensor written by a single grouped GEMM (its columns
//           alternate between the gates in groups that divide the head width, so any head width will do), the
//           gate biases are added here, and the backward also returns their gradient (column sums of du);
//   PLAIN   no token flags and a whole number of chunks: the masked arithmetic is not compiled in.
// The file also holds the raw affine scan operator (triton_scan.py:274-276), the TMA-staged kernels of the
// conv alone, and the self-test of the bounded wait.

#include "rglru_scan.cuh"

namespace rglru {

// ======================================================================
// Forward
// ======================================================================

template <typename IO, int TS, int LANES, int CH, int NSTAGE, bool CONV = false, bool MERGE = false, bool SPLIT = false>
struct FwdSmem {
  static constexpr int TC = LANES * TS;
  static constexpr int TILE = TC * CH * sizeof(IO);
  static constexpr int HALO = CONV ? 3 * CH * sizeof(IO) : 0;   // three rows in front of the x tile
  static constexpr int TILEX = TILE + HALO;
  static constexpr int OFF_G = TILEX + 2 * TILE;                // GeLU-branch tile of the merged variant
  static constexpr int STAGE = TILEX + 2 * TILE + (MERGE ? TILE : 0);
  static constexpr int OFF_AGG = NSTAGE * STAGE;
  static constexpr int OFF_EIN = OFF_AGG + ChainSmem<LANES, CH>::AGG;
  // The 32-lane shape splits a channel's chain over SEGS threads (segment totals: one float2 per segment and channel).
  static constexpr int SEGS = (LANES == 32 && CH == 32) ? 4 : 1;
  static constexpr int OFF_SEG = OFF_EIN + ChainSmem<LANES, CH>::EIN;
  static constexpr int OFF_BAR = OFF_SEG + SEGS * CH * 8;   // full[NSTAGE], ready[NSTAGE], dead flag
  static constexpr int OFF_SPLIT = OFF_BAR + 2 * NSTAGE * 8 + 16;
  static constexpr int BYTES = OFF_SPLIT + (SPLIT ? static_cast<int>(sizeof(SplitSmem<CH>)) : 0);
};

// Threads [0, LANES*NCV) compute; with TMA one extra warp issues every bulk copy so that
// no compute warp ever waits on the copy engine's instruction latency.
// MERGE: the kernel also reads the pre-activation of the block's GeLU branch and writes
// h_t * gelu(branch_t) (griffin/griffin.py:464, 520 of the reference) instead of h_t.
template <typename IO, int TS, int LANES, int CH, int NSTAGE, bool USE_TMA, bool CONV, bool MERGE, bool GROUPED, bool PLAIN = false,
          bool CARRY = false, bool PAIRED = false, bool SPLIT = false>
__device__ __forceinline__ void rglru_fwd_body(const FwdMaps& maps, const ScanFwdArgs& p) {
  using SM = FwdSmem<IO, TS, LANES, CH, NSTAGE, CONV, MERGE, SPLIT>;
  static_assert(!CONV || (SM::HALO % 128 == 0), "the halo must keep the result rows 128-byte aligned for TMA");
  constexpr int NCV = CH / CV;
  constexpr int TC = SM::TC;
  constexpr int ROWB = CH * sizeof(IO);
  // PAIRED: 64-byte tile rows (32 bf16 channels) put the four time-lanes of a warp on the same sixteen banks.  The
  // tile is then staged through 5-D tensor maps that view time as (eighth, half, step), t = 8 q + 4 h + j, and lay
  // it out as [q][j][h][channels]: rows t and t + 4 share one 128-byte line, a thread's four steps are 128 bytes
  // apart, and two neighbouring time-lanes fill a line between them, so a warp's access touches every bank once.
  static_assert(!PAIRED || (USE_TMA && PLAIN && !CONV && !MERGE && !GROUPED && TS == 4 && ROWB == 64 && TC % 8 == 0),
                "paired rows: plain TMA-staged kernel on 64-byte rows only");
  constexpr int RSTEP = PAIRED ? 2 * ROWB : ROWB;
  constexpr int NCOMP = LANES * NCV;
  extern __shared__ __align__(128) uint8_t smem[];
  float2* agg = reinterpret_cast<float2*>(smem + SM::OFF_AGG);
  float* ein = reinterpret_cast<float*>(smem + SM::OFF_EIN);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + SM::OFF_BAR);
  uint64_t* ready = full + NSTAGE;
  volatile int* dead = reinterpret_cast<volatile int*>(ready + NSTAGE);

  const int tid = threadIdx.x;
  const int lane_t = tid / NCV;
  const int vec = tid % NCV;
  const int b = blockIdx.y;
  const int d0 = blockIdx.x * CH;
  const int nchunks = (p.T + TC - 1) / TC;
  const int nsave = (p.T + SAVE_EVERY - 1) / SAVE_EVERY;
  // SPLIT: this CTA's chunks are rank, rank + nranks, ...; every CTA of the cluster goes through `rounds` rounds.
  static_assert(!SPLIT || (USE_TMA && !CONV && !CARRY), "the time split exists for the TMA-staged scan kernels");
  SplitChain<CH> split;
  if constexpr (SPLIT) split.init(reinterpret_cast<SplitSmem<CH>*>(smem + SM::OFF_SPLIT));
  const int rank = SPLIT ? static_cast<int>(split.rank) : 0, nranks = SPLIT ? static_cast<int>(split.size) : 1;
  const int rounds = SPLIT ? (nchunks + nranks - 1) / nranks : nchunks;
  const int mine = SPLIT ? (nchunks - rank + nranks - 1) / nranks : nchunks;   // chunks this CTA loads and stores
  static_assert(!GROUPED || USE_TMA, "the grouped gate layout is staged by TMA only");
  const GateTile<GROUPED, CH> gate(d0, p.gate_bw);

  auto issue = [&](int it) {
    const int sidx = it % NSTAGE;
    const int k = it * nranks + rank;
    uint8_t* st = smem + sidx * SM::STAGE;
    mbar_expect_tx(&full[sidx], SM::STAGE);
    if constexpr (PAIRED) {
      tma_load_5d(st, &maps.x, d0, 0, 0, k * (TC / 8), b, &full[sidx]);
      tma_load_5d(st + SM::TILEX, &maps.ur, d0, 0, 0, k * (TC / 8), b, &full[sidx]);
      tma_load_5d(st + SM::TILEX + SM::TILE, &maps.ui, d0, 0, 0, k * (TC / 8), b, &full[sidx]);
    } else {
      tma_load_3d(st, &maps.x, d0, k * TC - (CONV ? 3 : 0), b, &full[sidx]);   // rows before t = 0 read as zero
      gate.load(st + SM::TILEX, &maps.ur, 0, k * TC, b, &full[sidx]);
      gate.load(st + SM::TILEX + SM::TILE, &maps.ui, 1, k * TC, b, &full[sidx]);
      if (MERGE) tma_load_3d(st + SM::OFF_G, &maps.g, d0, k * TC, b, &full[sidx]);
    }
  };
  // Set-up by the thread that will issue the bulk copies, published by one early CTA barrier; after it the
  // producer warp and the compute warps go their own ways (the compute warps vote among themselves), so the
  // first loads are issued while the per-channel rates are worked out and nobody waits for the issuing thread.
  pdl_launch_dependents();
  if (USE_TMA ? (tid == NCOMP) : (tid == 0)) {
    *dead = 0;
    if (USE_TMA) {
      for (int s = 0; s < NSTAGE; ++s) { mbar_init(&full[s], 1); mbar_init(&ready[s], NCOMP / 32); }
      if constexpr (SPLIT) { mbar_init(&split.sm->bar[0], 1); mbar_init(&split.sm->bar[1], 1); }
      mbar_fence_init();
      prefetch_map(&maps.x); prefetch_map(&maps.ur); prefetch_map(&maps.ui); prefetch_map(&maps.y);
      if (MERGE) prefetch_map(&maps.g);
      // While the kernel in front of this one on the stream drains, pull the first chunk towards L2.
      if constexpr (PAIRED) {
        tma_prefetch_5d(&maps.x, d0, 0, 0, rank * (TC / 8), b);
        tma_prefetch_5d(&maps.ur, d0, 0, 0, rank * (TC / 8), b);
        tma_prefetch_5d(&maps.ui, d0, 0, 0, rank * (TC / 8), b);
      } else {
        tma_prefetch_3d(&maps.x, d0, rank * TC - (CONV ? 3 : 0), b);
        gate.prefetch(&maps.ur, 0, rank * TC, b);
        gate.prefetch(&maps.ui, 1, rank * TC, b);
        if (MERGE) tma_prefetch_3d(&maps.g, d0, rank * TC, b);
      }
    }
  }
  if constexpr (SPLIT) cluster_sync_all();   // the barriers of every CTA are there before anybody sends
  else __syncthreads();
  pdl_wait();   // nothing above touches global memory; everything below may depend on the previous kernel

  if (USE_TMA && tid >= NCOMP) {
    // ---- producer warp: loads run NSTAGE-1 chunks ahead; a stage is refilled as soon as the
    // store of the results written into it has drained from shared memory.
    if (tid == NCOMP) {
      // Every CTA of the grid starts at once and asks for NSTAGE chunks; the first chunk is asked for alone and
      // the rest once it has landed, so that no CTA's first chunk queues behind other CTAs' later ones.
      issue(0);
      mbar_wait_or_flag(&full[0], 0, dead, p.status, DEV_TIMEOUT_LOAD);
      for (int it = 1; it < NSTAGE && it < mine; ++it) issue(it);
      for (int it = 0; it < mine; ++it) {
        const int sidx = it % NSTAGE, k = it * nranks + rank;
        mbar_wait_or_flag(&ready[sidx], (it / NSTAGE) & 1, dead, p.status, DEV_TIMEOUT_STORE);
        if constexpr (PAIRED) tma_store_5d(&maps.y, smem + sidx * SM::STAGE, d0, 0, 0, k * (TC / 8), b);
        else if (!CARRY) tma_store_3d(&maps.y, smem + sidx * SM::STAGE + SM::HALO, d0, k * TC, b);
        tma_commit();
        if (it + NSTAGE < mine) {
          tma_wait_read<0>();
          issue(it + NSTAGE);
        }
      }
      tma_wait_all<0>();
    }
    if constexpr (SPLIT) { __syncwarp(); cluster_sync_all(); }
    return;
  }

  float2 K[2];
  {
    const int d = d0 + vec * CV;
    K[0] = make_float2(decay_rate(p.lambda, d, p.D, p.c), decay_rate(p.lambda, d + 1, p.D, p.c));
    K[1] = make_float2(decay_rate(p.lambda, d + 2, p.D, p.c), decay_rate(p.lambda, d + 3, p.D, p.c));
  }
  const bool poly = bar_compute_and(NCOMP, fmaxf(fmaxf(K[0].x, K[0].y), fmaxf(K[1].x, K[1].y)) <= -POLY_RANGE);

  if (blockIdx.x == 0 && blockIdx.y == 0 && tid == 0 && p.ticket) *p.ticket = 0u;   // consumed by the backward kernel

  ConvTaps ct;
  if (CONV) load_taps(p.conv_w, p.conv_b, d0 + vec * CV, p.D, ct);
  GateBias gb;
  if (GROUPED) load_gate_bias<sizeof(IO) == 2>(p.gate_bias, d0 + vec * CV, p.D, p.gate_bw, gb);

  // Level-two chain: SEGS threads per channel (thread tid: channel d0 + tid % CH, lane segment tid / CH), each
  // of which carries the channel's state across chunks (identical copies).
  constexpr int SEGS = SM::SEGS, SEGL = LANES / SEGS;
  static_assert(SEGS * CH <= NCOMP && (SEGS * CH) % 32 == 0, "chain threads are whole warps of the compute group");
  float2* segtot = reinterpret_cast<float2*>(smem + SM::OFF_SEG);
  const bool chain_thread = tid < SEGS * CH;
  const int cch = tid % CH, seg = tid / CH;
  float carry = 0.0f;
  const int dch = d0 + cch;
  if (chain_thread && dch < p.D && p.h0) carry = p.h0[static_cast<size_t>(b) * p.D + dch];
  // Product of the decays over the sequence: with the final state it is the affine map h0 -> h_last of this
  // call, which is what a caller that splits one sequence over several calls (or GPUs) needs to chain them.
  const bool want_prod = p.decay_prod != nullptr;
  float prod_all = 1.0f;

  const int off0 = PAIRED ? ((lane_t >> 1) * TS) * RSTEP + (lane_t & 1) * ROWB + vec * Pack<IO>::BYTES
                          : (lane_t * TS) * ROWB + vec * Pack<IO>::BYTES;

  for (int it = 0; it < rounds; ++it) {
    const int k = it * nranks + rank;
    const bool idle = SPLIT && it >= mine;     // last round: no chunk left for this CTA, it only takes part in the exchange
    if constexpr (SPLIT) { if (tid == 0) split.arm(it); }
    const int stage = USE_TMA ? (it % NSTAGE) : 0;
    uint8_t* tiles = smem + stage * SM::STAGE;
    const int t0 = k * TC;
    uint32_t fl[(TS + 3) / 4];
    const bool masked = !PLAIN && ((p.tok != nullptr) || (t0 + TC > p.T));
    if (masked) load_flags<TS>(p.tok, b, p.T, t0 + lane_t * TS, fl);

    float2 P[TS][2], S[TS][2];
    if (!idle) {
    if (USE_TMA) {
      mbar_wait_or_flag(&full[stage], (it / NSTAGE) & 1, dead, p.status, DEV_TIMEOUT_LOAD);
    } else {
      tile_load_plain<IO, CH>(tiles, p.x, b, t0 - (CONV ? 3 : 0), d0, TC + (CONV ? 3 : 0), p.T, p.D);
      tile_load_plain<IO, CH>(tiles + SM::TILEX, p.ur, b, t0, d0, TC, p.T, p.D);
      tile_load_plain<IO, CH>(tiles + SM::TILEX + SM::TILE, p.ui, b, t0, d0, TC, p.T, p.D);
      if (MERGE) tile_load_plain<IO, CH>(tiles + SM::OFF_G, p.g, b, t0, d0, TC, p.T, p.D);
      bar_compute(NCOMP);
    }

    const uint8_t* tx = tiles;
    const uint8_t* tr = tiles + SM::TILEX;
    const uint8_t* ti = tiles + SM::TILEX + SM::TILE;
    float2 hist_v[3][2];
    const float2 (*hist)[2] = nullptr;
    if (CONV && k == 0 && lane_t == 0 && p.conv_state) {   // history carried from an earlier call
      load_hist<IO>(p.conv_state, b, d0 + vec * CV, p.D, hist_v);
      hist = hist_v;
    }
    if (masked && any_flag(fl)) {
      if (poly) fwd_local<IO, TS, CH, true, true, CONV, GROUPED, RSTEP>(tx, tr, ti, off0, K, fl, ct, hist, gb, P, S);
      else fwd_local<IO, TS, CH, true, false, CONV, GROUPED, RSTEP>(tx, tr, ti, off0, K, fl, ct, hist, gb, P, S);
    } else {
      if (poly) fwd_local<IO, TS, CH, false, true, CONV, GROUPED, RSTEP>(tx, tr, ti, off0, K, fl, ct, hist, gb, P, S);
      else fwd_local<IO, TS, CH, false, false, CONV, GROUPED, RSTEP>(tx, tr, ti, off0, K, fl, ct, hist, gb, P, S);
    }
    {
      float4* dst = reinterpret_cast<float4*>(agg + lane_t * CH + vec * CV);
      dst[0] = make_float4(P[TS - 1][0].x, S[TS - 1][0].x, P[TS - 1][0].y, S[TS - 1][0].y);
      dst[1] = make_float4(P[TS - 1][1].x, S[TS - 1][1].x, P[TS - 1][1].y, S[TS - 1][1].y);
    }
    }
    bar_compute(NCOMP);

    if (chain_thread) {
      float2 ag[SEGL];
#pragma unroll
      for (int j = 0; j < SEGL; ++j) ag[j] = idle ? make_float2(1.0f, 0.0f) : agg[(seg * SEGL + j) * CH + cch];
      auto emit = [&](int lane, float e) {       // state entering a lane; every SAVE_EVERY steps also kept for the backward
        if (((lane * TS) % SAVE_EVERY) == 0) {
          const int t = t0 + lane * TS;
          if (p.states && t < p.T && dch < p.D)
            p.states[(static_cast<size_t>(b) * nsave + t / SAVE_EVERY) * p.D + dch] = e;
        }
        ein[lane * CH + cch] = e;
      };
      if (SEGS == 1 && !SPLIT) {
        float e = carry;
#pragma unroll
        for (int j = 0; j < LANES; ++j) {
          emit(j, e);
          e = fmaf(ag[j].x, e, ag[j].y);
        }
        carry = e;
        if (want_prod) {
#pragma unroll
          for (int j = 0; j < LANES; ++j) prod_all *= ag[j].x;
        }
      } else {
        // Each thread composes its segment from the identity, keeping the map (pp, sp) that takes the state
        // entering the segment to the state entering each of its lanes; the segment totals are exchanged through
        // shared memory and every thread chains the few totals in front of it.
        float pp[SEGL], sp[SEGL];
        float pa = 1.0f, sa = 0.0f;
#pragma unroll
        for (int j = 0; j < SEGL; ++j) {
          pp[j] = pa;
          sp[j] = sa;
          sa = fmaf(ag[j].x, sa, ag[j].y);
          pa *= ag[j].x;
        }
        float enter;
        if constexpr (!SPLIT) {
          segtot[seg * CH + cch] = make_float2(pa, sa);
          bar_chain(SEGS * CH);
          float e = carry;
          enter = carry;
#pragma unroll
          for (int sgm = 0; sgm < SEGS; ++sgm) {
            const float2 tot = segtot[sgm * CH + cch];
            if (sgm == seg) enter = e;
            e = fmaf(tot.x, e, tot.y);
            prod_all *= tot.x;
          }
          carry = e;
        } else {
          float2 before = make_float2(1.0f, 0.0f), tot = make_float2(pa, sa);   // map of the segments before this one / of the chunk
          if constexpr (SEGS > 1) {
            segtot[seg * CH + cch] = tot;
            bar_chain(SEGS * CH);
            tot = make_float2(1.0f, 0.0f);
#pragma unroll
            for (int sgm = 0; sgm < SEGS; ++sgm) {
              const float2 t = segtot[sgm * CH + cch];
              if (sgm == seg) before = tot;
              tot = make_float2(tot.x * t.x, fmaf(t.x, tot.y, t.y));
            }
          }
          split.send(it, cch, tot, seg, SEGS);
          enter = fmaf(before.x, split.receive(it, cch, carry, prod_all, dead, p.status), before.y);
        }
        if (!idle) {
#pragma unroll
          for (int j = 0; j < SEGL; ++j) emit(seg * SEGL + j, fmaf(pp[j], enter, sp[j]));
        }
      }
    }
    bar_compute(NCOMP);
    if (idle) break;

    {
      const float4 e4 = *reinterpret_cast<const float4*>(ein + lane_t * CH + vec * CV);
      const float2 e[2] = {make_float2(e4.x, e4.y), make_float2(e4.z, e4.w)};
      uint8_t* ty = tiles + SM::HALO;  // y overwrites the x tile in place (past its halo rows)
#pragma unroll
      for (int st = 0; st < TS; ++st) {
        float2 yv[2];
#pragma unroll
        for (int cp = 0; cp < 2; ++cp) yv[cp] = fma2(P[st][cp], e[cp], S[st][cp]);
        if constexpr (SPLIT) {   // the final state is the last step's output to the bit, not the folded carry
          if (p.h_last && t0 + lane_t * TS + st == p.T - 1) {
            float* hl = p.h_last + static_cast<size_t>(b) * p.D + d0 + vec * CV;
            const float v[4] = {yv[0].x, yv[0].y, yv[1].x, yv[1].y};
#pragma unroll
            for (int ch = 0; ch < 4; ++ch)
              if (d0 + vec * CV + ch < p.D) hl[ch] = v[ch];
          }
        }
        if (MERGE) {
          float2 gv[2];
          Pack<IO>::unpack2(Pack<IO>::load(tiles + SM::OFF_G + off0 + st * RSTEP), gv);
#pragma unroll
          for (int cp = 0; cp < 2; ++cp) yv[cp] = mul2(yv[cp], mul2(gv[cp], gelu_sigmoid2<sizeof(IO) == 2>(gv[cp])));
        }
        Pack<IO>::store2(ty + off0 + st * RSTEP, yv);
      }
    }
    if (USE_TMA) {
      fence_async_smem();        // make this thread's results visible to the bulk store
      __syncwarp();
      if ((tid & 31) == 0) mbar_arrive(&ready[stage]);   // one arrival per warp
    } else {
      bar_compute(NCOMP);
      if (!CARRY) tile_store_plain<IO, CH>(tiles + SM::HALO, p.y, b, t0, d0, TC, p.T, p.D);
      bar_compute(NCOMP);
    }
  }
  if constexpr (SPLIT) {
    __syncwarp();
    cluster_sync_all();        // no CTA leaves while another may still send to it
    if (rank != 0) return;
  }
  if (!SPLIT && tid < CH && dch < p.D && p.h_last) p.h_last[static_cast<size_t>(b) * p.D + dch] = carry;   // segment 0's copy
  if (tid < CH && dch < p.D && want_prod) p.decay_prod[static_cast<size_t>(b) * p.D + dch] = prod_all;
}

// PLAIN: no token flags and a whole number of chunks, so the masked arithmetic is not compiled in.
// CARRY: the carry-only pass of a time-split sequence: no output tensor, nothing is stored but h_last and decay_prod.
// PAIRED: 64-byte tile rows staged two to a 128-byte line through 5-D tensor maps (see rglru_fwd_body).
template <typename IO, int TS, int LANES, int CH, int NSTAGE, bool USE_TMA, bool CONV, bool MERGE, bool GROUPED, bool PLAIN = false,
          bool CARRY = false, bool PAIRED = false, bool SPLIT = false>
__global__ void __launch_bounds__(LANES*(CH / CV) + (USE_TMA ? 32 : 0))
    rglru_fwd_kernel(const __grid_constant__ FwdMaps maps, const ScanFwdArgs p) {
  rglru_fwd_body<IO, TS, LANES, CH, NSTAGE, USE_TMA, CONV, MERGE, GROUPED, PLAIN, CARRY, PAIRED, SPLIT>(maps, p);
}
// The same kernel capped at 96 registers, which lets two 9-warp CTAs share an SM's register files (five warps
// on one scheduler partition).  Used for the merged / grouped variants, which otherwise take about 112.
template <typename IO, int TS, int LANES, int CH, int NSTAGE, bool USE_TMA, bool CONV, bool MERGE, bool GROUPED, bool PLAIN = false,
          bool SPLIT = false>
__global__ void __maxnreg__(96)
    rglru_fwd_kernel_capped(const __grid_constant__ FwdMaps maps, const ScanFwdArgs p) {
  rglru_fwd_body<IO, TS, LANES, CH, NSTAGE, USE_TMA, CONV, MERGE, GROUPED, PLAIN, false, false, SPLIT>(maps, p);
}

// ======================================================================
// Backward
// ======================================================================

template <typename IO, int TS, int LANES, int CH, int NSTAGE, bool CONV = false, bool MERGE = false, bool SPLIT = false>
struct BwdSmem {
  static constexpr int TC = LANES * TS;
  static constexpr int TILE = TC * CH * sizeof(IO);
  static constexpr int HALO = CONV ? 3 * CH * sizeof(IO) : 0;   // three rows in front of the x tile
  static constexpr int TILEX = TILE + HALO;
  static constexpr int OFF_X = TILE, OFF_UR = TILE + TILEX, OFF_UI = 2 * TILE + TILEX;   // after the dy tile
  static constexpr int OFF_G = 3 * TILE + TILEX;                // GeLU-branch tile of the merged variant
  static constexpr int STAGE = 3 * TILE + TILEX + (MERGE ? TILE : 0);
  // Lane aggregates as three float planes [LANES][CH]: decay product, local state, local reverse carry.
  static constexpr int PLANE = LANES * CH * 4;
  static constexpr int OFF_AGGP = NSTAGE * STAGE;
  static constexpr int OFF_AGGS = OFF_AGGP + PLANE;
  static constexpr int OFF_AGGC = OFF_AGGS + PLANE;
  static constexpr int OFF_EINF = OFF_AGGC + PLANE;
  static constexpr int OFF_EINR = OFF_EINF + PLANE;
  static constexpr int OFF_BAR = OFF_EINR + PLANE;   // full[NSTAGE], ready[NSTAGE], dead flag
  static constexpr int OFF_SPLIT = OFF_BAR + 2 * NSTAGE * 8 + 16;
  static constexpr int BYTES = OFF_SPLIT + (SPLIT ? static_cast<int>(sizeof(SplitSmem<CH>)) : 0);
};

// SELF_ISSUE: no producer warp.  One thread of the last compute warp (not a chain thread) issues the bulk
// copies right after the first barrier of a chunk: by then every thread has finished, and fenced, the results
// of the chunk before, so that chunk's tiles can leave and the stage of the chunk before it, whose store has
// been read out of shared memory by now, can be refilled.  No barrier is added; loads run NSTAGE - 2 chunks
// ahead.  A whole number of warps per scheduler partition leaves every thread 128 registers at 512 threads.
// PLAIN: the caller passed no token flags and the sequence is a whole number of chunks, so no step is ever
// masked; the masked arithmetic is not compiled in (half the code, and registers allotted for this path alone).
// CARRY: the carry-only pass of a time-split sequence: no gradient tensors, nothing is stored but dh0.
template <typename IO, int TS, int LANES, int CH, int NSTAGE, bool USE_TMA, bool CONV, bool MERGE, bool GROUPED,
          bool SELF_ISSUE = false, bool PLAIN = false, bool CARRY = false, bool SPLIT = false>
__global__ void __launch_bounds__(LANES*(CH / CV) + ((USE_TMA && !SELF_ISSUE) ? 32 : 0),
                                  (SELF_ISSUE && CH == 32) ? 2 : 1)
    rglru_bwd_kernel(const __grid_constant__ BwdMaps maps, const ScanBwdArgs p) {
  using SM = BwdSmem<IO, TS, LANES, CH, NSTAGE, CONV, MERGE, SPLIT>;
  static_assert(!CONV || (SM::HALO % 128 == 0), "the halo must keep the result rows 128-byte aligned for TMA");
  constexpr int NCV = CH / CV;
  constexpr int TC = SM::TC;
  static_assert(TC % SAVE_EVERY == 0, "backward chunks must start on a saved state");
  static_assert(!SELF_ISSUE || !USE_TMA || NSTAGE >= 3, "without a producer warp a stage is refilled two chunks after its use");
  constexpr int ROWB = CH * sizeof(IO);
  constexpr int NCOMP = LANES * NCV;
  extern __shared__ __align__(128) uint8_t smem[];
  float* aggP = reinterpret_cast<float*>(smem + SM::OFF_AGGP);
  float* aggS = reinterpret_cast<float*>(smem + SM::OFF_AGGS);
  float* aggC = reinterpret_cast<float*>(smem + SM::OFF_AGGC);
  float* einF = reinterpret_cast<float*>(smem + SM::OFF_EINF);
  float* einR = reinterpret_cast<float*>(smem + SM::OFF_EINR);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + SM::OFF_BAR);
  uint64_t* ready = full + NSTAGE;
  volatile int* dead = reinterpret_cast<volatile int*>(ready + NSTAGE);

  const int tid = threadIdx.x;
  const int lane_t = tid / NCV;
  const int vec = tid % NCV;
  const int b = blockIdx.y;
  const int d0 = blockIdx.x * CH;
  const int nchunks = (p.T + TC - 1) / TC;
  const int nsave = (p.T + SAVE_EVERY - 1) / SAVE_EVERY;
  // SPLIT: in processing order (from the end of the sequence) this CTA's chunks are rank, rank + nranks, ...
  static_assert(!SPLIT || (USE_TMA && !CONV && !CARRY), "the time split exists for the TMA-staged scan kernels");
  SplitChain<CH> split;
  if constexpr (SPLIT) split.init(reinterpret_cast<SplitSmem<CH>*>(smem + SM::OFF_SPLIT));
  const int rank = SPLIT ? static_cast<int>(split.rank) : 0, nranks = SPLIT ? static_cast<int>(split.size) : 1;
  const int rounds = SPLIT ? (nchunks + nranks - 1) / nranks : nchunks;
  const int mine = SPLIT ? (nchunks - rank + nranks - 1) / nranks : nchunks;   // chunks this CTA loads and stores
  static_assert(!GROUPED || USE_TMA, "the grouped gate layout is staged by TMA only");
  const GateTile<GROUPED, CH> gate(d0, p.gate_bw);

  auto issue = [&](int q) {  // this CTA's q-th chunk in processing order, which runs from the end of the sequence
    const int k = nchunks - 1 - (q * nranks + rank);
    const int sidx = q % NSTAGE;
    uint8_t* st = smem + sidx * SM::STAGE;
    mbar_expect_tx(&full[sidx], SM::STAGE);
    tma_load_3d(st, &maps.dy, d0, k * TC, b, &full[sidx]);
    tma_load_3d(st + SM::OFF_X, &maps.x, d0, k * TC - (CONV ? 3 : 0), b, &full[sidx]);
    gate.load(st + SM::OFF_UR, &maps.ur, 0, k * TC, b, &full[sidx]);
    gate.load(st + SM::OFF_UI, &maps.ui, 1, k * TC, b, &full[sidx]);
    if (MERGE) tma_load_3d(st + SM::OFF_G, &maps.g, d0, k * TC, b, &full[sidx]);
  };
  auto store = [&](int q) {
    const int k = nchunks - 1 - (q * nranks + rank);
    uint8_t* st = smem + (q % NSTAGE) * SM::STAGE;
    if (!CARRY) {
      tma_store_3d(&maps.dx, st + SM::OFF_X + SM::HALO, d0, k * TC, b);
      gate.store(&maps.dur, st + SM::OFF_UR, 0, k * TC, b);
      gate.store(&maps.dui, st + SM::OFF_UI, 1, k * TC, b);
      if (MERGE) tma_store_3d(&maps.dg, st + SM::OFF_G, d0, k * TC, b);
    }
    tma_commit();
  };
  // Set-up by the thread that will issue the bulk copies (the producer warp's first lane, or with SELF_ISSUE
  // the first lane of the last compute warp), published by one early CTA barrier; after it the producer warp
  // and the compute warps go their own ways (the compute warps vote among themselves), so the first loads are
  // issued while the per-channel rates are worked out.
  const bool issuer = USE_TMA && tid == (SELF_ISSUE ? NCOMP - 32 : NCOMP);
  const bool self_issuer = SELF_ISSUE && issuer;
  pdl_launch_dependents();
  if (USE_TMA ? issuer : (tid == 0)) {
    *dead = 0;
    if (USE_TMA) {
      for (int s = 0; s < NSTAGE; ++s) { mbar_init(&full[s], 1); mbar_init(&ready[s], NCOMP / 32); }
      if constexpr (SPLIT) { mbar_init(&split.sm->bar[0], 1); mbar_init(&split.sm->bar[1], 1); }
      mbar_fence_init();
      prefetch_map(&maps.dy); prefetch_map(&maps.x); prefetch_map(&maps.ur); prefetch_map(&maps.ui);
      prefetch_map(&maps.dx); prefetch_map(&maps.dur); prefetch_map(&maps.dui);
      if (MERGE) { prefetch_map(&maps.g); prefetch_map(&maps.dg); }
      // While the kernel in front of this one on the stream drains, pull the first chunk (the last in time)
      // towards L2.
      const int kl = nchunks - 1 - rank;
      tma_prefetch_3d(&maps.dy, d0, kl * TC, b);
      tma_prefetch_3d(&maps.x, d0, kl * TC - (CONV ? 3 : 0), b);
      gate.prefetch(&maps.ur, 0, kl * TC, b);
      gate.prefetch(&maps.ui, 1, kl * TC, b);
      if (MERGE) tma_prefetch_3d(&maps.g, d0, kl * TC, b);
    }
  }
  if constexpr (SPLIT) cluster_sync_all();   // the barriers of every CTA are there before anybody sends
  else __syncthreads();
  pdl_wait();   // nothing above touches global memory; everything below may depend on the previous kernel

  if (USE_TMA && !SELF_ISSUE && tid >= NCOMP) {
    // ---- producer warp (chunks are walked from the end of the sequence to its start)
    if (tid == NCOMP) {
      // the first chunk is asked for alone, the rest once it has landed (see the forward kernel)
      issue(0);
      mbar_wait_or_flag(&full[0], 0, dead, p.status, DEV_TIMEOUT_LOAD);
      for (int q = 1; q < NSTAGE && q < mine; ++q) issue(q);
      for (int q = 0; q < mine; ++q) {
        const int sidx = q % NSTAGE;
        mbar_wait_or_flag(&ready[sidx], (q / NSTAGE) & 1, dead, p.status, DEV_TIMEOUT_STORE);
        store(q);
        if (q + NSTAGE < mine) {
          tma_wait_read<0>();
          issue(q + NSTAGE);
        }
      }
      tma_wait_all<0>();
    }
    if constexpr (SPLIT) { __syncwarp(); cluster_sync_all(); }
    return;
  }

  if (self_issuer) issue(0);    // the first chunk before this thread's share of the prologue, the rest after it
  float2 K[2];
  {
    const int d = d0 + vec * CV;
    K[0] = make_float2(decay_rate(p.lambda, d, p.D, p.c), decay_rate(p.lambda, d + 1, p.D, p.c));
    K[1] = make_float2(decay_rate(p.lambda, d + 2, p.D, p.c), decay_rate(p.lambda, d + 3, p.D, p.c));
  }
  const bool poly = bar_compute_and(NCOMP, fmaxf(fmaxf(K[0].x, K[0].y), fmaxf(K[1].x, K[1].y)) <= -POLY_RANGE);

  // Threads 0..63 chain the forward lane aggregates, threads 64..127 the reverse ones.
  const int cch = tid & (CH - 1);
  const int dch = d0 + cch;
  const bool fwd_chain = tid < CH;
  const bool rev_chain = tid >= CH && tid < 2 * CH;
  float carry_rev = 0.0f;
  if (rev_chain && dch < p.D && p.dh_last) carry_rev = p.dh_last[static_cast<size_t>(b) * p.D + dch];

  ConvTaps ct;
  if (CONV) load_taps(p.conv_w, p.conv_b, d0 + vec * CV, p.D, ct);
  GateBias gb;
  if (GROUPED) load_gate_bias<sizeof(IO) == 2>(p.gate_bias, d0 + vec * CV, p.D, p.gate_bw, gb);

  float2 dlam[2] = {f2(0.0f), f2(0.0f)};
  float2 dsr[2] = {f2(0.0f), f2(0.0f)}, dsi[2] = {f2(0.0f), f2(0.0f)};   // grouped layout: sums over time of du_r, du_i
  const int off0 = (lane_t * TS) * ROWB + vec * Pack<IO>::BYTES;

  for (int q = 0; q < rounds; ++q) {
    const int k = nchunks - 1 - (q * nranks + rank);
    const bool idle = SPLIT && q >= mine;     // last round: no chunk left for this CTA, it only takes part in the exchange
    if constexpr (SPLIT) { if (tid == 0) split.arm(q); }
    const int stage = USE_TMA ? (q % NSTAGE) : 0;
    uint8_t* tiles = smem + stage * SM::STAGE;
    const int t0 = k * TC;
    uint32_t fl[(TS + 3) / 4];
    const bool masked = !PLAIN && ((p.tok != nullptr) || (t0 + TC > p.T));
    if (masked && !idle) load_flags<TS>(p.tok, b, p.T, t0 + lane_t * TS, fl);

    // State entering this chunk (saved by the forward kernel; chunk 0 starts from h0).
    float enter = 0.0f;
    if (fwd_chain && dch < p.D && !idle) {
      if (k == 0) enter = p.h0 ? p.h0[static_cast<size_t>(b) * p.D + dch] : 0.0f;
      else enter = p.states[(static_cast<size_t>(b) * nsave + t0 / SAVE_EVERY) * p.D + dch];
    }

    BwdRegs<IO, TS> R;
    bool flagged = false;
    if (!idle) {
    if (USE_TMA) {
      mbar_wait_or_flag(&full[stage], (q / NSTAGE) & 1, dead, p.status, DEV_TIMEOUT_LOAD);
      if (self_issuer && q == 0)      // the first chunk was asked for alone; now that it has landed, the rest
        for (int qq = 1; qq < NSTAGE && qq < mine; ++qq) issue(qq);
    } else {
      tile_load_plain<IO, CH>(tiles, p.dy, b, t0, d0, TC, p.T, p.D);
      tile_load_plain<IO, CH>(tiles + SM::OFF_X, p.x, b, t0 - (CONV ? 3 : 0), d0, TC + (CONV ? 3 : 0), p.T, p.D);
      tile_load_plain<IO, CH>(tiles + SM::OFF_UR, p.ur, b, t0, d0, TC, p.T, p.D);
      tile_load_plain<IO, CH>(tiles + SM::OFF_UI, p.ui, b, t0, d0, TC, p.T, p.D);
      if (MERGE) tile_load_plain<IO, CH>(tiles + SM::OFF_G, p.g, b, t0, d0, TC, p.T, p.D);
      bar_compute(NCOMP);
    }

    float2 prod[2], sfwd[2], crev[2];
    flagged = masked && any_flag(fl);
    {
      uint8_t* tdy = tiles;
      uint8_t* tg = tiles + SM::OFF_G;
      const uint8_t* tx = tiles + SM::OFF_X;
      const uint8_t* tr = tiles + SM::OFF_UR;
      const uint8_t* ti = tiles + SM::OFF_UI;
      float2 hist_v[3][2];
      const float2 (*hist)[2] = nullptr;
      if (CONV && k == 0 && lane_t == 0 && p.conv_state) {
        load_hist<IO>(p.conv_state, b, d0 + vec * CV, p.D, hist_v);
        hist = hist_v;
      }
      if (flagged) {
        if (poly) bwd_local<IO, TS, CH, true, true, CONV, MERGE, GROUPED>(tdy, tg, tx, tr, ti, off0, K, fl, ct, hist, gb, R, prod, sfwd, crev);
        else bwd_local<IO, TS, CH, true, false, CONV, MERGE, GROUPED>(tdy, tg, tx, tr, ti, off0, K, fl, ct, hist, gb, R, prod, sfwd, crev);
      } else {
        if (poly) bwd_local<IO, TS, CH, false, true, CONV, MERGE, GROUPED>(tdy, tg, tx, tr, ti, off0, K, fl, ct, hist, gb, R, prod, sfwd, crev);
        else bwd_local<IO, TS, CH, false, false, CONV, MERGE, GROUPED>(tdy, tg, tx, tr, ti, off0, K, fl, ct, hist, gb, R, prod, sfwd, crev);
      }
    }
    {
      const int ao = lane_t * CH + vec * CV;
      *reinterpret_cast<float4*>(aggP + ao) = make_float4(prod[0].x, prod[0].y, prod[1].x, prod[1].y);
      *reinterpret_cast<float4*>(aggS + ao) = make_float4(sfwd[0].x, sfwd[0].y, sfwd[1].x, sfwd[1].y);
      *reinterpret_cast<float4*>(aggC + ao) = make_float4(crev[0].x, crev[0].y, crev[1].x, crev[1].y);
    }
    }
    bar_compute(NCOMP);
    if (self_issuer && q >= 1) {
      store(q - 1);
      if (q >= 2 && q - 2 + NSTAGE < mine) {
        tma_wait_read<1>();      // all but the store just committed have been read out: the stage of chunk q-2 is free
        issue(q - 2 + NSTAGE);
      }
    }

    if ((fwd_chain && !idle) || rev_chain) {
      const float* plane = fwd_chain ? aggS : aggC;
      float* ein = fwd_chain ? einF : einR;
      float ap[LANES], as[LANES];
#pragma unroll
      for (int j = 0; j < LANES; ++j) { ap[j] = aggP[j * CH + cch]; as[j] = plane[j * CH + cch]; }
      if (fwd_chain) {
        float e = enter;
#pragma unroll
        for (int j = 0; j < LANES; ++j) {
          ein[j * CH + cch] = e;
          e = fmaf(ap[j], e, as[j]);
        }
      } else if constexpr (!SPLIT) {
        float e = carry_rev;
#pragma unroll
        for (int j = LANES - 1; j >= 0; --j) {
          ein[j * CH + cch] = e;
          e = fmaf(ap[j], e, as[j]);
        }
        carry_rev = e;
      } else {
        // Compose the chunk from the identity, leaving in (ap, as) the map that takes the carry entering the chunk
        // (at its end) to the carry entering each lane.
        float pa = 1.0f, sa = 0.0f, unused = 1.0f;
        if (!idle) {
#pragma unroll
          for (int j = LANES - 1; j >= 0; --j) {
            const float pj = ap[j], sj = as[j];
            ap[j] = pa;
            as[j] = sa;
            sa = fmaf(pj, sa, sj);
            pa *= pj;
          }
        }
        split.send(q, cch, make_float2(pa, sa), 0, 1);
        const float e = split.receive(q, cch, carry_rev, unused, dead, p.status);
        if (!idle) {
#pragma unroll
          for (int j = 0; j < LANES; ++j) ein[j * CH + cch] = fmaf(ap[j], e, as[j]);
        }
      }
    }
    bar_compute(NCOMP);
    if (idle) break;

    {
      const float4 f4 = *reinterpret_cast<const float4*>(einF + lane_t * CH + vec * CV);
      const float4 r4 = *reinterpret_cast<const float4*>(einR + lane_t * CH + vec * CV);
      const float2 hin[2] = {make_float2(f4.x, f4.y), make_float2(f4.z, f4.w)};
      const float2 cin[2] = {make_float2(r4.x, r4.y), make_float2(r4.z, r4.w)};
      if (flagged) bwd_apply<IO, TS, CH, true, CONV, MERGE, GROUPED>(tiles, SM::OFF_X + SM::HALO, SM::OFF_UR, SM::OFF_UI, SM::OFF_G, off0, K, hin, cin, R, dlam, dsr, dsi);
      else bwd_apply<IO, TS, CH, false, CONV, MERGE, GROUPED>(tiles, SM::OFF_X + SM::HALO, SM::OFF_UR, SM::OFF_UI, SM::OFF_G, off0, K, hin, cin, R, dlam, dsr, dsi);
    }
    if (USE_TMA && SELF_ISSUE) {
      fence_async_smem();          // the stage leaves after the next barrier all threads pass
    } else if (USE_TMA) {
      fence_async_smem();
      __syncwarp();
      if ((tid & 31) == 0) mbar_arrive(&ready[stage]);   // one arrival per warp
    } else {
      bar_compute(NCOMP);
      if (!CARRY) {
        tile_store_plain<IO, CH>(tiles + SM::OFF_X + SM::HALO, p.dx, b, t0, d0, TC, p.T, p.D);
        tile_store_plain<IO, CH>(tiles + SM::OFF_UR, p.dur, b, t0, d0, TC, p.T, p.D);
        tile_store_plain<IO, CH>(tiles + SM::OFF_UI, p.dui, b, t0, d0, TC, p.T, p.D);
        if (MERGE) tile_store_plain<IO, CH>(tiles + SM::OFF_G, p.dg, b, t0, d0, TC, p.T, p.D);
      }
      bar_compute(NCOMP);
    }
  }

  if (rev_chain && rank == 0 && dch < p.D && p.dh0) p.dh0[static_cast<size_t>(b) * p.D + dch] = carry_rev;

  // Per-row partial of sum_t dl * r: fold the time-lanes in a fixed order.
  bar_compute(NCOMP);
  if (self_issuer) {
    // (in an idle last round the barrier of that round has already sent the last chunk's results off)
    if (mine == rounds) store(mine - 1);     // the last chunk's results; the issuing thread drains its stores on its way out
  }
  auto drain = [&]() { if (USE_TMA && SELF_ISSUE && self_issuer) tma_wait_all<0>(); };
  *reinterpret_cast<float4*>(einF + lane_t * CH + vec * CV) = make_float4(dlam[0].x, dlam[0].y, dlam[1].x, dlam[1].y);
  if (GROUPED) {   // the chain planes are free now: the two gate sums go through them the same way
    *reinterpret_cast<float4*>(einR + lane_t * CH + vec * CV) = make_float4(dsr[0].x, dsr[0].y, dsr[1].x, dsr[1].y);
    *reinterpret_cast<float4*>(aggP + lane_t * CH + vec * CV) = make_float4(dsi[0].x, dsi[0].y, dsi[1].x, dsi[1].y);
  }
  bar_compute(NCOMP);
  static_assert(!GROUPED || NCOMP >= 3 * CH, "one thread per channel and sum");
  if (tid < (GROUPED ? 3 * CH : CH) && dch < p.D) {
    const int which = tid / CH;                       // 0: dLambda partial, 1: sum du_r, 2: sum du_i
    const float* plane = which == 0 ? einF : (which == 1 ? einR : aggP);
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < LANES; ++j) acc += plane[j * CH + cch];
    if constexpr (SPLIT) { st_cluster_f32(cluster_map(&split.sm->sums[rank][tid], 0), acc); }
    else if (which == 0) p.dlam_part[static_cast<size_t>(b) * p.D + dch] = acc;
    else if (p.dgate_part) p.dgate_part[static_cast<size_t>(b) * 2 * p.D + grouped_col(dch, p.gate_bw) + (which - 1) * p.gate_bw] = acc;
  }
  if constexpr (SPLIT) {     // rank 0 folds the sums of the cluster in rank order
    __syncwarp();
    cluster_sync_all();      // (nothing is sent to any CTA after this)
    if (rank != 0) { drain(); return; }
    if (tid < (GROUPED ? 3 * CH : CH) && dch < p.D) {
      const int which = tid / CH;
      float acc = 0.0f;
      for (int r = 0; r < nranks; ++r) acc += split.sm->sums[r][tid];
      if (which == 0) p.dlam_part[static_cast<size_t>(b) * p.D + dch] = acc;
      else if (p.dgate_part) p.dgate_part[static_cast<size_t>(b) * 2 * p.D + grouped_col(dch, p.gate_bw) + (which - 1) * p.gate_bw] = acc;
    }
  }
  if (!p.ticket) { drain(); return; }   // the caller folds the rows with rglru_dlambda_kernel

  // The CTA that finishes last folds the per-row partials into dLambda (rows in index order, so the
  // result does not depend on which CTA that is) and re-arms the ticket for the next backward call.
  // The ticket is one acquire-release atomic by one thread between two CTA barriers: the barrier in front makes
  // the partial rows every thread of this CTA stored part of what the release publishes, the barrier behind makes
  // what the acquire saw (the other CTAs' rows) visible to every thread that goes on to read them, past L1.
  __shared__ int s_last;
  bar_compute(NCOMP);
  if (tid == 0) {
    const unsigned total = gridDim.x * gridDim.y;
    unsigned before;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(before) : "l"(p.ticket), "r"(1u) : "memory");
    s_last = (before == total - 1u) ? 1 : 0;
  }
  bar_compute(NCOMP);
  if (!s_last) { drain(); return; }
  // Rows are added in index order whatever the load order; loads go out eight rows at a time so that the
  // fold costs a few round trips to L2, not one per row.  (Lambda and the caller's buffers need not lie on 16-byte boundaries.)
  const uintptr_t ends = reinterpret_cast<uintptr_t>(p.lambda) | reinterpret_cast<uintptr_t>(p.dlambda) | reinterpret_cast<uintptr_t>(p.dlam_part);
  if ((p.D & 3) == 0 && (ends & 15u) == 0) {
    for (int d = tid * 4; d < p.D; d += NCOMP * 4) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int r0 = 0; r0 < p.B; r0 += 8) {
        float4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          v[j] = (r0 + j < p.B) ? __ldcg(reinterpret_cast<const float4*>(p.dlam_part + static_cast<size_t>(r0 + j) * p.D + d))
                                : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 8; ++j) { acc.x += v[j].x; acc.y += v[j].y; acc.z += v[j].z; acc.w += v[j].w; }
      }
      const float4 lam = *reinterpret_cast<const float4*>(p.lambda + d);
      float4 out;
      out.x = (1.0f / (1.0f + expf(lam.x))) * p.c * acc.x;
      out.y = (1.0f / (1.0f + expf(lam.y))) * p.c * acc.y;
      out.z = (1.0f / (1.0f + expf(lam.z))) * p.c * acc.z;
      out.w = (1.0f / (1.0f + expf(lam.w))) * p.c * acc.w;
      *reinterpret_cast<float4*>(p.dlambda + d) = out;
    }
  } else {
    for (int d = tid; d < p.D; d += NCOMP) {
      float acc = 0.0f;
      for (int r = 0; r < p.B; ++r) acc += __ldcg(p.dlam_part + static_cast<size_t>(r) * p.D + d);
      const float lam = p.lambda[d];
      p.dlambda[d] = (1.0f / (1.0f + expf(lam))) * p.c * acc;
    }
  }
  if (GROUPED && p.dgate && p.dgate_part) {     // gate-bias gradient: column sums of du over the batch rows
    const int N2 = 2 * p.D;                     // a multiple of 4: groups of four channels or more
    for (int d = tid * 4; d < N2; d += NCOMP * 4) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int r0 = 0; r0 < p.B; r0 += 8) {
        float4 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
          v[j] = (r0 + j < p.B) ? __ldcg(reinterpret_cast<const float4*>(p.dgate_part + static_cast<size_t>(r0 + j) * N2 + d))
                                : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 8; ++j) { acc.x += v[j].x; acc.y += v[j].y; acc.z += v[j].z; acc.w += v[j].w; }
      }
      *reinterpret_cast<float4*>(p.dgate + d) = acc;
    }
  }
  if (tid == 0) *p.ticket = 0u;
  drain();
}

// out[n] = sum_b part[b, n], rows added in index order (gate-bias gradient when the batch is too large for the
// backward kernel's own fold).
__global__ void rglru_colsum_kernel(const float* __restrict__ part, float* __restrict__ out, int B, int N) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  float acc = 0.0f;
  for (int b = 0; b < B; ++b) acc += part[static_cast<size_t>(b) * N + n];
  out[n] = acc;
}

// dLambda[d] = d/dLambda of sum dl * r * c * logsigmoid(Lambda) = sigmoid(-Lambda_d) * c * sum_b partial[b, d],
// rows added in index order.
__global__ void rglru_dlambda_kernel(const float* __restrict__ part, const float* __restrict__ lambda,
                                     float* __restrict__ dlambda, int B, int D, float c) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= D) return;
  float acc = 0.0f;
  for (int b = 0; b < B; ++b) acc += part[static_cast<size_t>(b) * D + d];
  const float lam = lambda[d];
  const float sig_neg = 1.0f / (1.0f + expf(lam));
  dlambda[d] = sig_neg * c * acc;
}

// ======================================================================
// Raw affine scan h_t = a_t h_{t-1} + b_t on fp32 tensors (operator-level drop-in
// for griffin/triton_scan.py:274-276).  Same two-level structure, no gate math.
// ======================================================================

// 32-channel tiles (whole 128-byte lines) in four stages, two CTAs per SM: against one CTA per SM on 64-channel tiles,
// B = 3, T = 1999, D = 1000 takes 16 + 25 us instead of 33 + 45 us with the time split, B = 6, T = 2048, D = 1024
// 28 + 47 instead of 37 + 51 us without it.
constexpr int CH = 32;
constexpr int NCV = CH / CV;
constexpr int RAW_TS = 4;
constexpr int RAW_LANES = 16;
constexpr int RAW_NT = RAW_LANES * NCV;
constexpr int RAW_TC = RAW_LANES * RAW_TS;
constexpr int RAW_TILE = RAW_TC * CH * 4;
constexpr int RAW_STAGES = 4;

// The decays of this operator are the caller's and may be of any size, so the map of a whole chunk is not always what
// the steps it is made of are: a product of 64 decays above one overflows, or takes the digits of a state that the steps
// would have left small (h = 4 h - 3 stays at 1 for ever, 4^64 1 - (4^64 - 1) does not), and one that underflows turns an
// infinite state into NaN.  Maps of decays up to one do neither.  So a channel whose round has a lane's product above one,
// or a state that is not finite, is chained lane by lane instead, the ranks of the cluster one after another, each
// handing the state behind its chunk to all: the same arithmetic as the unsplit kernel's.  CH is one warp, so which
// channels these are is a ballot, and every CTA of the cluster, having the same pairs, comes to the same answer.
struct RawSerial {
  float exact[MAX_SPLIT][CH];    // state behind rank r's chunk of this round
  uint64_t bar[MAX_SPLIT];
};
static_assert(CH == 32, "the channels of a tile are one warp");

// The chain leaves the state entering a lane where the lane's aggregate was (.x of its pair), so that a split backward
// with two stages stays below half an SM's shared memory.
template <int NSTAGE, int NTILE, bool SPLIT>
struct RawSmem {
  static constexpr int STAGE = NTILE * RAW_TILE;
  static constexpr int OFF_AGG = NSTAGE * STAGE;
  static constexpr int OFF_BAR = OFF_AGG + ChainSmem<RAW_LANES, CH>::AGG;
  static constexpr int OFF_SPLIT = OFF_BAR + NSTAGE * 8 + 16;
  static constexpr int OFF_SERIAL = OFF_SPLIT + static_cast<int>(offsetof(SplitSmem<CH>, sums));
  static constexpr int BYTES = SPLIT ? OFF_SERIAL + static_cast<int>(sizeof(RawSerial)) : OFF_SPLIT;
};
// The states (carries) of a thread's four channels that enter its lane.
__device__ __forceinline__ void raw_entering(const float2* agg, int at, float2 (&e)[2]) {
  const float4 a = *reinterpret_cast<const float4*>(agg + at), b = *reinterpret_cast<const float4*>(agg + at + 2);
  e[0] = make_float2(a.x, a.z);
  e[1] = make_float2(b.x, b.z);
}
// Level two of a chunk for one channel (thread): chain the lane aggregates onto the carry (lanes in increasing time order,
// or decreasing with REV), leave every lane's entering state in place and return the state behind the chunk.  `idle`: this
// CTA has no chunk in the round.
template <bool REV, bool SPLIT>
__device__ __forceinline__ float raw_chain(float2* agg, float& carry, SplitChain<CH>& split, RawSerial* serial, int& serial_rounds,
                                          int it, bool idle, bool& alive) {
  constexpr int LANES = RAW_LANES;
  const int tid = threadIdx.x;
  float2 ag[LANES];
#pragma unroll
  for (int j = 0; j < LANES; ++j) ag[j] = idle ? make_float2(1.0f, 0.0f) : agg[j * CH + tid];
  auto chain = [&](float e) {       // lane by lane from the state entering the chunk; returns the state behind it
#pragma unroll
    for (int q = 0; q < LANES; ++q) {
      const int j = REV ? LANES - 1 - q : q;
      if (!idle) agg[j * CH + tid].x = e;
      e = fmaf(ag[j].x, e, ag[j].y);
    }
    return e;
  };
  if constexpr (!SPLIT) {
    return carry = chain(carry);
  } else {
    float2 m = make_float2(1.0f, 0.0f);        // the map of the whole chunk
    bool composable = true;
#pragma unroll
    for (int q = 0; q < LANES; ++q) {
      const float2 a = ag[REV ? LANES - 1 - q : q];
      composable = composable && fabsf(a.x) <= 1.0f;
      m = make_float2(m.x * a.x, fmaf(a.x, m.y, a.y));
    }
    if (!composable) m.x = __int_as_float(0x7f800000);      // tells every rank
    split.send(it, tid, m, 0, 1);
    const float before = carry;
    bool contractive;
    const float e = split.receive(it, tid, carry, contractive, alive);
    const bool steady = contractive && fabsf(carry) <= FLT_MAX;     // (a state that is not finite stays so to the end of the round)
    const unsigned wild = __ballot_sync(0xffffffffu, !steady);
    float behind = e;                          // state behind this CTA's chunk
    if (steady) behind = chain(e);
    if (wild) {
      if (tid == 0)
        for (uint32_t r = 0; r < split.size; ++r) mbar_expect_tx(&serial->bar[r], 4 * __popc(wild));
      __syncwarp();
      float state = before;
      for (uint32_t r = 0; r < split.size; ++r) {
        if (r == split.rank && !steady) {
          behind = state = chain(state);
          for (uint32_t to = 0; to < split.size; ++to)
            st_async_f32(cluster_map(&serial->exact[r][tid], to), state, cluster_map(&serial->bar[r], to));
        }
        __syncwarp();
        if (alive) alive = mbar_wait_bounded(&serial->bar[r], serial_rounds & 1);
        if (!steady) state = serial->exact[r][tid];
      }
      if (!steady) carry = state;
      ++serial_rounds;
    }
    return behind;
  }
}

template <int NSTAGE, bool USE_TMA, bool SPLIT>
__global__ void __launch_bounds__(RAW_NT) rawscan_fwd_kernel(const __grid_constant__ RawFwdMaps maps, const RawScanArgs p) {
  using SM = RawSmem<NSTAGE, 2, SPLIT>;
  constexpr int TS = RAW_TS, TC = RAW_TC, ROWB = CH * 4;
  extern __shared__ __align__(128) uint8_t smem[];
  float2* agg = reinterpret_cast<float2*>(smem + SM::OFF_AGG);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::OFF_BAR);
  const int tid = threadIdx.x, lane_t = tid / NCV, vec = tid % NCV;
  const int b = blockIdx.y, d0 = blockIdx.x * CH;
  const int nchunks = (p.T + TC - 1) / TC;
  SplitChain<CH> split;
  if constexpr (SPLIT) split.init(reinterpret_cast<SplitSmem<CH>*>(smem + SM::OFF_SPLIT));
  [[maybe_unused]] RawSerial* serial = reinterpret_cast<RawSerial*>(smem + SM::OFF_SERIAL);      // SPLIT only
  [[maybe_unused]] int serial_rounds = 0;
  const int rank = SPLIT ? static_cast<int>(split.rank) : 0, nranks = SPLIT ? static_cast<int>(split.size) : 1;
  const int rounds = SPLIT ? (nchunks + nranks - 1) / nranks : nchunks;
  const int mine = SPLIT ? (nchunks - rank + nranks - 1) / nranks : nchunks;   // chunks this CTA loads and stores

  auto issue = [&](int it) {
    const int sidx = it % NSTAGE, k = it * nranks + rank;
    uint8_t* st = smem + sidx * SM::STAGE;
    mbar_expect_tx(&bars[sidx], 2 * RAW_TILE);
    tma_load_3d(st, &maps.drive, d0, k * TC, b, &bars[sidx]);
    tma_load_3d(st + RAW_TILE, &maps.decay, d0, k * TC, b, &bars[sidx]);
  };
  pdl_launch_dependents();
  if (USE_TMA) {
    if (tid == 0) {
      for (int s = 0; s < NSTAGE; ++s) mbar_init(&bars[s], 1);
      if constexpr (SPLIT) {
        mbar_init(&split.sm->bar[0], 1);
        mbar_init(&split.sm->bar[1], 1);
        for (int r = 0; r < MAX_SPLIT; ++r) mbar_init(&serial->bar[r], 1);
      }
      mbar_fence_init();
    }
    if constexpr (SPLIT) cluster_sync_all();
    else __syncthreads();
  }
  pdl_wait();
  if (USE_TMA && tid == 0)
    for (int it = 0; it < NSTAGE && it < mine; ++it) issue(it);
  float carry = 0.0f;
  const int dch = d0 + tid;
  if (tid < CH && dch < p.D && p.h0) carry = p.h0[static_cast<size_t>(b) * p.D + dch];
  const int off0 = (lane_t * TS) * ROWB + vec * 16;
  bool alive = true;

  for (int it = 0; it < rounds; ++it) {
    const int k = it * nranks + rank;
    const bool idle = SPLIT && it >= mine;
    if constexpr (SPLIT) { if (tid == 0) split.arm(it); }
    const int stage = USE_TMA ? (it % NSTAGE) : 0;
    uint8_t* tiles = smem + stage * SM::STAGE;
    const int t0 = k * TC;
    if (USE_TMA) {
      if (!idle && alive) alive = mbar_wait_bounded(&bars[stage], (it / NSTAGE) & 1);
    } else {
      tile_load_plain<float, CH>(tiles, p.drive, b, t0, d0, TC, p.T, p.D);
      tile_load_plain<float, CH>(tiles + RAW_TILE, p.decay, b, t0, d0, TC, p.T, p.D);
      __syncthreads();
    }
    float2 P[TS][2], S[TS][2];
    {
      float2 pp[2] = {f2(1.0f), f2(1.0f)}, ss[2] = {f2(0.0f), f2(0.0f)};
#pragma unroll
      for (int st = 0; st < TS; ++st) {
        float2 bv[2], av[2];
        Pack<float>::unpack2(Pack<float>::load(tiles + off0 + st * ROWB), bv);
        Pack<float>::unpack2(Pack<float>::load(tiles + RAW_TILE + off0 + st * ROWB), av);
        const float live = (t0 + lane_t * TS + st < p.T) ? 1.0f : 0.0f;  // steps past T carry the state through
#pragma unroll
        for (int cp = 0; cp < 2; ++cp) {
          const float2 a = fma2(av[cp], f2(live), f2(1.0f - live));
          const float2 bb = mul2(bv[cp], f2(live));
          pp[cp] = mul2(pp[cp], a);
          ss[cp] = fma2(a, ss[cp], bb);
          P[st][cp] = pp[cp];
          S[st][cp] = ss[cp];
        }
      }
    }
    {
      float4* dst = reinterpret_cast<float4*>(agg + lane_t * CH + vec * CV);
      dst[0] = make_float4(P[TS - 1][0].x, S[TS - 1][0].x, P[TS - 1][0].y, S[TS - 1][0].y);
      dst[1] = make_float4(P[TS - 1][1].x, S[TS - 1][1].x, P[TS - 1][1].y, S[TS - 1][1].y);
    }
    alive = __syncthreads_and(alive);
    if (!SPLIT && !alive) break;
    if (tid < CH) raw_chain<false, SPLIT>(agg, carry, split, serial, serial_rounds, it, idle, alive);
    __syncthreads();
    if (idle) break;
    {
      float2 e[2];
      raw_entering(agg, lane_t * CH + vec * CV, e);
#pragma unroll
      for (int st = 0; st < TS; ++st) {
        float2 yv[2];
#pragma unroll
        for (int cp = 0; cp < 2; ++cp) yv[cp] = fma2(P[st][cp], e[cp], S[st][cp]);
        Pack<float>::store2(tiles + off0 + st * ROWB, yv);
      }
    }
    if (USE_TMA) {
      fence_async_smem();
      __syncthreads();
      if (tid == 0) {
        tma_store_3d(&maps.out, tiles, d0, t0, b);
        tma_commit();
        const int prev = it - 1;
        if (prev >= 0 && prev + NSTAGE < mine) {
          tma_wait_read<1>();
          issue(prev + NSTAGE);
        }
      }
    } else {
      __syncthreads();
      tile_store_plain<float, CH>(tiles, p.out, b, t0, d0, TC, p.T, p.D);
      __syncthreads();
    }
  }
  if constexpr (SPLIT) { __syncwarp(); cluster_sync_all(); }     // no CTA leaves while another may still send to it
  if (USE_TMA && tid == 0) tma_wait_all<0>();
  if (USE_TMA && !alive && tid < CH) atomicExch(p.status, DEV_TIMEOUT_LOAD);
}

// Backward of the raw scan.  Tiles per chunk: d_out, decay, and the forward output
// shifted one step back in time (row t holds h_{t-1}; the row before t = 0 is h0).
template <int NSTAGE, bool USE_TMA, bool SPLIT>
__global__ void __launch_bounds__(RAW_NT) rawscan_bwd_kernel(const __grid_constant__ RawBwdMaps maps, const RawScanArgs p) {
  using SM = RawSmem<NSTAGE, 3, SPLIT>;
  constexpr int TS = RAW_TS, TC = RAW_TC, ROWB = CH * 4;
  extern __shared__ __align__(128) uint8_t smem[];
  float2* agg = reinterpret_cast<float2*>(smem + SM::OFF_AGG);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::OFF_BAR);
  const int tid = threadIdx.x, lane_t = tid / NCV, vec = tid % NCV;
  const int b = blockIdx.y, d0 = blockIdx.x * CH;
  const int nchunks = (p.T + TC - 1) / TC;
  SplitChain<CH> split;
  if constexpr (SPLIT) split.init(reinterpret_cast<SplitSmem<CH>*>(smem + SM::OFF_SPLIT));
  [[maybe_unused]] RawSerial* serial = reinterpret_cast<RawSerial*>(smem + SM::OFF_SERIAL);      // SPLIT only
  [[maybe_unused]] int serial_rounds = 0;
  const int rank = SPLIT ? static_cast<int>(split.rank) : 0, nranks = SPLIT ? static_cast<int>(split.size) : 1;
  const int rounds = SPLIT ? (nchunks + nranks - 1) / nranks : nchunks;
  const int mine = SPLIT ? (nchunks - rank + nranks - 1) / nranks : nchunks;   // chunks this CTA loads and stores

  auto issue = [&](int q) {
    const int k = nchunks - 1 - (q * nranks + rank);
    const int sidx = q % NSTAGE;
    uint8_t* st = smem + sidx * SM::STAGE;
    mbar_expect_tx(&bars[sidx], 3 * RAW_TILE);
    tma_load_3d(st, &maps.dout, d0, k * TC, b, &bars[sidx]);
    tma_load_3d(st + RAW_TILE, &maps.decay, d0, k * TC, b, &bars[sidx]);
    tma_load_3d(st + 2 * RAW_TILE, &maps.out, d0, k * TC - 1, b, &bars[sidx]);
  };
  pdl_launch_dependents();
  if (USE_TMA) {
    if (tid == 0) {
      for (int s = 0; s < NSTAGE; ++s) mbar_init(&bars[s], 1);
      if constexpr (SPLIT) {
        mbar_init(&split.sm->bar[0], 1);
        mbar_init(&split.sm->bar[1], 1);
        for (int r = 0; r < MAX_SPLIT; ++r) mbar_init(&serial->bar[r], 1);
      }
      mbar_fence_init();
    }
    if constexpr (SPLIT) cluster_sync_all();
    else __syncthreads();
  }
  pdl_wait();
  if (USE_TMA && tid == 0)
    for (int it = 0; it < NSTAGE && it < mine; ++it) issue(it);
  float carry = 0.0f;  // a_t g_t flowing towards earlier steps
  const int dch = d0 + tid;
  const int off0 = (lane_t * TS) * ROWB + vec * 16;
  bool alive = true;

  for (int q = 0; q < rounds; ++q) {
    const int k = nchunks - 1 - (q * nranks + rank);
    const bool idle = SPLIT && q >= mine;
    if constexpr (SPLIT) { if (tid == 0) split.arm(q); }
    const int stage = USE_TMA ? (q % NSTAGE) : 0;
    uint8_t* tiles = smem + stage * SM::STAGE;
    const int t0 = k * TC;
    if (USE_TMA) {
      if (!idle && alive) alive = mbar_wait_bounded(&bars[stage], (q / NSTAGE) & 1);
    } else {
      tile_load_plain<float, CH>(tiles, p.dout, b, t0, d0, TC, p.T, p.D);
      tile_load_plain<float, CH>(tiles + RAW_TILE, p.decay, b, t0, d0, TC, p.T, p.D);
      tile_load_plain<float, CH>(tiles + 2 * RAW_TILE, p.out_in, b, t0 - 1, d0, TC, p.T, p.D);
      __syncthreads();
    }
    float2 av[TS][2], gv[TS][2], hv[TS][2];
    float2 qq[2] = {f2(1.0f), f2(1.0f)}, cc[2] = {f2(0.0f), f2(0.0f)};
#pragma unroll
    for (int st = 0; st < TS; ++st) {
      Pack<float>::unpack2(Pack<float>::load(tiles + off0 + st * ROWB), gv[st]);
      Pack<float>::unpack2(Pack<float>::load(tiles + RAW_TILE + off0 + st * ROWB), av[st]);
      Pack<float>::unpack2(Pack<float>::load(tiles + 2 * RAW_TILE + off0 + st * ROWB), hv[st]);
    }
    if (k == 0 && lane_t == 0) {  // the state entering t = 0
      float h0v[CV];
#pragma unroll
      for (int ch = 0; ch < CV; ++ch) {
        const int d = d0 + vec * CV + ch;
        h0v[ch] = (p.h0 && d < p.D) ? p.h0[static_cast<size_t>(b) * p.D + d] : 0.0f;
      }
      hv[0][0] = make_float2(h0v[0], h0v[1]);
      hv[0][1] = make_float2(h0v[2], h0v[3]);
    }
#pragma unroll
    for (int st = TS - 1; st >= 0; --st)
#pragma unroll
      for (int cp = 0; cp < 2; ++cp) {
        cc[cp] = mul2(av[st][cp], add2(gv[st][cp], cc[cp]));
        qq[cp] = mul2(qq[cp], av[st][cp]);
      }
    {
      float4* dst = reinterpret_cast<float4*>(agg + lane_t * CH + vec * CV);
      dst[0] = make_float4(qq[0].x, cc[0].x, qq[0].y, cc[0].y);
      dst[1] = make_float4(qq[1].x, cc[1].x, qq[1].y, cc[1].y);
    }
    alive = __syncthreads_and(alive);
    if (!SPLIT && !alive) break;
    if (tid < CH) {
      const float behind = raw_chain<true, SPLIT>(agg, carry, split, serial, serial_rounds, q, idle, alive);
      // (the first steps' own chunk has it to the bit, the folded carry to a rounding or two)
      if (alive && k == 0 && dch < p.D && p.dh0) p.dh0[static_cast<size_t>(b) * p.D + dch] = behind;
    }
    __syncthreads();
    if (idle) break;
    {
      float2 c[2];
      raw_entering(agg, lane_t * CH + vec * CV, c);
#pragma unroll
      for (int st = TS - 1; st >= 0; --st) {
        float2 da[2], db[2];
#pragma unroll
        for (int cp = 0; cp < 2; ++cp) {
          const float2 g = add2(gv[st][cp], c[cp]);
          c[cp] = mul2(av[st][cp], g);
          db[cp] = g;
          da[cp] = mul2(g, hv[st][cp]);
        }
        Pack<float>::store2(tiles + off0 + st * ROWB, db);
        Pack<float>::store2(tiles + RAW_TILE + off0 + st * ROWB, da);
      }
    }
    if (USE_TMA) {
      fence_async_smem();
      __syncthreads();
      if (tid == 0) {
        tma_store_3d(&maps.ddrive, tiles, d0, t0, b);
        tma_store_3d(&maps.ddecay, tiles + RAW_TILE, d0, t0, b);
        tma_commit();
        const int qp = q - 1;
        if (qp >= 0 && qp + NSTAGE < mine) {
          tma_wait_read<1>();
          issue(qp + NSTAGE);
        }
      }
    } else {
      __syncthreads();
      tile_store_plain<float, CH>(tiles, p.ddrive, b, t0, d0, TC, p.T, p.D);
      tile_store_plain<float, CH>(tiles + RAW_TILE, p.ddecay, b, t0, d0, TC, p.T, p.D);
      __syncthreads();
    }
  }
  if constexpr (SPLIT) { __syncwarp(); cluster_sync_all(); }     // no CTA leaves while another may still send to it
  if (USE_TMA && tid == 0) tma_wait_all<0>();
  if (USE_TMA && !alive && tid < CH) atomicExch(p.status, DEV_TIMEOUT_LOAD);
}

// ======================================================================
// The conv alone (griffin/griffin.py:474-487 of the reference), staged like the scan:
// a CTA owns 64 channels of one batch row and walks the sequence in 64-step chunks
// that a producer warp moves through shared memory with TMA; there is no cross-thread
// dependence, so the only synchronisation is the mbarrier pipeline itself.
// Used when B * ceil(D / 64) CTAs fill the machine; otherwise the per-run kernels of
// rglru_conv.cu, which also split the time axis, are the better fit.
// ======================================================================

template <typename IO, int NSTAGE>
struct ConvFwdSmem {
  static constexpr int TS = 4, LANES = 16, CH = 64, TC = LANES * TS;
  static constexpr int TILE = TC * CH * sizeof(IO);
  static constexpr int HALO = 3 * CH * sizeof(IO);
  static constexpr int TILEX = TILE + HALO;     // input rows t0-3 .. t0+TC-1
  static constexpr int STAGE = TILEX + TILE;    // + the result tile
  static constexpr int OFF_BAR = NSTAGE * STAGE;
  static constexpr int BYTES = OFF_BAR + 2 * NSTAGE * 8 + 16;
};

template <typename IO, int NSTAGE>
__global__ void __launch_bounds__(288) conv_tma_fwd_kernel(const __grid_constant__ ConvMaps maps, const ConvTmaArgs p) {
  using SM = ConvFwdSmem<IO, NSTAGE>;
  constexpr int TS = SM::TS, CH = SM::CH, TC = SM::TC, NCV = CH / CV, NCOMP = SM::LANES * NCV;
  constexpr int ROWB = CH * sizeof(IO);
  extern __shared__ __align__(128) uint8_t smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + SM::OFF_BAR);
  uint64_t* ready = full + NSTAGE;
  volatile int* dead = reinterpret_cast<volatile int*>(ready + NSTAGE);
  const int tid = threadIdx.x, lane_t = tid / NCV, vec = tid % NCV;
  const int b = blockIdx.y, d0 = blockIdx.x * CH;
  const int nchunks = (p.T + TC - 1) / TC;

  if (tid == 0) {
    *dead = 0;
    for (int s = 0; s < NSTAGE; ++s) { mbar_init(&full[s], 1); mbar_init(&ready[s], NCOMP / 32); }
    mbar_fence_init();
  }
  __syncthreads();

  if (tid >= NCOMP) {
    if (tid == NCOMP) {
      prefetch_map(&maps.in0); prefetch_map(&maps.out0);
      auto issue = [&](int k) {
        const int sidx = k % NSTAGE;
        mbar_expect_tx(&full[sidx], SM::TILEX);
        tma_load_3d(smem + sidx * SM::STAGE, &maps.in0, d0, k * TC - 3, b, &full[sidx]);   // rows before t = 0 read as zero
      };
      for (int k = 0; k < NSTAGE && k < nchunks; ++k) issue(k);
      for (int k = 0; k < nchunks; ++k) {
        const int sidx = k % NSTAGE;
        mbar_wait_or_flag(&ready[sidx], (k / NSTAGE) & 1, dead, p.status, DEV_TIMEOUT_STORE);
        tma_store_3d(&maps.out0, smem + sidx * SM::STAGE + SM::TILEX, d0, k * TC, b);
        tma_commit();
        if (k + NSTAGE < nchunks) {
          tma_wait_read<0>();
          issue(k + NSTAGE);
        }
      }
      tma_wait_all<0>();
    }
    return;
  }

  ConvTaps ct;
  load_taps(p.w, p.bias, d0 + vec * CV, p.D, ct, p.half_w, p.half_b);
  const int off0 = (lane_t * TS) * ROWB + vec * Pack<IO>::BYTES;

  for (int k = 0; k < nchunks; ++k) {
    const int stage = k % NSTAGE;
    uint8_t* tiles = smem + stage * SM::STAGE;
    const int t0 = k * TC;
    uint32_t fl[1];
    const bool masked = (p.tok != nullptr) || (t0 + TC > p.T);
    if (masked) load_flags_word(p.tok, b, p.T, t0 + lane_t * TS, fl);
    float2 hist_v[3][2];
    const float2 (*hist)[2] = nullptr;
    if (k == 0 && lane_t == 0 && p.state) {
      load_hist<IO>(p.state, b, d0 + vec * CV, p.D, hist_v);
      hist = hist_v;
    }
    mbar_wait_or_flag(&full[stage], (k / NSTAGE) & 1, dead, p.status, DEV_TIMEOUT_LOAD);
    float2 xc[TS][2];
    const bool flagged = masked && any_flag(fl);
    if (flagged) conv_front<IO, TS, CH, true>(tiles, off0, ct, fl, hist, xc);
    else conv_front<IO, TS, CH, false>(tiles, off0, ct, fl, hist, xc);
    uint8_t* to = tiles + SM::TILEX;
#pragma unroll
    for (int st = 0; st < TS; ++st) {
      if (flagged && ((fl[0] >> (8 * st)) & TOK_INACTIVE)) { xc[st][0] = f2(0.0f); xc[st][1] = f2(0.0f); }   // padding emits zero
      Pack<IO>::store2(to + off0 + st * ROWB, xc[st]);
    }
    fence_async_smem();
    __syncwarp();
    if ((tid & 31) == 0) mbar_arrive(&ready[stage]);
  }
}

// The TS steps of one thread in the conv backward.  Two sliding four-row windows: ga = upstream gradient of
// tokens (step .. step+3), xa = input at times (step-3 .. step); each step loads one new row of each.
// `fb` holds the flag bytes of the TS + 3 tokens whose gradient is read; `dstate` (first lane of the first
// chunk only) receives the gradient of the carried history, whose rows only tokens 0 .. 2 reach.
template <typename IO, int TS, int CH, bool MASKED>
__device__ __forceinline__ void conv_bwd_steps(const uint8_t* tg, const uint8_t* tx, uint8_t* tdx, int off0,
                                               const ConvTaps& ct, const uint32_t (&fb)[TS + 3], const float2 (*hist)[2],
                                               IO* dstate, int D, int channels_left, float2 (&gw)[5][2]) {
  constexpr int ROWB = CH * sizeof(IO);
  auto grad_row = [&](int j, float2 (&v)[2]) {
    Pack<IO>::unpack2(Pack<IO>::load(tg + off0 + j * ROWB), v);
    if (MASKED && (fb[j] & TOK_INACTIVE)) { v[0] = f2(0.0f); v[1] = f2(0.0f); }
  };
  auto reach_of = [&](int j) { return MASKED ? 3 - static_cast<int>(fb[j] & TOK_CUT_MASK) : 3; };
  float2 ga[4][2], xa[4][2];
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    grad_row(j, ga[j]);
    Pack<IO>::unpack2(Pack<IO>::load(tx + off0 + j * ROWB), xa[j]);
    if (hist) { xa[j][0] = hist[j][0]; xa[j][1] = hist[j][1]; }
  }
  if (dstate) {
#pragma unroll
    for (int slot = 0; slot < 3; ++slot) {
      float2 acc[2] = {f2(0.0f), f2(0.0f)};
#pragma unroll
      for (int u = 0; u <= slot; ++u) {               // token u reads time slot-3 with lag u + 3 - slot
        const int lag = u + 3 - slot;
        const float m = reach_of(u) >= lag ? 1.0f : 0.0f;
#pragma unroll
        for (int cp = 0; cp < 2; ++cp) acc[cp] = fma2(mul2(ct.w[3 - lag][cp], f2(m)), ga[u][cp], acc[cp]);
      }
      const float v4[4] = {acc[0].x, acc[0].y, acc[1].x, acc[1].y};
#pragma unroll
      for (int ch = 0; ch < 4; ++ch)
        if (ch < channels_left) dstate[static_cast<size_t>(slot) * D + ch] = Pack<IO>::from_float(v4[ch]);
    }
  }
#pragma unroll
  for (int st = 0; st < TS; ++st) {
    grad_row(st + 3, ga[3]);
    Pack<IO>::unpack2(Pack<IO>::load(tx + off0 + (st + 3) * ROWB), xa[3]);   // input at the step's own time
    float2 dx[2];
#pragma unroll
    for (int cp = 0; cp < 2; ++cp) {
      if (MASKED) {
        float2 a = mul2(ct.w[3][cp], ga[0][cp]);
        a = fma2(mul2(ct.w[2][cp], f2(reach_of(st + 1) >= 1 ? 1.0f : 0.0f)), ga[1][cp], a);
        a = fma2(mul2(ct.w[1][cp], f2(reach_of(st + 2) >= 2 ? 1.0f : 0.0f)), ga[2][cp], a);
        dx[cp] = fma2(mul2(ct.w[0][cp], f2(reach_of(st + 3) >= 3 ? 1.0f : 0.0f)), ga[3][cp], a);
      } else {
        float2 a = mul2(ct.w[3][cp], ga[0][cp]);
        a = fma2(ct.w[2][cp], ga[1][cp], a);
        a = fma2(ct.w[1][cp], ga[2][cp], a);
        dx[cp] = fma2(ct.w[0][cp], ga[3][cp], a);
      }
    }
    Pack<IO>::store2(tdx + off0 + st * ROWB, dx);
    // tap gradients of the step's own token (its flag decides how far back it reaches)
    const int reach = reach_of(st);
#pragma unroll
    for (int cp = 0; cp < 2; ++cp) {
      const float2 g0 = ga[0][cp];
      gw[4][cp] = add2(gw[4][cp], g0);
      gw[3][cp] = fma2(g0, xa[3][cp], gw[3][cp]);
      if (MASKED) {
        gw[2][cp] = fma2(mul2(g0, f2(reach >= 1 ? 1.0f : 0.0f)), xa[2][cp], gw[2][cp]);
        gw[1][cp] = fma2(mul2(g0, f2(reach >= 2 ? 1.0f : 0.0f)), xa[1][cp], gw[1][cp]);
        gw[0][cp] = fma2(mul2(g0, f2(reach >= 3 ? 1.0f : 0.0f)), xa[0][cp], gw[0][cp]);
      } else {
        gw[2][cp] = fma2(g0, xa[2][cp], gw[2][cp]);
        gw[1][cp] = fma2(g0, xa[1][cp], gw[1][cp]);
        gw[0][cp] = fma2(g0, xa[0][cp], gw[0][cp]);
      }
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      ga[j][0] = ga[j + 1][0]; ga[j][1] = ga[j + 1][1];
      xa[j][0] = xa[j + 1][0]; xa[j][1] = xa[j + 1][1];
    }
  }
}

// Backward of the conv.  Per chunk: the upstream gradient rows t0 .. t0+TC+2 (three rows of look-ahead, zero
// past T), the input rows t0-3 .. t0+TC-1, and the result tile.
//   dx[t]     = sum_lag w[3-lag] g[t+lag] [token t+lag reaches back lag steps]
//   dw[3-lag] += g[t] x[t-lag] [token t reaches back lag steps],   db += g[t]
// with g zero on padding.  The tap gradients stay in registers over the whole sequence and are folded
// across the CTA's time-lanes in a fixed order at the end: one partial row [5, D] per batch row.
template <typename IO, int NSTAGE>
struct ConvBwdSmem {
  static constexpr int TS = 4, LANES = 16, CH = 64, TC = LANES * TS;
  static constexpr int TILE = TC * CH * sizeof(IO);
  static constexpr int HALO = 3 * CH * sizeof(IO);
  static constexpr int TILEX = TILE + HALO;
  static constexpr int OFF_X = TILEX, OFF_DX = 2 * TILEX;
  static constexpr int STAGE = 2 * TILEX + TILE;
  static constexpr int OFF_BAR = NSTAGE * STAGE;
  static constexpr int BYTES = OFF_BAR + 2 * NSTAGE * 8 + 16;
  static_assert(NSTAGE * STAGE >= LANES * 5 * CH * 4, "the final fold reuses the stage memory");
};

template <typename IO, int NSTAGE>
__global__ void __maxnreg__(96) conv_tma_bwd_kernel(const __grid_constant__ ConvMaps maps, const ConvTmaArgs p) {
  using SM = ConvBwdSmem<IO, NSTAGE>;
  constexpr int TS = SM::TS, CH = SM::CH, TC = SM::TC, NCV = CH / CV, NCOMP = SM::LANES * NCV, LANES = SM::LANES;
  constexpr int ROWB = CH * sizeof(IO);
  extern __shared__ __align__(128) uint8_t smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + SM::OFF_BAR);
  uint64_t* ready = full + NSTAGE;
  volatile int* dead = reinterpret_cast<volatile int*>(ready + NSTAGE);
  const int tid = threadIdx.x, lane_t = tid / NCV, vec = tid % NCV;
  const int b = blockIdx.y, d0 = blockIdx.x * CH;
  const int nchunks = (p.T + TC - 1) / TC;

  if (tid == 0) {
    *dead = 0;
    for (int s = 0; s < NSTAGE; ++s) { mbar_init(&full[s], 1); mbar_init(&ready[s], NCOMP / 32); }
    mbar_fence_init();
  }
  __syncthreads();

  if (tid >= NCOMP) {
    if (tid == NCOMP) {
      prefetch_map(&maps.in0); prefetch_map(&maps.in1); prefetch_map(&maps.out0);
      auto issue = [&](int k) {
        const int sidx = k % NSTAGE;
        uint8_t* st = smem + sidx * SM::STAGE;
        mbar_expect_tx(&full[sidx], 2 * SM::TILEX);
        tma_load_3d(st, &maps.in0, d0, k * TC, b, &full[sidx]);                   // gradient, rows past T read as zero
        tma_load_3d(st + SM::OFF_X, &maps.in1, d0, k * TC - 3, b, &full[sidx]);   // input, rows before 0 read as zero
      };
      for (int k = 0; k < NSTAGE && k < nchunks; ++k) issue(k);
      for (int k = 0; k < nchunks; ++k) {
        const int sidx = k % NSTAGE;
        mbar_wait_or_flag(&ready[sidx], (k / NSTAGE) & 1, dead, p.status, DEV_TIMEOUT_STORE);
        tma_store_3d(&maps.out0, smem + sidx * SM::STAGE + SM::OFF_DX, d0, k * TC, b);
        tma_commit();
        if (k + NSTAGE < nchunks) {
          tma_wait_read<0>();
          issue(k + NSTAGE);
        }
      }
      tma_wait_all<0>();
    }
    bar_all(NCOMP + 32);   // the final fold below reuses stage memory: every bulk store has left it
    return;
  }

  ConvTaps ct;
  load_taps(p.w, nullptr, d0 + vec * CV, p.D, ct, p.half_w);
  float2 gw[5][2];
#pragma unroll
  for (int q = 0; q < 5; ++q) { gw[q][0] = f2(0.0f); gw[q][1] = f2(0.0f); }
  const int off0 = (lane_t * TS) * ROWB + vec * Pack<IO>::BYTES;

  for (int k = 0; k < nchunks; ++k) {
    const int stage = k % NSTAGE;
    uint8_t* tiles = smem + stage * SM::STAGE;
    const int t0 = k * TC;
    // flag bytes of the TS + 3 tokens whose gradient this thread reads (steps at or past T count as padding)
    uint32_t fb[TS + 3];
    const bool masked = (p.tok != nullptr) || (t0 + TC + 3 > p.T);
    {
      const int t_first = t0 + lane_t * TS;
      const uint8_t* fp = p.tok ? p.tok + static_cast<size_t>(b) * p.T + t_first : nullptr;
      if (masked && fp && t_first + 8 <= p.T && (reinterpret_cast<uintptr_t>(fp) & 3u) == 0) {
        const uint32_t w0 = *reinterpret_cast<const uint32_t*>(fp);       // two aligned words cover the seven tokens
        const uint32_t w1 = *reinterpret_cast<const uint32_t*>(fp + 4);
#pragma unroll
        for (int j = 0; j < TS + 3; ++j) fb[j] = ((j < 4 ? w0 : w1) >> (8 * (j & 3))) & 0xffu;
      } else {
#pragma unroll
        for (int j = 0; j < TS + 3; ++j) {
          fb[j] = 0u;
          if (masked) {
            const int t = t_first + j;
            fb[j] = t < p.T ? (p.tok ? p.tok[static_cast<size_t>(b) * p.T + t] : 0u) : TOK_INACTIVE;
          }
        }
      }
    }
    float2 hist_v[3][2];
    const bool use_hist = (k == 0 && lane_t == 0 && p.state != nullptr);
    if (use_hist) load_hist<IO>(p.state, b, d0 + vec * CV, p.D, hist_v);
    mbar_wait_or_flag(&full[stage], (k / NSTAGE) & 1, dead, p.status, DEV_TIMEOUT_LOAD);

    IO* dstate = nullptr;
    if (k == 0 && lane_t == 0 && p.d_state)
      dstate = static_cast<IO*>(p.d_state) + static_cast<size_t>(b) * 3 * p.D + d0 + vec * CV;
    const float2 (*hist)[2] = use_hist ? hist_v : nullptr;
    if (masked && any_flag(fb)) conv_bwd_steps<IO, TS, CH, true>(tiles, tiles + SM::OFF_X, tiles + SM::OFF_DX, off0, ct, fb, hist, dstate,
                                                 p.D, p.D - (d0 + vec * CV), gw);
    else conv_bwd_steps<IO, TS, CH, false>(tiles, tiles + SM::OFF_X, tiles + SM::OFF_DX, off0, ct, fb, hist, dstate,
                                           p.D, p.D - (d0 + vec * CV), gw);
    fence_async_smem();
    __syncwarp();
    if ((tid & 31) == 0) mbar_arrive(&ready[stage]);
  }

  // Fold the time-lanes in index order; the stage memory is free once the producer has drained its stores.
  bar_all(NCOMP + 32);
  float* red = reinterpret_cast<float*>(smem);          // [LANES][5][CH]
#pragma unroll
  for (int q = 0; q < 5; ++q)
    *reinterpret_cast<float4*>(red + (lane_t * 5 + q) * CH + vec * CV) = make_float4(gw[q][0].x, gw[q][0].y, gw[q][1].x, gw[q][1].y);
  bar_compute(NCOMP);
  for (int idx = tid; idx < 5 * CH; idx += NCOMP) {
    const int q = idx / CH, cc = idx % CH;
    if (d0 + cc >= p.D) continue;
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < LANES; ++j) acc += red[(j * 5 + q) * CH + cc];
    p.part[(static_cast<size_t>(b) * 5 + q) * p.D + d0 + cc] = acc;
  }
}

// ======================================================================
// Self-test of the bounded wait: one CTA waits on an mbarrier that nothing ever completes, with a limit of
// `limit` SM cycles.  The wait must give up, set the device status word, and let every thread reach the
// barrier and the final store below -- the behaviour the pipelined kernels rely on when a copy never lands.
// ======================================================================
__global__ void __launch_bounds__(64) wait_selftest_kernel(int* status, int* finished, long long limit) {
  __shared__ uint64_t bar;
  __shared__ int dead_flag;
  volatile int* dead = &dead_flag;
  if (threadIdx.x == 0) {
    dead_flag = 0;
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  __syncthreads();
  mbar_wait_or_flag(&bar, 0, dead, status, DEV_TIMEOUT_SELFTEST, limit);
  __syncthreads();                       // every thread gets here: barriers stay matched after a timeout
  if (threadIdx.x == 0 && finished) *finished = 1;
}
cudaError_t launch_wait_selftest(int* status, int* finished, long long limit_cycles, cudaStream_t s) {
  wait_selftest_kernel<<<1, 64, 0, s>>>(status, finished, limit_cycles);
  return cudaGetLastError();
}

// ======================================================================
// Launchers
// ======================================================================

// CTA shapes.  CH channels x (LANES * TS) time-steps per chunk, LANES * CH / 4 compute threads.
//   64 x 64  : the default; grids large enough to put two or more forward CTAs on every SM.
//   32 x 128 : half-width forward tiles double the number of CTAs for small grids, so that two CTAs
//              (two independent barrier domains) still share an SM and overlap their phases.
struct Shape64x16x4 { static constexpr int CH = 64, LANES = 16, TS = 4; };
struct Shape32x32x4 { static constexpr int CH = 32, LANES = 32, TS = 4; };

// Kernel variants.  Forward: 0 = 64 x 64 tiles, 2 = 32 x 128 tiles.  Backward: 0 = 64 x 64 tiles with a
// producer warp, 3 = the same tiles with the bulk copies issued by a compute thread (SELF_ISSUE).  The numbers
// are what RGLRU_FWD_VARIANT / RGLRU_BWD_VARIANT accept (they force one variant for a whole process; the
// test-suite uses them to run every variant over the parity cases); anything else means "choose by shape".
static bool fwd_variant_exists(int v) { return v == 0 || v == 2; }
static bool bwd_variant_exists(int v) { return v == 0 || v == 3; }

// Whether a forward call takes the paired-row tile layout: the 32-channel shape on bf16 tensors without token
// flags over a whole number of 128-step chunks.  The API encodes 5-D tensor maps exactly when this says so.
bool scan_fwd_paired(int variant, bool bf16, const void* tok, int T) {
  return variant == 2 && bf16 && tok == nullptr && T % 128 == 0;
}
int scan_fwd_box_rows(int v) { return v == 2 ? 128 : 64; }
int scan_fwd_box_cols(int v) { return v == 2 ? 32 : 64; }
int scan_bwd_box_rows(int) { return 64; }
int scan_bwd_box_cols(int) { return 64; }

static int env_override(const char* name) {
  const char* v = getenv(name);
  return (v && v[0] >= '0' && v[0] <= '9' && v[1] == 0) ? (v[0] - '0') : -1;
}

// Measured on B200 (T = 2048, D = 1024): half-width forward tiles win while 64-channel tiles cannot fill the 148 SMs
// (bf16 B = 8, 128 tiles: 28 us against 48 us) and lose once they can (B = 16: 52 us against 50 us); for fp32, whose
// stages leave one CTA per SM, they win as long as there is an SM for each of them (B = 4, 64 tiles: 25 us against 43;
// B = 5: 47 against 44).  The backward runs one CTA per SM either way; without the
// producer warp it is 1 to 2 % faster for bf16 tensors (eight warps leave every thread its registers).
int scan_fwd_variant(int B, int T, int D, bool bf16) {
  static const int forced = env_override("RGLRU_FWD_VARIANT");
  if (fwd_variant_exists(forced)) return forced;
  const long long tiles = static_cast<long long>(B) * ((D + 63) / 64);
  return (tiles <= (bf16 ? 160 : 74) && T >= 256) ? 2 : 0;
}
int scan_bwd_variant(int B, int T, int D, bool bf16) {
  static const int forced = env_override("RGLRU_BWD_VARIANT");
  if (bwd_variant_exists(forced)) return forced;
  (void)B; (void)T; (void)D;
  return bf16 ? 3 : 0;
}

// One forward (backward) kernel instantiation with its launch shape.  Kern::get() is the kernel, prepared for its
// dynamic shared memory.
template <typename IO, typename V, int STAGES, bool USE_TMA, bool CONV = false, bool MERGE = false, bool GROUPED = false,
          bool PLAIN = false, bool CARRY = false, bool PAIRED = false, bool SPLIT = false>
struct FwdKern {
  static constexpr int ST = USE_TMA ? STAGES : 1;
  static constexpr bool CAPPED = USE_TMA && !CONV && (MERGE || GROUPED || SPLIT);
  static constexpr int THREADS = V::LANES * (V::CH / CV) + (USE_TMA ? 32 : 0);
  static constexpr int BYTES = FwdSmem<IO, V::TS, V::LANES, V::CH, ST, CONV, MERGE, SPLIT>::BYTES;
  static constexpr int CH = V::CH;
  static constexpr bool IS_SPLIT = SPLIT;
  static_assert(BYTES <= 232448, "shared memory of one CTA");
  using Fn = void (*)(FwdMaps, ScanFwdArgs);
  static Fn get(cudaError_t& e) {
    Fn kern;
    if constexpr (CAPPED) kern = rglru_fwd_kernel_capped<IO, V::TS, V::LANES, V::CH, ST, USE_TMA, CONV, MERGE, GROUPED, PLAIN, SPLIT>;
    else kern = rglru_fwd_kernel<IO, V::TS, V::LANES, V::CH, ST, USE_TMA, CONV, MERGE, GROUPED, PLAIN, CARRY, PAIRED, SPLIT>;
    e = set_smem<FwdKern>(kern, BYTES);
    return kern;
  }
};
template <typename IO, typename V, int STAGES, bool USE_TMA, bool CONV = false, bool MERGE = false, bool GROUPED = false,
          bool SELF_ISSUE = false, bool PLAIN = false, bool CARRY = false, bool SPLIT = false>
struct BwdKern {
  static constexpr int ST = USE_TMA ? STAGES : 1;
  static constexpr int THREADS = V::LANES * (V::CH / CV) + ((USE_TMA && !SELF_ISSUE) ? 32 : 0);
  static constexpr int BYTES = BwdSmem<IO, V::TS, V::LANES, V::CH, ST, CONV, MERGE, SPLIT>::BYTES;
  static constexpr int CH = V::CH;
  static constexpr bool IS_SPLIT = SPLIT, IS_GROUPED = GROUPED;
  static_assert(BYTES <= 232448, "shared memory of one CTA");
  using Fn = void (*)(BwdMaps, ScanBwdArgs);
  static Fn get(cudaError_t& e) {
    Fn kern = rglru_bwd_kernel<IO, V::TS, V::LANES, V::CH, ST, USE_TMA, CONV, MERGE, GROUPED, SELF_ISSUE, PLAIN, CARRY, SPLIT>;
    e = set_smem<BwdKern>(kern, BYTES);
    return kern;
  }
};

template <typename K>
static cudaError_t launch_fwd(const FwdMaps& maps, const ScanFwdArgs& a, cudaStream_t s) {
  cudaError_t e;
  auto kern = K::get(e);
  if (e != cudaSuccess) return e;
  dim3 grid((a.D + K::CH - 1) / K::CH, a.B);
  return launch_pdl(kern, grid, K::THREADS, K::BYTES, s, maps, a, K::IS_SPLIT ? a.split : 1);
}
template <typename IO, typename V, int STAGES, bool USE_TMA, bool CONV = false, bool MERGE = false, bool GROUPED = false,
          bool PLAIN = false, bool CARRY = false, bool PAIRED = false>
static cudaError_t launch_fwd_t(const FwdMaps& maps, const ScanFwdArgs& a, cudaStream_t s) {
  return launch_fwd<FwdKern<IO, V, STAGES, USE_TMA, CONV, MERGE, GROUPED, PLAIN, CARRY, PAIRED>>(maps, a, s);
}

// The time-split kernels.  Three (merged: two) stages leave the bf16 forward small enough for two CTAs per SM.
template <typename IO, bool PLAIN>
using SplitFwd = FwdKern<IO, Shape64x16x4, 3, true, false, false, false, PLAIN, false, false, true>;
template <typename IO, bool MERGE>
using SplitGroupedFwd = FwdKern<IO, Shape64x16x4, MERGE ? 2 : 3, true, false, MERGE, true, false, false, false, true>;

template <typename IO>
static cudaError_t launch_fwd_io(bool use_tma, int variant, const FwdMaps& maps, const ScanFwdArgs& a, cudaStream_t s) {
  constexpr bool H = sizeof(IO) == 2;
  if (a.y == nullptr)   // carry-only pass: one shape, masked arithmetic
    return use_tma ? launch_fwd_t<IO, Shape64x16x4, H ? 4 : 3, true, false, false, false, false, true>(maps, a, s)
                   : launch_fwd_t<IO, Shape64x16x4, 1, false, false, false, false, false, true>(maps, a, s);
  if (!use_tma) return launch_fwd_t<IO, Shape64x16x4, 1, false>(maps, a, s);
  const bool plain = a.tok == nullptr && a.T % 128 == 0;   // no step of any chunk is masked
  if (a.split > 1) {
    return plain ? launch_fwd<SplitFwd<IO, true>>(maps, a, s) : launch_fwd<SplitFwd<IO, false>>(maps, a, s);
  }
  if (plain && variant == 0) return launch_fwd_t<IO, Shape64x16x4, H ? 4 : 3, true, false, false, false, true>(maps, a, s);
  if (plain && variant == 2) {
    if constexpr (H) {   // 64-byte rows: the paired-row layout when the caller could encode its 5-D maps
      if (a.paired) return launch_fwd_t<IO, Shape32x32x4, 4, true, false, false, false, true, false, true>(maps, a, s);
    }
    return launch_fwd_t<IO, Shape32x32x4, H ? 4 : 3, true, false, false, false, true>(maps, a, s);
  }
  if (variant == 2) return launch_fwd_t<IO, Shape32x32x4, H ? 4 : 3, true>(maps, a, s);
  return launch_fwd_t<IO, Shape64x16x4, H ? 4 : 3, true>(maps, a, s);
}

cudaError_t launch_scan_fwd(bool bf16, bool use_tma, int variant, const FwdMaps& maps, const ScanFwdArgs& a,
                            cudaStream_t s) {
  return bf16 ? launch_fwd_io<__nv_bfloat16>(use_tma, variant, maps, a, s) : launch_fwd_io<float>(use_tma, variant, maps, a, s);
}

template <typename K>
static cudaError_t launch_bwd(const BwdMaps& maps, const ScanBwdArgs& a, cudaStream_t s) {
  cudaError_t e;
  auto kern = K::get(e);
  if (e != cudaSuccess) return e;
  dim3 grid((a.D + K::CH - 1) / K::CH, a.B);
  e = launch_pdl(kern, grid, K::THREADS, K::BYTES, s, maps, a, K::IS_SPLIT ? a.split : 1);
  if (e != cudaSuccess || a.ticket || !a.dlambda) return e;
  rglru_dlambda_kernel<<<(a.D + 255) / 256, 256, 0, s>>>(a.dlam_part, a.lambda, a.dlambda, a.B, a.D, a.c);
  if (K::IS_GROUPED && a.dgate && a.dgate_part)
    rglru_colsum_kernel<<<(2 * a.D + 255) / 256, 256, 0, s>>>(a.dgate_part, a.dgate, a.B, 2 * a.D);
  return cudaGetLastError();
}

template <typename IO, typename V, int STAGES, bool USE_TMA, bool CONV = false, bool MERGE = false, bool GROUPED = false,
          bool SELF_ISSUE = false, bool PLAIN = false, bool CARRY = false>
static cudaError_t launch_bwd_t(const BwdMaps& maps, const ScanBwdArgs& a, cudaStream_t s) {
  return launch_bwd<BwdKern<IO, V, STAGES, USE_TMA, CONV, MERGE, GROUPED, SELF_ISSUE, PLAIN, CARRY>>(maps, a, s);
}

template <typename IO, bool PLAIN>
using SplitBwd = BwdKern<IO, Shape64x16x4, sizeof(IO) == 2 ? 5 : 3, true, false, false, false, sizeof(IO) == 2, PLAIN, false, true>;
template <typename IO, bool MERGE>
using SplitGroupedBwd = BwdKern<IO, Shape64x16x4, sizeof(IO) == 2 ? (MERGE ? 4 : 5) : (MERGE ? 2 : 3), true, false, MERGE, true,
                                sizeof(IO) == 2 && !MERGE, false, false, true>;

template <typename IO>
static cudaError_t launch_bwd_io(bool use_tma, int variant, const BwdMaps& maps, const ScanBwdArgs& a, cudaStream_t s) {
  constexpr bool H = sizeof(IO) == 2;
  if (a.dx == nullptr)   // carry-only pass: producer-warp shape, masked arithmetic
    return use_tma ? launch_bwd_t<IO, Shape64x16x4, H ? 4 : 3, true, false, false, false, false, false, true>(maps, a, s)
                   : launch_bwd_t<IO, Shape64x16x4, 1, false, false, false, false, false, false, true>(maps, a, s);
  if (!use_tma) return launch_bwd_t<IO, Shape64x16x4, 1, false>(maps, a, s);
  const bool plain = a.tok == nullptr && a.T % 64 == 0;   // no step of any chunk is masked
  if (a.split > 1) {
    return plain ? launch_bwd<SplitBwd<IO, true>>(maps, a, s) : launch_bwd<SplitBwd<IO, false>>(maps, a, s);
  }
  if (variant == 3) {   // bulk copies issued by a compute thread: loads run NSTAGE - 2 chunks ahead, so one more stage
    if (plain) return launch_bwd_t<IO, Shape64x16x4, H ? 5 : 3, true, false, false, false, true, true>(maps, a, s);
    return launch_bwd_t<IO, Shape64x16x4, H ? 5 : 3, true, false, false, false, true>(maps, a, s);
  }
  if (plain) return launch_bwd_t<IO, Shape64x16x4, H ? 4 : 3, true, false, false, false, false, true>(maps, a, s);
  return launch_bwd_t<IO, Shape64x16x4, H ? 4 : 3, true>(maps, a, s);
}

cudaError_t launch_scan_bwd(bool bf16, bool use_tma, int variant, const BwdMaps& maps, const ScanBwdArgs& a,
                            cudaStream_t s) {
  return bf16 ? launch_bwd_io<__nv_bfloat16>(use_tma, variant, maps, a, s) : launch_bwd_io<float>(use_tma, variant, maps, a, s);
}

// Conv folded into the load stage: one shape (64 channels x 64 steps); the x map's box has three more rows.
cudaError_t launch_conv_scan_fwd(bool bf16, bool use_tma, const FwdMaps& maps, const ScanFwdArgs& a, cudaStream_t s) {
  if (bf16)
    return use_tma ? launch_fwd_t<__nv_bfloat16, Shape64x16x4, 4, true, true>(maps, a, s)
                   : launch_fwd_t<__nv_bfloat16, Shape64x16x4, 1, false, true>(maps, a, s);
  return use_tma ? launch_fwd_t<float, Shape64x16x4, 3, true, true>(maps, a, s)
                 : launch_fwd_t<float, Shape64x16x4, 1, false, true>(maps, a, s);
}
cudaError_t launch_conv_scan_bwd(bool bf16, bool use_tma, const BwdMaps& maps, const ScanBwdArgs& a, cudaStream_t s) {
  if (bf16)
    return use_tma ? launch_bwd_t<__nv_bfloat16, Shape64x16x4, 4, true, true, false, false, true>(maps, a, s)
                   : launch_bwd_t<__nv_bfloat16, Shape64x16x4, 1, false, true>(maps, a, s);
  return use_tma ? launch_bwd_t<float, Shape64x16x4, 3, true, true>(maps, a, s)
                 : launch_bwd_t<float, Shape64x16x4, 1, false, true>(maps, a, s);
}

// Branch merge folded into the store stage (forward) and the load stage (backward), with or without the
// conv fold: one shape (64 channels x 64 steps).  One more tile per stage, so fp32 backward keeps two stages.
template <typename IO, bool CONV>
static cudaError_t launch_merge_fwd_t(bool use_tma, const FwdMaps& maps, const ScanFwdArgs& a, cudaStream_t s) {
  constexpr bool H = sizeof(IO) == 2;
  return use_tma ? launch_fwd_t<IO, Shape64x16x4, H ? (CONV ? 4 : 3) : 3, true, CONV, true>(maps, a, s)
                 : launch_fwd_t<IO, Shape64x16x4, 1, false, CONV, true>(maps, a, s);
}
template <typename IO, bool CONV>
static cudaError_t launch_merge_bwd_t(bool use_tma, const BwdMaps& maps, const ScanBwdArgs& a, cudaStream_t s) {
  constexpr bool H = sizeof(IO) == 2;
  if (!use_tma) return launch_bwd_t<IO, Shape64x16x4, 1, false, CONV, true>(maps, a, s);
  // bf16: four stages without a producer warp (eight warps leave these variants the registers they need);
  // fp32 fits two stages only, which the producer warp needs to keep a load ahead
  if constexpr (H) return launch_bwd_t<IO, Shape64x16x4, 4, true, CONV, true, false, true>(maps, a, s);
  else return launch_bwd_t<IO, Shape64x16x4, 2, true, CONV, true>(maps, a, s);
}
cudaError_t launch_merge_fwd(bool bf16, bool use_tma, bool conv, const FwdMaps& maps, const ScanFwdArgs& a, cudaStream_t s) {
  if (bf16) return conv ? launch_merge_fwd_t<__nv_bfloat16, true>(use_tma, maps, a, s)
                        : launch_merge_fwd_t<__nv_bfloat16, false>(use_tma, maps, a, s);
  return conv ? launch_merge_fwd_t<float, true>(use_tma, maps, a, s) : launch_merge_fwd_t<float, false>(use_tma, maps, a, s);
}
cudaError_t launch_merge_bwd(bool bf16, bool use_tma, bool conv, const BwdMaps& maps, const ScanBwdArgs& a, cudaStream_t s) {
  if (bf16) return conv ? launch_merge_bwd_t<__nv_bfloat16, true>(use_tma, maps, a, s)
                        : launch_merge_bwd_t<__nv_bfloat16, false>(use_tma, maps, a, s);
  return conv ? launch_merge_bwd_t<float, true>(use_tma, maps, a, s) : launch_merge_bwd_t<float, false>(use_tma, maps, a, s);
}

// Grouped gate layout (one [B, T, 2 D] gate tensor, biases added in the kernel), with or without the
// branch merge; TMA staging only, one shape (64 channels x 64 steps).
template <typename IO, bool MERGE>
static cudaError_t launch_grouped_fwd_t(const FwdMaps& maps, const ScanFwdArgs& a, cudaStream_t s) {
  constexpr bool H = sizeof(IO) == 2;
  constexpr int ST = H ? (MERGE ? 3 : 4) : 3;
  if (a.split > 1) return launch_fwd<SplitGroupedFwd<IO, MERGE>>(maps, a, s);
  return launch_fwd_t<IO, Shape64x16x4, ST, true, false, MERGE, true>(maps, a, s);
}
template <typename IO, bool MERGE>
static cudaError_t launch_grouped_bwd_t(const BwdMaps& maps, const ScanBwdArgs& a, cudaStream_t s) {
  constexpr bool H = sizeof(IO) == 2;
  // Measured on B200 at B = 16, T = 2048, D = 1024 bf16: with the branch merge (five loads and four stores per
  // chunk) the producer warp wins although the kernel then spills a little at its 168-register limit (162 us
  // against 169 us with the copies issued by a compute thread); without the merge the compute-thread variant does.
  constexpr bool SELF = H && !MERGE;
  constexpr int ST = SELF ? 5 : (H ? 4 : (MERGE ? 2 : 3));
  if (a.split > 1) return launch_bwd<SplitGroupedBwd<IO, MERGE>>(maps, a, s);
  return launch_bwd_t<IO, Shape64x16x4, ST, true, false, MERGE, true, SELF>(maps, a, s);
}
cudaError_t launch_grouped_fwd(bool bf16, bool merge, const FwdMaps& maps, const ScanFwdArgs& a, cudaStream_t s) {
  if (bf16) return merge ? launch_grouped_fwd_t<__nv_bfloat16, true>(maps, a, s) : launch_grouped_fwd_t<__nv_bfloat16, false>(maps, a, s);
  return merge ? launch_grouped_fwd_t<float, true>(maps, a, s) : launch_grouped_fwd_t<float, false>(maps, a, s);
}
cudaError_t launch_grouped_bwd(bool bf16, bool merge, const BwdMaps& maps, const ScanBwdArgs& a, cudaStream_t s) {
  if (bf16) return merge ? launch_grouped_bwd_t<__nv_bfloat16, true>(maps, a, s) : launch_grouped_bwd_t<__nv_bfloat16, false>(maps, a, s);
  return merge ? launch_grouped_bwd_t<float, true>(maps, a, s) : launch_grouped_bwd_t<float, false>(maps, a, s);
}
int grouped_box_cols() { return Shape64x16x4::CH; }

// CTAs that share one (batch row, channel tile) along time in a call of this shape, 1 for none (see pick_split).  The
// plain forward has the 32-channel shape to fall back on, which fills the machine twice as well as 64-channel tiles:
// pairs of CTAs do not beat it, three or more do (bf16, T = 2048, D = 1024, unsplit 32-channel / split: B = 6 27 / 33 us
// in pairs, B = 5 27 / 25 us in threes, B = 1 19 / 11 us in eights; fp32 B = 4 25 / 31 in pairs, B = 2 24 / 18 in fours).
template <bool MERGE, bool GROUPED>
static int split_of(bool fwd, bool bf16, int B, int T, int D) {
  const long long tiles = static_cast<long long>(B) * ((D + 63) / 64);
  const int nchunks = (T + 63) / 64;
  using H = __nv_bfloat16;
  if constexpr (GROUPED) {
    if (fwd) return bf16 ? pick_split<SplitGroupedFwd<H, MERGE>>(tiles, nchunks) : pick_split<SplitGroupedFwd<float, MERGE>>(tiles, nchunks);
    return bf16 ? pick_split<SplitGroupedBwd<H, MERGE>>(tiles, nchunks) : pick_split<SplitGroupedBwd<float, MERGE>>(tiles, nchunks);
  } else {
    if (fwd) return bf16 ? pick_split<SplitFwd<H, false>>(tiles, nchunks) : pick_split<SplitFwd<float, false>>(tiles, nchunks);
    return bf16 ? pick_split<SplitBwd<H, false>>(tiles, nchunks) : pick_split<SplitBwd<float, false>>(tiles, nchunks);
  }
}
int scan_split(bool fwd, bool bf16, int B, int T, int D) {
  static const bool forced = fwd_variant_exists(env_override("RGLRU_FWD_VARIANT")) || bwd_variant_exists(env_override("RGLRU_BWD_VARIANT"));
  if (forced) return 1;
  const int split = split_of<false, false>(fwd, bf16, B, T, D);
  return fwd && split < 3 ? 1 : split;      // see scan_fwd_variant
}
// In the layer the gate tensor has just been written and much of it is still in L2.  There the bf16 forward without the branch
// product is faster unsplit than in pairs (D = 1024, forward of the layer unsplit / pairs: 96 tiles T = 2048 53 / 57 us,
// T = 1200 34 / 38, 128 tiles T = 2048 57 / 60, T = 512 23 / 25, T = 16384 406 / 414, 16 tiles T = 128 10 / 12; three and more
// win: 80 tiles 51 / 45, 64 tiles 48 / 36).
// With the product (96 tiles 151 / 146, 128 tiles 182 / 174 in the block), and for fp32 (60 tiles 88 / 84), pairs win too.
int grouped_split(bool fwd, bool bf16, bool merge, int B, int T, int D) {
  if (merge) return split_of<true, true>(fwd, bf16, B, T, D);
  const int split = split_of<false, true>(fwd, bf16, B, T, D);
  return fwd && bf16 && split < 3 ? 1 : split;
}

int raw_box_rows() { return RAW_TC; }
int raw_box_cols() { return CH; }

template <int NSTAGE, bool USE_TMA, bool SPLIT>
struct RawFwdKern {
  static constexpr int THREADS = RAW_NT, BYTES = RawSmem<NSTAGE, 2, SPLIT>::BYTES;
  using Fn = void (*)(RawFwdMaps, RawScanArgs);
  static Fn get(cudaError_t& e) {
    Fn kern = rawscan_fwd_kernel<NSTAGE, USE_TMA, SPLIT>;
    e = set_smem<RawFwdKern>(kern, BYTES);
    return kern;
  }
};
template <int NSTAGE, bool USE_TMA, bool SPLIT>
struct RawBwdKern {
  static constexpr int THREADS = RAW_NT, BYTES = RawSmem<NSTAGE, 3, SPLIT>::BYTES;
  using Fn = void (*)(RawBwdMaps, RawScanArgs);
  static Fn get(cudaError_t& e) {
    Fn kern = rawscan_bwd_kernel<NSTAGE, USE_TMA, SPLIT>;
    e = set_smem<RawBwdKern>(kern, BYTES);
    return kern;
  }
};
template <typename K, typename Maps>
static cudaError_t launch_raw(const Maps& maps, const RawScanArgs& a, int split, cudaStream_t s) {
  cudaError_t e;
  auto kern = K::get(e);
  if (e != cudaSuccess) return e;
  return launch_pdl(kern, dim3((a.D + CH - 1) / CH, a.B), K::THREADS, K::BYTES, s, maps, a, split);
}
using RawSplitFwd = RawFwdKern<RAW_STAGES, true, true>;
using RawSplitBwd = RawBwdKern<RAW_STAGES, true, true>;
int raw_split(bool fwd, int B, int T, int D) {
  const long long tiles = static_cast<long long>(B) * ((D + CH - 1) / CH);
  const int nchunks = (T + RAW_TC - 1) / RAW_TC;
  return fwd ? pick_split<RawSplitFwd>(tiles, nchunks) : pick_split<RawSplitBwd>(tiles, nchunks);
}
cudaError_t launch_raw_fwd(bool use_tma, const RawFwdMaps& maps, const RawScanArgs& a, cudaStream_t s) {
  if (!use_tma) return launch_raw<RawFwdKern<1, false, false>>(maps, a, 1, s);
  const int split = raw_split(true, a.B, a.T, a.D);
  return split > 1 ? launch_raw<RawSplitFwd>(maps, a, split, s) : launch_raw<RawFwdKern<RAW_STAGES, true, false>>(maps, a, 1, s);
}
cudaError_t launch_raw_bwd(bool use_tma, const RawBwdMaps& maps, const RawScanArgs& a, cudaStream_t s) {
  if (!use_tma) return launch_raw<RawBwdKern<1, false, false>>(maps, a, 1, s);
  const int split = raw_split(false, a.B, a.T, a.D);
  return split > 1 ? launch_raw<RawSplitBwd>(maps, a, split, s) : launch_raw<RawBwdKern<RAW_STAGES, true, false>>(maps, a, 1, s);
}

int conv_tma_box_rows() { return 64 + 3; }
int conv_tma_box_cols() { return 64; }

template <typename IO>
static cudaError_t conv_tma_fwd_t(const ConvMaps& maps, const ConvTmaArgs& a, cudaStream_t s) {
  constexpr int ST = sizeof(IO) == 2 ? 4 : 3;
  auto kern = conv_tma_fwd_kernel<IO, ST>;
  constexpr int bytes = ConvFwdSmem<IO, ST>::BYTES;
  cudaError_t e = set_smem<KernelTag<ConvFwdSmem<IO, ST>>>(kern, bytes);
  if (e != cudaSuccess) return e;
  kern<<<dim3((a.D + 63) / 64, a.B), 288, bytes, s>>>(maps, a);
  return cudaGetLastError();
}
cudaError_t launch_conv_tma_fwd(bool bf16, const ConvMaps& maps, const ConvTmaArgs& a, cudaStream_t s) {
  return bf16 ? conv_tma_fwd_t<__nv_bfloat16>(maps, a, s) : conv_tma_fwd_t<float>(maps, a, s);
}
template <typename IO>
static cudaError_t conv_tma_bwd_t(const ConvMaps& maps, const ConvTmaArgs& a, cudaStream_t s) {
  constexpr int ST = sizeof(IO) == 2 ? 4 : 2;   // about 100 KB either way: two CTAs per SM
  auto kern = conv_tma_bwd_kernel<IO, ST>;
  constexpr int bytes = ConvBwdSmem<IO, ST>::BYTES;
  static_assert(bytes <= 232448, "shared memory of one CTA");
  cudaError_t e = set_smem<KernelTag<ConvBwdSmem<IO, ST>>>(kern, bytes);
  if (e != cudaSuccess) return e;
  kern<<<dim3((a.D + 63) / 64, a.B), 288, bytes, s>>>(maps, a);
  return cudaGetLastError();
}
cudaError_t launch_conv_tma_bwd(bool bf16, const ConvMaps& maps, const ConvTmaArgs& a, cudaStream_t s) {
  return bf16 ? conv_tma_bwd_t<__nv_bfloat16>(maps, a, s) : conv_tma_bwd_t<float>(maps, a, s);
}

}  // namespace rglru
