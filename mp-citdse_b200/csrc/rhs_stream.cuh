// rhs_stream.cuh -- the dipole-coupling pass of one right-hand-side
// evaluation, streaming every dipole block through shared memory once.
//
// Replaces the 4 strided cblas_dgemv calls per dipole block of
// MatVecV/MatVecL::operator() (src/tdse/tdse.cpp:28-68, :99-139), which read
// each block four times (Re/Im x D/D^T).  Here each element D[r][c] of block
// L is read once from HBM and used twice:
//   row partial  P_row[r] += D[r][c] * y_{L+1}[c]   (D_L y_{L+1} -> block L)
//   col partial  P_col[c] += D[r][c] * y_L[r]       (D_L^T y_L   -> block L+1)
// with y complex and D real, 4 DFMA per element.
//
// Layout: one persistent CTA per SM.  Warp 8 is the producer: one lane
// issues 2-D TMA loads of 16x256 tiles (with an L2 evict-first hint: the
// blocks are streamed once per pass) plus a 1-D bulk copy of the tile's 16
// stage-vector rows into a kStages-deep shared-memory ring (full/empty
// mbarriers).  Warps 0-7 consume: warp w takes rows 2w and 2w+1
// of each tile; lane l holds the 8 columns {64j + 2l, 64j + 2l + 1}, j<4, of
// the current strip.
//   - Row partials are complete for the strip after a reduce-scatter across
//     the warp, two tiles at a time where the strip has two (9 shuffles and
//     one chain of latencies for both, not 12 and two); they are staged in
//     shared memory (two buffers of kRpRows rows) and written to
//     RP[strip][row] by one bulk store per run of consecutive rows.
//   - Column partials accumulate in registers while the CTA walks down a
//     strip; when the strip (or the CTA's range) ends, the 8 warps' partials
//     are summed in shared memory (warps 0..3, each with its partner 4..7)
//     and stored as one slot CP[slot][0..255].
// Every output is written by exactly one thread in a fixed order, so repeated
// runs give identical bits.
//
// What bounds it: blocks beyond L2 the HBM stream; blocks that fit the tile
// rate from L2 and, per pass, about 6 us of the combine pass and of latencies
// at both ends.  The consumers have to stay well ahead of the ring: with one
// tile at a time (a select per operand for the timed-out case, two shuffle
// chains) they cost 17-20 % over the bare stream.  Measured, 60 steps on
// 18,000 states (491 MB of blocks): 63.5 -> 57.7 ms; 150 steps on 5,712
// states (52 MB): 30.5 -> 25.5 ms.
// kPrefill: tiles requested while the previous kernel, the combine pass, is
// still at work.  Their loads queue before the combine's own, whose latency
// everything waits for: 1 / 2 / 3 / 4 tiles give 25.5 / 25.7 / 26.1 / 26.5 ms
// on the 52 MB blocks, and no difference beyond the noise on the 491 MB ones.
// kStages: 3 / 4 / 6 stages give 59.0 / 57.7 / 59.6 ms on the large blocks and
// 25.6 / 25.7 / 25.9 ms on the small ones, at two tiles of prefill.
#pragma once
#include <cuda.h>

#include "dev_util.cuh"
#include "plan.h"
#include "stream_types.h"

namespace mpc {


__device__ __forceinline__ double2 ld_y(const double2* y, int idx) {
  return __ldg(y + idx);
}

__global__ void __launch_bounds__(kStreamThreads, 1)
    k_rhs_stream(const __grid_constant__ StreamArgs a, const __grid_constant__ TmapSet tm) {
  extern __shared__ __align__(1024) unsigned char smem[];
  double* tiles = reinterpret_cast<double*>(smem);
  double2* yrows = reinterpret_cast<double2*>(smem + kStages * kTileBytes);
  double2* red = reinterpret_cast<double2*>(smem + kStages * (kTileBytes + kYRowBytes));
  double2* rpbuf =
      reinterpret_cast<double2*>(smem + kStages * (kTileBytes + kYRowBytes) + kRedBytes);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * (kTileBytes + kYRowBytes) +
                                               kRedBytes + kRpStageBytes);
  uint64_t* empty = full + kStages;

  const Geometry& g = a.g;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int t_begin = (int)((long long)g.ntiles * blockIdx.x / gridDim.x);
  const int t_end = (int)((long long)g.ntiles * (blockIdx.x + 1) / gridDim.x);

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1 + (s == 0 ? a.skew : 0u));
      mbar_init(&empty[s], kConsumerWarps);
    }
    fence_mbar_init();
  }
  __syncthreads();
  pdl_trigger();
  if (t_begin >= t_end) {
    pdl_wait();
    return;
  }

  if (warp == kConsumerWarps) {
    // ---------------- producer ----------------
    if (lane != 0) {
      pdl_wait();
      return;
    }
    const uint64_t stream_policy = make_evict_first_policy();
    const uint64_t keep_policy = make_evict_last_policy();
    const int keep_end = t_begin + (int)(a.keep_frac * (float)(t_end - t_begin));
    // The dipole blocks do not change between launches: the first kPrefill
    // tiles are requested before waiting for the previous kernel;
    // their stage-vector rows (written by that kernel) only after it.
    const int pre = min(t_end - t_begin, kPrefill);
    for (int i = 0; i < pre; ++i) {
      int b, s, rt;
      decode_tile(g, t_begin + i, b, s, rt);
      mbar_arrive_expect_tx(&full[i], kTileBytes + kYRowBytes);
      tma_load_2d_hint(tiles + i * (kTileR * kStripW), &tm.m[b], &full[i], s * kStripW,
                       rt * kTileR, t_begin + i < keep_end ? keep_policy : stream_policy);
    }
    pdl_wait();
    int issued = 0;
    bool late = false;   // the consumers gave up
    for (int t = t_begin; t < t_end; ++t, ++issued) {
      const int stage = issued % kStages;
      const int round = issued / kStages;
      int b, s, rt;
      decode_tile(g, t, b, s, rt);
      if (issued >= pre) {
        if (round > 0 && !mbar_wait_bounded(&empty[stage], (round - 1) & 1, a.status)) {
          late = true;
          break;
        }
        mbar_arrive_expect_tx(&full[stage], kTileBytes + kYRowBytes);
        tma_load_2d_hint(tiles + stage * (kTileR * kStripW), &tm.m[b], &full[stage],
                         s * kStripW, rt * kTileR, t < keep_end ? keep_policy : stream_policy);
      }
      // the tile's 16 rows of the stage vector (the vector carries a zeroed
      // tail of kVecPad entries, so the last tile never reads past it)
      bulk_load(yrows + stage * kTileR, a.y + g.blk[b].row_off + rt * kTileR, kYRowBytes,
                &full[stage]);
    }
    // Do not leave while a load is in flight: wait until every issued tile
    // was released by the consumers, or, once they gave up, until it landed,
    // with one limit for all that is left.
    unsigned long long deadline = late ? globaltimer_ns() + kWaitLimitNs : 0;
    for (int i = (issued > kStages ? issued - kStages : 0); i < issued; ++i) {
      const int stage = i % kStages;
      const int round = i / kStages;
      if (!late && !mbar_wait_bounded(&empty[stage], round & 1, a.status)) {
        late = true;
        deadline = globaltimer_ns() + kWaitLimitNs;
      }
      if (late) mbar_wait_until(&full[stage], round & 1, deadline);
    }
    return;
  }

  // ---------------- consumers ----------------
  pdl_wait();
  double2 ycol[8];
  double2 cacc[8];
  int cur_b = -1, cur_s = -1;
  int slot = a.cta_slot0[blockIdx.x] - 1;
  const int ctid = threadIdx.x;  // 0..255 among consumers

  auto flush_cols = [&](int b) {
    // warp partials -> shared in two halves (a whole set would cost the ring a
    // stage), then a fixed-order sum
    double2* mine = red + (warp % kRedWarps) * kStripW + 2 * lane;
    if (warp < kRedWarps) {
#pragma unroll
      for (int j = 0; j < 8; ++j) mine[64 * (j / 2) + j % 2] = cacc[j];
    }
    named_bar_sync(1, kConsumerWarps * 32);
    if (warp >= kRedWarps) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        double2 v = mine[64 * (j / 2) + j % 2];
        v.x += cacc[j].x;
        v.y += cacc[j].y;
        mine[64 * (j / 2) + j % 2] = v;
      }
    }
    named_bar_sync(1, kConsumerWarps * 32);
    double2 acc = red[ctid];
#pragma unroll
    for (int w = 1; w < kRedWarps; ++w) {
      const double2 v = red[w * kStripW + ctid];
      acc.x += v.x;
      acc.y += v.y;
    }
    a.CP[(long long)slot * kStripW + ctid] = acc;
    named_bar_sync(1, kConsumerWarps * 32);
    (void)b;
  };

  // Row partials of the current run of consecutive rows [seg_r0, seg_r0 +
  // seg_n) of strip seg_s of block seg_b, staged in rpbuf[rp_cur]; flushed by
  // one bulk store when the run ends or the buffer is full.  The store of
  // the other buffer must have read its rows before that buffer is reused.
  int rp_cur = 0, seg_b = -1, seg_s = 0, seg_r0 = 0, seg_n = 0;
  auto flush_rows = [&]() {
    if (seg_n == 0) return;
    fence_proxy_async_smem();
    named_bar_sync(2, kConsumerWarps * 32);
    if (ctid == 0) {
      const BlockGeom& sb = g.blk[seg_b];
      const int nv = min(seg_n, sb.nrow - seg_r0);  // rows past the block's end are not stored
      bulk_store(a.RP + sb.rp_off + (long long)seg_s * sb.nrow + seg_r0, rpbuf + rp_cur * kRpRows,
                 (uint32_t)nv * 16u);
      bulk_commit();
      bulk_wait_read<1>();
    }
    named_bar_sync(2, kConsumerWarps * 32);
    rp_cur ^= 1;
    seg_n = 0;
  };

  // After a timed-out wait a lane keeps walking its tiles, on whatever the slots
  // hold, so that its warp stays together in the reductions (another lane's wait
  // may have come through) and reaches each named barrier; the raised status
  // makes the host discard the result.  Slots are released by lane 0, as long as
  // its own waits come through: the producer stops at its next wait for one.
  // (The warp's vote on each wait instead: +0.4 % on 52 MB of blocks.)
  bool dead = false;
  int stage = 0, phase = 0;  // of the next tile
  // The next tile: this warp's two rows' sums over its columns into w (row
  // 2 warp: re, im; row 2 warp + 1: re, im), its columns' into cacc.
  auto tile = [&](double* w) {
    if (!dead && !mbar_wait_bounded(&full[stage], phase, a.status)) dead = true;
    // rows past the block's end meet zero-filled dipole rows, so their
    // (finite) stage-vector entries contribute nothing
    const double2 yr0 = yrows[stage * kTileR + 2 * warp];
    const double2 yr1 = yrows[stage * kTileR + 2 * warp + 1];
    const double* T = tiles + stage * (kTileR * kStripW);
    const double* T0 = T + (2 * warp) * kStripW + 2 * lane;
    const double* T1 = T0 + kStripW;
    double2 ra = make_double2(0.0, 0.0), rb = make_double2(0.0, 0.0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double2 d0 = *reinterpret_cast<const double2*>(T0 + 64 * j);
      const double2 d1 = *reinterpret_cast<const double2*>(T1 + 64 * j);
      const double2 c0 = ycol[2 * j], c1 = ycol[2 * j + 1];
      ra.x = fma(d0.x, c0.x, ra.x); ra.x = fma(d0.y, c1.x, ra.x);
      ra.y = fma(d0.x, c0.y, ra.y); ra.y = fma(d0.y, c1.y, ra.y);
      rb.x = fma(d1.x, c0.x, rb.x); rb.x = fma(d1.y, c1.x, rb.x);
      rb.y = fma(d1.x, c0.y, rb.y); rb.y = fma(d1.y, c1.y, rb.y);
      double2& q0 = cacc[2 * j];
      double2& q1 = cacc[2 * j + 1];
      q0.x = fma(d0.x, yr0.x, q0.x); q0.x = fma(d1.x, yr1.x, q0.x);
      q0.y = fma(d0.x, yr0.y, q0.y); q0.y = fma(d1.x, yr1.y, q0.y);
      q1.x = fma(d0.y, yr0.x, q1.x); q1.x = fma(d1.y, yr1.x, q1.x);
      q1.y = fma(d0.y, yr0.y, q1.y); q1.y = fma(d1.y, yr1.y, q1.y);
    }
    __syncwarp();
    if (lane == 0 && !dead) mbar_arrive(&empty[stage]);
    if (++stage == kStages) {
      stage = 0;
      phase ^= 1;
    }
    w[0] = ra.x;
    w[1] = ra.y;
    w[2] = rb.x;
    w[3] = rb.y;
  };
  // A reduce-scatter step over lane bit OFF: half of the 2 N values stay.
  auto halve = [&](double* v, int n, int off) {
    const bool up = (lane & off) != 0;
    for (int i = 0; i < n; ++i) {
      const double keep = up ? v[i + n] : v[i], send = up ? v[i] : v[i + n];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  };
  int t = t_begin;
  int b, s, rt;
  if (t < t_end) decode_tile(g, t, b, s, rt);
  while (t < t_end) {
    const BlockGeom& bg = g.blk[b];
    // two tiles of the strip at a time where there are two: their chains and
    // shuffles overlap, and the eight sums reduce in nine shuffles, not twelve
    const int two = t + 1 < t_end && rt + 1 < bg.nrtiles ? 1 : 0;
    if (b != seg_b || s != seg_s || seg_n + kTileR * (1 + two) > kRpRows ||
        rt * kTileR != seg_r0 + seg_n) {
      flush_rows();
      seg_b = b;
      seg_s = s;
      seg_r0 = rt * kTileR;
    }
    const int rp_local = rt * kTileR - seg_r0;  // the first tile's first row in the buffer
    seg_n += kTileR * (1 + two);
    if (b != cur_b || s != cur_s) {
      if (cur_b >= 0) flush_cols(cur_b);
      ++slot;
      cur_b = b;
      cur_s = s;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int c = s * kStripW + 64 * j + 2 * lane + e;
          ycol[2 * j + e] = (c < bg.ncol) ? ld_y(a.y, bg.col_off + c) : make_double2(0.0, 0.0);
          cacc[2 * j + e] = make_double2(0.0, 0.0);
        }
      }
    }
    double w[8];
    tile(w);
    double* rp = reinterpret_cast<double*>(rpbuf + rp_cur * kRpRows + rp_local + 2 * warp);
    if (two) {
      tile(w + 4);
      // lane bits 16, 8, 4 -> tile, row, re/im
      halve(w, 4, 16);
      halve(w, 2, 8);
      halve(w, 1, 4);
      double z = w[0];
      z += __shfl_xor_sync(0xffffffffu, z, 2);
      z += __shfl_xor_sync(0xffffffffu, z, 1);
      if ((lane & 3) == 0)
        rp[(lane & 16 ? 2 * kTileR : 0) + (lane & 8 ? 2 : 0) + (lane & 4 ? 1 : 0)] = z;
      t += 2;
      rt += 2;
    } else {
      // lane bits 16, 8 -> row, re/im
      halve(w, 2, 16);
      halve(w, 1, 8);
      double z = w[0];
      z += __shfl_xor_sync(0xffffffffu, z, 4);
      z += __shfl_xor_sync(0xffffffffu, z, 2);
      z += __shfl_xor_sync(0xffffffffu, z, 1);
      if ((lane & 7) == 0) rp[(lane & 16 ? 2 : 0) + (lane & 8 ? 1 : 0)] = z;
      ++t;
      ++rt;
    }
    if (rt >= bg.nrtiles && t < t_end) decode_tile(g, t, b, s, rt);
  }
  flush_rows();
  if (cur_b >= 0) flush_cols(cur_b);
  if (ctid == 0) bulk_wait<0>();  // the last stores complete before the grid does
}

}  // namespace mpc
