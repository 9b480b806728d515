// flow_batch.cuh -- many pulses on a system whose coupling fits on chip: one
// persistent cooperative launch for all steps of all pulses, each right-hand
// side an FP64 tensor-core product (mma.sync m8n8k4 .f64) whose left operand,
// the coupling, never leaves the registers.
//
// Layout.  The CTAs form ng column groups; a group's CTAs together hold every
// row once, and each group works on its own pulses, in chunks of 8.  A CTA's
// rows lie in one state block L, so they all couple to the same window
// (blocks L-1 and L+1).  Its 8 compute warps split the window: warp w takes
// every 8th group of 4 window rows, and keeps the MT x KT m8k4 fragments of its
// share of the coupling in registers.  A window element (one pulse, re and im)
// is one 16-byte load per lane straight into the right operand's fragment
// layout: lane (k, pulse) of a 4 x 8 tile feeds one m8n8 tile with the real
// parts and one with the imaginary parts.  So a step of the loop is one load
// and 2 MT DMMAs, with no shared memory in between; the warps' partial sums
// meet in shared memory once per item, where one thread per (row, pulse) does
// the rest of the item in FP64.
//
// Why: the stage GEMM (batch_stage.cuh) reloads coupling tiles for every
// product and leaves most SMs idle below about 128 pulses (90 tiles at 48
// pulses); here every SM holds its share for the whole run whatever the width,
// and the chunks hide each other's exchange.
//
// Exchange as in resident_flow.cuh: rows are published with 16-byte stores and
// polled by their readers in buffers preset to kEmpty; a chunk's buffers
// rotate by step, a helper warp presets them and does the per-pulse control
// (norms, times, fields, step sizes) from all CTAs' partial sums, redundantly
// and identically in every CTA.
//
// Modes: 0 fixed step (12 Horner products, the reference's semantics),
// 1 adaptive (13 stages, embedded error, per-pulse step control), 2 the
// transposed Horner products of the objective gradient.
#pragma once
#include <cuda_runtime.h>

#include "batch_types.h"
#include "dev_util.cuh"
#include "plan.h"
#include "resident_flow.cuh"
#include "rkf78.h"

namespace mpc {

constexpr int CP = 8;               // pulses per chunk
constexpr int kMaxChunks = 32;      // chunks per column group and launch
constexpr int kMaxMT = 6;           // 8-row tiles per CTA

struct FbCta {
  int L, row0, nrows;
  int grp, idx;      // column group, index within it
  int cfg;           // which MT x KT instance
};

struct FbArgs {
  const double* D;
  const double* eps;
  const FbCta* cta;
  int gp;                 // CTAs per column group
  int ng;                 // column groups
  int nch;                // chunks of this launch: chunk c belongs to group c % ng
  const int* cid;         // [nch][CP] pulse ids (-1: empty slot)
  const int* csteps;      // [nch] steps of the chunk's longest pulse (descending per group)
  double2* V;             // [nch][slots][ntot][CP] vectors in flight
  int slots;
  int mt;                 // most 8-row tiles of a CTA
  double* part;           // [nch][2][gp][2 * CP] norm (and error) partials
  unsigned long long* ctr;  // [nch] helpers' arrivals
  unsigned* status;
  double2* xst;           // [nch][ntot][CP] the step's x
  const double2* in;      // start states by pulse id, [id][ntot]
  double2* out;           // final states by pulse id
  const mpc_pulse* pulse; // by pulse id
  const double* t0;       // by pulse id
  const int* nsteps;      // by pulse id
  const double* Ftab;     // [step][ldf] by pulse id, or null: the pulses' own fields
  int ldf;
  double dt;
  int gauge;
  int pop_index;
  long long hist_ld;
  double* pop_hist;       // [id][hist_ld]
  double* norm_hist;      // [id][hist_ld]
  // the objective gradient (null when unused).  Chunk vectors [nch][ntot][CP]
  // lie cvec apart, the same vector of all chunks:
  const double2* start;   // the first step's state, instead of `in`, ...
  const double* start_nrm;  // ... and its norm by pulse id, hist_ld apart (null: 1)
  double2* ckpt;          // slot k: x after k * ckpt_every steps, not yet renormalised
  int ckpt_every;
  double2* seg_v;         // step n >= seg_from: slot (n - seg_from) * 13 + m holds v_m, + 12 x_n
  int seg_from;
  long long cvec;
  int len;                // mode 2: steps swept, the last first
  const double* norms;    // mode 2: [id][hist_ld] norm of step n
  double2* lam;           // mode 2: dJ/dx in and out
  double2* xb;            // mode 2: the sum over m of G_m vbar_m
  double* fs;             // mode 2: [nch][ntot][CP] dJ/dF of the step so far
  double* fpart;          // mode 2: [len][nch][gp][CP]
  // adaptive steps
  const double* t_end;    // by pulse id
  double h0, dt_max, rtol, atol;
  int max_attempts;
  double2* kst;           // [12] slopes, cvec apart; null: in shared memory
  double2* xnew;          // the attempt's x_new
  int* nacc;              // results by pulse id
  int* nrej;
  double* tf;
  int* gave_up;
  BarrierCfg bc;
  Geometry g;
};

__device__ __forceinline__ void dmma884(double* c, double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// What the helper tells the compute warps about a chunk.
struct FbCtl {
  double2 nrm[kMaxChunks][CP];   // norm of x and its reciprocal
  double F[kMaxChunks][CP];      // the step's field
  double t[kMaxChunks][CP];
  int id[kMaxChunks][CP];
  int ns[kMaxChunks][CP];        // the pulse's steps
  int nst[kMaxChunks];           // the chunk's steps
  volatile int step[kMaxChunks]; // control is done up to this step
  volatile int progress;         // (step, chunk) pairs the compute warps finished
  volatile int hdead, mexit;
  volatile int mdead[2];         // a wait ran out, by item parity
};

// What adaptive steps need besides.
constexpr int kMaxAdapt = 16;       // chunks per column group and launch
struct FbAdapt {
  double F[kMaxAdapt][kNumStages][CP];   // the attempt's stage fields
  double h[kMaxAdapt][CP];      // proposed next step
  double hatt[kMaxAdapt][CP];   // step of the attempt
  double t_end[kMaxAdapt][CP];
  int acc[kMaxAdapt][CP];       // the last attempt was accepted
  int ret[kMaxAdapt][CP];       // the pulse ended with it
  int done[kMaxAdapt][CP];      // 1 at t_end, 2 gave up, 3 empty slot
  int lastst[kMaxAdapt][CP];    // the attempt ends at t_end
  int cnt[kMaxAdapt][3][CP];    // accepted, rejected, attempts
  int alive[kMaxAdapt];         // the chunk has pulses left
};

struct FbView {
  FlowWin w;
  int r0;           // first row within block L
  int nrows, row0, L, nc, grp, idx;
  long long cpitch; // V elements per chunk
  long long spitch; // V elements per slot
};

__device__ __forceinline__ const double2* fb_slot(const FbArgs& a, const FbView& u, int c, int slot) {
  return a.V + u.cpitch * (c * a.ng + u.grp) + u.spitch * slot;
}

// ---- one item: the coupling of one chunk's window, summed over the warps ----
template <int MT, int KT>
struct FbTile {
  // Window loads go out in batches, one batch ahead of the DMMAs: single loads
  // issued a few steps ahead share their scoreboards with the DMMAs, whose
  // waits then also wait for the loads (400 cycles per step, measured, against
  // 270 in batches of 3 to 6 and 192 of DMMA).  The rest is L2: all of a
  // group's CTAs read the same fresh lines at about the same time, at 12 bytes
  // per cycle and SM in such bursts (27 when the SMs stream apart).  Tried: a
  // copy ring in shared memory (cp.async) instead of registers (twice as slow:
  // what is not there yet is sent for again), the coupling in shared memory
  // and longer batches (+20 to +50 %), separate epilogue warps (+2 %).
  static constexpr int BD = MT * KT > 60 || KT <= 6 ? 3 : 4;
  static constexpr int NB = (KT + BD - 1) / BD;
  double A[MT][KT];
  double2 b[2][BD];
  int nj;                      // groups of 4 window rows of this warp
  int klast, nlo;              // the last lanes' rows are clamped to the window
  int k0;
  long long lo, up;            // element offsets of the two blocks' rows

  __device__ __forceinline__ void init(const FbArgs& a, const FbView& u, int warp, int lane) {
    const int K = u.w.K();
    nj = max(0, (K - 4 * warp + 4 * FW - 1) / (4 * FW));
    klast = K - 1;
    nlo = u.w.nlo;
    k0 = 4 * warp + (lane & 3);
    lo = (long long)u.w.lo0 * CP + (lane >> 2);
    up = (long long)(u.w.up0 - u.w.nlo) * CP + (lane >> 2);
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int j = 0; j < KT; ++j) {
        const int lr = m * 8 + (lane >> 2), k = k0 + 4 * FW * j;
        A[m][j] = (lr < u.nrows && k < K)
                      ? flow_coupling(a.g, a.D, a.gauge, u.L, u.r0 + lr, u.w, k)
                      : 0.0;
      }
  }
  // this lane's element of the warp's j-th group (past the window: its last
  // row, against a zero coupling)
  __device__ __forceinline__ const double2* at(const double2* src, int j) const {
    const int k = min(k0 + 4 * FW * j, klast);
    return src + (k < nlo ? lo : up) + k * CP;
  }
  __device__ __forceinline__ void load(const double2* src, int nb) {
#pragma unroll
    for (int i = 0; i < BD; ++i)
      if (nb * BD + i < KT && nb * BD + i < nj) b[nb & 1][i] = ld_relaxed2(at(src, nb * BD + i));
  }
  __device__ __forceinline__ void prefetch(const double2* src) { load(src, 0); }
  static __device__ __forceinline__ bool missing(double2 v) { return is_empty(v.x) || is_empty(v.y); }

  // acc = coupling x window, polling what is not there yet; the first batch has
  // been sent for
  __device__ __forceinline__ void run(const double2* src, double (&acc)[MT][4], volatile int* dead,
                                      unsigned* status, unsigned long long limit_ns) {
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[m][v] = 0.0;
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
      if (nb * BD >= nj) break;
      double2* y = b[nb & 1];
      unsigned long long t0 = 0;
      for (unsigned it = 0;; ++it) {
        bool miss = false;
#pragma unroll
        for (int i = 0; i < BD; ++i)
          if (nb * BD + i < KT && nb * BD + i < nj) miss = miss || missing(y[i]);
        if (!__any_sync(0xffffffffu, miss)) break;
        // (by vote: the word may change between two lanes' reads)
        if (__any_sync(0xffffffffu, *dead != 0)) break;
#pragma unroll
        for (int i = 0; i < BD; ++i)
          if (nb * BD + i < KT && nb * BD + i < nj && missing(y[i]))
            y[i] = ld_relaxed2(at(src, nb * BD + i));
        if ((it & 255u) == 255u) {
          const unsigned long long t = globaltimer_ns();
          if (t0 == 0) t0 = t;
          if (t - t0 > limit_ns) {
            *dead = 1;
            atomicOr(status, ST_WAIT_TIMEOUT);
          }
        }
      }
      __syncwarp();
      if (nb + 1 < NB) load(src, nb + 1);
#pragma unroll
      for (int i = 0; i < BD; ++i) {
        if (nb * BD + i >= KT || nb * BD + i >= nj) continue;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          dmma884(acc[m], A[m][nb * BD + i], y[i].x);
          dmma884(acc[m] + 2, A[m][nb * BD + i], y[i].y);
        }
      }
    }
  }
  // partial sums to red[warp * MT * 64 + row * 8 + pulse]
  static __device__ __forceinline__ void put(const double (&acc)[MT][4], double2* red, int warp,
                                             int lane) {
    double2* r = red + warp * (MT * 64) + (lane >> 2) * 8 + 2 * (lane & 3);
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      r[m * 64] = make_double2(acc[m][0], acc[m][2]);
      r[m * 64 + 1] = make_double2(acc[m][1], acc[m][3]);
    }
  }
};

// The coupling sum of element e, the warps' parts in order.
template <int MT>
__device__ __forceinline__ double2 fb_sum(const double2* red, int e) {
  double2 s[FW];
#pragma unroll
  for (int q = 0; q < FW; ++q) s[q] = red[q * (MT * 64) + e];
  double2 t;
  t.x = ((s[0].x + s[1].x) + (s[2].x + s[3].x)) + ((s[4].x + s[5].x) + (s[6].x + s[7].x));
  t.y = ((s[0].y + s[1].y) + (s[2].y + s[3].y)) + ((s[4].y + s[5].y) + (s[6].y + s[7].y));
  return t;
}

// M(F) v of one row: e its energy, W its coupling sum.
__device__ __forceinline__ double2 fb_m(int gauge, double e, double F, double2 v, double2 W) {
  if (gauge == 0)  // -i (e v + F W)
    return make_double2(fma(F, W.y, e * v.y), -fma(F, W.x, e * v.x));
  return make_double2(fma(F, W.x, e * v.y), fma(F, W.y, -e * v.x));  // -i e v + F W
}

// Waits until the helper is done with chunk c up to `step`; false if the
// helper gave up (its own waits are bounded).  What the helper wrote before its
// word is plain shared memory: the fence orders the reads after the spin.
__device__ __forceinline__ bool fb_await(FbCtl& ctl, int c, int step) {
  bool ok = true;
  while (ok && ctl.step[c] < step)
    if (ctl.hdead || ctl.mexit) ok = ctl.step[c] >= step;
  __threadfence_block();
  return ok;
}

// The compute warps have finished one more (step, chunk) pair, said by their
// thread 0 after the CTA's barrier.
__device__ __forceinline__ void fb_tell(FbCtl& ctl) {
  __threadfence_block();
  ctl.progress = ctl.progress + 1;
}

// ---------------------------------------------------------------------------
// fixed step: slots 2 x 11 Horner vectors by step parity, then 3 x x_{n+1}
// ---------------------------------------------------------------------------
constexpr int kFixSlots = 25;
__device__ __forceinline__ int fix_v(int step, int p) { return (step & 1) * 11 + p; }
__device__ __forceinline__ int fix_x(int step) { return 22 + (step + 3) % 3; }   // x_{step+1}

// x_step of one element is formed from the unnormalised z; the pulse's
// population and, at its end, its final state go out.
__device__ __forceinline__ double2 fix_begin(const FbArgs& a, FbCtl& ctl, int c, int q, int row,
                                             int step, double2 z) {
  const double2 x = quot2(z, ctl.nrm[c][q]);
  const int id = ctl.id[c][q];
  if (id >= 0 && step <= ctl.ns[c][q]) {
    if (a.pop_hist && row == a.pop_index && step > 0)
      a.pop_hist[(long long)id * a.hist_ld + step] =
          __dadd_rn(__dmul_rn(x.x, x.x), __dmul_rn(x.y, x.y));
    if (step == ctl.ns[c][q]) a.out[(long long)id * a.g.ntot + row] = x;
  }
  return x;
}

template <int MT, int KT>
__device__ void fb_fixed_main(const FbArgs& a, FbCtl& ctl, const FbView& u, double2* red,
                              double (*red8)[CP], int tid) {
  constexpr int NE = (MT * 64 + FT - 1) / FT;   // elements per thread, of one pulse
  const int warp = tid >> 5, lane = tid & 31, q = tid & 7;
  FbTile<MT, KT> tile;
  tile.init(a, u, warp, lane);
  const double h = a.dt;
  const int ne = u.nrows * CP;
  auto slot = [&](int c, int s) {
    return a.V + u.cpitch * (c * a.ng + u.grp) + u.spitch * s + (long long)u.row0 * CP;
  };
  auto chunk = [&](int c) { return ((long long)(c * a.ng + u.grp) * a.g.ntot + u.row0) * CP; };
  // the start states, as given
  for (int c = 0; c < u.nc; ++c)
    for (int e = tid; e < ne; e += FT) {
      const int id = ctl.id[c][q];
      double2 x = make_double2(0.0, 0.0);
      if (id >= 0)
        x = a.start ? a.start[chunk(c) + e] : a.in[(long long)id * a.g.ntot + u.row0 + (e >> 3)];
      publish(slot(c, fix_x(-1)) + e, x);
    }
  // items: per step, per product, the chunks with steps left (the longest first)
  int it = 0, act = u.nc;
  bool primed = false;
  for (int step = 0;; ++step) {
    while (act > 0 && ctl.nst[act - 1] <= step) {
      // the last state of a chunk that has finished
      const int c = --act;
      if (!fb_await(ctl, c, step)) ctl.mdead[it & 1] = 1;
      for (int e = tid; e < ne; e += FT)
        fix_begin(a, ctl, c, q, u.row0 + (e >> 3), step, __ldcg(slot(c, fix_x(step - 1)) + e));
    }
    if (act == 0) return;
#pragma unroll 1
    for (int p = 0; p < kFlowProducts; ++p) {
      const bool last = p == kFlowProducts - 1;
      const double gm = f_G[11 - p], sc = p == 0 ? f_G[12] : 1.0;
#pragma unroll 1
      for (int c = 0; c < act; ++c, ++it) {
        const int in_slot = p == 0 ? fix_x(step - 1) : fix_v(step, p - 1);
        const double2* src = fb_slot(a, u, c, in_slot);
        if (!primed) tile.prefetch(src);
        double acc[MT][4];
        tile.run(src, acc, &ctl.mdead[it & 1], a.status, a.bc.wait_ns);
        // the next item's first loads, where its buffer is known to be preset
        primed = act > 1;
        if (primed) {
          const double2* next = nullptr;
          if (c + 1 < act)
            next = fb_slot(a, u, c + 1, in_slot);
          else if (!last)
            next = fb_slot(a, u, 0, fix_v(step, p));
          else if (ctl.nst[0] > step + 1)
            next = fb_slot(a, u, 0, fix_x(step));
          primed = next != nullptr;
          if (primed) tile.prefetch(next);
        }
        double2* rb = red + (it & 1) * (FW * MT * 64);
        tile.put(acc, rb, warp, lane);
        // this thread's own elements of x and of the product's input
        double2 xo[NE], vo[NE];
        const double2* own = slot(c, in_slot);
        double2* xs = a.xst + chunk(c);
        double2* keep = a.seg_v && step >= a.seg_from
                            ? a.seg_v + a.cvec * (13LL * (step - a.seg_from)) + chunk(c)
                            : nullptr;
#pragma unroll
        for (int i = 0; i < NE; ++i) {
          const int e = tid + i * FT;
          if (e < ne) {
            vo[i] = __ldcg(own + e);
            if (p > 0) xo[i] = xs[e];
          }
        }
        named_bar_sync(kBarMain, FT);
        if (ctl.mdead[it & 1]) return;
        if (p == 0 && !fb_await(ctl, c, step)) ctl.mdead[(it + 1) & 1] = 1;
        const double F = ctl.F[c][q];
        double2* dst = slot(c, last ? fix_x(step) : fix_v(step, p));
        double nsq = 0.0;
#pragma unroll
        for (int i = 0; i < NE; ++i) {
          const int e = tid + i * FT;
          if (e >= ne) continue;
          const int row = u.row0 + (e >> 3);
          double2 W = fb_sum<MT>(rb, e), x = xo[i], v = vo[i];
          if (p == 0) {
            if (a.ckpt && step % a.ckpt_every == 0)
              a.ckpt[a.cvec * (step / a.ckpt_every) + chunk(c) + e] = v;
            x = fix_begin(a, ctl, c, q, row, step, v);
            xs[e] = x;
            if (keep) keep[12 * a.cvec + e] = x;
            v = make_double2(sc * x.x, sc * x.y);   // v_12 = G_12 x
            W = quot2(W, ctl.nrm[c][q]);
            W.x *= sc;
            W.y *= sc;
          }
          const double2 m = fb_m(a.gauge, a.eps[row], F, v, W);
          const double2 o = make_double2(fma(h, m.x, gm * x.x), fma(h, m.y, gm * x.y));
          publish(dst + e, o);
          if (keep && !last) keep[(11 - p) * a.cvec + e] = o;
          nsq += fma(o.x, o.x, o.y * o.y);
        }
        if (last) {
          // the CTA's norm partial per pulse: a thread's rows, the lanes of its
          // pulse, the warps in order
          nsq += __shfl_xor_sync(0xffffffffu, nsq, 8);
          nsq += __shfl_xor_sync(0xffffffffu, nsq, 16);
          if (lane < CP) red8[warp][lane] = nsq;
          named_bar_sync(kBarMain, FT);
          if (tid < CP) {
            double t = red8[0][tid];
#pragma unroll
            for (int k = 1; k < FW; ++k) t += red8[k][tid];
            st_relaxed1(a.part + (((long long)(c * a.ng + u.grp) * 2 + (step & 1)) * a.gp + u.idx) *
                                     (2 * CP) + tid,
                        canonical(t));
          }
          __syncwarp();
          if (tid == 0) fb_tell(ctl);
        }
      }
    }
  }
}

// Waits, as a warp, until *ctr reaches `target`; false after limit_ns.
__device__ __forceinline__ bool fb_count(const unsigned long long* ctr, unsigned long long target,
                                         int lane, unsigned long long limit_ns) {
  bool ok = true;
  if (lane == 0) {
    unsigned long long v = 0, t0 = 0;
    for (unsigned i = 0;; ++i) {
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(ctr) : "memory");
      if (v >= target) break;
      if ((i & 1023u) == 1023u) {
        const unsigned long long t = globaltimer_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > limit_ns) {
          ok = false;
          break;
        }
      }
    }
  }
  return __shfl_sync(0xffffffffu, ok, 0);
}
__device__ __forceinline__ void fb_arrive(unsigned long long* ctr) {
  asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(ctr), "l"(1ull) : "memory");
}
// Waits, in the helper, for the compute warps' `events`-th (step, chunk) pair.
__device__ __forceinline__ bool fb_progress(FbCtl& ctl, int events) {
  bool ok = true;
  while (ok && ctl.progress < events) ok = ctl.mexit == 0 || ctl.progress >= events;
  __threadfence_block();
  return __all_sync(0xffffffffu, ok);
}

// Per chunk and step: the norms from all CTAs' partials, the pulses' times and
// next fields, the presets.  One warp; lane = (quarter of the CTAs, pulse).
__device__ void fb_fixed_helper(const FbArgs& a, FbCtl& ctl, const FbView& u, int lane) {
  const int q = lane & 7;
  auto field = [&](int c, int step) {
    const int id = ctl.id[c][q];
    if (id < 0 || step >= ctl.ns[c][q]) return 0.0;
    if (a.Ftab) return a.Ftab[(long long)step * a.ldf + id];
    return dev_field(a.pulse[id], ctl.t[c][q] + a.dt);
  };
  for (int c = 0; c < u.nc; ++c) {
    if (lane < CP) {
      const double n0 = a.start_nrm && ctl.id[c][q] >= 0
                            ? a.start_nrm[(long long)ctl.id[c][q] * a.hist_ld]
                            : 1.0;
      ctl.nrm[c][q] = make_double2(n0, 1.0 / n0);
      ctl.t[c][q] = ctl.id[c][q] >= 0 && a.t0 ? a.t0[ctl.id[c][q]] : 0.0;
      ctl.F[c][q] = field(c, 0);
    }
    __syncwarp();
    __threadfence_block();
    if (lane == 0) ctl.step[c] = 0;
  }
  int events = 0;
  for (int n = 0;; ++n) {   // event n: step n of a chunk is complete
    bool any = false;
    for (int c = 0; c < u.nc && ctl.nst[c] > n; ++c) {
      any = true;
      ++events;
      bool ok = fb_progress(ctl, events);
      if (!ok) return;
      const int gc = c * a.ng + u.grp;
      if (n > 0)   // everyone's presets of event n - 1 are made
        ok = fb_count(a.ctr + gc, (unsigned long long)n * a.gp + a.bc.skew, lane, a.bc.wait_ns);
      double sum = 0.0;
      const double* pp = a.part + ((long long)gc * 2 + (n & 1)) * a.gp * (2 * CP);
      for (int b0 = lane >> 3; ok && b0 < a.gp; b0 += 32) {
        double v[8];
        unsigned long long t0 = 0;
        for (unsigned i = 0;; ++i) {
          bool ready = true;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            v[j] = b0 + 4 * j < a.gp ? ld_relaxed1(pp + (b0 + 4 * j) * (2 * CP) + q) : 0.0;
#pragma unroll
          for (int j = 0; j < 8; ++j) ready = ready && !is_empty(v[j]);
          if (ready) break;
          if ((i & 255u) == 255u) {
            const unsigned long long t = globaltimer_ns();
            if (t0 == 0) t0 = t;
            if (t - t0 > a.bc.wait_ns) {
              ok = false;
              break;
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) sum += v[j];
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0) {
          atomicOr(a.status, ST_WAIT_TIMEOUT);
          ctl.hdead = 1;
        }
        return;
      }
      sum += __shfl_xor_sync(0xffffffffu, sum, 8);
      sum += __shfl_xor_sync(0xffffffffu, sum, 16);
      if (lane < CP) {
        const int id = ctl.id[c][q];
        double nrm = sqrt(sum);
        if (id < 0) nrm = 1.0;
        if (id >= 0 && n < ctl.ns[c][q]) {
          ctl.t[c][q] += a.dt;
          if (u.idx == 0) {
            if (a.norm_hist) a.norm_hist[(long long)id * a.hist_ld + n] = nrm;
            // (the objective gives such a pulse its NaN, beside the others' numbers)
            if (!a.seg_v && (!(nrm > 0.0) || !isfinite(nrm))) atomicOr(a.status, ST_NONFINITE);
          }
        }
        ctl.nrm[c][q] = make_double2(nrm, 1.0 / nrm);
        ctl.F[c][q] = field(c, n + 1);
        st_relaxed1(a.part + (((long long)gc * 2 + ((n + 1) & 1)) * a.gp + u.idx) * (2 * CP) + q,
                    __longlong_as_double((long long)kEmpty));
      }
      __syncwarp();
      __threadfence_block();
      if (lane == 0) ctl.step[c] = n + 1;
      // every CTA is past step n of this chunk: its Horner vectors, and x_n
      double2* base = a.V + u.cpitch * gc + (long long)u.row0 * CP;
      const int ne = u.nrows * CP;
      for (int s = 0; s <= 11; ++s) {
        double2* d = base + u.spitch * (s < 11 ? fix_v(n, s) : fix_x(n - 1));
        for (int e = lane; e < ne; e += 32) st_relaxed2(d + e, empty2());
      }
      __syncwarp();
      if (lane == 0) fb_arrive(a.ctr + gc);
    }
    if (!any) return;
  }
}

// ---------------------------------------------------------------------------
// the objective gradient's sweep (see k_flow_adjoint for the transposed
// products): slots 3 x 12, ring m % 3 of the m-th swept step, vbar_p
// ---------------------------------------------------------------------------
constexpr int kAdjSlots = 36;
__device__ __forceinline__ int adj_v(int m, int p) { return (m % 3) * 12 + p; }

template <int MT, int KT>
__device__ void fb_adj_main(const FbArgs& a, FbCtl& ctl, const FbView& u, double2* red,
                            double (*red8)[CP], int tid) {
  constexpr int NE = (MT * 64 + FT - 1) / FT;
  const int warp = tid >> 5, lane = tid & 31, q = tid & 7;
  FbTile<MT, KT> tile;
  tile.init(a, u, warp, lane);
  const double h = a.dt;
  const int ne = u.nrows * CP;
  auto slot = [&](int c, int s) {
    return a.V + u.cpitch * (c * a.ng + u.grp) + u.spitch * s + (long long)u.row0 * CP;
  };
  auto chunk = [&](int c) { return ((long long)(c * a.ng + u.grp) * a.g.ntot + u.row0) * CP; };
  // zbar = lambda / ||z_n|| of the step with local index n
  auto zbar = [&](int c, int n, double2 l) {
    const int id = ctl.id[c][q];
    const double nz = id >= 0 ? a.norms[(long long)id * a.hist_ld + n] : 1.0;
    return quot2(l, make_double2(nz, 1.0 / nz));
  };
  for (int c = 0; c < u.nc; ++c)
    for (int e = tid; e < ne; e += FT)
      publish(slot(c, adj_v(0, 0)) + e, zbar(c, a.len - 1, a.lam[chunk(c) + e]));
  int it = 0;
  bool primed = false;
  for (int m = 0; m < a.len; ++m) {
    const int n = a.len - 1 - m;   // the step, counted from the segment's start
#pragma unroll 1
    for (int p = 0; p < kFlowProducts; ++p) {
      const bool last = p == kFlowProducts - 1;
      const double gm = f_G[p], sc = last ? f_G[12] : 1.0;
#pragma unroll 1
      for (int c = 0; c < u.nc; ++c, ++it) {
        if (p == 0 && !fb_await(ctl, c, m - 1)) ctl.mdead[it & 1] = 1;
        const double2* src = fb_slot(a, u, c, adj_v(m, p));
        if (!primed) tile.prefetch(src);
        double acc[MT][4];
        tile.run(src, acc, &ctl.mdead[it & 1], a.status, a.bc.wait_ns);
        // (a step's first product waits for the helper's word, chunk by chunk)
        primed = u.nc > 1 && (c + 1 < u.nc ? p > 0 : !last);
        if (primed)
          tile.prefetch(c + 1 < u.nc ? fb_slot(a, u, c + 1, adj_v(m, p))
                                     : fb_slot(a, u, 0, adj_v(m, p + 1)));
        double2* rb = red + (it & 1) * (FW * MT * 64);
        tile.put(acc, rb, warp, lane);
        double2 vo[NE], vk[NE], xo[NE];
        double fo[NE];
        const double2* own = slot(c, adj_v(m, p));
        const double2* kept = a.seg_v + a.cvec * (13LL * n + p + 1) + chunk(c);
        double2* xs = a.xb + chunk(c);
        double* fv = a.fs + chunk(c);
#pragma unroll
        for (int i = 0; i < NE; ++i) {
          const int e = tid + i * FT;
          if (e < ne) {
            vo[i] = __ldcg(own + e);
            vk[i] = kept[e];
            if (p > 0) {
              xo[i] = xs[e];
              fo[i] = fv[e];
            }
          }
        }
        named_bar_sync(kBarMain, FT);
        if (ctl.mdead[it & 1]) return;
        const double F = ctl.id[c][q] >= 0 ? a.Ftab[(long long)n * a.ldf + ctl.id[c][q]] : 0.0;
        double fsum = 0.0;
#pragma unroll
        for (int i = 0; i < NE; ++i) {
          const int e = tid + i * FT;
          if (e >= ne) continue;
          const double2 W = fb_sum<MT>(rb, e), vb = vo[i];
          const double2 m1 = a.gauge == 0 ? make_double2(W.y, -W.x) : W;
          const double2 mv = fb_m(a.gauge, a.eps[u.row0 + (e >> 3)], F, vb, W);
          const double2 o = make_double2(-h * mv.x, -h * mv.y);   // vbar_{p+1}
          double2 x = p > 0 ? xo[i] : make_double2(0.0, 0.0);
          x.x = fma(gm, vb.x, x.x);
          x.y = fma(gm, vb.y, x.y);
          double f = p > 0 ? fo[i] : 0.0;
          f -= sc * fma(m1.x, vk[i].x, m1.y * vk[i].y);   // v_12 = G_12 x
          if (!last) {
            publish(slot(c, adj_v(m, p + 1)) + e, o);
            xs[e] = x;
            fv[e] = f;
          } else {
            const double2 l = make_double2(fma(f_G[12], o.x, x.x), fma(f_G[12], o.y, x.y));
            fsum += f * h;
            if (m + 1 < a.len)
              publish(slot(c, adj_v(m + 1, 0)) + e, zbar(c, n - 1, l));
            else
              a.lam[chunk(c) + e] = l;
          }
        }
        if (last) {
          fsum += __shfl_xor_sync(0xffffffffu, fsum, 8);
          fsum += __shfl_xor_sync(0xffffffffu, fsum, 16);
          if (lane < CP) red8[warp][lane] = fsum;
          named_bar_sync(kBarMain, FT);
          if (tid < CP) {
            double t = red8[0][tid];
#pragma unroll
            for (int k = 1; k < FW; ++k) t += red8[k][tid];
            a.fpart[(((long long)n * a.nch + c * a.ng + u.grp) * a.gp + u.idx) * CP + tid] = t;
          }
          if (tid == 0) fb_tell(ctl);
        }
      }
    }
  }
}

// Once every CTA is past a chunk's m-th step its ring is preset, for the step
// m + 3; the arrival of the next step publishes that.
__device__ void fb_adj_helper(const FbArgs& a, FbCtl& ctl, const FbView& u, int lane) {
  int events = 0;
  for (int m = 0; m < a.len; ++m)
    for (int c = 0; c < u.nc; ++c) {
      if (!fb_progress(ctl, ++events)) return;
      const int gc = c * a.ng + u.grp;
      __syncwarp();
      if (lane == 0) fb_arrive(a.ctr + gc);
      if (!fb_count(a.ctr + gc, (unsigned long long)(m + 1) * a.gp + a.bc.skew, lane,
                    a.bc.wait_ns)) {
        if (lane == 0) {
          atomicOr(a.status, ST_WAIT_TIMEOUT);
          ctl.hdead = 1;
        }
        return;
      }
      double2* base = a.V + u.cpitch * gc + (long long)u.row0 * CP;
      const int ne = u.nrows * CP;
      for (int p = 0; p < 12; ++p) {
        double2* d = base + u.spitch * adj_v(m, p);
        for (int e = lane; e < ne; e += 32) st_relaxed2(d + e, empty2());
      }
      __syncwarp();
      __threadfence_block();
      if (lane == 0) ctl.step[c] = m + 1;
    }
}

// ---------------------------------------------------------------------------
// adaptive steps: slots 2 x 13 stage inputs by attempt parity
// ---------------------------------------------------------------------------
constexpr int kAdaptSlots = 26;
__device__ __forceinline__ int ada_y(int att, int s) { return (att & 1) * kNumStages + s; }

static __constant__ double f_A[13][13];
static __constant__ double f_B8[13];
static __constant__ double f_E[13];   // b8 - b7
static __constant__ double f_C[13];

__device__ __forceinline__ double fb_nanmax(double m, double e) {
  return (m != m) ? m : ((e != e) ? e : fmax(m, e));
}

template <int MT, int KT>
__device__ void fb_adapt_main(const FbArgs& a, FbCtl& ctl, FbAdapt& ad, const FbView& u,
                              double2* red, double2* kshm, double (*red8)[CP], double (*rede)[CP],
                              int tid) {
  constexpr int NE = (MT * 64 + FT - 1) / FT;
  const int warp = tid >> 5, lane = tid & 31, q = tid & 7;
  FbTile<MT, KT> tile;
  tile.init(a, u, warp, lane);
  const int ne = u.nrows * CP;
  auto slot = [&](int c, int s) {
    return a.V + u.cpitch * (c * a.ng + u.grp) + u.spitch * s + (long long)u.row0 * CP;
  };
  auto chunk = [&](int c) { return ((long long)(c * a.ng + u.grp) * a.g.ntot + u.row0) * CP; };
  for (int c = 0; c < u.nc; ++c)
    for (int e = tid; e < ne; e += FT) {
      const int id = ctl.id[c][q];
      a.xst[chunk(c) + e] = id >= 0 ? a.in[(long long)id * a.g.ntot + u.row0 + (e >> 3)]
                                    : make_double2(0.0, 0.0);
    }
  unsigned live = u.nc >= 32 ? 0xffffffffu : (1u << u.nc) - 1u;
  int it = 0;
  bool primed = false;
  for (int att = 0;; ++att) {
    // ---- the attempt's start states out: x_new / ||x_new|| where the last
    // attempt was accepted; finished pulses leave ----
    for (int c = 0; c < u.nc; ++c) {
      if (!(live >> c & 1u)) continue;
      const bool ok = fb_await(ctl, c, att);
      if (!ok) ctl.mdead[it & 1] = 1;
      const int id = ctl.id[c][q];
      for (int e = tid; e < ne && ok; e += FT) {
        double2 x = a.xst[chunk(c) + e];
        if (ad.acc[c][q]) {
          x = quot2(a.xnew[chunk(c) + e], ctl.nrm[c][q]);
          a.xst[chunk(c) + e] = x;
        }
        if (ad.ret[c][q]) a.out[(long long)id * a.g.ntot + u.row0 + (e >> 3)] = x;
        if (ad.alive[c]) publish(slot(c, ada_y(att, 0)) + e, x);
      }
      if (ok && !ad.alive[c]) live &= ~(1u << c);
    }
    if (!live) return;
#pragma unroll 1
    for (int s = 0; s < kNumStages; ++s) {
      const bool last = s == kNumStages - 1;
#pragma unroll 1
      for (unsigned todo = live; todo; todo &= todo - 1) {
        const int c = __ffs(todo) - 1;
        const unsigned after = todo & (todo - 1);
        const double2* src = fb_slot(a, u, c, ada_y(att, s));
        if (!primed) tile.prefetch(src);
        double acc[MT][4];
        tile.run(src, acc, &ctl.mdead[it & 1], a.status, a.bc.wait_ns);
        primed = (live & (live - 1)) && (after || !last);
        if (primed)
          tile.prefetch(after ? fb_slot(a, u, __ffs(after) - 1, ada_y(att, s))
                              : fb_slot(a, u, __ffs(live) - 1, ada_y(att, s + 1)));
        double2* rb = red + (it & 1) * (FW * MT * 64);
        tile.put(acc, rb, warp, lane);
        double2 xo[NE], vo[NE];
        const double2* own = slot(c, ada_y(att, s));
        double2* ks = kshm ? kshm + c * (kNumStages - 1) * ne : a.kst + chunk(c);
        const long long kp = kshm ? ne : a.cvec;
#pragma unroll
        for (int i = 0; i < NE; ++i) {
          const int e = tid + i * FT;
          if (e < ne) {
            vo[i] = __ldcg(own + e);
            xo[i] = a.xst[chunk(c) + e];
          }
        }
        named_bar_sync(kBarMain, FT);
        if (ctl.mdead[it & 1]) return;
        const double F = ad.F[c][s][q], hq = ad.hatt[c][q];
        double nsq = 0.0, em = 0.0;
#pragma unroll
        for (int i = 0; i < NE; ++i) {
          const int e = tid + i * FT;
          if (e >= ne) continue;
          const double2 x = xo[i];
          const double2 k = fb_m(a.gauge, a.eps[u.row0 + (e >> 3)], F, vo[i], fb_sum<MT>(rb, e));
          if (!last) ks[s * kp + e] = k;
          double2 o = x;
          if (!last) {
#pragma unroll
            for (int j = 0; j < kNumStages - 1; ++j) {
              const double cj = f_A[s + 1][j];
              if (j > s || cj == 0.0) continue;
              const double2 w = j == s ? k : ks[j * kp + e];
              const double cf = hq * cj;
              o.x = fma(cf, w.x, o.x);
              o.y = fma(cf, w.y, o.y);
            }
            publish(slot(c, ada_y(att, s + 1)) + e, o);
          } else {
            double2 er = make_double2(0.0, 0.0);
#pragma unroll
            for (int j = 0; j < kNumStages; ++j) {
              const double bj = f_B8[j], ej = f_E[j];
              if (bj == 0.0 && ej == 0.0) continue;
              const double2 w = j == kNumStages - 1 ? k : ks[j * kp + e];
              if (bj != 0.0) {
                o.x = fma(hq * bj, w.x, o.x);
                o.y = fma(hq * bj, w.y, o.y);
              }
              if (ej != 0.0) {
                er.x = fma(hq * ej, w.x, er.x);
                er.y = fma(hq * ej, w.y, er.y);
              }
            }
            const double ax = sqrt(x.x * x.x + x.y * x.y), an = sqrt(o.x * o.x + o.y * o.y);
            const double ae = sqrt(er.x * er.x + er.y * er.y);
            em = fb_nanmax(em, ae / (a.atol + a.rtol * fmax(ax, an)));
            a.xnew[chunk(c) + e] = o;
            nsq += o.x * o.x + o.y * o.y;
          }
        }
        if (last) {
          nsq += __shfl_xor_sync(0xffffffffu, nsq, 8);
          nsq += __shfl_xor_sync(0xffffffffu, nsq, 16);
          em = fb_nanmax(em, __shfl_xor_sync(0xffffffffu, em, 8));
          em = fb_nanmax(em, __shfl_xor_sync(0xffffffffu, em, 16));
          if (lane < CP) {
            red8[warp][lane] = nsq;
            rede[warp][lane] = em;
          }
          named_bar_sync(kBarMain, FT);
          if (tid < CP) {
            double t = red8[0][tid], m = rede[0][tid];
#pragma unroll
            for (int k = 1; k < FW; ++k) {
              t += red8[k][tid];
              m = fb_nanmax(m, rede[k][tid]);
            }
            double* pp = a.part + (((long long)(c * a.ng + u.grp) * 2 + (att & 1)) * a.gp + u.idx) *
                                      (2 * CP) + tid;
            st_relaxed1(pp, canonical(t));
            st_relaxed1(pp + CP, canonical(m));
          }
          __syncwarp();
          if (tid == 0) fb_tell(ctl);
        }
        ++it;
      }
    }
  }
}

// Per chunk and attempt: norm and error over all CTAs, accept or reject, the
// next step and its stage fields (the controller of the stage-GEMM path,
// k_batch_control, run redundantly and identically in every CTA).
__device__ void fb_adapt_helper(const FbArgs& a, FbCtl& ctl, FbAdapt& ad, const FbView& u,
                                int lane) {
  const int q = lane & 7;
  auto retire = [&](int c) {
    const int id = ctl.id[c][q];
    ad.ret[c][q] = 1;
    if (u.idx == 0) {
      a.nacc[id] = ad.cnt[c][0][q];
      a.nrej[id] = ad.cnt[c][1][q];
      a.tf[id] = ctl.t[c][q];
      a.gave_up[id] = ad.done[c][q] == 2;
    }
  };
  // the attempt's step (capped at the time left), its fields, who is left
  auto prepare = [&](int c, int att) {
    if (lane < CP) {
      double hatt = 0.0;
      if (!ad.done[c][q]) {
        hatt = ad.h[c][q];
        const double rem = ad.t_end[c][q] - ctl.t[c][q];
        ad.lastst[c][q] = hatt >= rem;
        if (hatt >= rem) hatt = rem;
      }
      ad.hatt[c][q] = hatt;
    }
    __syncwarp();
    for (int s = lane >> 3; s < kNumStages; s += 4) {
      const int id = ctl.id[c][q];
      ad.F[c][s][q] =
          ad.done[c][q] ? 0.0 : dev_field(a.pulse[id], ctl.t[c][q] + f_C[s] * ad.hatt[c][q]);
    }
    const bool any = __any_sync(0xffffffffu, ad.done[c][q] == 0);
    if (lane == 0) ad.alive[c] = any;
    __syncwarp();
    __threadfence_block();
    if (lane == 0) ctl.step[c] = att;
  };
  for (int c = 0; c < u.nc; ++c) {
    if (lane < CP) {
      const int id = ctl.id[c][q];
      ctl.nrm[c][q] = make_double2(1.0, 1.0);
      ad.acc[c][q] = ad.ret[c][q] = 0;
      ad.cnt[c][0][q] = ad.cnt[c][1][q] = ad.cnt[c][2][q] = 0;
      ad.h[c][q] = a.h0;
      ctl.t[c][q] = id >= 0 ? a.t0[id] : 0.0;
      ad.t_end[c][q] = id >= 0 ? a.t_end[id] : 0.0;
      ad.done[c][q] = id < 0 ? 3 : ctl.t[c][q] >= ad.t_end[c][q] ? 1 : 0;
      if (ad.done[c][q] == 1) retire(c);
    }
    __syncwarp();
    prepare(c, 0);
  }
  unsigned live = 0;
  for (int c = 0; c < u.nc; ++c)
    if (ad.alive[c]) live |= 1u << c;
  int events = 0;
  for (int n = 0; live; ++n)
    for (unsigned todo = live; todo; todo &= todo - 1) {
      const int c = __ffs(todo) - 1;
      if (!fb_progress(ctl, ++events)) return;
      const int gc = c * a.ng + u.grp;
      bool ok = true;
      if (n > 0)
        ok = fb_count(a.ctr + gc, (unsigned long long)n * a.gp + a.bc.skew, lane, a.bc.wait_ns);
      double sum = 0.0, em = 0.0;
      const double* pp = a.part + ((long long)gc * 2 + (n & 1)) * a.gp * (2 * CP);
      for (int b0 = lane >> 3; ok && b0 < a.gp; b0 += 16) {
        double v[4], w[4];
        unsigned long long t0 = 0;
        for (unsigned i = 0;; ++i) {
          bool ready = true;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const bool in = b0 + 4 * j < a.gp;
            v[j] = in ? ld_relaxed1(pp + (b0 + 4 * j) * (2 * CP) + q) : 0.0;
            w[j] = in ? ld_relaxed1(pp + (b0 + 4 * j) * (2 * CP) + CP + q) : 0.0;
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) ready = ready && !is_empty(v[j]) && !is_empty(w[j]);
          if (ready) break;
          if ((i & 255u) == 255u) {
            const unsigned long long t = globaltimer_ns();
            if (t0 == 0) t0 = t;
            if (t - t0 > a.bc.wait_ns) {
              ok = false;
              break;
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          sum += v[j];
          em = fb_nanmax(em, w[j]);
        }
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (lane == 0) {
          atomicOr(a.status, ST_WAIT_TIMEOUT);
          ctl.hdead = 1;
        }
        return;
      }
      sum += __shfl_xor_sync(0xffffffffu, sum, 8);
      sum += __shfl_xor_sync(0xffffffffu, sum, 16);
      em = fb_nanmax(em, __shfl_xor_sync(0xffffffffu, em, 8));
      em = fb_nanmax(em, __shfl_xor_sync(0xffffffffu, em, 16));
      if (lane < CP) {
        ad.acc[c][q] = ad.ret[c][q] = 0;
        if (!ad.done[c][q]) {
          const double nrm = sqrt(sum), hh = ad.hatt[c][q];
          double fac = 5.0;
          if (em != 0.0) fac = fmin(fmax(0.9 / sqrt(sqrt(sqrt(em))), 0.2), 5.0);
          ++ad.cnt[c][2][q];
          if (em <= 1.0 && nrm > 0.0 && isfinite(nrm)) {
            ctl.t[c][q] = ad.lastst[c][q] ? ad.t_end[c][q] : ctl.t[c][q] + hh;
            ++ad.cnt[c][0][q];
            ad.acc[c][q] = 1;
            ctl.nrm[c][q] = make_double2(nrm, 1.0 / nrm);
            ad.h[c][q] = fmin(hh * fac, a.dt_max);
            if (ad.lastst[c][q]) ad.done[c][q] = 1;
          } else {
            ++ad.cnt[c][1][q];
            ad.h[c][q] = hh * fmin(fac, 1.0);
          }
          if (!ad.done[c][q] &&
              (ad.cnt[c][2][q] >= a.max_attempts ||
               ad.h[c][q] < 1e-13 * fmax(1.0, fabs(ad.t_end[c][q]))))
            ad.done[c][q] = 2;
          if (ad.done[c][q]) retire(c);
        }
        double* mine = a.part + (((long long)gc * 2 + ((n + 1) & 1)) * a.gp + u.idx) * (2 * CP) + q;
        st_relaxed1(mine, __longlong_as_double((long long)kEmpty));
        st_relaxed1(mine + CP, __longlong_as_double((long long)kEmpty));
      }
      __syncwarp();
      prepare(c, n + 1);
      if (!ad.alive[c]) {
        live &= ~(1u << c);
        continue;
      }
      // every CTA is past attempt n of this chunk
      double2* base = a.V + u.cpitch * gc + (long long)u.row0 * CP;
      const int ne = u.nrows * CP;
      for (int s = 0; s < kNumStages; ++s) {
        double2* d = base + u.spitch * ada_y(n, s);
        for (int e = lane; e < ne; e += 32) st_relaxed2(d + e, empty2());
      }
      __syncwarp();
      if (lane == 0) fb_arrive(a.ctr + gc);
    }
}

template <int MODE>
__global__ void __launch_bounds__(FTHREADS, 1) k_flow_batch(const __grid_constant__ FbArgs a) {
  extern __shared__ __align__(16) unsigned char bsm[];
  const FbCta me = a.cta[blockIdx.x];
  FbCtl& ctl = *reinterpret_cast<FbCtl*>(bsm);
  double2* red = reinterpret_cast<double2*>(bsm + (sizeof(FbCtl) + 15) / 16 * 16);
  // mode 1: the control's second part, then the slopes if they fit
  FbAdapt& ad = *reinterpret_cast<FbAdapt*>(red + 2 * FW * a.mt * 64);
  double2* kshm = MODE == 1 && !a.kst
                      ? reinterpret_cast<double2*>(reinterpret_cast<unsigned char*>(&ad) +
                                                   (sizeof(FbAdapt) + 15) / 16 * 16)
                      : nullptr;
  __shared__ double red8[FW][CP], rede[FW][CP];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  FbView u;
  u.w = flow_window(a.g, me.L);
  u.L = me.L;
  u.row0 = me.row0;
  u.nrows = me.nrows;
  u.r0 = me.row0 - a.g.state_off[me.L];
  u.grp = me.grp;
  u.idx = me.idx;
  u.nc = (a.nch - me.grp + a.ng - 1) / a.ng;
  u.spitch = (long long)a.g.ntot * CP;
  u.cpitch = u.spitch * a.slots;
  for (int i = tid; i < u.nc * CP; i += FTHREADS) {
    const int c = i / CP, q = i % CP, id = a.cid[(c * a.ng + me.grp) * CP + q];
    ctl.id[c][q] = id;
    ctl.ns[c][q] = id >= 0 && a.nsteps ? a.nsteps[id] : 0;
    if (q == 0) {
      ctl.nst[c] = a.csteps[c * a.ng + me.grp];
      ctl.step[c] = MODE == 2 ? 0 : -1;
    }
  }
  if (tid == 0) {
    ctl.progress = 0;
    ctl.hdead = ctl.mexit = 0;
    ctl.mdead[0] = ctl.mdead[1] = 0;
  }
  __syncthreads();
#define FB_CONFIGS(X) \
  X(0, 1, 6) X(1, 2, 6) X(2, 4, 6) X(3, 2, 10) X(4, 4, 10) X(5, 6, 10) X(6, 2, 13) X(7, 5, 13) \
  X(8, 2, 19) X(9, 3, 19) X(10, 2, 25) X(11, 3, 25)
  if (warp >= FW) {
    regs_dec<40>();
    if (warp == FW) {
      if constexpr (MODE == 2)
        fb_adj_helper(a, ctl, u, lane);
      else if constexpr (MODE == 1)
        fb_adapt_helper(a, ctl, ad, u, lane);
      else
        fb_fixed_helper(a, ctl, u, lane);
    }
    return;
  }
  regs_inc<232>();
#define FB_RUN(I, MT, KT) \
  case I: \
    if constexpr (MODE == 2) fb_adj_main<MT, KT>(a, ctl, u, red, red8, tid); \
    else if constexpr (MODE == 1) fb_adapt_main<MT, KT>(a, ctl, ad, u, red, kshm, red8, rede, tid); \
    else fb_fixed_main<MT, KT>(a, ctl, u, red, red8, tid); \
    break;
  switch (me.cfg) { FB_CONFIGS(FB_RUN) }
#undef FB_RUN
  if (tid == 0) ctl.mexit = 1;
}

// Shared memory of a launch whose CTAs have at most mt 8-row tiles: control, two
// buffers of partial sums, and for adaptive steps their control and, where
// they fit, the slopes of all a group's chunks (`rows` rows per CTA).  The
// slopes are read up to nine times per item: from shared memory an attempt of 48
// pulses on 1752 states takes 173 us, from global memory 188.
inline size_t flowb_smem(int mode, int mt, int slope_chunks = 0, int rows = 0) {
  return (sizeof(FbCtl) + 15) / 16 * 16 + sizeof(double2) * 2 * FW * mt * 64 +
         (mode == 1 ? (sizeof(FbAdapt) + 15) / 16 * 16 : 0) +
         sizeof(double2) * (kNumStages - 1) * (size_t)slope_chunks * rows * CP;
}

}  // namespace mpc
