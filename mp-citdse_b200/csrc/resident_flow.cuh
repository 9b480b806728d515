// resident_flow.cuh -- the fixed-step propagation and its adjoint for systems
// whose coupling fits on chip: one persistent cooperative launch for all
// steps, CTAs exchanging vectors through L2 without grid barriers.
//
// Layout.  CTA c owns a contiguous range of rows of ONE state block L, so all
// its rows couple to the same window: blocks L-1 and L+1 of the vector.  Their
// coupling rows (column r of D_{L-1} and row r of D_L, the latter negated in
// the velocity gauge) stay in registers for the whole launch: warp (rg, cg)
// holds the rows of row group rg restricted to every CG-th 32-column slice of
// the window, RW rows x CPL columns per lane (or, for systems whose rows do
// not fit the registers, in shared memory, read once per product).  CG is
// chosen per CTA so that end blocks (half the window, twice the rows) use the
// same RW x CPL tile.
//
// A step is the 12 Horner products of the RKF78 stability polynomial
// (v_12 = G_12 x, v_m = h M(F) v_{m+1} + G_m x, x_new = v_0): with the field
// frozen over a step this is the 13-stage step exactly, with one product
// fewer and no slopes to keep.
//
// Exchange.  Every product is a dependency of every row on its two neighbour
// blocks; what bounds the kernel is the latency of that exchange, not bytes or
// flops.  The owner of a row publishes its new element with one 16-byte
// store; the readers poll the elements themselves, whose buffers are preset to
// a bit pattern no published value has (kEmpty, an all-ones NaN; a computed NaN
// with those bits is published as another NaN).  One L2 round trip per product,
// against the store + fence + atomic + poll + load of a grid barrier.
// Buffers rotate by step; a helper warp, off the critical path, presets a
// step's buffers once every CTA is past it and meets the other helpers at a
// counter before its CTA may read them again.
//
// Renormalisation.  x_new is published unnormalised, its norm's partials next to
// it; the helper warp sums all CTAs' partials while the compute warps poll the
// window, and the window's elements are divided as they enter the next step
// (by every reader alike, so a run cut into several calls has the same bits).
//
// Measured, per step: 1752 states (6 blocks of 292) 20.9 us (22.0 before the
// fences at the spins), 3480 states (9 blocks of 384-388) 30.4 us, against 64.9 and 89.5 us for 13 stages with a grid
// barrier each and every row re-reading the window from shared memory; a
// gradient of 192 steps (3492 states) 14.4 ms against 45.6 ms.  Of a product's
// 3,560 cycles at 1752 states and 22.0 us about 2,600 are the exchange (publish, poll, the
// slowest of a CTA's polls), 690 the sums, 500 the row update.  Tried: two FMA
// chains per sum (no change), a pause of 50 ns between polls (+5 %), a delay
// of 400 / 800 / 1200 cycles before the first poll (-3 / +2 / +12 %).
#pragma once
#include <cuda_runtime.h>

#include "dev_util.cuh"
#include "plan.h"
#include "rkf78.h"

namespace mpc {

constexpr int FW = 8;              // compute warps
constexpr int FT = FW * 32;        // compute threads (one more warp helps)
// One more warpgroup, of which one warp helps: with a warpgroup of its own its
// registers can be handed to the compute warps (setmaxnreg), which hold the
// coupling: 2 x 128 x 232 + 128 x 40 = 384 x 168, the launch's total.
constexpr int FTHREADS = FT + 128;
constexpr int kHelpBar = FT + 32;  // compute warps and the helper warp
constexpr int kFlowProducts = 12;
constexpr int kFlowMaxRows = FT;   // one thread per row in the row update
constexpr unsigned long long kEmpty = ~0ull;
// Norm partials lie a cache line apart and are polled only once the reader's
// own CTA has published its own: 148 writers of 8 bytes each on ten lines that
// 148 readers poll all the time took 8,000 cycles to get through.
constexpr int kPartPitch = 16;     // doubles

struct FlowCta {
  int L;        // state block
  int row0;     // first row (global state index)
  int nrows;
  int cg;       // column groups (1, 2, 4, 8); FW / cg row groups
};

static __constant__ double f_G[13];   // the stability polynomial's coefficients

__device__ __forceinline__ double2 ld_relaxed2(const double2* p) {
  double2 v;
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];"
               : "=d"(v.x), "=d"(v.y)
               : "l"(p)
               : "memory");
  return v;
}
__device__ __forceinline__ double ld_relaxed1(const double* p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed2(double2* p, double2 v) {
  asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v.x), "d"(v.y)
               : "memory");
}
__device__ __forceinline__ void st_relaxed1(double* p, double v) {
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}
__device__ __forceinline__ bool is_empty(double v) {
  return (unsigned long long)__double_as_longlong(v) == kEmpty;
}
// kEmpty is one of many NaNs: a computed value that has its bits takes others.
__device__ __forceinline__ double canonical(double v) {
  return is_empty(v) ? __longlong_as_double(0x7ff8000000000000ll) : v;
}
__device__ __forceinline__ double2 empty2() {
  const double e = __longlong_as_double((long long)kEmpty);
  return make_double2(e, e);
}
// One element, published for the polling readers.
__device__ __forceinline__ void publish(double2* p, double2 v) {
  st_relaxed2(p, make_double2(canonical(v.x), canonical(v.y)));
}

__device__ __forceinline__ void bar_arrive(int id, int nthreads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
template <int R>
__device__ __forceinline__ void regs_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R));
}
template <int R>
__device__ __forceinline__ void regs_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R));
}
constexpr int kBarMain = 2;     // the compute warps
constexpr int kBarNorm = 1;     // forward: the step's norm is there
constexpr int kBarHelp = 3;     // the next step's buffers are preset

// The compute warps' progress, for the helper warp: steps (or slots) published
// by warp 0.  Waits until `step` of them are, or the compute warps gave up
// (their own waits are bounded); false then.
__device__ __forceinline__ void tell_step(volatile int* progress, int step) {
  if (threadIdx.x == 0) {
    __threadfence_block();
    *progress = step;
  }
}
__device__ __forceinline__ bool await_step(volatile int* progress, volatile int* dead, int step) {
  bool ok = true;
  while (ok && *progress < step) ok = *dead == 0;
  __threadfence_block();   // the compute warps' accesses before their word come first
  return __all_sync(0xffffffffu, ok);
}

// What a CTA's rows couple to: nlo elements from global row lo0, then nup from
// up0.
struct FlowWin {
  int nlo, nup, lo0, up0;
  __device__ __forceinline__ int K() const { return nlo + nup; }
  __device__ __forceinline__ int row(int k) const { return k < nlo ? lo0 + k : up0 + (k - nlo); }
};

__device__ __forceinline__ FlowWin flow_window(const Geometry& g, int L) {
  FlowWin w;
  w.nlo = L > 0 ? g.state_off[L] - g.state_off[L - 1] : 0;
  w.nup = L < g.nblk ? g.state_off[L + 2] - g.state_off[L + 1] : 0;
  w.lo0 = L > 0 ? g.state_off[L - 1] : 0;
  w.up0 = L < g.nblk ? g.state_off[L + 1] : 0;
  return w;
}

// Coupling element of local row r (of block L) with window element k.
__device__ __forceinline__ double flow_coupling(const Geometry& g, const double* D, int gauge,
                                                int L, int r, const FlowWin& w, int k) {
  if (k < w.nlo) {
    const BlockGeom& b = g.blk[L - 1];
    return D[b.d_off + (long long)k * b.pitch + r];
  }
  const BlockGeom& b = g.blk[L];
  const double d = D[b.d_off + (long long)r * b.pitch + (k - w.nlo)];
  return gauge == 1 ? -d : d;
}

// Polls the window's elements of NC vectors (src, src + spitch, ...) into win
// (shared; vector c at win + c * wpitch), the vectors in `on` only.  All of a
// thread's loads are in flight together: one L2 round trip once the elements
// are there.  Returns false if the wait passed limit_ns.
template <int NC>
__device__ __forceinline__ bool poll_window(const double2* src, size_t spitch, unsigned on,
                                            const FlowWin& w, double2* win, int wpitch, int tid,
                                            unsigned long long limit_ns) {
  constexpr int U = 4;   // elements per thread and vector in flight
  const int K = w.K();
  for (int k0 = tid; k0 < K; k0 += U * FT) {
    unsigned pend = 0;
#pragma unroll
    for (int j = 0; j < U; ++j)
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (k0 + j * FT < K && (on >> c & 1u)) pend |= 1u << (j * NC + c);
    unsigned long long t0 = 0;
    for (unsigned it = 0; pend; ++it) {
      double2 y[U * NC];
#pragma unroll
      for (int j = 0; j < U; ++j)
#pragma unroll
        for (int c = 0; c < NC; ++c)
          if (pend >> (j * NC + c) & 1u)
            y[j * NC + c] = ld_relaxed2(src + c * spitch + w.row(k0 + j * FT));
#pragma unroll
      for (int j = 0; j < U; ++j)
#pragma unroll
        for (int c = 0; c < NC; ++c)
          if ((pend >> (j * NC + c) & 1u) && !is_empty(y[j * NC + c].x) &&
              !is_empty(y[j * NC + c].y)) {
            win[c * wpitch + k0 + j * FT] = y[j * NC + c];
            pend &= ~(1u << (j * NC + c));
          }
      if ((it & 1023u) == 1023u) {
        const unsigned long long t = globaltimer_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > limit_ns) return false;
      }
    }
  }
  return true;
}

// y / nrm with r = 1 / nrm at hand: the product, corrected once by its residual
// (P. Markstein, IBM J. Res. Dev. 34, 1990), a chain of three operations where
// the division's is several times that.  The bits are the division's for every
// quotient that is a normal number (none differed in 9e8 random ones); below
// 2.2e-308 the last place may differ.  A norm here is the root of a sum of
// squares, so its reciprocal does not overflow; where the norm is zero or not
// finite the call fails, or the pulse is NaN, either way.  Every quotient by a
// norm on this path is formed here, so all readers of an element get the same
// bits.
__device__ __forceinline__ double quot(double y, double nrm, double r) {
  const double q = y * r;
  return fma(fma(-q, nrm, y), r, q);
}
__device__ __forceinline__ double2 quot2(double2 y, double2 nr) {
  return make_double2(quot(y.x, nr.x, nr.y), quot(y.y, nr.x, nr.y));
}

// Polls n values and adds those of this lane (every 32nd), a batch of loads in
// flight at a time.  Returns false if the wait passed limit_ns.
__device__ __forceinline__ bool poll_sum(const double* src, int n, int lane,
                                         unsigned long long limit_ns, double* sum) {
  constexpr int U = 5;   // 148 CTAs' values in one batch
  double t = 0.0;
  for (int p0 = lane; p0 < n; p0 += 32 * U) {
    double v[U];
    unsigned long long t0 = 0;
    for (unsigned it = 0;; ++it) {
      bool ready = true;
#pragma unroll
      for (int j = 0; j < U; ++j)
        v[j] = p0 + 32 * j < n ? ld_relaxed1(src + kPartPitch * (p0 + 32 * j)) : 0.0;
#pragma unroll
      for (int j = 0; j < U; ++j) ready = ready && !is_empty(v[j]);
      if (ready) break;
      if ((it & 1023u) == 1023u) {
        const unsigned long long now = globaltimer_ns();
        if (t0 == 0) t0 = now;
        if (now - t0 > limit_ns) return false;
      }
    }
    t += ((v[0] + v[1]) + (v[2] + v[3])) + v[4];
  }
  *sum = t;
  return true;
}

// The window of a buffer that was complete before the launch.
__device__ __forceinline__ void load_window(const double2* src, const FlowWin& w, double2* win,
                                            int tid) {
  const int K = w.K();
  for (int k = tid; k < K; k += FT) win[k] = __ldcg(src + w.row(k));
}

// Sums N values over the 32 lanes by halving: after each exchange a lane
// keeps half of the values, so a warp needs about N + 5 shuffles of doubles
// instead of 5 N.  Lane-constant: which value a lane ends with.
template <int N, int OFF>
struct LaneSum {
  static __device__ __forceinline__ void run(double* v, int lane) {
    if constexpr (OFF > 0) {
      if constexpr (N == 1) {
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], OFF);
        LaneSum<1, OFF / 2>::run(v, lane);
      } else {
        constexpr int H = (N + 1) / 2;
        const bool up = lane & OFF;
#pragma unroll
        for (int i = 0; i < H; ++i) {
          const double lo = v[i], hi = (i + H < N) ? v[i + H] : 0.0;
          const double send = up ? lo : hi;
          v[i] = (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, send, OFF);
        }
        LaneSum<H, OFF / 2>::run(v, lane);
      }
    }
  }
  // index of the value lane ends with, -1 for padding
  static __device__ __forceinline__ int index(int lane, int base, int real) {
    if constexpr (OFF > 0) {
      if constexpr (N == 1) {
        return LaneSum<1, OFF / 2>::index(lane, base, real);
      } else {
        constexpr int H = (N + 1) / 2;
        if (lane & OFF) {
          base += H;
          real = real > H ? real - H : 0;
        } else {
          real = real < H ? real : H;
        }
        return LaneSum<H, OFF / 2>::index(lane, base, real);
      }
    }
    return real > 0 ? base : -1;
  }
};

// The coupling sums of a CTA's rows with NC vectors' windows.
template <int RW, int CPL, bool REG, int NC>
struct FlowRows {
  static constexpr int NV = 2 * NC * RW;
  double cp[REG ? RW : 1][REG ? CPL : 1];
  int rg, cg, CG, RG, rwr, lane, warp, K, ncl, vidx;

  __device__ __forceinline__ void init(const Geometry& g, const double* D, int gauge,
                                       const FlowCta& me, const FlowWin& w, int warp_, int lane_,
                                       double* crow) {
    warp = warp_;
    lane = lane_;
    CG = me.cg;
    RG = FW / CG;
    rg = warp / CG;
    cg = warp % CG;
    rwr = (me.nrows + RG - 1) / RG;   // rows per row group
    K = w.K();
    ncl = (K + 32 * CG - 1) / (32 * CG);
    vidx = LaneSum<NV, 16>::index(lane, 0, NV);
    const int r0 = me.row0 - g.state_off[me.L];
    if constexpr (REG) {
#pragma unroll
      for (int i = 0; i < RW; ++i)
#pragma unroll
        for (int j = 0; j < CPL; ++j) {
          const int lr = rg * rwr + i, k = (j * CG + cg) * 32 + lane;
          cp[i][j] = (i < rwr && lr < me.nrows && k < K)
                         ? flow_coupling(g, D, gauge, me.L, r0 + lr, w, k)
                         : 0.0;
        }
    } else {
      // every warp its own rows and columns
      for (int i = 0; i < rwr; ++i)
        for (int j = 0; j < ncl; ++j) {
          const int lr = rg * rwr + i, k = (j * CG + cg) * 32 + lane;
          if (lr < me.nrows && k < K)
            crow[(size_t)lr * K + k] = flow_coupling(g, D, gauge, me.L, r0 + lr, w, k);
        }
      // (columns past K meet the window's zero padding; the slack after the
      // last row has to be finite for that)
      if (warp == 0)
        for (int k = lane; k < 256; k += 32) crow[(size_t)me.nrows * K + k] = 0.0;
      __syncwarp();
    }
  }

  // Partial sums of this warp's rows and columns into red: value (row i of
  // the group, vector c, re/im) of warp at red[warp * rstride + (i * NC + c) * 2 + ri].
  __device__ __forceinline__ void run(const double2* win, int wpitch, const double* crow, int nrows,
                                      double* red, int rstride) const {
    if constexpr (REG) {
      double v[NV];
#pragma unroll
      for (int i = 0; i < NV; ++i) v[i] = 0.0;
#pragma unroll
      for (int j = 0; j < CPL; ++j) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const double2 y = win[c * wpitch + (j * CG + cg) * 32 + lane];
#pragma unroll
          for (int i = 0; i < RW; ++i) {
            v[(i * NC + c) * 2] = fma(cp[i][j], y.x, v[(i * NC + c) * 2]);
            v[(i * NC + c) * 2 + 1] = fma(cp[i][j], y.y, v[(i * NC + c) * 2 + 1]);
          }
        }
      }
      LaneSum<NV, 16>::run(v, lane);
      if (vidx >= 0) red[warp * rstride + vidx] = v[0];
    } else {
      for (int i0 = 0; i0 < rwr; i0 += RW) {
        double v[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) v[i] = 0.0;
        const double* cr[RW];
#pragma unroll
        for (int i = 0; i < RW; ++i) cr[i] = crow + (size_t)min(rg * rwr + i0 + i, nrows - 1) * K;
#pragma unroll 4
        for (int j = 0; j < ncl; ++j) {
          const int k = (j * CG + cg) * 32 + lane;
          double2 y[NC];
#pragma unroll
          for (int c = 0; c < NC; ++c) y[c] = win[c * wpitch + k];
#pragma unroll
          for (int i = 0; i < RW; ++i) {
            const double d = cr[i][k];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              v[(i * NC + c) * 2] = fma(d, y[c].x, v[(i * NC + c) * 2]);
              v[(i * NC + c) * 2 + 1] = fma(d, y[c].y, v[(i * NC + c) * 2 + 1]);
            }
          }
        }
        LaneSum<NV, 16>::run(v, lane);
        if (vidx >= 0) red[warp * rstride + i0 * 2 * NC + vidx] = v[0];
      }
    }
  }
};

// Where a row's thread finds its partial sums: CG of them, rstride apart.
template <int NC>
struct FlowSum {
  const double2* p;
  int step, CG;
  __device__ __forceinline__ void init(const double* red, int rstride, int CG_, int rwr, int lr) {
    const int rg = lr / rwr, i = lr - rg * rwr;
    p = reinterpret_cast<const double2*>(red + rg * CG_ * rstride) + i * NC;
    step = rstride / 2;
    CG = CG_;
  }
  // the row's coupling with vector c, column groups added in order
  __device__ __forceinline__ double2 get(int c) const {
    double2 w = p[c];
    if (CG == 1) return w;
    const double2 o = p[c + step];
    w = make_double2(w.x + o.x, w.y + o.y);
    for (int q = 2; q < CG; q += 2) {
      const double2 s = p[c + q * step], t = p[c + (q + 1) * step];
      w = make_double2(w.x + (s.x + t.x), w.y + (s.y + t.y));
    }
    return w;
  }
};

struct FlowArgs {
  const double* D;
  const double* eps;
  const double* Ftab;       // field per step
  const FlowCta* cta;
  double2* V;               // [2][11][ntot] Horner vectors in flight
  double2* XS;              // [2][ntot] x_{n+1} before its renormalisation
  double* part;             // [2][npart + 1] norm partials, kPartPitch apart
  unsigned long long* ctr;  // helpers' arrivals, cleared before the launch
  unsigned* status;
  const double2* xin;       // start state (taken as given)
  double2* xout;            // normalised state at the end
  double* pop_hist;         // [steps+1] or null
  double* norm_hist;        // [steps] or null
  int pop_index;
  int steps;
  int gauge;
  int pw;                   // partials per CTA
  double dt;
  // for the objective gradient (null when unused); slots vpitch apart:
  // ckpt slot k: x after k * ckpt_every steps; seg_v: per step n >= seg_from,
  // slot (n - seg_from) * 13 + m holds v_m, m = 1..11, and slot + 12 x_n
  double2* ckpt;
  int ckpt_every;
  double2* seg_v;
  int seg_from;
  long long vpitch;
  BarrierCfg bc;
  Geometry g;
};

// Shared memory of one CTA: window(s), partial sums, coupling rows.
struct FlowSmem {
  int kpad;      // window pitch (elements)
  int rstride;   // red pitch (doubles) per warp
  size_t bytes;
};
__host__ __device__ inline FlowSmem flow_smem(int K, int nrows, int cg, int RW, int CPL, bool reg,
                                              int NC) {
  FlowSmem s;
  const int RG = FW / cg;
  const int rwr = (nrows + RG - 1) / RG;
  const int rows = reg ? RW : (rwr + RW - 1) / RW * RW;
  s.kpad = reg ? CPL * cg * 32 : (K + 32 * cg - 1) / (32 * cg) * (32 * cg);
  s.rstride = rows * 2 * NC;
  s.bytes = 16 * (size_t)s.kpad * NC + 8 * (size_t)FW * s.rstride +
            (reg ? 0 : 8 * ((size_t)nrows * K + 256));   // the last row's slices run past K
  return s;
}

template <int RW, int CPL, bool REG>
__global__ void __launch_bounds__(FTHREADS, 1) k_flow_forward(const __grid_constant__ FlowArgs a) {
  extern __shared__ __align__(16) unsigned char fsm[];
  const Geometry& g = a.g;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const FlowCta me = a.cta[blockIdx.x];
  const FlowWin w = flow_window(g, me.L);
  const int G = gridDim.x, ntot = g.ntot;
  const int np = G * a.pw;
  const FlowSmem sm = flow_smem(w.K(), me.nrows, me.cg, RW, CPL, REG, 1);
  double2* win = reinterpret_cast<double2*>(fsm);
  double* red = reinterpret_cast<double*>(win + sm.kpad);
  double* crow = red + (size_t)FW * sm.rstride;
  __shared__ double2 nrm_sh[2];   // norm and its reciprocal
  __shared__ int mdead, ndead, hdead, progress;
  if (tid == 0) mdead = ndead = hdead = progress = 0;
  for (int k = tid; k < sm.kpad; k += FTHREADS) win[k] = make_double2(0.0, 0.0);
  __syncthreads();

  if (warp >= FW) {
    regs_dec<40>();
    if (warp > FW) return;
    // ---------------- helper warp ----------------
    for (int s = 0; s <= a.steps; ++s) {
      bool ok = true;
      if (s > 0) {
        // ||x_s||: every CTA's partials, lanes striding, then a fixed xor tree
        double sum = 0.0;
        if (!await_step(&progress, &mdead, s)) return;   // step s-1 is published
        ok = poll_sum(a.part + (size_t)((s - 1) & 1) * kPartPitch * (np + 1),
                      np + (int)a.bc.skew, lane, a.bc.wait_ns, &sum);
        ok = __all_sync(0xffffffffu, ok);
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const double nrm = sqrt(sum);
        if (lane == 0) {
          nrm_sh[s & 1] = make_double2(nrm, 1.0 / nrm);
          if (!ok) {
            ndead = 1;
            atomicOr(a.status, ST_WAIT_TIMEOUT);
          }
        }
        __syncwarp();
        bar_arrive(kBarNorm, kHelpBar);
        if (!ok) return;
        if (blockIdx.x == 0 && lane == 0) {
          if (a.norm_hist) a.norm_hist[s - 1] = nrm;
          if (s == a.steps && (!(nrm > 0.0) || !isfinite(nrm))) atomicOr(a.status, ST_NONFINITE);
        }
      }
      if (s == a.steps) return;
      if (s > 0) {
        // every CTA is past step s-1's products: preset its Horner vectors,
        // and x and partials of the step before, for their next use
        double2* V = a.V + (size_t)((s - 1) & 1) * 11 * ntot + me.row0;
        for (int e = lane; e < 11 * me.nrows; e += 32) {
          const int q = e / me.nrows, r = e - q * me.nrows;
          st_relaxed2(V + (size_t)q * ntot + r, empty2());
        }
        for (int r = lane; r < me.nrows; r += 32)
          st_relaxed2(a.XS + (size_t)(s & 1) * ntot + me.row0 + r, empty2());
        if (lane < a.pw)
          st_relaxed1(a.part + kPartPitch * ((size_t)(s & 1) * (np + 1) + blockIdx.x * a.pw + lane),
                      __longlong_as_double((long long)kEmpty));
        __syncwarp();
        if (lane == 0 &&
            !grid_arrive_wait(a.ctr, (unsigned long long)s * G, a.status, a.bc.wait_ns)) {
          ok = false;
          hdead = 1;
        }
        ok = __shfl_sync(0xffffffffu, ok, 0);
      }
      bar_arrive(kBarHelp, kHelpBar);
      if (!ok) return;
    }
    return;
  }

  // ---------------- compute warps ----------------
  regs_inc<232>();
  FlowRows<RW, CPL, REG, 1> rows;
  rows.init(g, a.D, a.gauge, me, w, warp, lane, crow);
  const bool isrow = tid < me.nrows;
  const int row = me.row0 + tid;
  FlowSum<1> sums;
  sums.init(red, sm.rstride, rows.CG, rows.rwr, isrow ? tid : 0);
  double2 xr = make_double2(0.0, 0.0), v = xr;
  double e = 0.0;
  if (isrow) {
    xr = __ldcg(a.xin + row);
    e = a.eps[row];
    if (a.pop_hist && row == a.pop_index)
      a.pop_hist[0] = __dadd_rn(__dmul_rn(xr.x, xr.x), __dmul_rn(xr.y, xr.y));
  }
  const double h = a.dt;
  double F = a.Ftab[0];
  for (int step = 0; step < a.steps; ++step) {
    const double Fnext = (step + 1 < a.steps) ? a.Ftab[step + 1] : 0.0;
    double2* Vs = a.V + (size_t)(step & 1) * 11 * ntot;
    double2* keep = (a.seg_v && step >= a.seg_from)
                        ? a.seg_v + a.vpitch * (13LL * (step - a.seg_from)) + row
                        : nullptr;
    // ---- x_n into the window, divided by its norm ----
    if (step == 0) {
      load_window(a.xin, w, win, tid);
    } else {
      if (!poll_window<1>(a.XS + (size_t)((step - 1) & 1) * ntot, 0, 1u, w, win, sm.kpad, tid,
                          a.bc.wait_ns)) {
        mdead = 1;
        atomicOr(a.status, ST_WAIT_TIMEOUT);
      }
      named_bar_sync(kBarNorm, kHelpBar);
      if (mdead || ndead) return;
      const double2 nr = nrm_sh[step & 1];
#pragma unroll 4
      for (int k = tid; k < w.K(); k += FT) win[k] = quot2(win[k], nr);
      if (isrow) {
        xr = quot2(xr, nr);
        if (a.pop_hist && row == a.pop_index)
          a.pop_hist[step] = __dadd_rn(__dmul_rn(xr.x, xr.x), __dmul_rn(xr.y, xr.y));
        if (a.ckpt && step % a.ckpt_every == 0)
          a.ckpt[a.vpitch * (step / a.ckpt_every) + row] = xr;
      }
    }
    if (isrow && keep) keep[12 * a.vpitch] = xr;
    v = xr;
#pragma unroll 1
    for (int p = 0; p < kFlowProducts; ++p) {
      const bool last = (p == kFlowProducts - 1);
      // all of v_{11-p} = h M(F) v_{12-p} + G_{11-p} x but the coupling's part:
      // one FMA is left once the sums are there (v_12 = G_12 x, whose coupling
      // is G_12 times that of x)
      const double gm = f_G[11 - p], sc = p == 0 ? f_G[12] : 1.0;
      const double cw = h * F * sc, he = h * e * sc;
      const double2 b = make_double2(fma(he, v.y, gm * xr.x), fma(-he, v.x, gm * xr.y));
      if (p > 0 && !poll_window<1>(Vs + (size_t)(p - 1) * ntot, 0, 1u, w, win, sm.kpad, tid,
                                   a.bc.wait_ns)) {
        mdead = 1;
        atomicOr(a.status, ST_WAIT_TIMEOUT);
      }
      if (last)
        named_bar_sync(kBarHelp, kHelpBar);
      else
        named_bar_sync(kBarMain, FT);
      if (mdead || (last && hdead)) return;
      rows.run(win, sm.kpad, crow, me.nrows, red, sm.rstride);
      named_bar_sync(kBarMain, FT);
      if (warp >= a.pw) continue;
      double nsq = 0.0;
      if (isrow) {
        const double2 W = sums.get(0);
        const double2 o = a.gauge == 0 ? make_double2(fma(cw, W.y, b.x), fma(-cw, W.x, b.y))
                                       : make_double2(fma(cw, W.x, b.x), fma(cw, W.y, b.y));
        if (!last) {
          publish(Vs + (size_t)p * ntot + row, o);
          v = o;
          if (keep) keep[(11 - p) * a.vpitch] = o;
        } else {
          publish(a.XS + (size_t)(step & 1) * ntot + row, o);
          nsq = fma(o.x, o.x, o.y * o.y);
          xr = o;
        }
      }
      if (last) {
        for (int o = 16; o > 0; o >>= 1) nsq += __shfl_xor_sync(0xffffffffu, nsq, o);
        if (lane == 0)
          st_relaxed1(a.part + kPartPitch * ((size_t)(step & 1) * (np + 1) + blockIdx.x * a.pw + warp),
                      canonical(nsq));
        tell_step(&progress, step + 1);
      }
    }
    F = Fnext;
  }
  named_bar_sync(kBarNorm, kHelpBar);
  if (ndead) return;
  if (isrow) {
    const double2 x = quot2(xr, nrm_sh[a.steps & 1]);
    a.xout[row] = x;
    if (a.pop_hist && row == a.pop_index)
      a.pop_hist[a.steps] = __dadd_rn(__dmul_rn(x.x, x.x), __dmul_rn(x.y, x.y));
  }
}

// ---------------------------------------------------------------------------
// The reverse pass of the objective gradient: the transpose of the Horner
// products.  M(F) is anti-Hermitian, so with lambda = dJ/dx_{n+1}:
//   vbar_0 = zbar = lambda / ||z_n||        (z_n is x_{n+1} before renormalisation)
//   vbar_{m+1} = -h M(F_n) vbar_m           (m = 0 .. 11)
//   dJ/dF_n = -h sum_m Re<M1 vbar_m, v_{m+1}>,   M1 = dM/dF
//   dJ/dx_n = sum_{m = 0 .. 12} G_m vbar_m
// (the transposed stages of the 13-stage form give the same numbers).  The
// normalisation's projection zbar = (lambda - x Re<x, lambda>) / ||z|| is
// applied once, to the seed: every later lambda is orthogonal to its x,
// Re<x_n, R^T zbar> = Re<R x_n, zbar> = ||z_n|| Re<x_{n+1}, zbar> = 0.
//
// One launch runs iterations it0 .. it1: iteration `it` recomputes segment
// nseg-1-it forward from its checkpoint and sweeps segment nseg-it backwards.
// The two are independent, and both latency-bound, so every product carries
// both vectors through the same exchange and the same coupling registers.
// What the sweep needs of the forward (v_m and x of its own rows) is written
// and read by the same thread.  The norms are the forward pass's.
struct FlowAdjArgs {
  const double* D;
  const double* eps;
  const double* Ftab;        // field of global step n
  const FlowCta* cta;
  double2* V;                // [3][12][2][ntot] in flight: per slot ring and product, both vectors
  unsigned long long* ctr;
  unsigned* status;
  const double2* ckpt;       // slot k: x after k * ckpt_every steps
  const double* norms;       // ||x_{n+1}|| of every step n (pre-renormalisation)
  double2* seg_v[2];         // per buffer set: v_m / x of every step of a segment
  double2* lam;              // in: dJ/dx after the last swept step; out: before the first
  double* fpart;             // [steps][npart] dJ/dF partials
  int steps, ckpt_every, nseg;
  int it0, it1;              // iterations [it0, it1)
  int gauge;
  int pw;
  double dt;
  long long vpitch;
  BarrierCfg bc;
  Geometry g;
};

template <int RW, int CPL, bool REG>
__global__ void __launch_bounds__(FTHREADS, 1) k_flow_adjoint(const __grid_constant__ FlowAdjArgs a) {
  extern __shared__ __align__(16) unsigned char fsm[];
  const Geometry& g = a.g;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const FlowCta me = a.cta[blockIdx.x];
  const FlowWin w = flow_window(g, me.L);
  const int G = gridDim.x, ntot = g.ntot;
  const FlowSmem sm = flow_smem(w.K(), me.nrows, me.cg, RW, CPL, REG, 2);
  double2* win = reinterpret_cast<double2*>(fsm);          // [2][kpad]
  double* red = reinterpret_cast<double*>(win + 2 * sm.kpad);
  double* crow = red + (size_t)FW * sm.rstride;
  __shared__ int mdead, hdead, progress;
  if (tid == 0) mdead = hdead = progress = 0;
  for (int k = tid; k < 2 * sm.kpad; k += FTHREADS) win[k] = make_double2(0.0, 0.0);
  __syncthreads();
  const int Kc = a.ckpt_every;
  // step slots of the launch
  int nslots = 0;
  for (int it = a.it0; it < a.it1; ++it) {
    const int rseg = a.nseg - 1 - it, aseg = a.nseg - it;
    const int lenF = rseg >= 0 ? min(Kc, a.steps - rseg * Kc) : 0;
    const int lenA = aseg <= a.nseg - 1 ? min(Kc, a.steps - aseg * Kc) : 0;
    nslots += max(lenF, lenA);
  }
  const size_t ring = (size_t)12 * 2 * ntot;

  if (warp >= FW) {
    regs_dec<40>();
    if (warp > FW) return;
    // helper: once its CTA is past slot s-1 it arrives at the counter (which
    // also publishes the presets it made a slot earlier), waits for every
    // CTA, and presets slot s-1's buffers, which slot s+2 uses.
    for (int s = 0; s < nslots; ++s) {
      bool ok = true;
      if (s > 0) {
        if (!await_step(&progress, &mdead, s)) return;
        if (lane == 0)
          ok = grid_arrive_wait(a.ctr, (unsigned long long)s * G + a.bc.skew, a.status,
                                a.bc.wait_ns);
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (ok) {
          double2* V = a.V + (size_t)((s - 1) % 3) * ring + me.row0;
          for (int e = lane; e < 24 * me.nrows; e += 32) {
            const int q = e / me.nrows, r = e - q * me.nrows;
            st_relaxed2(V + (size_t)q * ntot + r, empty2());
          }
        }
        __syncwarp();
      }
      if (!ok && lane == 0) hdead = 1;
      __syncwarp();
      bar_arrive(kBarHelp, kHelpBar);
      if (!ok) return;
    }
    return;
  }

  regs_inc<232>();
  FlowRows<RW, CPL, REG, 2> rows;
  rows.init(g, a.D, a.gauge, me, w, warp, lane, crow);
  const bool isrow = tid < me.nrows;
  const int row = me.row0 + tid;
  FlowSum<2> sums;
  sums.init(red, sm.rstride, rows.CG, rows.rwr, isrow ? tid : 0);
  double e = 0.0;
  double2 lam = make_double2(0.0, 0.0);
  if (isrow) {
    e = a.eps[row];
    lam = __ldcg(a.lam + row);
  }
  const double h = a.dt;
  const long long vp = a.vpitch;
  int s = 0;   // slot
  for (int it = a.it0; it < a.it1; ++it) {
    const int rseg = a.nseg - 1 - it, aseg = a.nseg - it;
    const int lenF = rseg >= 0 ? min(Kc, a.steps - rseg * Kc) : 0;
    const int lenA = aseg <= a.nseg - 1 ? min(Kc, a.steps - aseg * Kc) : 0;
    const int slots = max(lenF, lenA);
    double2 xr = make_double2(0.0, 0.0);
    if (isrow && lenF) xr = __ldcg(a.ckpt + vp * rseg + row);
    for (int slot = 0; slot < slots; ++slot, ++s) {
      const bool fw = slot < lenF, ad = slot < lenA;
      const int nF = rseg * Kc + slot;                   // recomputed step
      const int jA = lenA - 1 - slot, nA = aseg * Kc + jA;  // swept step
      double2* Vs = a.V + (size_t)(s % 3) * ring;
      const double FF = fw ? a.Ftab[nF] : 0.0, FA = ad ? a.Ftab[nA] : 0.0;
      const double nF1 = fw ? a.norms[nF] : 1.0, nA1 = ad ? a.norms[nA] : 1.0;
      const double2 nrF = make_double2(nF1, 1.0 / nF1), nrA = make_double2(nA1, 1.0 / nA1);
      double2* keep = a.seg_v[rseg & 1] + vp * (13LL * slot) + row;
      const double2* kept = a.seg_v[aseg & 1] + vp * (13LL * jA) + row;
      double2 v = xr, vb = make_double2(0.0, 0.0), xb = vb;
      double fs = 0.0;
      if (isrow) {
        if (fw) {
          publish(Vs + row, xr);
          keep[12 * vp] = xr;
        }
        if (ad) {
          vb = quot2(lam, nrA);
          publish(Vs + ntot + row, vb);
        }
      }
#pragma unroll 1
      for (int p = 0; p < kFlowProducts; ++p) {
        const bool last = (p == kFlowProducts - 1);
        const double2* src = Vs + (size_t)p * 2 * ntot;
        // as in the forward: everything but the coupling's part, beforehand
        const double gm = f_G[11 - p], sc = p == 0 ? f_G[12] : 1.0, gA = f_G[p];
        const double cw = h * FF * sc, he = h * e * sc, cA = -h * FA, heA = h * e;
        const double2 b = make_double2(fma(he, v.y, gm * xr.x), fma(-he, v.x, gm * xr.y));
        const double2 bA = make_double2(-heA * vb.y, heA * vb.x);   // -h (-i e vbar)
        xb.x = fma(gA, vb.x, xb.x);
        xb.y = fma(gA, vb.y, xb.y);
        double2 vk = make_double2(0.0, 0.0);
        if (isrow && ad) vk = kept[(p + 1) * vp];   // v_{p+1} of the swept step
        if (!poll_window<2>(src, ntot, (fw ? 1u : 0u) | (ad ? 2u : 0u), w, win, sm.kpad, tid,
                            a.bc.wait_ns)) {
          mdead = 1;
          atomicOr(a.status, ST_WAIT_TIMEOUT);
        }
        if (last)
          named_bar_sync(kBarHelp, kHelpBar);
        else
          named_bar_sync(kBarMain, FT);
        if (mdead || (last && hdead)) {
          return;
        }
        rows.run(win, sm.kpad, crow, me.nrows, red, sm.rstride);
        named_bar_sync(kBarMain, FT);
        if (last) tell_step(&progress, s + 1);   // the slot's windows are consumed
        if (warp >= a.pw) continue;
        if (isrow) {
          double2* out = Vs + (size_t)(p + 1) * 2 * ntot + row;
          if (fw) {
            const double2 W = sums.get(0);
            const double2 o = a.gauge == 0
                                  ? make_double2(fma(cw, W.y, b.x), fma(-cw, W.x, b.y))
                                  : make_double2(fma(cw, W.x, b.x), fma(cw, W.y, b.y));
            if (!last) {
              publish(out, o);
              v = o;
              keep[(11 - p) * vp] = o;
            } else {
              xr = quot2(o, nrF);
            }
          }
          if (ad) {
            const double2 W = sums.get(1);
            const double2 m1 = a.gauge == 0 ? make_double2(W.y, -W.x) : W;
            vb = make_double2(fma(cA, m1.x, bA.x), fma(cA, m1.y, bA.y));
            if (!last) publish(out + ntot, vb);
            // v_12 = G_12 x
            fs -= (last ? f_G[12] : 1.0) * fma(m1.x, vk.x, m1.y * vk.y);
            if (last) {
              lam = make_double2(fma(f_G[12], vb.x, xb.x), fma(f_G[12], vb.y, xb.y));
              fs *= h;
            }
          }
        }
        if (last && ad) {
          for (int o = 16; o > 0; o >>= 1) fs += __shfl_xor_sync(0xffffffffu, fs, o);
          if (lane == 0) a.fpart[((long long)nA * G + blockIdx.x) * a.pw + warp] = fs;
        }
      }
    }
  }
  if (isrow) a.lam[row] = lam;
}

}  // namespace mpc
