// resident.cu -- the resident path: fixed-step propagation and the objective
// gradient's reverse pass for systems whose coupling fits on chip, one
// persistent cooperative launch each (kernels in resident_flow.cuh).  This
// file splits the rows over the CTAs, picks the kernels' register tiles and
// launches them.
// Same semantics as the streaming path (tdse::propV / propL,
// src/tdse/tdse.cpp:186-215): F frozen at t+dt, 8th-order RKF78, c /= ||c||.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <vector>

#include "ctx.h"
#include "dev_util.cuh"
#include "plan.h"
#include "resident_flow.cuh"
#include "rkf78.h"

using namespace mpc;

namespace {

// A kernel instance: RW rows x CPL window columns per lane, the coupling in
// registers (reg) or, for rows too long or too many for them, in shared
// memory.
struct FlowKernel {
  int RW, CPL;
  bool reg;
  const void* fn;
};

#define FWD(RW, CPL) {RW, CPL, true, reinterpret_cast<const void*>(&k_flow_forward<RW, CPL, true>)}
#define ADJ(RW, CPL) {RW, CPL, true, reinterpret_cast<const void*>(&k_flow_adjoint<RW, CPL, true>)}
const FlowKernel kForward[] = {
    FWD(1, 4), FWD(2, 6), FWD(3, 10), FWD(4, 10), FWD(5, 12), FWD(6, 13),
    {6, 0, false, reinterpret_cast<const void*>(&k_flow_forward<6, 1, false>)}};
const FlowKernel kAdjoint[] = {
    ADJ(1, 4), ADJ(2, 6), ADJ(3, 10), ADJ(4, 10),
    {6, 0, false, reinterpret_cast<const void*>(&k_flow_adjoint<6, 1, false>)}};
#undef FWD
#undef ADJ

// dJ/dF_n = sum over the CTAs' partials of step n: one warp per step, lanes
// striding, then a fixed xor tree.
__global__ void k_flow_fbar(const double* fpart, int steps, int np, double* fbar) {
  const int n = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (n >= steps) return;
  double t = 0.0;
  for (int p = lane; p < np; p += 32) t += fpart[(long long)n * np + p];
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) fbar[n] = t;
}

// lambda_N = (1 - x x^T) dJ/dx_N, x = x_N (unit norm): yield -> 2 x on the
// states at or above the threshold, target -> 2 x_t.  One CTA; the projection
// is the last step's normalisation adjoint.
__global__ void k_flow_seed(const double2* x, const double* eps, double2* lam, int target,
                            double thr, int ntot) {
  __shared__ double sh[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto seed = [&](int i) {
    const double2 v = x[i];
    const bool on = target < 0 ? eps[i] >= thr : i == target;
    return on ? make_double2(2.0 * v.x, 2.0 * v.y) : make_double2(0.0, 0.0);
  };
  double d = 0.0;
  for (int i = threadIdx.x; i < ntot; i += blockDim.x) {
    const double2 v = x[i], l = seed(i);
    d += fma(v.x, l.x, v.y * l.y);
  }
  for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
  if (lane == 0) sh[warp] = d;
  __syncthreads();
  d = 0.0;
  for (int q = 0; q < (int)(blockDim.x >> 5); ++q) d += sh[q];
  for (int i = threadIdx.x; i < ntot; i += blockDim.x) {
    const double2 v = x[i], l = seed(i);
    lam[i] = make_double2(fma(-d, v.x, l.x), fma(-d, v.y, l.y));
  }
}

constexpr size_t kFlowStatic = 256;   // the kernels' static shared memory, rounded up

int window_len(const Geometry& g, int L) {
  return (L > 0 ? g.state_off[L] - g.state_off[L - 1] : 0) +
         (L < g.nblk ? g.state_off[L + 2] - g.state_off[L + 1] : 0);
}

// CTAs to blocks: each CTA's rows lie in one block, and the next CTA always
// goes to the block whose rows per CTA x window length (its product's work,
// with 64 columns' worth for the row itself) is largest, so that end blocks,
// with half the window, get twice the rows.  At
// least 4 rows per CTA on average: fewer, larger CTAs poll less for the same
// latency.
bool split_rows(const Geometry& g, int sms, std::vector<FlowCta>& ctas) {
  const int nb = g.nstate_blk;
  const int G = std::min(sms, std::max(nb, (g.ntot + 3) / 4));
  if (nb > G) return false;
  std::vector<int> cnt(nb, 1);
  for (int used = nb; used < G; ++used) {
    int best = -1;
    double most = 0.0;
    for (int L = 0; L < nb; ++L) {
      const int nL = g.state_off[L + 1] - g.state_off[L];
      if (cnt[L] >= nL) continue;
      const double work = (double)nL / cnt[L] * (window_len(g, L) + 64);
      if (work > most) {
        most = work;
        best = L;
      }
    }
    if (best < 0) break;
    ++cnt[best];
  }
  ctas.clear();
  for (int L = 0; L < nb; ++L) {
    const int o = g.state_off[L], nL = g.state_off[L + 1] - o;
    for (int j = 0; j < cnt[L]; ++j) {
      const int r0 = (int)((long long)nL * j / cnt[L]), r1 = (int)((long long)nL * (j + 1) / cnt[L]);
      ctas.push_back({L, o + r0, r1 - r0, 1});
      if (r1 - r0 > kFlowMaxRows) return false;
    }
  }
  return true;
}

// Sets every CTA's column groups for kernel k; false if a CTA does not fit.
// In registers: the most column groups (the fewest reads of the window from
// shared memory) whose rows per row group still fit.  From shared memory: the
// fewest reads of window and coupling together (a pass over the window per
// RW rows of a group).
bool fit_kernel(const Geometry& g, const FlowKernel& k, int NC, size_t limit,
                std::vector<FlowCta>& ctas, size_t* smem) {
  *smem = 0;
  for (FlowCta& c : ctas) {
    const int K = window_len(g, c.L);
    int best = 0;
    double cost = 1e300;
    for (int cg = FW; cg >= 1; cg /= 2) {
      const int RG = FW / cg, rwr = (c.nrows + RG - 1) / RG;
      if (k.reg) {
        if (rwr > k.RW || K > 32 * cg * k.CPL) continue;
        best = cg;
        break;
      }
      const int passes = (rwr + k.RW - 1) / k.RW;
      const double t = passes * (0.125 * NC * RG * K + 400.0);
      if (t < cost &&
          flow_smem(K, c.nrows, cg, k.RW, k.CPL, false, NC).bytes + kFlowStatic <= limit) {
        cost = t;
        best = cg;
      }
    }
    if (!best) return false;
    c.cg = best;
    const FlowSmem s = flow_smem(K, c.nrows, best, k.RW, k.CPL, k.reg, NC);
    if (s.bytes + kFlowStatic > limit) return false;
    *smem = std::max(*smem, s.bytes);
  }
  return true;
}

// One kernel's launch: the instance, each CTA's layout (device), its shared
// memory.
struct FlowLaunch {
  const void* fn = nullptr;
  FlowCta* ctas = nullptr;
  size_t smem = 0;
};

template <size_t N>
bool plan_kernel(const Geometry& g, const FlowKernel (&list)[N], int NC, size_t limit,
                 std::vector<FlowCta> ctas, FlowLaunch* out) {
  for (const FlowKernel& k : list) {
    size_t smem = 0;
    if (!fit_kernel(g, k, NC, limit, ctas, &smem)) continue;
    int per_sm = 0;
    if (!mpc_allow_smem(k.fn, (int)limit) ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k.fn, FTHREADS, smem) !=
            cudaSuccess ||
        per_sm < 1) {
      cudaGetLastError();
      continue;
    }
    if (cudaMalloc(&out->ctas, sizeof(FlowCta) * ctas.size()) != cudaSuccess ||
        cudaMemcpy(out->ctas, ctas.data(), sizeof(FlowCta) * ctas.size(),
                   cudaMemcpyHostToDevice) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    out->fn = k.fn;
    out->smem = smem;
    return true;
  }
  return false;
}

}  // namespace

struct mpc_resident_state {
  bool ok = false;
  bool adj_ok = false;
  bool one_launch = true;        // the reverse pass in one launch
  int G = 0;
  int pw = 1;                    // partials per CTA (32 rows each)
  FlowLaunch fwd, adj;
  unsigned long long* ctr = nullptr;   // helpers' arrivals
  double2* V = nullptr;          // [3][12][2][ntot]: vectors in flight (both kernels)
  double* part = nullptr;        // [2][G * pw + 1], kPartPitch apart
  double2* XS = nullptr;         // [2][ntot]
  double* fpart = nullptr;
  size_t fpart_n = 0;
};

// All the dynamic shared memory a block may have: the attribute belongs to the
// function, so a context must not set it to its own, smaller need.
bool mpc_allow_smem(const void* fn, int optin) {
  cudaFuncAttributes at{};
  const bool ok = cudaFuncGetAttributes(&at, fn) == cudaSuccess &&
                  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       optin - (int)at.sharedSizeBytes) == cudaSuccess;
  if (!ok) cudaGetLastError();
  return ok;
}

// Sets up the resident path if the system fits; returns true when usable.
bool mpc_resident_setup(mpc_ctx* c) {
  if (c->resident) return c->resident->ok;
  mpc_resident_state* r = new mpc_resident_state();
  c->resident = r;
  if (std::getenv("MPC_NO_RESIDENT")) return false;
  int coop = 0, optin = 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
  if (!coop) return false;
  std::vector<FlowCta> ctas;
  if (!split_rows(c->g, c->num_sms, ctas)) return false;
  if (!plan_kernel(c->g, kForward, 1, optin, ctas, &r->fwd)) return false;
  r->G = (int)ctas.size();
  int rows = 1;
  for (const FlowCta& t : ctas) rows = std::max(rows, t.nrows);
  r->pw = (rows + 31) / 32;
  const size_t n = c->g.ntot;
  if (cudaMemcpyToSymbol(f_G, rkf78::G, sizeof rkf78::G) != cudaSuccess ||
      cudaMalloc(&r->ctr, sizeof(unsigned long long)) != cudaSuccess ||
      cudaMalloc(&r->V, sizeof(double2) * 72 * n) != cudaSuccess ||
      cudaMalloc(&r->XS, sizeof(double2) * 2 * n) != cudaSuccess ||
      cudaMalloc(&r->part, sizeof(double) * 2 * kPartPitch * ((size_t)r->G * r->pw + 1)) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  r->adj_ok = plan_kernel(c->g, kAdjoint, 2, optin, ctas, &r->adj);
  r->one_launch = std::getenv("MPC_NO_FUSED_ADJOINT") == nullptr;
  r->ok = true;
  return true;
}

void mpc_resident_free(mpc_ctx* c) {
  if (!c || !c->resident) return;
  mpc_resident_state* r = c->resident;
  cudaFree(r->fwd.ctas);
  cudaFree(r->adj.ctas);
  cudaFree(r->ctr);
  cudaFree(r->V);
  cudaFree(r->XS);
  cudaFree(r->part);
  cudaFree(r->fpart);
  delete r;
  c->resident = nullptr;
}

namespace {

int launch_forward(mpc_ctx* c, FlowArgs& a) {
  mpc_resident_state* r = c->resident;
  const size_t n = c->g.ntot;
  a.D = c->d_D;
  a.eps = c->d_eps;
  a.cta = r->fwd.ctas;
  a.V = r->V;
  a.XS = r->XS;
  a.part = r->part;
  a.ctr = r->ctr;
  a.status = c->d_status;
  a.gauge = (c->gauge == 'l') ? 0 : 1;
  a.pw = r->pw;
  a.bc = mpc_barrier_cfg(c);
  a.g = c->g;
  CK(cudaMemsetAsync(r->ctr, 0, sizeof(unsigned long long), c->stream));
  CK(cudaMemsetAsync(r->V, 0xff, sizeof(double2) * 22 * n, c->stream));
  CK(cudaMemsetAsync(r->XS, 0xff, sizeof(double2) * 2 * n, c->stream));
  CK(cudaMemsetAsync(r->part, 0xff, sizeof(double) * 2 * kPartPitch * ((size_t)r->G * r->pw + 1), c->stream));
  void* args[] = {&a};
  ProfScope ps(c, MPC_KERNEL_RESIDENT);
  CK(cudaLaunchCooperativeKernel(r->fwd.fn, dim3(r->G), dim3(FTHREADS), args, r->fwd.smem,
                                 c->stream));
  return MPC_OK;
}

}  // namespace

// Runs `steps` steps of the fixed-step loop on the state in c->d_x with the
// field table already in c->d_Ftab; histories into c->d_pop / c->d_nrm.
int mpc_resident_run(mpc_ctx* c, double dt, int steps, int pop_index) {
  FlowArgs a{};
  a.Ftab = c->d_Ftab;
  a.xin = c->d_x;
  a.xout = c->d_x;   // written once every CTA is past its last step
  a.pop_hist = c->d_pop;
  a.norm_hist = c->d_nrm;
  a.pop_index = pop_index;
  a.steps = steps;
  a.dt = dt;
  return launch_forward(c, a);
}

// The objective's forward pass from x_in for `steps` steps with the field
// table Ftab: the result into x_out, every step's norm, the state every
// ckpt_every steps, and from step seg_from on every
// step's Horner vectors (seg_v); slots vpitch complex apart.
int mpc_resident_forward_ex(mpc_ctx* c, const double2* x_in, double2* x_out, const double* Ftab,
                            double dt, int steps, double* norm_hist, double2* ckpt,
                            int ckpt_every, double2* seg_v, int seg_from, long long vpitch) {
  FlowArgs a{};
  a.Ftab = Ftab;
  a.xin = x_in;
  a.xout = x_out;
  a.norm_hist = norm_hist;
  a.pop_index = -1;
  a.steps = steps;
  a.dt = dt;
  a.ckpt = ckpt;
  a.ckpt_every = ckpt_every;
  a.seg_v = seg_v;
  a.seg_from = seg_from;
  a.vpitch = vpitch;
  return launch_forward(c, a);
}

bool mpc_resident_adjoint_ok(mpc_ctx* c) { return c->resident && c->resident->adj_ok; }

// The whole reverse pass (k_flow_adjoint): lam = lambda_N in, lambda_0 out,
// dJ/dF of every step into fbar; segment a's Horner vectors live in
// seg_v[a & 1]; last_kept: the forward left the last segment's there.
int mpc_resident_backward(mpc_ctx* c, const double2* ckpt, const double* norms, int steps,
                          int ckpt_every, const double* Ftab, double dt, double2* const* seg_v,
                          bool last_kept, double2* lam, double* fbar, long long vpitch) {
  mpc_resident_state* r = c->resident;
  if (!r || !r->adj_ok) return mpc_fail(MPC_ERR_ARG, "resident adjoint unavailable");
  const int np = r->G * r->pw;
  if (r->fpart_n < (size_t)steps * np) {
    cudaFree(r->fpart);
    r->fpart = nullptr;
    r->fpart_n = 0;
    CK(cudaMalloc(&r->fpart, sizeof(double) * (size_t)steps * np));
    r->fpart_n = (size_t)steps * np;
  }
  FlowAdjArgs a{};
  a.D = c->d_D;
  a.eps = c->d_eps;
  a.Ftab = Ftab;
  a.cta = r->adj.ctas;
  a.V = r->V;
  a.ctr = r->ctr;
  a.status = c->d_status;
  a.ckpt = ckpt;
  a.norms = norms;
  a.seg_v[0] = seg_v[0];
  a.seg_v[1] = seg_v[1];
  a.lam = lam;
  a.fpart = r->fpart;
  a.steps = steps;
  a.ckpt_every = ckpt_every;
  a.nseg = (steps + ckpt_every - 1) / ckpt_every;
  a.gauge = (c->gauge == 'l') ? 0 : 1;
  a.pw = r->pw;
  a.dt = dt;
  a.vpitch = vpitch;
  a.bc = mpc_barrier_cfg(c);
  a.g = c->g;
  // iteration 0 only recomputes the last segment
  const int first = last_kept ? 1 : 0, end = a.nseg + 1;
  for (int it = first; it < end;) {
    a.it0 = it;
    a.it1 = r->one_launch ? end : it + 1;
    CK(cudaMemsetAsync(r->ctr, 0, sizeof(unsigned long long), c->stream));
    CK(cudaMemsetAsync(r->V, 0xff, sizeof(double2) * 72 * c->g.ntot, c->stream));
    void* args[] = {&a};
    ProfScope ps(c, MPC_KERNEL_RESIDENT);
    CK(cudaLaunchCooperativeKernel(r->adj.fn, dim3(r->G), dim3(FTHREADS), args, r->adj.smem,
                                   c->stream));
    it = a.it1;
  }
  k_flow_fbar<<<(steps * 32 + 127) / 128, 128, 0, c->stream>>>(r->fpart, steps, np, fbar);
  CK(cudaGetLastError());
  ++c->launches;
  return MPC_OK;
}

// lambda_N of the objective at x (see k_flow_seed).
int mpc_resident_seed(mpc_ctx* c, const double2* x, double2* lam, int target) {
  k_flow_seed<<<1, 512, 0, c->stream>>>(x, c->d_eps, lam, target, c->yield_thr, c->g.ntot);
  CK(cudaGetLastError());
  ++c->launches;
  return MPC_OK;
}
