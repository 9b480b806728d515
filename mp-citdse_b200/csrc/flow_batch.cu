// flow_batch.cu -- host side of the persistent batched kernels
// (flow_batch.cuh): the split of the rows over the CTAs and of the pulses
// over column groups and chunks, the work space, the launches.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <numeric>
#include <vector>

#include "batch_types.h"
#include "ctx.h"
#include "flow_batch.cuh"
#include "flow_batch.h"

using namespace mpc;

namespace {

constexpr int kMaxGroups = 4;
const void* const kKernels[] = {reinterpret_cast<const void*>(&k_flow_batch<0>),
                                reinterpret_cast<const void*>(&k_flow_batch<1>),
                                reinterpret_cast<const void*>(&k_flow_batch<2>)};
const int kSlots[] = {kFixSlots, kAdaptSlots, kAdjSlots};

int window_len(const Geometry& g, int L) {
  return (L > 0 ? g.state_off[L] - g.state_off[L - 1] : 0) +
         (L < g.nblk ? g.state_off[L + 2] - g.state_off[L + 1] : 0);
}

// The kernels' instances, 8-row tiles x groups of 4 window rows per warp (the
// cases of k_flow_batch's switch); a CTA takes the cheapest that holds its rows.
struct FbConfig {
  int mt, kt;
};
const FbConfig kConfigs[] = {{1, 6},  {2, 6},  {4, 6},  {2, 10}, {4, 10}, {6, 10},
                             {2, 13}, {5, 13}, {2, 19}, {3, 19}, {2, 25}, {3, 25}};

int config_for(int rows, int K) {
  int best = -1;
  for (int i = 0; i < (int)(sizeof kConfigs / sizeof kConfigs[0]); ++i) {
    const FbConfig& f = kConfigs[i];
    if (rows > 8 * f.mt || K > 4 * FW * f.kt) continue;
    if (best < 0 || f.mt * f.kt < kConfigs[best].mt * kConfigs[best].kt) best = i;
  }
  return best;
}
// its DMMA work: the window groups that are there, all tiles of the instance
int config_cost(int i, int K) { return kConfigs[i].mt * ((K + 4 * FW - 1) / (4 * FW)); }

// One column group's CTAs: every block starts with the fewest CTAs whose
// registers hold its rows; then the block whose CTAs cost most gets as many
// more as its next cheaper instance needs, while there are any.
bool split_group(const Geometry& g, int gp, std::vector<FbCta>& ctas, int* cost) {
  const int nb = g.nstate_blk;
  std::vector<int> cnt(nb), cfg(nb);
  int used = 0;
  for (int L = 0; L < nb; ++L) {
    const int nL = g.state_off[L + 1] - g.state_off[L], K = window_len(g, L);
    cnt[L] = 0;
    for (int n = 1; n <= std::min(nL, gp) && !cnt[L]; ++n) {
      cfg[L] = config_for((nL + n - 1) / n, K);
      if (cfg[L] >= 0) cnt[L] = n;
    }
    if (!cnt[L]) return false;
    used += cnt[L];
  }
  if (used > gp) return false;
  auto work = [&](int L) { return config_cost(cfg[L], window_len(g, L)); };
  while (true) {
    int top = 0;
    for (int L = 1; L < nb; ++L)
      if (work(L) > work(top)) top = L;
    const int nL = g.state_off[top + 1] - g.state_off[top], K = window_len(g, top);
    int n = cnt[top] + 1, f = -1;
    for (; n <= nL && used - cnt[top] + n <= gp; ++n) {
      f = config_for((nL + n - 1) / n, K);
      if (f >= 0 && config_cost(f, K) < work(top)) break;
      f = -1;
    }
    if (f < 0) break;
    used += n - cnt[top];
    cnt[top] = n;
    cfg[top] = f;
  }
  ctas.clear();
  *cost = 0;
  for (int L = 0; L < nb; ++L) {
    const int o = g.state_off[L], nL = g.state_off[L + 1] - o;
    for (int j = 0; j < cnt[L]; ++j) {
      const int r0 = (int)((long long)nL * j / cnt[L]), r1 = (int)((long long)nL * (j + 1) / cnt[L]);
      ctas.push_back({L, o + r0, r1 - r0, 0, (int)ctas.size(), cfg[L]});
    }
    *cost = std::max(*cost, work(L));
  }
  return true;
}

// Microseconds of a product for the chunks of one column group: items of 64
// cycles per unit of DMMA work and about 2,500 for loads, sums and the rest
// (1752 states 5,750 cycles at 57 units, 3492 states 8,000 at 75, 500 states
// 3,100 at 14), or the exchange, about 4,500, when there are too few chunks to
// hide it.
double product_us(int cost, int chunks_per_group) {
  return std::max(chunks_per_group * (64.0 * cost + 2500.0), 64.0 * cost + 4500.0) / 1900.0;
}

// The stage GEMM's product at B pulses: measured 47 us at 1752 states and 256
// pulses, 23 at 64; 103 and 44 at 3492 states; 17 at 500 states and 256 pulses.
double gemm_us(const Geometry& g, int B) {
  double s = 0.0;
  for (int L = 0; L < g.nblk; ++L) s += (double)g.blk[L].nrow * g.blk[L].ncol;
  return 14.0 + 8.0 * s * B / 26e6;
}

struct Group {
  bool ok = false;
  int gp = 0;       // CTAs per group
  int cost = 0;
  int mt = 0, rows = 0;   // of its largest CTA
  FbCta* ctas = nullptr;
};

template <class T>
int grow(T** p, size_t* cap, size_t n) {
  if (*cap >= n) return MPC_OK;
  cudaFree(*p);
  *p = nullptr;
  *cap = 0;
  CK(cudaMalloc(p, sizeof(T) * n));
  *cap = n;
  return MPC_OK;
}

}  // namespace

struct mpc_flowb_state {
  bool tried = false, ok = false;
  size_t optin = 0;          // shared memory a CTA may have
  Group grp[kMaxGroups + 1];
  // work space, kept between calls and grown on demand
  double2* V = nullptr;
  size_t V_n = 0;
  double* part = nullptr;
  size_t part_n = 0;
  unsigned long long* ctr = nullptr;
  size_t ctr_n = 0;
  double2* xst = nullptr;
  size_t xst_n = 0;
  double2* kst = nullptr;    // adaptive steps: slopes and x_new
  size_t kst_n = 0;
  double2* io = nullptr;     // start and final states by pulse id
  size_t io_n = 0;
  int* ints = nullptr;       // chunk ids, chunk steps, pulse steps
  size_t ints_n = 0;
  mpc_pulse* pulse = nullptr;
  size_t pulse_n = 0;
  double* t0 = nullptr;
  size_t t0_n = 0;
  double* hist = nullptr;    // population and norm histories
  size_t hist_n = 0;
  // the batched objective's last forward pass (kept for its backward pass, so
  // in buffers of its own)
  int oB = 0, osteps = 0, ockpt = 0, ong = 0, onch = 0;
  bool okept = false;        // seg_v holds the last segment
  double odt = 0.0;
  int* oint = nullptr;
  size_t oint_n = 0;
  double2* oio = nullptr;    // start states, x_N [B][n]
  size_t oio_n = 0;
  double* oF = nullptr;      // fields [steps][B]
  size_t oF_n = 0;
  double* onorm = nullptr;   // [B][steps]
  size_t onorm_n = 0;
  double2* ockp = nullptr;   // checkpoints
  size_t ockp_n = 0;
  double2* oseg = nullptr;   // a segment's vectors
  size_t oseg_n = 0;
  double2* olam = nullptr;   // lambda, then the sums of G_m vbar_m
  size_t olam_n = 0;
  double* ofs = nullptr;
  size_t ofs_n = 0;
  double* ofp = nullptr;     // dJ/dF partials of a segment
  size_t ofp_n = 0;
  double* ofb = nullptr;     // dJ/dF [steps][B]
  size_t ofb_n = 0;
};

bool mpc_flowb_setup(mpc_ctx* c) {
  if (!c->flowb) c->flowb = new mpc_flowb_state();
  mpc_flowb_state* f = c->flowb;
  if (f->tried) return f->ok;
  f->tried = true;
  if (std::getenv("MPC_NO_RESIDENT")) return false;
  int coop = 0, optin = 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
  if (!coop) return false;
  f->optin = optin;
  double A[13][13], B8[13], E[13], Cn[13];
  for (int i = 0; i < 13; ++i) {
    for (int j = 0; j < 13; ++j) A[i][j] = rkf78::A[i][j];
    B8[i] = rkf78::B8[i];
    E[i] = rkf78::B8[i] - rkf78::B7[i];
    Cn[i] = rkf78::C[i];
  }
  if (cudaMemcpyToSymbol(f_G, rkf78::G, sizeof rkf78::G) != cudaSuccess ||
      cudaMemcpyToSymbol(f_A, A, sizeof A) != cudaSuccess ||
      cudaMemcpyToSymbol(f_B8, B8, sizeof B8) != cudaSuccess ||
      cudaMemcpyToSymbol(f_E, E, sizeof E) != cudaSuccess ||
      cudaMemcpyToSymbol(f_C, Cn, sizeof Cn) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  for (int ng = 1; ng <= kMaxGroups; ++ng) {
    Group& g = f->grp[ng];
    std::vector<FbCta> one, all;
    if (!split_group(c->g, c->num_sms / ng, one, &g.cost)) continue;
    g.gp = (int)one.size();
    for (int k = 0; k < ng; ++k)
      for (FbCta t : one) {
        t.grp = k;
        all.push_back(t);
        g.mt = std::max(g.mt, kConfigs[t.cfg].mt);
        g.rows = std::max(g.rows, t.nrows);
      }
    int per_sm = 0;
    bool fits = true;
    for (int mode = 0; mode < 3 && fits; ++mode)
      fits = mpc_allow_smem(kKernels[mode], optin) &&
             cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kKernels[mode], FTHREADS,
                                                           flowb_smem(mode, g.mt)) == cudaSuccess &&
             per_sm >= 1;
    if (!fits || cudaMalloc(&g.ctas, sizeof(FbCta) * all.size()) != cudaSuccess ||
        cudaMemcpy(g.ctas, all.data(), sizeof(FbCta) * all.size(), cudaMemcpyHostToDevice) !=
            cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    g.ok = true;
    f->ok = true;
  }
  return f->ok;
}

void mpc_flowb_objective_release(mpc_ctx* c) {
  mpc_flowb_state* f = c->flowb;
  if (!f) return;
  auto drop = [](auto** p, size_t* cap) {
    cudaFree(*p);
    *p = nullptr;
    *cap = 0;
  };
  drop(&f->oint, &f->oint_n);
  drop(&f->oio, &f->oio_n);
  drop(&f->oF, &f->oF_n);
  drop(&f->onorm, &f->onorm_n);
  drop(&f->ockp, &f->ockp_n);
  drop(&f->oseg, &f->oseg_n);
  drop(&f->olam, &f->olam_n);
  drop(&f->ofs, &f->ofs_n);
  drop(&f->ofp, &f->ofp_n);
  drop(&f->ofb, &f->ofb_n);
}

void mpc_flowb_free(mpc_ctx* c) {
  if (!c || !c->flowb) return;
  mpc_flowb_state* f = c->flowb;
  for (Group& g : f->grp) cudaFree(g.ctas);
  cudaFree(f->V);
  cudaFree(f->part);
  cudaFree(f->ctr);
  cudaFree(f->xst);
  cudaFree(f->kst);
  cudaFree(f->io);
  cudaFree(f->ints);
  cudaFree(f->pulse);
  cudaFree(f->t0);
  cudaFree(f->hist);
  mpc_flowb_objective_release(c);
  delete f;
  c->flowb = nullptr;
}

namespace {

// The column groups for nch chunks.
int pick_groups(const mpc_flowb_state* f, int nch) {
  int best = 0;
  double t = 1e300;
  for (int ng = 1; ng <= kMaxGroups; ++ng) {
    if (!f->grp[ng].ok || ng > nch) continue;
    const double x = product_us(f->grp[ng].cost, (nch + ng - 1) / ng);
    if (x < t) {
      t = x;
      best = ng;
    }
  }
  return best ? best : 1;
}

}  // namespace

namespace {

// One launch of nch chunks on ng column groups, its work space preset.
int launch(mpc_ctx* c, FbArgs& a, int ng, int nch, int mode, int slope_chunks = 0) {
  const int slots = kSlots[mode];
  mpc_flowb_state* f = c->flowb;
  const Group& grp = f->grp[ng];
  const size_t n = c->g.ntot;
  const size_t vn = (size_t)nch * slots * n * CP, pn = (size_t)nch * 2 * grp.gp * 2 * CP;
  int rc;
  if ((rc = grow(&f->V, &f->V_n, vn)) || (rc = grow(&f->part, &f->part_n, pn)) ||
      (rc = grow(&f->ctr, &f->ctr_n, (size_t)nch)) || (rc = grow(&f->xst, &f->xst_n, nch * n * CP)))
    return rc;
  CK(cudaMemsetAsync(f->V, 0xff, sizeof(double2) * vn, c->stream));
  CK(cudaMemsetAsync(f->part, 0xff, sizeof(double) * pn, c->stream));
  CK(cudaMemsetAsync(f->ctr, 0, sizeof(unsigned long long) * nch, c->stream));
  a.D = c->d_D;
  a.eps = c->d_eps;
  a.slots = slots;
  a.status = c->d_status;
  a.gauge = (c->gauge == 'l') ? 0 : 1;
  a.g = c->g;
  a.cta = grp.ctas;
  a.gp = grp.gp;
  a.mt = grp.mt;
  a.ng = ng;
  a.nch = nch;
  a.V = f->V;
  a.part = f->part;
  a.ctr = f->ctr;
  a.xst = f->xst;
  a.bc = mpc_barrier_cfg(c);
  void* args[] = {&a};
  ProfScope ps(c, MPC_KERNEL_BATCH_STAGE);
  CK(cudaLaunchCooperativeKernel(kKernels[mode], dim3(ng * grp.gp), dim3(FTHREADS), args,
                                 flowb_smem(mode, grp.mt, slope_chunks, grp.rows), c->stream));
  return MPC_OK;
}

// lambda_N of every pulse, projected as k_flow_seed does (one CTA per pulse).
__global__ void k_fb_seed(const int* cid, const double2* x, const double* eps, double2* lam,
                          int target, double thr, int ntot) {
  const int gc = blockIdx.x / CP, q = blockIdx.x % CP, id = cid[blockIdx.x];
  __shared__ double sh[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double2* xp = x + (long long)max(id, 0) * ntot;
  auto seed = [&](int i) {
    const bool on = id >= 0 && (target < 0 ? eps[i] >= thr : i == target);
    return on ? make_double2(2.0 * xp[i].x, 2.0 * xp[i].y) : make_double2(0.0, 0.0);
  };
  double d = 0.0;
  for (int i = threadIdx.x; i < ntot; i += blockDim.x) {
    const double2 v = xp[i], l = seed(i);
    d += fma(v.x, l.x, v.y * l.y);
  }
  for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
  if (lane == 0) sh[warp] = d;
  __syncthreads();
  d = 0.0;
  for (int k = 0; k < (int)(blockDim.x >> 5); ++k) d += sh[k];
  for (int i = threadIdx.x; i < ntot; i += blockDim.x) {
    double2 l = make_double2(0.0, 0.0);
    if (id >= 0) {
      const double2 v = xp[i], s = seed(i);
      l = make_double2(fma(-d, v.x, s.x), fma(-d, v.y, s.y));
    }
    lam[((long long)gc * ntot + i) * CP + q] = l;
  }
}

// dJ/dF_n per pulse from the CTAs' partials: a warp per step and chunk.
__global__ void k_fb_fbar(const double* fpart, const int* cid, int len, int nch, int gp,
                          double* fbar, int B) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= len * nch) return;
  const int n = w / nch, gc = w % nch, q = lane & 7;
  double t = 0.0;
  for (int k = lane >> 3; k < gp; k += 4) t += fpart[((long long)w * gp + k) * CP + q];
  t += __shfl_xor_sync(0xffffffffu, t, 8);
  t += __shfl_xor_sync(0xffffffffu, t, 16);
  const int id = cid[gc * CP + q];
  if (lane < CP && id >= 0) fbar[(long long)n * B + id] = t;
}

size_t obj_bytes(const mpc_ctx* c, int B, int steps, int ckpt) {
  const size_t nch = (B + CP - 1) / CP, vec = 16 * nch * (size_t)c->g.ntot * CP;
  const size_t nseg = (steps + ckpt - 1) / ckpt;
  return vec * (nseg + 13 * (size_t)ckpt + kAdjSlots + 6) + 32 * (size_t)steps * B +
         8 * nch * CP * (size_t)ckpt * c->num_sms;
}

}  // namespace

// The batched objective runs here: faster than the stage GEMM, one launch.
bool mpc_flowb_objective_wanted(mpc_ctx* c, int B) {
  if (!mpc_flowb_wanted(c, B)) return false;
  const int nch = (B + CP - 1) / CP;
  return nch <= kMaxChunks * pick_groups(c->flowb, nch);
}

size_t mpc_flowb_objective_bytes(const mpc_ctx* c, int B, int steps, int ckpt) {
  return obj_bytes(c, B, steps, ckpt);
}

// ckpt_every <= 0: the longest interval whose buffers fit in 85 % of the free
// device memory.
int mpc_flowb_auto_ckpt(mpc_ctx* c, int B, int steps, int* ckpt) {
  mpc_flowb_state* f = c->flowb;
  size_t free_b = 0, total_b = 0;
  CK(cudaMemGetInfo(&free_b, &total_b));
  const double own = 16.0 * (f->ockp_n + f->oseg_n + f->V_n + f->xst_n + f->olam_n);
  const double budget = 0.85 * ((double)free_b + own);
  int k = steps;
  while (k > 1 && (double)obj_bytes(c, B, steps, k) > budget) k = (k + 1) / 2;
  if ((double)obj_bytes(c, B, steps, k) > budget)
    return mpc_fail(MPC_ERR_NOMEM, "the batched objective needs %.3g GB, %.3g GB free",
                    obj_bytes(c, B, steps, k) / 1e9, free_b / 1e9);
  *ckpt = k;
  return MPC_OK;
}

namespace {

FbArgs obj_args(mpc_ctx* c) {
  mpc_flowb_state* f = c->flowb;
  FbArgs a{};
  a.cid = f->oint;
  a.csteps = f->oint + (size_t)f->onch * CP;
  a.nsteps = a.csteps + f->onch;
  a.in = f->oio;
  a.out = f->oio + (size_t)f->oB * c->g.ntot;
  a.Ftab = f->oF;
  a.ldf = f->oB;
  a.dt = f->odt;
  a.pop_index = -1;
  a.hist_ld = f->osteps;
  a.norm_hist = f->onorm;
  a.seg_v = f->oseg;
  a.cvec = (long long)f->onch * c->g.ntot * CP;
  return a;
}

// Steps [n0, n0 + len) of all pulses run: chunk and pulse step counts.
int obj_steps(mpc_ctx* c, int len) {
  mpc_flowb_state* f = c->flowb;
  std::vector<int> v((size_t)f->onch + f->oB, len);
  CK(cudaMemcpyAsync(f->oint + (size_t)f->onch * CP, v.data(), sizeof(int) * v.size(),
                     cudaMemcpyHostToDevice, c->stream));
  CK(cudaStreamSynchronize(c->stream));   // v is pageable and goes away
  return MPC_OK;
}

int obj_status(mpc_ctx* c, const char* where) {
  unsigned st = 0;
  CK(cudaMemcpyAsync(&st, c->d_status, sizeof st, cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  if (!st) return MPC_OK;
  CK(cudaMemsetAsync(c->d_status, 0, sizeof(unsigned), c->stream));
  return mpc_fail(MPC_ERR_DEVICE, "kernel status 0x%x during the %s", st, where);
}

}  // namespace

// Forward pass of the batched objective: fields F host [steps][B], start
// states ct0 host [B][n], final states into xN host [B][n].
int mpc_flowb_objective(mpc_ctx* c, int B, const double* F, double dt, int steps, int ckpt,
                        const double* ct0, double2* xN) {
  mpc_flowb_state* f = c->flowb;
  const size_t n = c->g.ntot;
  const int nch = (B + CP - 1) / CP, nseg = (steps + ckpt - 1) / ckpt;
  const size_t vec = (size_t)nch * n * CP;
  int rc;
  std::vector<int> cid((size_t)nch * CP, -1);
  for (int i = 0; i < B; ++i) cid[i] = i;
  f->oB = B;
  f->osteps = steps;
  f->ockpt = ckpt;
  f->onch = nch;
  f->ong = pick_groups(f, nch);
  f->odt = dt;
  f->okept = false;
  // a larger set does not lie beside the smaller one it replaces
  if (f->ockp_n < vec * nseg || f->oseg_n < vec * 13 * std::min(ckpt, steps))
    mpc_flowb_objective_release(c);
  if ((rc = grow(&f->oint, &f->oint_n, (size_t)nch * (CP + 1) + B)) ||
      (rc = grow(&f->oio, &f->oio_n, 2 * B * n)) ||
      (rc = grow(&f->oF, &f->oF_n, (size_t)steps * B)) ||
      (rc = grow(&f->onorm, &f->onorm_n, (size_t)steps * B)) ||
      (rc = grow(&f->ockp, &f->ockp_n, vec * nseg)) ||
      (rc = grow(&f->oseg, &f->oseg_n, vec * 13 * std::min(ckpt, steps))) ||
      (rc = grow(&f->olam, &f->olam_n, 2 * vec)) || (rc = grow(&f->ofs, &f->ofs_n, vec)) ||
      (rc = grow(&f->ofp, &f->ofp_n,
                 (size_t)std::min(ckpt, steps) * nch * f->grp[f->ong].gp * CP)) ||
      (rc = grow(&f->ofb, &f->ofb_n, (size_t)steps * B)))
    return rc;
  CK(cudaMemcpyAsync(f->oio, ct0, sizeof(double2) * B * n, cudaMemcpyHostToDevice, c->stream));
  CK(cudaMemcpyAsync(f->oF, F, sizeof(double) * (size_t)steps * B, cudaMemcpyHostToDevice,
                     c->stream));
  CK(cudaMemcpyAsync(f->oint, cid.data(), sizeof(int) * cid.size(), cudaMemcpyHostToDevice,
                     c->stream));
  if ((rc = obj_steps(c, steps))) return rc;
  FbArgs a = obj_args(c);
  a.ckpt = f->ockp;
  a.ckpt_every = ckpt;
  a.seg_from = (nseg - 1) * ckpt;
  if ((rc = launch(c, a, f->ong, nch, 0))) return rc;
  CK(cudaMemcpyAsync(xN, a.out, sizeof(double2) * B * n, cudaMemcpyDeviceToHost, c->stream));
  f->okept = true;
  return obj_status(c, "batched forward pass");
}

// Its reverse pass: dJ/dF into fb host [steps][B].
int mpc_flowb_objective_backward(mpc_ctx* c, int target, double* fb) {
  mpc_flowb_state* f = c->flowb;
  const size_t n = c->g.ntot;
  const int B = f->oB, nch = f->onch, steps = f->osteps, ckpt = f->ockpt;
  const int nseg = (steps + ckpt - 1) / ckpt;
  const size_t vec = (size_t)nch * n * CP;
  int rc;
  k_fb_seed<<<nch * CP, 256, 0, c->stream>>>(f->oint, f->oio + (size_t)B * n, c->d_eps, f->olam,
                                             target, c->yield_thr, (int)n);
  CK(cudaGetLastError());
  ++c->launches;
  int lens = -1;   // the step counts on the device
  for (int seg = nseg - 1; seg >= 0; --seg) {
    const int n0 = seg * ckpt, len = std::min(ckpt, steps - n0);
    if (!(f->okept && seg == nseg - 1)) {
      // recompute the segment's vectors, from the checkpoint and its norm
      if (lens != len && (rc = obj_steps(c, lens = len))) return rc;
      FbArgs a = obj_args(c);
      a.start = f->ockp + vec * seg;
      a.start_nrm = n0 > 0 ? f->onorm + (n0 - 1) : nullptr;
      a.Ftab = f->oF + (size_t)n0 * B;
      a.norm_hist = f->onorm + n0;   // the same norms again
      a.out = f->oio;                // (the start states are not needed any more)
      if ((rc = launch(c, a, f->ong, nch, 0))) return rc;
    }
    FbArgs a = obj_args(c);
    a.Ftab = f->oF + (size_t)n0 * B;
    a.norms = f->onorm + n0;
    a.len = len;
    a.lam = f->olam;
    a.xb = f->olam + vec;
    a.fs = f->ofs;
    a.fpart = f->ofp;
    if ((rc = launch(c, a, f->ong, nch, 2))) return rc;
    k_fb_fbar<<<(len * nch * 32 + 127) / 128, 128, 0, c->stream>>>(
        f->ofp, f->oint, len, nch, f->grp[f->ong].gp, f->ofb + (size_t)n0 * B, B);
    CK(cudaGetLastError());
    ++c->launches;
  }
  f->okept = f->okept && nseg == 1;   // the recomputes overwrote the last segment
  CK(cudaMemcpyAsync(fb, f->ofb, sizeof(double) * (size_t)steps * B, cudaMemcpyDeviceToHost,
                     c->stream));
  return obj_status(c, "batched adjoint pass");
}

// Whether B pulses run faster here than on the stage GEMM.  A switch that says
// how the GEMM is to run asks for the GEMM.
bool mpc_flowb_wanted(mpc_ctx* c, int B) {
  if (c->path == MPC_PATH_STREAMING || mpc_batch_pinned(c) || !mpc_flowb_setup(c)) return false;
  const mpc_flowb_state* f = c->flowb;
  const int nch = (B + CP - 1) / CP, ng = pick_groups(f, nch);
  return f->grp[ng].ok && product_us(f->grp[ng].cost, (nch + ng - 1) / ng) <= gemm_us(c->g, B);
}

bool mpc_flowb_fixed_wanted(mpc_ctx* c, int B) {
  return !c->no_persist && !c->force_persist && !c->force_tma && mpc_flowb_wanted(c, B);
}

int mpc_flowb_states(mpc_ctx* c, int B, double2** in) {
  mpc_flowb_state* f = c->flowb;
  int rc;
  if ((rc = grow(&f->io, &f->io_n, 2 * (size_t)B * c->g.ntot))) return rc;
  *in = f->io;
  return MPC_OK;
}

int mpc_flowb_tail(mpc_ctx* c, int B, const std::vector<int>& ids, const mpc_pulse* pulses,
                   const double* t, const int* left, const FixedStep& fx, double2* out) {
  mpc_flowb_state* f = c->flowb;
  int rc;
  // pulses by length, so that a chunk's end together
  std::vector<int> order(ids);
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return left[x] > left[y]; });
  const int nch_all = (int)(order.size() + CP - 1) / CP;
  std::vector<int> ints((size_t)nch_all * (CP + 1) + B, -1);
  int* cid = ints.data();
  int* cst = cid + (size_t)nch_all * CP;
  int* ns = cst + nch_all;
  std::copy(order.begin(), order.end(), cid);
  for (int k = 0; k < nch_all; ++k) cst[k] = left[order[(size_t)k * CP]];
  std::copy(left, left + B, ns);
  if ((rc = grow(&f->ints, &f->ints_n, ints.size())) ||
      (rc = grow(&f->pulse, &f->pulse_n, (size_t)B)) || (rc = grow(&f->t0, &f->t0_n, (size_t)B)))
    return rc;
  CK(cudaMemcpyAsync(f->ints, ints.data(), sizeof(int) * ints.size(), cudaMemcpyHostToDevice,
                     c->stream));
  CK(cudaMemcpyAsync(f->pulse, pulses, sizeof(mpc_pulse) * B, cudaMemcpyHostToDevice, c->stream));
  CK(cudaMemcpyAsync(f->t0, t, sizeof(double) * B, cudaMemcpyHostToDevice, c->stream));
  FbArgs a{};
  a.in = f->io;
  a.out = out;
  a.pulse = f->pulse;
  a.t0 = f->t0;
  a.nsteps = f->ints + (ns - cid);
  a.dt = fx.dt;
  a.pop_index = fx.pop_index;
  a.hist_ld = fx.hist_ld;
  a.pop_hist = fx.pop_hist;
  a.norm_hist = fx.norm_hist;
  // launches of at most kMaxChunks chunks per column group
  for (int k0 = 0; k0 < nch_all;) {
    const int ng = pick_groups(f, nch_all - k0);
    const int nch = std::min(nch_all - k0, kMaxChunks * ng);
    a.cid = f->ints + (size_t)k0 * CP;
    a.csteps = f->ints + (cst - cid) + k0;
    if ((rc = launch(c, a, ng, nch, 0))) return rc;
    k0 += nch;
  }
  CK(cudaStreamSynchronize(c->stream));   // the host arrays go away
  return MPC_OK;
}

// The fixed-step propagation of B pulses (mpc_batch_advance): ct host [B][n]
// in and out; pop_out / norm_out host, rows of `ld` and ld - 1 (or null).
int mpc_flowb_advance(mpc_ctx* c, int B, const mpc_pulse* pulses, const double* t0, double dt,
                      const int* steps, int pop_index, double* ct, double* pop_out,
                      double* norm_out, int max_steps) {
  mpc_flowb_state* f = c->flowb;
  const int n = c->g.ntot;
  int rc;
  const long long ld = (long long)max_steps + 1;
  const size_t hist = (size_t)B * ld;
  double2* in = nullptr;
  if ((rc = mpc_flowb_states(c, B, &in)) ||
      (rc = grow(&f->hist, &f->hist_n, (pop_out ? hist : 0) + (norm_out ? hist : 0) + 1)))
    return rc;
  double2* out = in + (size_t)B * n;
  CK(cudaMemcpyAsync(in, ct, sizeof(double2) * (size_t)B * n, cudaMemcpyHostToDevice, c->stream));
  FixedStep fx{};
  fx.dt = dt;
  fx.pop_index = pop_index;
  fx.hist_ld = ld;
  fx.pop_hist = pop_out ? f->hist : nullptr;
  fx.norm_hist = norm_out ? f->hist + (pop_out ? hist : 0) : nullptr;
  std::vector<int> ids(B);
  std::iota(ids.begin(), ids.end(), 0);
  if ((rc = mpc_flowb_tail(c, B, ids, pulses, t0, steps, fx, out))) return rc;
  std::vector<double> h(pop_out || norm_out ? (pop_out ? hist : 0) + (norm_out ? hist : 0) : 0);
  if (!h.empty())
    CK(cudaMemcpyAsync(h.data(), f->hist, sizeof(double) * h.size(), cudaMemcpyDeviceToHost,
                       c->stream));
  unsigned st = 0;
  CK(cudaMemcpyAsync(&st, c->d_status, sizeof st, cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  if (st) {
    CK(cudaMemsetAsync(c->d_status, 0, sizeof(unsigned), c->stream));
    return mpc_fail(MPC_ERR_DEVICE, "kernel status 0x%x in the batched propagation", st);
  }
  for (int b = 0; b < B; ++b) {
    if (pop_out) {
      const double* x = ct + 2 * ((size_t)b * n + pop_index);
      pop_out[b * ld] = x[0] * x[0] + x[1] * x[1];
      for (int k = 1; k <= steps[b]; ++k) pop_out[b * ld + k] = h[b * ld + k];
    }
    const double* hn = h.data() + (pop_out ? hist : 0);
    for (int k = 0; norm_out && k < steps[b]; ++k) norm_out[b * (ld - 1) + k] = hn[b * ld + k];
  }
  CK(cudaMemcpyAsync(ct, out, sizeof(double2) * (size_t)B * n, cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  return MPC_OK;
}

// The adaptive propagation of B pulses (mpc_batch_propagate); ct host [B][n] in
// and out, results by pulse (host).
int mpc_flowb_propagate(mpc_ctx* c, int B, const mpc_pulse* pulses, const double* t0,
                        const double* t_end, double h0, double dt_max, double rtol, double atol,
                        int max_attempts, double* ct, int* accepted, int* rejected,
                        double* t_final) {
  mpc_flowb_state* f = c->flowb;
  const size_t n = c->g.ntot;
  int rc;
  // pulses by the time they have to run: a chunk goes on until its last is done
  std::vector<int> order(B);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(),
                   [&](int x, int y) { return t_end[x] - t0[x] > t_end[y] - t0[y]; });
  const int nch_all = (B + CP - 1) / CP;
  std::vector<int> ints((size_t)nch_all * (CP + 1) + 3 * (size_t)B, 0);
  int* cid = ints.data();
  std::fill(cid, cid + (size_t)nch_all * CP, -1);
  std::copy(order.begin(), order.end(), cid);
  const size_t res = (size_t)nch_all * (CP + 1);   // nacc, nrej, gave_up
  if ((rc = grow(&f->ints, &f->ints_n, ints.size())) || (rc = grow(&f->pulse, &f->pulse_n, (size_t)B)) ||
      (rc = grow(&f->t0, &f->t0_n, 3 * (size_t)B)) || (rc = grow(&f->io, &f->io_n, 2 * B * n)))
    return rc;
  CK(cudaMemcpyAsync(f->io, ct, sizeof(double2) * B * n, cudaMemcpyHostToDevice, c->stream));
  CK(cudaMemcpyAsync(f->ints, ints.data(), sizeof(int) * ints.size(), cudaMemcpyHostToDevice,
                     c->stream));
  CK(cudaMemcpyAsync(f->pulse, pulses, sizeof(mpc_pulse) * B, cudaMemcpyHostToDevice, c->stream));
  CK(cudaMemcpyAsync(f->t0, t0, sizeof(double) * B, cudaMemcpyHostToDevice, c->stream));
  CK(cudaMemcpyAsync(f->t0 + B, t_end, sizeof(double) * B, cudaMemcpyHostToDevice, c->stream));
  FbArgs a{};
  a.in = f->io;
  a.out = f->io + B * n;
  a.pulse = f->pulse;
  a.t0 = f->t0;
  a.t_end = f->t0 + B;
  a.h0 = h0;
  a.dt_max = dt_max;
  a.rtol = rtol;
  a.atol = atol;
  a.max_attempts = max_attempts > 0 ? max_attempts : 1000000000;
  a.nacc = f->ints + res;
  a.nrej = a.nacc + B;
  a.gave_up = a.nrej + B;
  a.tf = f->t0 + 2 * (size_t)B;
  for (int k0 = 0; k0 < nch_all;) {
    const int ng = pick_groups(f, nch_all - k0);
    const int nch = std::min(nch_all - k0, kMaxAdapt * ng), per = (nch + ng - 1) / ng;
    const size_t vec = (size_t)nch * n * CP;
    const Group& grp = f->grp[ng];
    const bool shm = flowb_smem(1, grp.mt, per, grp.rows) + 1024 <= f->optin;
    if ((rc = grow(&f->kst, &f->kst_n, vec * kNumStages))) return rc;
    a.cid = f->ints + (size_t)k0 * CP;
    a.csteps = f->ints + (size_t)nch_all * CP;   // unused: zeros
    a.xnew = f->kst;
    a.kst = shm ? nullptr : f->kst + vec;
    a.cvec = (long long)vec;
    if ((rc = launch(c, a, ng, nch, 1, shm ? per : 0))) return rc;
    k0 += nch;
  }
  std::vector<double> tf(B);
  CK(cudaMemcpyAsync(ints.data() + res, f->ints + res, sizeof(int) * 3 * (size_t)B,
                     cudaMemcpyDeviceToHost, c->stream));
  CK(cudaMemcpyAsync(tf.data(), a.tf, sizeof(double) * B, cudaMemcpyDeviceToHost, c->stream));
  if ((rc = obj_status(c, "batched propagation"))) return rc;
  CK(cudaMemcpyAsync(ct, a.out, sizeof(double2) * B * n, cudaMemcpyDeviceToHost, c->stream));
  CK(cudaStreamSynchronize(c->stream));
  int gave_up = 0;
  for (int b = 0; b < B; ++b) {
    if (accepted) accepted[b] = ints[res + b];
    if (rejected) rejected[b] = ints[res + B + b];
    if (t_final) t_final[b] = tf[b];
    gave_up += ints[res + 2 * (size_t)B + b];
  }
  if (gave_up)
    return mpc_fail(MPC_ERR_DEVICE, "%d pulse(s) stopped after max_attempts step attempts",
                    gave_up);
  return MPC_OK;
}
