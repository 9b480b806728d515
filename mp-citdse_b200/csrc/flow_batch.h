// flow_batch.h -- the persistent batched propagation for systems whose
// coupling fits on chip (flow_batch.cu).
#pragma once
#include <cstddef>
#include <vector>

#include "batch_types.h"
#include "ctx.h"

bool mpc_flowb_setup(mpc_ctx* c);   // usable for this system
bool mpc_flowb_wanted(mpc_ctx* c, int B);   // and the faster path for B pulses
bool mpc_flowb_fixed_wanted(mpc_ctx* c, int B);   // idem, for fixed steps
void mpc_flowb_free(mpc_ctx* c);
int mpc_flowb_advance(mpc_ctx* c, int B, const mpc_pulse* pulses, const double* t0, double dt,
                      const int* steps, int pop_index, double* ct, double* pop_out,
                      double* norm_out, int max_steps);

// The batched objective on the same kernels (see flow_batch.cu).
bool mpc_flowb_objective_wanted(mpc_ctx* c, int B);
size_t mpc_flowb_objective_bytes(const mpc_ctx* c, int B, int steps, int ckpt);
int mpc_flowb_auto_ckpt(mpc_ctx* c, int B, int steps, int* ckpt);
int mpc_flowb_objective(mpc_ctx* c, int B, const double* F, double dt, int steps, int ckpt,
                        const double* ct0, double2* xN);
int mpc_flowb_objective_backward(mpc_ctx* c, int target, double* fb);
void mpc_flowb_objective_release(mpc_ctx* c);   // its buffers (a forward pass kept is lost)

int mpc_flowb_propagate(mpc_ctx* c, int B, const mpc_pulse* pulses, const double* t0,
                        const double* t_end, double h0, double dt_max, double rtol, double atol,
                        int max_attempts, double* ct, int* accepted, int* rejected,
                        double* t_final);

// The rest of a fixed-step batch that began on the stage GEMM: start states by
// pulse in the buffer mpc_flowb_states gives ([B][n], device), pulses `ids` with
// `left` steps from times t (host, by pulse); final states to out [B][n]
// (device), histories through fx's pointers.
int mpc_flowb_states(mpc_ctx* c, int B, double2** in);
int mpc_flowb_tail(mpc_ctx* c, int B, const std::vector<int>& ids, const mpc_pulse* pulses,
                   const double* t, const int* left, const mpc::FixedStep& fx, double2* out);
