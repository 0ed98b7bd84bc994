// FP64 vector kernels for the Lanczos recurrence and reorthogonalisation.
// All reductions are deterministic: fixed per-block slices, partials reduced
// in index order by the last block to finish (atomic ticket).
#pragma once

#include "common.cuh"

namespace dmrg {

constexpr int kVecThreads = 256;

// Scratch shared by the reductions of one context/solver.
struct ReduceScratch {
    DeviceBuffer partial;  // doubles, >= kMaxBlocks * kMaxVec
    DeviceBuffer ticket;   // unsigned counters
    int max_blocks = 0;
    int alloc(int blocks, int max_vectors);
};

// w = beta_w * w + sign * sum_k c[k] V_k   (c on the device, m <= kMaxVec)
int vec_combine(const double* V, int64_t ldv, int m, const double* c, double sign, double* w, double beta_w,
                int64_t n, int blocks, cudaStream_t st);
// Lanczos step: v_next = h / beta ; h = -beta * v_cur   (beta on the device)
int vec_lanczos_shift(const double* beta, const double* v_cur, double* h, double* v_next, int64_t n, int blocks,
                      cudaStream_t st);
// x /= ||x|| (two kernels: norm then scale); norm written to out[0]
int vec_normalize(double* x, int64_t n, double* out, ReduceScratch& rs, int blocks, cudaStream_t st);

constexpr int kMaxVec = 512;
constexpr int kTickets = 4;  // of a ReduceScratch
// ---- one Lanczos iteration ---------------------------------------------------
// The iteration i is read from state[kIterSlot] (a call with i >= niter does
// nothing), so one captured launch serves every iteration.  V: niter vectors of n,
// x = V_i the matvec's input, h += H x already:
//   alpha[i] = <x|h>;  h -= alpha[i] x;  beta[i] = ||h||;  unless i + 1 == niter:
//   V_{i+1} = h / beta[i], h = -beta[i] x;  V_{i+1} orthogonalised against V_0..V_i
//   by classical Gram-Schmidt twice, normalised;  x = V_{i+1};  and i += 1.
// `loop` (0: none): the captured loop's condition, left true while state[0] == 0 (no
// converged dimension) and iterations are left.
constexpr int kIterSlot = 4;
int lanczos_step_grid(int64_t n, int num_sms);  // CTAs of a step
// The kernel's shared-memory allowance on this device; once, ahead of any capture.
int lanczos_step_prepare();
// part: (2 niter + 3) * lanczos_step_grid(n, num_sms) doubles of scratch.
int vec_lanczos_step(double* x, double* h, double* V, int64_t n, int niter, double* alpha, double* beta, double* part,
                     int* state, cudaGraphConditionalHandle loop, int num_sms, cudaStream_t st);

}  // namespace dmrg
