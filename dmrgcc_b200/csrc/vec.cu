// FP64 vector kernels (see vec.cuh).  These are HBM-bound: each reads its
// operands once with coalesced grid-stride loops and reduces deterministically.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

#include "vec.cuh"

namespace dmrg {
namespace {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Sum over the block; result valid in thread 0.
__device__ double block_sum(double v) {
    __shared__ double s[kVecThreads / 32];
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) s[w] = v;
    __syncthreads();
    double r = 0.0;
    if (w == 0) {
        r = lane < kVecThreads / 32 ? s[lane] : 0.0;
        r = warp_sum(r);
    }
    __syncthreads();
    return r;
}

// Called by every thread of every block after thread 0 stored partial[blockIdx.x].
// The last block to arrive reduces the partials in index order into *out.
__device__ void last_block_finalize(double* partial, unsigned* ticket, double* out, bool take_sqrt) {
    __shared__ bool is_last;
    __threadfence();
    if (threadIdx.x == 0) is_last = (atomicAdd(ticket, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    double v = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) v += ((volatile double*)partial)[b];
    v = block_sum(v);
    if (threadIdx.x == 0) {
        *out = take_sqrt ? sqrt(v) : v;
        *ticket = 0u;
    }
}

__global__ void __launch_bounds__(kVecThreads) dot_kernel(const double* __restrict__ x, const double* __restrict__ y,
                                                          int64_t n, double* partial, unsigned* ticket, double* out,
                                                          int take_sqrt) {
    double acc = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        acc += x[i] * y[i];
    acc = block_sum(acc);
    if (threadIdx.x == 0) partial[blockIdx.x] = acc;
    last_block_finalize(partial, ticket, out, take_sqrt != 0);
}

// w = beta_w * w + sign * sum_k c[k] V_k
__global__ void __launch_bounds__(kVecThreads) combine_kernel(const double* __restrict__ V, int64_t ldv, int m,
                                                              const double* __restrict__ c, double sign,
                                                              double* __restrict__ w, double beta_w, int64_t n) {
    __shared__ double cs[kMaxVec];
    for (int k = threadIdx.x; k < m; k += blockDim.x) cs[k] = sign * c[k];
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double acc = beta_w == 0.0 ? 0.0 : beta_w * w[i];
        for (int k = 0; k < m; ++k) acc += cs[k] * V[(int64_t)k * ldv + i];
        w[i] = acc;
    }
}

__global__ void __launch_bounds__(kVecThreads) lanczos_shift_kernel(const double* __restrict__ beta,
                                                                    const double* __restrict__ v_cur,
                                                                    double* __restrict__ h,
                                                                    double* __restrict__ v_next, int64_t n) {
    const double b = *beta;
    const double inv = 1.0 / b;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        v_next[i] = h[i] * inv;
        h[i] = -b * v_cur[i];
    }
}

__global__ void __launch_bounds__(kVecThreads) scale_inv_kernel(double* __restrict__ x, const double* __restrict__ s,
                                                                int64_t n) {
    const double inv = 1.0 / *s;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        x[i] *= inv;
}

// ---------------------------------------------------------------------------
// One Lanczos iteration's vector work in one kernel (see vec_lanczos_step).
//
// The work is small (n doubles times a few passes over at most i + 1 vectors) and
// chains five reductions, each needed by the whole next pass, so it is bound by
// latency: as eight launches it took 45 us of an iteration at n = 2,037 and 60 us
// at n = 140,000.  The CTAs keep one slice each of all vectors and meet at a
// barrier per reduction instead: the hardware barrier of a cluster of 8 where the
// slices are short, else the grid barrier of a cooperative launch of one CTA per SM.
// The basis does not depend on the iteration's matvec, so its slices (as many as
// fit) are copied to shared memory while the first two reductions run.
// Reductions are deterministic (fixed slices, partials summed in a fixed order).
constexpr int kStepThreads = 512, kStepWarps = kStepThreads / 32;
constexpr int kStepCluster = 8;
// Up to here one cluster: its barrier takes a fraction of the grid's, but eight SMs
// read the basis.  Measured, us per iteration of a 20-iteration Lanczos run, cluster /
// grid: n = 2,037 37 / 43, 7,760 42 / 45, 21,425 78 / 58 (before: 64, 77, 106).
constexpr int64_t kClusterMax = 16384;
constexpr int64_t kStepShared = 24 * 1024;  // doubles of shared memory: w's slice (if it fits), then the basis

struct StepArgs {
    double *x, *h, *V;
    int64_t n;
    int niter;
    double *alpha, *beta;  // of every iteration
    double* part;          // (2 niter + 3) * grid partials
    int* state;
    int slice_in_smem, basis_in_smem;  // w's slice; vectors of the basis
    cudaGraphConditionalHandle loop;   // the captured loop's, or 0
};

__device__ __forceinline__ double warp_sum_all(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ void cp_async8(double* smem, const double* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}

template <bool CLUSTER>
__global__ void __launch_bounds__(kStepThreads) lanczos_step_kernel(const StepArgs a) {
    namespace cg = cooperative_groups;
    extern __shared__ double sm[];
    const int it = a.state[kIterSlot];
    if (it >= a.niter) return;  // the same for every CTA
    const int G = gridDim.x, rank = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto meet = [&]() {
        if (CLUSTER) cg::this_cluster().sync();
        else cg::this_grid().sync();
    };
    const int64_t chunk = (a.n + G - 1) / G, base = min((int64_t)rank * chunk, a.n);
    const int len = (int)(min(base + chunk, a.n) - base);
    // shared: warp partials, coefficients, CTA partials (cluster), w's slice, the basis
    double* red = sm;                         // kStepWarps * niter
    double* cs = red + kStepWarps * a.niter;  // niter
    double* mine = cs + a.niter;              // 2 niter + 3
    double* wsm = mine + 2 * a.niter + 3;
    double* basis = wsm + (a.slice_in_smem ? chunk : 0);
    double* x = a.x + base;
    double* h = a.h + base;
    const double* V = a.V + base;
    const int m = it + 1, kept = it + 1 < a.niter ? min(m, a.basis_in_smem) : 0;
    for (int k = 0; k < kept; ++k)
        for (int j = tid; j < len; j += kStepThreads) cp_async8(basis + (int64_t)k * chunk + j, V + (int64_t)k * a.n + j);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    // Partial `slot` of this CTA, and the warp's sum of all CTAs' (in every lane).
    auto put = [&](int slot, double v) {
        if (CLUSTER) mine[slot] = v;
        else a.part[(int64_t)slot * G + rank] = v;
    };
    auto get = [&](int slot) {
        double v = 0.0;
        if (CLUSTER) {
            if (lane < kStepCluster) v = cg::this_cluster().map_shared_rank(mine, lane)[slot];
        } else {
            for (int r = lane; r < G; r += 32) v += __ldcg(a.part + (int64_t)slot * G + r);
        }
        return warp_sum_all(v);
    };
    // Sum of the threads' v over all CTAs, the same in every thread.
    auto total = [&](double v, int slot) {
        v = warp_sum_all(v);
        if (lane == 0) red[warp] = v;
        __syncthreads();
        if (warp == 0) {
            v = warp_sum_all(lane < kStepWarps ? red[lane] : 0.0);
            if (lane == 0) put(slot, v);
        }
        meet();
        return get(slot);
    };
    double acc = 0.0;
#pragma unroll 4
    for (int j = tid; j < len; j += kStepThreads) acc += x[j] * h[j];
    const double al = total(acc, 0);
    acc = 0.0;
#pragma unroll 4
    for (int j = tid; j < len; j += kStepThreads) {
        const double v = h[j] - al * x[j];
        h[j] = v;
        acc += v * v;
    }
    const double be = sqrt(total(acc, 1));
    const bool last = it + 1 >= a.niter;  // the last vector slot is V[niter - 1]
    if (rank == 0 && tid == 0) {
        a.alpha[it] = al;
        a.beta[it] = be;
        // the next iteration (every CTA has read the counter); the captured loop goes on
        // while no converged dimension is known
        a.state[kIterSlot] = it + 1;
        if (a.loop) cudaGraphSetConditional(a.loop, !last && a.state[0] == 0 ? 1u : 0u);
    }
    if (!last) {
        // w = h / beta, h = -beta x
        double* next = a.V + (int64_t)m * a.n + base;
        double* w = a.slice_in_smem ? wsm : next;
        const double inv = 1.0 / be;
#pragma unroll 4
        for (int j = tid; j < len; j += kStepThreads) {
            w[j] = h[j] * inv;
            h[j] = -be * x[j];
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        // classical Gram-Schmidt against V_0 .. V_it, twice.  The dot products: the slice in
        // `segs` segments of at least 256 elements, a warp per segment and vector.
        const int segs = len >= 4096 ? 16 : len >= 2048 ? 8 : len >= 1024 ? 4 : len >= 512 ? 2 : 1;
        const int per = (len + segs - 1) / segs, seg = warp % segs, j0 = min(seg * per, len), j1 = min(j0 + per, len);
        for (int pass = 0; pass < 2; ++pass) {
            __syncthreads();  // w and the basis are complete
            const int slot = 3 + pass * a.niter;
            for (int k = warp / segs; k < m; k += kStepWarps / segs) {
                double s = 0.0;
                if (k < kept) {
                    const double* vk = basis + (int64_t)k * chunk;
#pragma unroll 4
                    for (int j = j0 + lane; j < j1; j += 32) s += vk[j] * w[j];
                } else {
                    const double* vk = V + (int64_t)k * a.n;
#pragma unroll 8
                    for (int j = j0 + lane; j < j1; j += 32) s += vk[j] * w[j];
                }
                s = warp_sum_all(s);
                if (lane == 0) red[k * segs + seg] = s;
            }
            __syncthreads();
            for (int k = tid; k < m; k += kStepThreads) {
                double s = 0.0;
                for (int q = 0; q < segs; ++q) s += red[k * segs + q];
                put(slot + k, s);
            }
            meet();
            for (int k = warp; k < m; k += kStepWarps) {
                const double s = get(slot + k);
                if (lane == 0) cs[k] = s;
            }
            __syncthreads();
            for (int j = tid; j < len; j += kStepThreads) {
                double v = w[j];
#pragma unroll 4
                for (int k = 0; k < kept; ++k) v -= cs[k] * basis[(int64_t)k * chunk + j];
#pragma unroll 8
                for (int k = kept; k < m; ++k) v -= cs[k] * V[(int64_t)k * a.n + j];
                w[j] = v;
            }
        }
        acc = 0.0;
        for (int j = tid; j < len; j += kStepThreads) acc += w[j] * w[j];  // its own elements
        __syncthreads();  // red is free
        const double scale = 1.0 / sqrt(total(acc, 2));
        for (int j = tid; j < len; j += kStepThreads) {
            const double v = w[j] * scale;
            next[j] = v;
            x[j] = v;
        }
    }
    if (CLUSTER) meet();  // no CTA leaves while another may read its partials
}

}  // namespace

int ReduceScratch::alloc(int blocks, int max_vectors) {
    max_blocks = blocks;
    DMRG_TRY(partial.alloc((size_t)blocks * (max_vectors > 0 ? max_vectors : 1) * sizeof(double)));
    if (!ticket.ptr) {
        DMRG_TRY(ticket.alloc(kTickets * sizeof(unsigned)));
        DMRG_TRY(ticket.zero());
    }
    return DMRG_OK;
}

int vec_combine(const double* V, int64_t ldv, int m, const double* c, double sign, double* w, double beta_w,
                int64_t n, int blocks, cudaStream_t st) {
    if (m > kMaxVec) return set_error(DMRG_E_ARG, "combine of %d > %d vectors", m, kMaxVec);
    DMRG_LAUNCH combine_kernel<<<blocks, kVecThreads, 0, st>>>(V, ldv, m, c, sign, w, beta_w, n);
    DMRG_CUDA_TRY(cudaGetLastError());
    return DMRG_OK;
}

int vec_lanczos_shift(const double* beta, const double* v_cur, double* h, double* v_next, int64_t n, int blocks,
                      cudaStream_t st) {
    DMRG_LAUNCH lanczos_shift_kernel<<<blocks, kVecThreads, 0, st>>>(beta, v_cur, h, v_next, n);
    DMRG_CUDA_TRY(cudaGetLastError());
    return DMRG_OK;
}

int vec_normalize(double* x, int64_t n, double* out, ReduceScratch& rs, int blocks, cudaStream_t st) {
    blocks = blocks < rs.max_blocks ? blocks : rs.max_blocks;
    DMRG_LAUNCH dot_kernel<<<blocks, kVecThreads, 0, st>>>(x, x, n, rs.partial.as<double>(), rs.ticket.as<unsigned>() + 2, out,
                                               1);
    DMRG_LAUNCH scale_inv_kernel<<<blocks, kVecThreads, 0, st>>>(x, out, n);
    DMRG_CUDA_TRY(cudaGetLastError());
    return DMRG_OK;
}

int lanczos_step_grid(int64_t n, int num_sms) {
    if (n <= kClusterMax) return kStepCluster;
    return (int)std::min<int64_t>(num_sms, (n + 1023) / 1024);
}

int lanczos_step_prepare() {
    static_assert(kStepShared * sizeof(double) <= 227 * 1024 && (kStepWarps + 3) * kMaxVec + 3 <= kStepShared,
                  "shared memory of a Lanczos step");
    static std::atomic<bool> done[64] = {};
    int dev = 0;
    DMRG_CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && done[dev].load(std::memory_order_acquire)) return DMRG_OK;
    for (auto kernel : {lanczos_step_kernel<true>, lanczos_step_kernel<false>})
        DMRG_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)(kStepShared * sizeof(double))));
    if (dev >= 0 && dev < 64) done[dev].store(true, std::memory_order_release);
    return DMRG_OK;
}

int vec_lanczos_step(double* x, double* h, double* V, int64_t n, int niter, double* alpha, double* beta, double* part,
                     int* state, cudaGraphConditionalHandle loop, int num_sms, cudaStream_t st) {
    if (niter > kMaxVec) return set_error(DMRG_E_ARG, "Lanczos dimension %d > %d", niter, kMaxVec);
    const int grid = lanczos_step_grid(n, num_sms);
    const int64_t slice = (n + grid - 1) / grid, tables = (kStepWarps + 3) * (int64_t)niter + 3;
    StepArgs a{x, h, V, n, niter, alpha, beta, part, state, 0, 0, loop};
    int64_t room = kStepShared - tables;
    if (slice <= room) {
        a.slice_in_smem = 1;
        room -= slice;
    }
    a.basis_in_smem = (int)std::min<int64_t>(room / std::max<int64_t>(slice, 1), niter);
    const bool cluster = n <= kClusterMax;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kStepThreads);
    cfg.dynamicSmemBytes = (size_t)(tables + (a.slice_in_smem + a.basis_in_smem) * slice) * sizeof(double);
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cluster) {
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kStepCluster;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    } else {
        attr.id = cudaLaunchAttributeCooperative;
        attr.val.cooperative = 1;
    }
    auto kernel = cluster ? lanczos_step_kernel<true> : lanczos_step_kernel<false>;
    count_launch();
    DMRG_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, a));
    return DMRG_OK;
}

}  // namespace dmrg
