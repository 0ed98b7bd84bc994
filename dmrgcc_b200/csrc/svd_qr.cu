// Batched Householder QR for the Jacobi SVD (see svd.cuh): panels of 16 columns,
// one launch per panel for all sectors.
//
// What bounds it: the chain of panels, each a chain of 16 column steps in one CTA.
// A launch therefore factors panel s in the CTA that has just updated it while the
// other CTAs update the rest, and a column lives in the registers of one warp, so
// that a column step has one barrier.  16 columns is the widest panel whose 1024
// rows fit the registers of one CTA.  Both factorisations at 17 sectors to
// 611 x 510 and 837 x 360: 64 launches, 1.68 ms (37 us while panels have more than
// 512 rows, 25 us and less below); to 33 columns: 6 launches, 80 us.  Forming Q and
// applying it: 136 and 239 us, bound by the DMMA rate of the SMs that hold the
// largest sectors' tiles.
#include <algorithm>

#include "svd.cuh"

namespace dmrg {
namespace {

constexpr int kNb = kQrPanel;        // columns of a panel, and of a tile that it is applied to
constexpr int kStepWarps = 8;        // qr_step_kernel: two panel columns per warp
constexpr int kApplyWarps = 16;      // qr_apply_kernel
constexpr int kMaxReg = 32;          // rows a lane holds in registers, at most (1024-row panels)
// Below this squared norm (columns under 1e-140 of a matrix whose largest entry is
// at least 1/2) the part of a column under the diagonal counts as zero: its square
// sum is near underflow and would give a reflector that is not orthogonal.
constexpr double kTiny2 = 1e-280;

struct QrSmem {
    union {
        double red[kApplyWarps][kNb * kNb];  // the warps' parts of V^T C
        double v[2][32 * kMaxReg];           // the current reflector, double-buffered
    };
    double t[kNb * kNb];                 // the panel's T
    double z[kNb * kNb], tz[kNb * kNb];  // V^T C and -T^(T) V^T C
    double s[kNb * kNb];                 // v_i . v_j (i < j) of the panel being factored
    double tau[kNb];
};

__device__ __forceinline__ void dmma_8x8x4(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// C <- (I - V T V^T) C, or (I - V T^T V^T) C with TRANSPOSED, for one tile of nc
// <= 16 columns.  V (m x nv, ld ldv) has its unit diagonal and the zeros above it
// stored; operands are read as DMMA fragments straight from global memory (column
// major: 32- and 64-byte pieces, L2 hits), the two products splitting the rows
// over the warps.  With `rt`, rows 0..15 of the result (finished rows of the
// factor) go to rt transposed (entry (row, c) at rt[c + row * ldr]) instead of C.
template <bool TRANSPOSED, int WARPS>
__device__ void apply_panel(const double* V, int ldv, int m, int nv, const double* __restrict__ T, double* C, int ldc,
                            int nc, double* rt, int ldr, QrSmem& S) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, fr = lane >> 2, fc = lane & 3;
    if (threadIdx.x < kNb * kNb) S.t[threadIdx.x] = T[threadIdx.x];
    double acc[2][2][2] = {};
    for (int r0 = warp * 32; r0 < m; r0 += 32 * WARPS) {
#pragma unroll
        for (int kk = 0; kk < 32; kk += 4) {
            const int r = r0 + kk + fc;
            double a[2], b[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                a[i] = r < m && i * 8 + fr < nv ? V[r + (int64_t)(i * 8 + fr) * ldv] : 0.0;
                b[i] = r < m && i * 8 + fr < nc ? C[r + (int64_t)(i * 8 + fr) * ldc] : 0.0;
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int n = 0; n < 2; ++n) dmma_8x8x4(acc[i][n][0], acc[i][n][1], a[i], b[n]);
        }
    }
    const int parts = min(WARPS, (m + 31) / 32);
    if (warp < parts) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int n = 0; n < 2; ++n)
                *reinterpret_cast<double2*>(&S.red[warp][(i * 8 + fr) * kNb + n * 8 + 2 * fc]) =
                    make_double2(acc[i][n][0], acc[i][n][1]);
    }
    __syncthreads();
    if (threadIdx.x < kNb * kNb) {
        double z = 0.0;
        for (int w = 0; w < parts; ++w) z += S.red[w][threadIdx.x];
        S.z[threadIdx.x] = z;
    }
    __syncthreads();
    if (threadIdx.x < kNb * kNb) {
        const int i = threadIdx.x / kNb, n = threadIdx.x % kNb;
        double y = 0.0;
#pragma unroll
        for (int l = 0; l < kNb; ++l) y += (TRANSPOSED ? S.t[l * kNb + i] : S.t[i * kNb + l]) * S.z[l * kNb + n];
        S.tz[threadIdx.x] = -y;
    }
    __syncthreads();
    double b[4][2];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int n = 0; n < 2; ++n) b[k][n] = S.tz[(4 * k + fc) * kNb + n * 8 + fr];
#pragma unroll 4
    for (int r0 = warp * 8; r0 < m; r0 += 8 * WARPS) {
        const int r = r0 + fr;
        double a[4], c[2][2];
#pragma unroll
        for (int k = 0; k < 4; ++k) a[k] = r < m && 4 * k + fc < nv ? V[r + (int64_t)(4 * k + fc) * ldv] : 0.0;
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int j = n * 8 + 2 * fc + h;
                c[n][h] = r < m && j < nc ? C[r + (int64_t)j * ldc] : 0.0;
            }
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int n = 0; n < 2; ++n) dmma_8x8x4(c[n][0], c[n][1], a[k], b[k][n]);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int j = n * 8 + 2 * fc + h;
                if (r < m && j < nc) {
                    if (rt && r < kNb) rt[j + (int64_t)r * ldr] = c[n][h];
                    else C[r + (int64_t)j * ldc] = c[n][h];
                }
            }
    }
    __syncthreads();
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The reflector of a column with entry alpha on the diagonal and squared norm ss
// below it: (I - tau v v^T) x = beta e, v = (1, scale * x_below).
__device__ __forceinline__ void reflector(double alpha, double ss, double& beta, double& tau, double& scale) {
    beta = alpha;
    tau = scale = 0.0;
    if (ss > kTiny2) {
        beta = -copysign(sqrt(alpha * alpha + ss), alpha);
        tau = (beta - alpha) / beta;
        scale = 1.0 / (alpha - beta);
    }
}

// Householder QR of a panel (m x nc, nc <= 16).  Warp w holds columns w and w + 8 in
// R registers a lane each (rows lane + 32 i).  Step j: the column's warp makes the
// reflector and publishes it in shared memory; after the step's one barrier every
// warp reads it once into registers and dots it with its two columns - a later
// column is updated, an earlier one (which holds its reflector by then) gives the
// entry v_i . v_j that T needs.  The warp of column j + 1 goes straight on to its
// reflector, so a step costs one dot product, one update and one norm of a column.
// (With one column a warp and the reflector read twice, the shared-memory wavefronts
// of 16 warps bound it: 37 us for 837 rows, 26 so.)  R
// (transposed) goes to rt.
template <int R>
__device__ void factor_panel(double* A, int lda, int m, int nc, double* rt, int ldr, QrSmem& S) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double x[2][R];
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int col = w + kStepWarps * c, r = lane + 32 * i;
            x[c][i] = col < nc && r < m ? A[r + (int64_t)col * lda] : 0.0;
        }
    const auto reflect = [&](double (&y)[R], int j) {
        double ss[4] = {lane > j ? y[0] * y[0] : 0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int i = 1; i < R; ++i) ss[i & 3] += y[i] * y[i];
        const double s = warp_sum((ss[0] + ss[1]) + (ss[2] + ss[3]));
        double beta, tau, scale;
        reflector(__shfl_sync(0xffffffffu, y[0], j), s, beta, tau, scale);
        if (lane <= j) rt[j + (int64_t)lane * ldr] = lane == j ? beta : y[0];
        double* v = S.v[j & 1];
        y[0] = lane > j ? y[0] * scale : lane == j ? 1.0 : 0.0;
        v[lane] = y[0];
#pragma unroll
        for (int i = 1; i < R; ++i) {
            y[i] *= scale;
            v[lane + 32 * i] = y[i];
        }
        if (lane == 0) S.tau[j] = tau;
    };
    for (int j = 0; j < nc; ++j) {
        if (w == (j & (kStepWarps - 1))) {
            if (j < kStepWarps) reflect(x[0], j);
            else reflect(x[1], j);
        }
        __syncthreads();
        double v[R];
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = S.v[j & 1][lane + 32 * i];
        double d[2][2] = {};
#pragma unroll
        for (int i = 0; i < R; ++i) {
            d[0][i & 1] += x[0][i] * v[i];
            d[1][i & 1] += x[1][i] * v[i];
        }
        const double d0 = warp_sum(d[0][0] + d[0][1]), d1 = warp_sum(d[1][0] + d[1][1]);
        const double tau = S.tau[j];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int col = w + kStepWarps * c;
            const double dc = c ? d1 : d0;
            if (col > j) {
                const double f = tau * dc;
#pragma unroll
                for (int i = 0; i < R; ++i) x[c][i] -= f * v[i];
            } else if (col < j && lane == 0) {
                S.s[col * kNb + j] = dc;
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int col = w + kStepWarps * c, r = lane + 32 * i;
            if (col < nc && r < m) A[r + (int64_t)col * lda] = x[c][i];
        }
}

// The same for panels of more rows than the registers hold, on the columns in
// global memory (the CTA's own writes, ordered by the steps' barriers).
__device__ void factor_panel_long(double* A, int lda, int m, int nc, double* rt, int ldr, QrSmem& S) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int j = 0; j < nc; ++j) {
        const double* v = A + (int64_t)j * lda;
        if (w == (j & (kStepWarps - 1))) {
            double* x = A + (int64_t)j * lda;
            double ss = 0.0;
            for (int r = lane; r < m; r += 32) ss += r > j ? x[r] * x[r] : 0.0;
            ss = warp_sum(ss);
            double beta, tau, scale;
            reflector(x[j], ss, beta, tau, scale);
            if (lane <= j) rt[j + (int64_t)lane * ldr] = lane == j ? beta : x[lane];
            __syncwarp();
            for (int r = lane; r < m; r += 32) x[r] = r > j ? x[r] * scale : r == j ? 1.0 : 0.0;
            if (lane == 0) S.tau[j] = tau;
        }
        __syncthreads();
        for (int col = w; col < nc; col += kStepWarps) {
            if (col == j) continue;
            double* x = A + (int64_t)col * lda;
            double d = 0.0;
#pragma unroll 4
            for (int r = lane; r < m; r += 32) d += x[r] * v[r];
            d = warp_sum(d);
            if (col > j) {
                const double f = S.tau[j] * d;
#pragma unroll 4
                for (int r = lane; r < m; r += 32) x[r] -= f * v[r];
            } else if (lane == 0) {
                S.s[col * kNb + j] = d;
            }
        }
        __syncwarp();
    }
}

// Step s of the factorisation of every problem's matrix M (rows x cols, ld rows)
// into reflectors (left in M) and R^T (to RT, cols x cols, its upper triangle left
// as it is): CTA (problem, y) applies the reflectors of panel s - 1 to the tile of
// 16 columns s + y; the one of the next panel (y = 0) then factors it and forms its
// T, while the others finish the update.
__global__ void __launch_bounds__(32 * kStepWarps) qr_step_kernel(const SvdProblem* __restrict__ probs, double* M, double* RT,
                                                           double* T, int s) {
    __shared__ __align__(16) QrSmem S;
    const SvdProblem p = probs[blockIdx.x];
    const int c0 = (s + (int)blockIdx.y) * kNb;
    if (c0 >= p.cols) return;
    const int nc = min(kNb, p.cols - c0);
    double* A = M + p.w_off + (int64_t)c0 * p.rows;
    double* rt = RT + p.q_off;
    double* t = T + p.t_off;
    if (s > 0) {
        const int k0 = (s - 1) * kNb;
        apply_panel<true, kStepWarps>(M + p.w_off + k0 + (int64_t)k0 * p.rows, p.rows, p.rows - k0, kNb, t + (s - 1) * kNb * kNb,
                          A + k0, p.rows, nc, rt + c0 + (int64_t)k0 * p.cols, p.cols, S);
    }
    if (blockIdx.y) return;
    if (threadIdx.x < kNb * kNb) S.s[threadIdx.x] = 0.0;
    if (threadIdx.x < kNb) S.tau[threadIdx.x] = 0.0;
    __syncthreads();
    const int m = p.rows - c0;
    A += c0;
    rt += c0 + (int64_t)c0 * p.cols;
    if (m <= 64) factor_panel<2>(A, p.rows, m, nc, rt, p.cols, S);
    else if (m <= 128) factor_panel<4>(A, p.rows, m, nc, rt, p.cols, S);
    else if (m <= 256) factor_panel<8>(A, p.rows, m, nc, rt, p.cols, S);
    else if (m <= 512) factor_panel<16>(A, p.rows, m, nc, rt, p.cols, S);
    else if (m <= 32 * kMaxReg) factor_panel<kMaxReg>(A, p.rows, m, nc, rt, p.cols, S);
    else factor_panel_long(A, p.rows, m, nc, rt, p.cols, S);
    __syncthreads();
    // T of the compact form I - V T V^T, upper triangular: lane i its row i,
    // T(i, j) = -tau_j sum_l T(i, l) (v_l . v_j)
    if (threadIdx.x < kNb) {
        const int i = threadIdx.x;
        double row[kNb];
#pragma unroll
        for (int j = 0; j < kNb; ++j) {
            double a = 0.0;
#pragma unroll
            for (int l = 0; l < j; ++l) a += row[l] * S.s[l * kNb + j];
            row[j] = i == j ? S.tau[j] : i < j ? -S.tau[j] * a : 0.0;
            t[s * kNb * kNb + i * kNb + j] = row[j];
        }
    }
}

// C <- H_0 H_1 ... C for the reflectors of every problem's M: one CTA per tile of
// 16 columns, which nothing but its own reflector blocks touch.  C (rows x cols, at
// w_off) starts as the identity (`src` null; the blocks whose rows lie below the
// tile's columns leave it as it is) or as src (cols x cols, at q_off) above zeros.
__global__ void __launch_bounds__(32 * kApplyWarps) qr_apply_kernel(const SvdProblem* __restrict__ probs, const double* M,
                                                            const double* __restrict__ T,
                                                            const double* __restrict__ src, double* C) {
    __shared__ __align__(16) QrSmem S;
    const SvdProblem p = probs[blockIdx.x];
    const int c0 = blockIdx.y * kNb;
    if (c0 >= p.cols) return;
    const int nc = min(kNb, p.cols - c0);
    double* c = C + p.w_off + (int64_t)c0 * p.rows;
    for (int64_t e = threadIdx.x; e < (int64_t)nc * p.rows; e += blockDim.x) {
        const int r = (int)(e % p.rows), j = (int)(e / p.rows);
        c[e] = src ? (r < p.cols ? src[p.q_off + r + (int64_t)(c0 + j) * p.cols] : 0.0) : (r == c0 + j ? 1.0 : 0.0);
    }
    __syncthreads();
    for (int k = src ? (p.cols - 1) / kNb : (int)blockIdx.y; k >= 0; --k) {
        const int k0 = k * kNb;
        apply_panel<false, kApplyWarps>(M + p.w_off + k0 + (int64_t)k0 * p.rows, p.rows, p.rows - k0, min(kNb, p.cols - k0),
                           T + p.t_off + k * kNb * kNb, c + k0, p.rows, nc, nullptr, 0, S);
    }
}

}  // namespace

int qr_factor(const SvdProblem* probs, int np, int max_cols, double* m, double* rt, double* t, cudaStream_t st) {
    const int panels = (max_cols + kNb - 1) / kNb;
    for (int s = 0; s < panels; ++s)
        DMRG_LAUNCH qr_step_kernel<<<dim3(np, panels - s), 32 * kStepWarps, 0, st>>>(probs, m, rt, t, s);
    DMRG_CUDA_TRY(cudaGetLastError());
    return DMRG_OK;
}

int qr_apply(const SvdProblem* probs, int np, int max_cols, const double* m, const double* t, const double* src,
             double* c, cudaStream_t st) {
    DMRG_LAUNCH qr_apply_kernel<<<dim3(np, (max_cols + kNb - 1) / kNb), 32 * kApplyWarps, 0, st>>>(probs, m, t, src, c);
    DMRG_CUDA_TRY(cudaGetLastError());
    return DMRG_OK;
}

}  // namespace dmrg
