// Batched one-sided block-Jacobi SVD (see svd.cuh).
#include <atomic>
#include <algorithm>
#include <cfloat>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "svd.cuh"

namespace dmrg {
namespace {

constexpr int kBlk = 32;        // columns per block
constexpr int kPair = 64;       // columns per pair
constexpr int kChunk = 32;      // rows per streamed chunk
constexpr int kThreads = 256;               // pair solve: one thread per 4x4 Gram block
constexpr int kSolveThreads = kThreads + 32;  // and a warp that finds the rotations
// Sweeps of a pair solve, at most, by the column blocks of the batch's largest sector
// (a round's solves run side by side, so the batch has one number).  More than four
// blocks: one, as a pair's other rounds undo its diagonality again (canonicalisation at
// D = 1024, 8 blocks: 8.7 ms with one, 9.5 with two, 10.2 with three).  Up to four: two,
// for three outer sweeps instead of five (D = 400 widened by half: 1.94 ms with one, 1.68
// with two).  Where the pair is the whole sector: three, for two outer sweeps, each a
// host round trip (D = 64: 0.94 ms with one, 0.80 with two, 0.74 with three).
int inner_sweeps(int blocks) { return blocks > 4 ? 1 : blocks > 2 ? 2 : 3; }
constexpr int kMaxSweeps = 40;
// The sweep cap in force (dmrg_svd_set_max_sweeps lowers it to provoke the
// did-not-converge path without touching the device).
std::atomic<int> g_max_sweeps{kMaxSweeps};
#ifndef DMRG_SVD_GRAM_MIN_ROWS
#define DMRG_SVD_GRAM_MIN_ROWS 64
#endif
constexpr int kGramMinRows = DMRG_SVD_GRAM_MIN_ROWS;  // rows of a Gram item, at least (multiple of 32)
// Columns whose norm is below kZeroRel * sqrt(rows) * ||A||_F are rounding
// residue of a rank-deficient matrix: they take part in no rotation and in no
// convergence test (their values are below any truncation threshold that is
// meaningful in FP64; rotating them only stirs rounding noise).
constexpr double kZeroRel = 4.0 * DBL_EPSILON;

constexpr int kQuads = kPair / 4;         // groups of four columns
constexpr int kClasses = (kPair - 1) / 3;  // partitions into groups of a sweep
constexpr int kSteps = kPair - 1;          // steps of the circle schedule (pair_schedule())

struct SvdSmem {
    double G[kPair * kPair], Q[kPair * kPair];  // Gram matrix, accumulated rotation
    double J[2][16 * kQuads];  // by parity: entry (a, b) of group g's 4x4 rotation at (4 a + b) * 16 + g
    int active[2];             // by parity: some group rotates
};

// The order of a pair solve's sweep.  The 64 columns are the points of the affine
// space of dimension 3 over the field of four elements (two bits a coordinate;
// addition is XOR): it has 84 lines of 4 points, any two points lie on exactly one,
// and the lines fall into 21 classes of 16 parallel lines, which partition the
// points.  A class's 16 groups of four columns are rotated at once, each through its
// six pairs; the 21 classes meet every pair once.  Group g of class c holds the
// columns base(g) ^ shift[a], a < 4.  The bases are chosen so that their low four
// bits are g: the columns of 16 neighbouring threads lie in 16 different 8-byte
// banks.
struct QuadClass {
    int shift[4];
    int c;
    __host__ __device__ explicit QuadClass(int c_) : c(c_) {
        const int d = c < 16 ? c | 16 : c < 20 ? (c - 16) | 4 : 1;  // the lines' direction
        const int wd = ((d >> 1) & 0x15) | (((d ^ (d >> 1)) & 0x15) << 1);  // times the field's generator
        shift[0] = 0;
        shift[1] = d;
        shift[2] = wd;
        shift[3] = d ^ wd;
    }
    __host__ __device__ int base(int g) const { return g | (c < 16 ? 0 : c < 20 ? g >> 2 : g & 3) << 4; }
};

// Seating of the columns in the circle schedule that dmrg_svd_pair_schedule reports and
// no kernel reads (the circle method of a round-robin tournament): at step r, seat 0 holds column 0 and seat s >= 1 holds column
// ((s - 1 - r) mod 63) + 1; seat lane j owns seats j and 63 - j, whose columns
// are the pair rotated at that step.  From one step to the next the column in
// seat s moves to seat s + 1 (seat 63 to seat 1; seat 0 stays), so a lane's two
// columns reach their next seats by one shuffle each way.
inline int seat_column(int seat, int r) {
    return seat == 0 ? 0 : ((seat - 1 - r) % kSteps + kSteps) % kSteps + 1;
}

__host__ __device__ __forceinline__ void rr_pair(int r, int i, int N, int& p, int& q) {
    if (i == 0) {
        p = 0;
        q = r % (N - 1) + 1;
    } else {
        p = (r + i) % (N - 1) + 1;
        q = (r - i + (N - 1)) % (N - 1) + 1;
    }
    if (p > q) {
        const int t = p;
        p = q;
        q = t;
    }
}

__device__ __forceinline__ void dmma_8x8x4(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// Stage 1 of a round: partial Gram matrices.  Item = (pair task, row range of W);
// 128 threads (2x2 warps, 32x32 each = 4x4 DMMA tiles); G_part = X^T X over the
// item's rows, X = the pair's 64 columns, streamed 32 rows at a time into a
// column-major shared tile (row pad 4: conflict-free stores and fragment reads).
constexpr int kGramLd = kChunk + 4;
__global__ void __launch_bounds__(128) gram_kernel(const SvdProblem* __restrict__ probs,
                                                   const SvdTask* __restrict__ tasks,
                                                   const SvdItem* __restrict__ items,
                                                   const int* __restrict__ colmap, const double* __restrict__ W,
                                                   double* __restrict__ gpart) {
    __shared__ double Xt[kPair * kGramLd];  // Xt[c][k]
    const SvdItem it = items[blockIdx.x];
    const SvdTask task = tasks[it.task];
    const SvdProblem p = probs[task.problem];
    const int colI = task.bi * kBlk, colJ = task.bj * kBlk;
    const double* Wp = W + p.w_off;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = warp >> 1, wn = warp & 1, fr = lane >> 2, fc = lane & 3;
    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    // thread: row k of each chunk in columns c = warp + 4e (e < 16); the column
    // offsets are looked up once, and the next chunk is loaded into registers
    // while the tensor cores work on the current one
    constexpr int kCols = kChunk * kPair / 128;
    static_assert(kChunk == 32 && kCols * 128 == kChunk * kPair, "one row per lane");
    const int k = lane;
    int64_t coff[kCols];
#pragma unroll
    for (int e = 0; e < kCols; ++e) {
        const int c = warp + 4 * e;
        const int vc = c < kBlk ? colI + c : colJ + c - kBlk;
        coff[e] = vc < p.cols ? (int64_t)colmap[p.perm_off + vc] * p.rows : -1;
    }
    double nxt[kCols];
#pragma unroll
    for (int e = 0; e < kCols; ++e) nxt[e] = (coff[e] >= 0 && it.r0 + k < it.r1) ? Wp[coff[e] + it.r0 + k] : 0.0;
    for (int k0 = it.r0; k0 < it.r1; k0 += kChunk) {
#pragma unroll
        for (int e = 0; e < kCols; ++e) Xt[(warp + 4 * e) * kGramLd + k] = nxt[e];
        __syncthreads();
        const int k1 = k0 + kChunk;
        if (k1 < it.r1) {
#pragma unroll
            for (int e = 0; e < kCols; ++e) nxt[e] = (coff[e] >= 0 && k1 + k < it.r1) ? Wp[coff[e] + k1 + k] : 0.0;
        }
#pragma unroll
        for (int kk = 0; kk < kChunk; kk += 4) {
            double a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = Xt[(wm * 32 + i * 8 + fr) * kGramLd + kk + fc];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Xt[(wn * 32 + j * 8 + fr) * kGramLd + kk + fc];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], a[i], b[j]);
        }
        __syncthreads();
    }
    double* g = gpart + (int64_t)blockIdx.x * kPair * kPair;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int row = wm * 32 + i * 8 + fr, col = wn * 32 + j * 8 + 2 * fc;
            g[row * kPair + col] = acc[i][j][0];
            g[row * kPair + col + 1] = acc[i][j][1];
        }
}

// Convergence measure of a sweep: one CTA per tile (problem, bi <= bj), the
// 32x32 block X_bi^T X_bj of the sector's Gram matrix over all rows (DMMA, 2x2
// warps of 16x16), reduced to the largest pair measure
// |g_ab| / (||A||_F max(|x_a|, |x_b|)) over its column pairs a < b (norms from
// the sweep's column norms), skipping columns at rounding level.
__global__ void __launch_bounds__(128) measure_kernel(const SvdProblem* __restrict__ probs,
                                                      const SvdTile* __restrict__ tiles,
                                                      const int* __restrict__ colmap, const double* __restrict__ W,
                                                      const double* __restrict__ norm, const double* __restrict__ fro2,
                                                      double* __restrict__ bm) {
    __shared__ double Xt[kPair * kGramLd];  // Xt[c][k]: c < 32 block bi, c >= 32 block bj
    __shared__ double red[4];
    const SvdTile tile = tiles[blockIdx.x];
    const SvdProblem p = probs[tile.problem];
    const int colI = tile.bi * kBlk, colJ = tile.bj * kBlk;
    const double* Wp = W + p.w_off;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = warp >> 1, wn = warp & 1, fr = lane >> 2, fc = lane & 3;
    double acc[2][2][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    constexpr int kCols = kChunk * kPair / 128;
    const int k = lane;
    int64_t coff[kCols];
#pragma unroll
    for (int e = 0; e < kCols; ++e) {
        const int c = warp + 4 * e;
        const int vc = c < kBlk ? colI + c : colJ + c - kBlk;
        coff[e] = vc < p.cols ? (int64_t)colmap[p.perm_off + vc] * p.rows : -1;
    }
    double nxt[kCols];
#pragma unroll
    for (int e = 0; e < kCols; ++e) nxt[e] = (coff[e] >= 0 && k < p.rows) ? Wp[coff[e] + k] : 0.0;
    for (int k0 = 0; k0 < p.rows; k0 += kChunk) {
#pragma unroll
        for (int e = 0; e < kCols; ++e) Xt[(warp + 4 * e) * kGramLd + k] = nxt[e];
        __syncthreads();
        const int k1 = k0 + kChunk;
        if (k1 < p.rows) {
#pragma unroll
            for (int e = 0; e < kCols; ++e) nxt[e] = (coff[e] >= 0 && k1 + k < p.rows) ? Wp[coff[e] + k1 + k] : 0.0;
        }
#pragma unroll
        for (int kk = 0; kk < kChunk; kk += 4) {
            double a[2], b[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) a[i] = Xt[(wm * 16 + i * 8 + fr) * kGramLd + kk + fc];
#pragma unroll
            for (int j = 0; j < 2; ++j) b[j] = Xt[(kBlk + wn * 16 + j * 8 + fr) * kGramLd + kk + fc];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], a[i], b[j]);
        }
        __syncthreads();
    }
    const double f2 = fro2[tile.problem];
    const double fro = sqrt(f2);
    const double zero2 = kZeroRel * kZeroRel * (double)p.rows * f2;
    double worst = 0.0;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int a = colI + wm * 16 + i * 8 + fr, b = colJ + wn * 16 + j * 8 + 2 * fc + h;
                if (a >= p.cols || b >= p.cols || a >= b) continue;
                const double na = norm[p.s_off + colmap[p.perm_off + a]], nb = norm[p.s_off + colmap[p.perm_off + b]];
                if (na * na <= zero2 || nb * nb <= zero2) continue;
                worst = fmax(worst, fabs(acc[i][j][h]) / (fro * fmax(na, nb)));
            }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) worst = fmax(worst, __shfl_xor_sync(0xffffffffu, worst, o));
    if (lane == 0) red[warp] = worst;
    __syncthreads();
    if (threadIdx.x == 0) bm[blockIdx.x] = fmax(fmax(red[0], red[1]), fmax(red[2], red[3]));
}

// The rotation (c, s) of two columns with Gram entries daa, dbb and apq that
// annihilates apq; the identity if its measure calls for none.
__device__ __forceinline__ bool angle(double daa, double dbb, double apq, double zero2, double tol2f, double& c, double& s) {
    const bool on = daa > zero2 && dbb > zero2 && apq * apq > tol2f * fmax(daa, dbb);
    // The rotation with tan = sign(x) y / (|x| + sqrt(x^2 + y^2)),
    // x = dbb - daa, y = 2 apq (the smaller root of the Jacobi
    // equation), as c = u / sqrt(u^2 + y^2), s = sign(x) y / sqrt(u^2 + y^2)
    // with u = |x| + sqrt(x^2 + y^2): no division.  (Where the pair is rotated,
    // apq^2 > tol2f zero2 is far from underflow, and so are both sums.)
    const double xd = dbb - daa, y = 2.0 * apq, h = fma(xd, xd, y * y);
    const double u = fma(h, rsqrt(h), fabs(xd));
    const double rn = rsqrt(fma(u, u, y * y));
    c = on ? u * rn : 1.0;
    s = on ? (xd >= 0.0 ? y : -y) * rn : 0.0;
    return on;
}

// Applies it to A and to the columns of two rows of the accumulated 4x4 rotation.
template <int p, int q>
__device__ __forceinline__ void rotate4(double (&A)[4][4], double (&J)[2][4], double c, double s) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (k == p || k == q) continue;
        double& ap = k < p ? A[k][p] : A[p][k];
        double& aq = k < q ? A[k][q] : A[q][k];
        const double f = c * ap - s * aq, g = s * ap + c * aq;
        ap = f;
        aq = g;
    }
    const double daa = A[p][p], apq = A[p][q], dbb = A[q][q];
    const double pp = c * daa - s * apq, pq = c * apq - s * dbb, qp = s * daa + c * apq, qq = s * apq + c * dbb;
    A[p][p] = c * pp - s * pq;
    A[p][q] = s * pp + c * pq;
    A[q][q] = s * qp + c * qq;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const double f = c * J[k][p] - s * J[k][q], g = s * J[k][p] + c * J[k][q];
        J[k][p] = f;
        J[k][q] = g;
    }
}

// The two disjoint pairs (p, q) and (r, t) of a group: the lower of its two lanes (h = 0)
// finds the first one's rotation, the upper the second's, and they exchange them.  (With
// both in every lane, the roots' branches stand in line: canonicalisation at D = 1024
// 9.09 ms, 8.70 so.)
template <int p, int q, int r, int t>
__device__ __forceinline__ bool rotate_pairs(double (&A)[4][4], double (&J)[2][4], int h, double zero2, double tol2f) {
    double c, s;
    const bool on = angle(h ? A[r][r] : A[p][p], h ? A[t][t] : A[q][q], h ? A[r][t] : A[p][q], zero2, tol2f, c, s);
    const double co = __shfl_xor_sync(0xffffffffu, c, 16), so = __shfl_xor_sync(0xffffffffu, s, 16);
    rotate4<p, q>(A, J, h ? co : c, h ? so : s);
    rotate4<r, t>(A, J, h ? c : co, h ? s : so);
    return on;
}

// The class's 16 rotations, by one warp: lane g and lane g + 16 work on group g, each
// on all of its 4x4 Gram block and on two rows of its rotation.
__device__ void find_rotations(SvdSmem& S, int par, const QuadClass& qc, int lane, double zero2, double tol2f) {
    const int g = lane & 15, h = lane >> 4, b0 = qc.base(g);
    double A[4][4], J[2][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = a; b < 4; ++b) A[a][b] = S.G[(b0 ^ qc.shift[a]) * kPair + (b0 ^ qc.shift[b])];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int b = 0; b < 4; ++b) J[k][b] = 2 * h + k == b ? 1.0 : 0.0;
    bool any = rotate_pairs<0, 1, 2, 3>(A, J, h, zero2, tol2f);
    any |= rotate_pairs<0, 2, 1, 3>(A, J, h, zero2, tol2f);
    any |= rotate_pairs<0, 3, 1, 2>(A, J, h, zero2, tol2f);
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int b = 0; b < 4; ++b) S.J[par][((2 * h + k) * 4 + b) * kQuads + g] = J[k][b];
    any = __any_sync(0xffffffffu, any);
    if (lane == 0) S.active[par] = any ? 1 : 0;
}

// Stage 2: one CTA per pair task.  Sums the task's partial Gram matrices (fixed
// order), measures the pair's convergence, and (unless converged) runs a few
// cyclic Jacobi sweeps on the 64x64 Gram matrix, writing the accumulated 64x64
// rotation to rot[task - first] and skip[task - first] = 0.
//
// A chain of dependent steps in one CTA, bound by their latency and by the
// shared-memory passes over G.  A step rotates the 16 groups of four columns of a
// class (QuadClass) through their six pairs each and applies the 4x4 rotations to G
// and Q: 21 steps a sweep, each one
// pass over G and two barriers.  (Rotating 32 disjoint pairs at a time, 63 passes over
// G a sweep, took 76 us for one sweep at D = 1024, 47 so, and the same number of outer
// sweeps or one fewer.)  The next class's rotations, a chain of three
// pair rotations, are found beside the update of Q.
__global__ void __launch_bounds__(kSolveThreads) solve_kernel(const SvdProblem* __restrict__ probs,
                                                              const SvdTask* __restrict__ tasks, int first,
                                                              int inner_sweeps, const double* __restrict__ gpart,
                                                              const double* __restrict__ fro2,
                                                              double* __restrict__ rot, int* __restrict__ skip) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SvdSmem& S = *reinterpret_cast<SvdSmem*>(smem_raw);
    const int t = first + blockIdx.x;
    const SvdTask task = tasks[t];
    const SvdProblem p = probs[task.problem];
    const double tol = 2.0 * DBL_EPSILON * sqrt((double)p.rows);
    const double zero2 = kZeroRel * kZeroRel * (double)p.rows * fro2[task.problem];
    const int tid = threadIdx.x, lane = tid & 31;
    const bool worker = tid < kThreads;
    if (worker) {
        // the partials in a fixed order (c ascending) per entry; the entries of
        // a thread are independent, so all of a partial's loads are in flight
        constexpr int kElems = kPair * kPair / kThreads;
        static_assert(kPair * kPair % kThreads == 0, "even split");
        double v[kElems];
#pragma unroll
        for (int u = 0; u < kElems; ++u) v[u] = 0.0;
        const double* gp = gpart + (int64_t)task.g_first * kPair * kPair + tid;
#pragma unroll 2
        for (int c = 0; c < task.g_count; ++c, gp += kPair * kPair)
#pragma unroll
            for (int u = 0; u < kElems; ++u) v[u] += gp[u * kThreads];
#pragma unroll
        for (int u = 0; u < kElems; ++u) {
            const int idx = tid + u * kThreads;
            S.G[idx] = v[u];
            S.Q[idx] = idx / kPair == idx % kPair ? 1.0 : 0.0;
        }
    }
    __syncthreads();

    // ---- convergence measure over the pair: |g_ij| / (||A||_F max(|x_i|, |x_j|)),
    // the size (relative to ||A||_F) of the perturbation of A that leaving the pair
    // unrotated amounts to.  Below tol the pair is as converged as a backward
    // stable SVD can tell (for two columns of norm ~||A|| this is the usual
    // relative test; a column far below ||A|| needs only an angle ~tol ||A|| / |x|).
    // Here and for the rotations the bound is half of tol, in squared form, so that
    // every pair that measure_kernel calls unconverged is rotated whatever the
    // rounding of either expression.  A step that rotates nothing skips the update,
    // and the solve ends once a sweep leaves every measure at or below the bound.
    const double tol2f = 0.25 * tol * tol * fro2[task.problem];
    const auto unconverged = [&] {
        bool off = false;
#pragma unroll 5
        for (int idx = tid; idx < kPair * kPair; idx += kSolveThreads) {
            const int a = idx / kPair, b = idx % kPair;
            const double ga = S.G[a * kPair + a], gb = S.G[b * kPair + b], g = S.G[idx];
            off |= a < b && ga > zero2 && gb > zero2 && g * g > tol2f * fmax(ga, gb);
        }
        return __syncthreads_or(off) != 0;
    };
    const bool rotate = unconverged();
    if (tid == 0) skip[blockIdx.x] = rotate ? 0 : 1;
    if (!rotate) return;

    const int gi = tid >> 4, gj = tid & 15;  // a worker's Gram block; for Q: rows 4 gi .. 4 gi + 3, group gj
    if (!worker) find_rotations(S, 0, QuadClass(0), lane, zero2, tol2f);
    __syncthreads();
    int par = 0;
    for (int sweep = 0; sweep < inner_sweeps; ++sweep) {
        bool rotated = false;
        for (int c = 0; c < kClasses; ++c, par ^= 1) {
            const QuadClass qc(c);
            const bool active = S.active[par];  // the same verdict for every thread
            double jj[4][4];
            int col[4];
            if (worker && active) {
                const double* J = S.J[par];
#pragma unroll
                for (int e = 0; e < 16; ++e) jj[e >> 2][e & 3] = J[e * kQuads + gj];
                const int bi = qc.base(gi), bj = qc.base(gj);
#pragma unroll
                for (int b = 0; b < 4; ++b) col[b] = bj ^ qc.shift[b];
                // B <- J_i^T B J_j, row by row of B, in place: nobody else touches the block
                double x[4][4];
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    double y[4];
#pragma unroll
                    for (int b = 0; b < 4; ++b) y[b] = S.G[(bi ^ qc.shift[a]) * kPair + col[b]];
#pragma unroll
                    for (int b = 0; b < 4; ++b)
                        x[a][b] = y[0] * jj[0][b] + y[1] * jj[1][b] + y[2] * jj[2][b] + y[3] * jj[3][b];
                }
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    const double j0 = J[a * kQuads + gi], j1 = J[(4 + a) * kQuads + gi], j2 = J[(8 + a) * kQuads + gi],
                                 j3 = J[(12 + a) * kQuads + gi];
#pragma unroll
                    for (int b = 0; b < 4; ++b)
                        S.G[(bi ^ qc.shift[a]) * kPair + col[b]] =
                            j0 * x[0][b] + j1 * x[1][b] + j2 * x[2][b] + j3 * x[3][b];
                }
            }
            __syncthreads();
            // the next class's rotations beside the update of Q
            if (!worker) {
                find_rotations(S, par ^ 1, QuadClass(c + 1 == kClasses ? 0 : c + 1), lane, zero2, tol2f);
            } else if (active) {
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    double* q = S.Q + (4 * gi + a) * kPair;
                    double y[4];
#pragma unroll
                    for (int b = 0; b < 4; ++b) y[b] = q[col[b]];
#pragma unroll
                    for (int b = 0; b < 4; ++b)
                        q[col[b]] = y[0] * jj[0][b] + y[1] * jj[1][b] + y[2] * jj[2][b] + y[3] * jj[3][b];
                }
            }
            rotated |= active;
            __syncthreads();
        }
        if (!rotated || sweep + 1 == inner_sweeps) break;  // uniform: every thread saw the same flags
        if (!unconverged()) break;
    }
    double* R = rot + (int64_t)blockIdx.x * kPair * kPair;
    for (int idx = tid; idx < kPair * kPair; idx += kSolveThreads) R[idx] = S.Q[idx];
}

// Stage 3: item = (pair task, segment, row range): the pair's 64 columns of W
// (segment 0) or of the accumulated rotation (segment 1), rows [r0, r1) with
// r1 - r0 <= 64, are multiplied by the task's 64x64 rotation (DMMA, in place).
// Shared tiles: Xt[c][row] and R[c][col], row pad 4 (conflict-free).
constexpr int kRotLd = kPair + 4;
constexpr size_t kRotSmem = 2 * sizeof(double) * kPair * kRotLd;
__global__ void __launch_bounds__(128) rotate_kernel(const SvdProblem* __restrict__ probs,
                                                     const SvdTask* __restrict__ tasks,
                                                     const SvdItem* __restrict__ items, int first,
                                                     const double* __restrict__ rot, const int* __restrict__ skip,
                                                     const int* __restrict__ colmap, double* __restrict__ W,
                                                     double* __restrict__ Qacc) {
    extern __shared__ __align__(16) double rsm[];
    double* Xt = rsm;                   // [64 cols][kRotLd]
    double* R = rsm + kPair * kRotLd;   // [64][kRotLd]
    const SvdItem it = items[blockIdx.x];
    if (skip[it.task - first]) return;
    const SvdTask task = tasks[it.task];
    const SvdProblem p = probs[task.problem];
    const int colI = task.bi * kBlk, colJ = task.bj * kBlk;
    double* base = it.seg == 0 ? W + p.w_off : Qacc + p.q_off;
    const int ld = it.seg == 0 ? p.rows : p.cols;
    const double* Rg = rot + (int64_t)(it.task - first) * kPair * kPair;
    for (int idx = threadIdx.x; idx < kPair * kPair; idx += 128) {
        const int c = idx / kPair, k = idx % kPair;  // consecutive threads: consecutive rows of a column
        const int vc = c < kBlk ? colI + c : colJ + c - kBlk;
        const bool v = vc < p.cols && it.r0 + k < it.r1;
        Xt[c * kRotLd + k] = v ? base[(int64_t)colmap[p.perm_off + vc] * ld + it.r0 + k] : 0.0;
        R[c * kRotLd + k] = Rg[idx];
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wm = warp >> 1, wn = warp & 1, fr = lane >> 2, fc = lane & 3;
    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll 4
    for (int kk = 0; kk < kPair; kk += 4) {
        double a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = Xt[(kk + fc) * kRotLd + wm * 32 + i * 8 + fr];  // X[row][c]
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = R[(kk + fc) * kRotLd + wn * 32 + j * 8 + fr];   // R[c][col]
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int row = wm * 32 + i * 8 + fr, col = wn * 32 + j * 8 + 2 * fc;
            Xt[col * kRotLd + row] = acc[i][j][0];
            Xt[(col + 1) * kRotLd + row] = acc[i][j][1];
        }
    __syncthreads();
    for (int idx = threadIdx.x; idx < kPair * kPair; idx += 128) {
        const int c = idx / kPair, k = idx % kPair;
        const int vc = c < kBlk ? colI + c : colJ + c - kBlk;
        if (vc < p.cols && it.r0 + k < it.r1) base[(int64_t)colmap[p.perm_off + vc] * ld + it.r0 + k] = Xt[c * kRotLd + k];
    }
}

// Scales each working matrix whose largest magnitude is below 1/2 by the power
// of two that brings it into [0.5, 1), and records the exponent e (0: left
// as is).  Only exponents change, so the scaling is exact; the Gram matrices,
// thresholds and rotations then never meet underflow, however small the
// sector's values (a sector that carries a negligible weight of the state
// reaches 1e-100 and below, whose squares underflow).  unscale_kernel undoes
// it on the result.  Three kernels over grid (problems, kSlices): the slices'
// largest magnitudes; the scaling (each slice takes the problem's maximum over
// the slice maxima) with the slices' sums of squares; the squared Frobenius
// norms, summing the slices in a fixed order.
constexpr int kSlices = 32;
__device__ __forceinline__ void slice_range(int64_t cnt, int slice, int64_t& b, int64_t& e) {
    b = cnt * slice / kSlices;
    e = cnt * (slice + 1) / kSlices;
}

__device__ __forceinline__ double block_reduce(double v, bool take_max) {
    __shared__ double red[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double u = __shfl_xor_sync(0xffffffffu, v, o);
        v = take_max ? fmax(v, u) : v + u;
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) r = take_max ? fmax(r, red[k]) : r + red[k];
    return r;
}

__global__ void __launch_bounds__(256) slice_max_kernel(const SvdProblem* __restrict__ probs,
                                                        const double* __restrict__ W, double* __restrict__ part) {
    const SvdProblem p = probs[blockIdx.x];
    const double* w = W + p.w_off;
    int64_t b, e;
    slice_range((int64_t)p.rows * p.cols, blockIdx.y, b, e);
    double mx = 0.0;
    for (int64_t i = b + threadIdx.x; i < e; i += blockDim.x) mx = fmax(mx, fabs(w[i]));
    mx = block_reduce(mx, true);
    if (threadIdx.x == 0) part[blockIdx.x * kSlices + blockIdx.y] = mx;
}

__global__ void __launch_bounds__(256) prescale_kernel(const SvdProblem* __restrict__ probs, double* __restrict__ W,
                                                       const double* __restrict__ part_max, int* __restrict__ expo,
                                                       double* __restrict__ part_ss) {
    const SvdProblem p = probs[blockIdx.x];
    double m = 0.0;
    for (int k = 0; k < kSlices; ++k) m = fmax(m, part_max[blockIdx.x * kSlices + k]);
    int ex = 0;
    if (m > 0.0 && m < 0.5) frexp(m, &ex);  // m = f 2^e, f in [0.5, 1), e <= -1
    if (blockIdx.y == 0 && threadIdx.x == 0) expo[blockIdx.x] = ex;
    double* w = W + p.w_off;
    int64_t b, e;
    slice_range((int64_t)p.rows * p.cols, blockIdx.y, b, e);
    double ss = 0.0;
    for (int64_t i = b + threadIdx.x; i < e; i += blockDim.x) {
        const double v = ex ? ldexp(w[i], -ex) : w[i];
        if (ex) w[i] = v;
        ss += v * v;
    }
    ss = block_reduce(ss, false);
    if (threadIdx.x == 0) part_ss[blockIdx.x * kSlices + blockIdx.y] = ss;
}

// Undoes prescale_kernel on the final working matrix and the sorted singular
// values.  Grid (problems, slices).
__global__ void __launch_bounds__(256) unscale_kernel(const SvdProblem* __restrict__ probs, const int* __restrict__ expo,
                                                      double* __restrict__ W, double* __restrict__ sig) {
    const SvdProblem p = probs[blockIdx.x];
    const int e = expo[blockIdx.x];
    if (e == 0) return;
    double* w = W + p.w_off;
    const int64_t cnt = (int64_t)p.rows * p.cols;
    for (int64_t i = (int64_t)blockIdx.y * blockDim.x + threadIdx.x; i < cnt; i += (int64_t)gridDim.y * blockDim.x)
        w[i] = ldexp(w[i], e);
    if (blockIdx.y == 0)
        for (int j = threadIdx.x; j < p.cols; j += blockDim.x) sig[p.s_off + j] = ldexp(sig[p.s_off + j], e);
}

// Squared Frobenius norm of each working matrix: its slices' sums in order.
__global__ void fro2_kernel(const double* __restrict__ part_ss, int np, double* __restrict__ fro2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= np) return;
    double s = 0.0;
    for (int k = 0; k < kSlices; ++k) s += part_ss[i * kSlices + k];
    fro2[i] = s;
}

// H <- W with its columns in the given order.  Grid (problems, kSlices).
__global__ void __launch_bounds__(256) order_columns_kernel(const SvdProblem* __restrict__ probs,
                                                            const int* __restrict__ order,
                                                            const double* __restrict__ W, double* __restrict__ H) {
    const SvdProblem p = probs[blockIdx.x];
    int64_t b, e;
    slice_range((int64_t)p.rows * p.cols, blockIdx.y, b, e);
    for (int64_t i = b + threadIdx.x; i < e; i += blockDim.x) {
        const int64_t c = i / p.rows;
        H[p.w_off + i] = W[p.w_off + (int64_t)order[p.perm_off + c] * p.rows + (i - c * p.rows)];
    }
}

// Q <- P Qx: row i of the accumulated rotation belongs to column order[i] of W.
// Grid (problems, kSlices).
__global__ void __launch_bounds__(256) order_rows_kernel(const SvdProblem* __restrict__ probs,
                                                         const int* __restrict__ order,
                                                         const double* __restrict__ Qx, double* __restrict__ Q) {
    const SvdProblem p = probs[blockIdx.x];
    int64_t b, e;
    slice_range((int64_t)p.cols * p.cols, blockIdx.y, b, e);
    for (int64_t i = b + threadIdx.x; i < e; i += blockDim.x) {
        const int64_t c = i / p.cols;
        Q[p.q_off + c * p.cols + order[p.perm_off + (i - c * p.cols)]] = Qx[p.q_off + i];
    }
}

// Column norms of every working matrix, one warp per column (fixed reduction order).
__global__ void __launch_bounds__(256) colnorm_kernel(const SvdProblem* __restrict__ probs,
                                                      const double* __restrict__ W, double* __restrict__ norm) {
    const SvdProblem p = probs[blockIdx.x];
    const int lane = threadIdx.x & 31;
    const int j = blockIdx.y * 8 + (threadIdx.x >> 5);
    if (j >= p.cols) return;
    const double* col = W + p.w_off + (int64_t)j * p.rows;
    double s = 0.0;
    for (int k = lane; k < p.rows; k += 32) s += col[k] * col[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) norm[p.s_off + j] = sqrt(s);
}

// Descending order of the column norms (ties by column index): order[rank] = column;
// with `sig`, also the sorted values.  Grid (problems, column slices of 256).
__global__ void __launch_bounds__(256) rank_kernel(const SvdProblem* __restrict__ probs,
                                                   const double* __restrict__ norm, int* __restrict__ order,
                                                   double* __restrict__ sig) {
    const SvdProblem p = probs[blockIdx.x];
    const double* t = norm + p.s_off;
    for (int j = blockIdx.y * blockDim.x + threadIdx.x; j < p.cols; j += gridDim.y * blockDim.x) {
        // a NaN ranks as the largest, so that the order is a permutation for any input
        const double v = t[j], kv = isnan(v) ? INFINITY : v;
        int rank = 0;
        for (int o = 0; o < p.cols; ++o) {
            const double u = isnan(t[o]) ? INFINITY : t[o];
            rank += (u > kv) || (u == kv && o < j);
        }
        order[p.perm_off + rank] = j;
        if (sig) sig[p.s_off + rank] = v;
    }
}

// Sign convention for each singular triplet (rank j, sorted): the left singular
// vector u_j is taken with its largest-magnitude component positive; components
// within a relative 1e-6 of the largest count as equal and the first decides.
// u_j is column perm[j] of W (scaled by 1/s_j) when W = A, of Q when W = A^T.
// One warp per rank.
__global__ void __launch_bounds__(256) sign_kernel(const SvdProblem* __restrict__ probs, const double* __restrict__ W,
                                                   const double* __restrict__ Q, const int* __restrict__ perm,
                                                   double* __restrict__ sign) {
    const SvdProblem p = probs[blockIdx.x];
    const int lane = threadIdx.x & 31;
    const int j = blockIdx.y * 8 + (threadIdx.x >> 5);
    if (j >= p.cols) return;
    const int k = perm[p.perm_off + j];
    const double* u = p.transposed ? Q + p.q_off + (int64_t)k * p.m : W + p.w_off + (int64_t)k * p.m;
    double mx = 0.0;
    for (int i = lane; i < p.m; i += 32) mx = fmax(mx, fabs(u[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    int first = p.m;
    for (int i = lane; i < p.m; i += 32)
        if (mx > 0.0 && fabs(u[i]) >= mx * (1.0 - 1e-6)) {
            first = i;
            break;
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) first = min(first, __shfl_xor_sync(0xffffffffu, first, o));
    if (lane == 0) sign[p.s_off + j] = (first < p.m && u[first] < 0.0) ? -1.0 : 1.0;
}

// The circle schedule of a 64-column sweep, which dmrg_svd_pair_schedule reports (the
// device's order is QuadClass's).  Step r rotates the 32 column pairs
// seated at the 32 seat lanes (seat_column); chosen here is which lane of the
// Gram update takes which pair and which of its two columns the lane addresses
// first.  Entry (r, lane) = a | b << 6 | flip << 12 | j << 13 | jflip << 18:
// a < b the pair's columns, flip = the lane addresses b first, j = the pair's
// seat lane, jflip = the column in seat j is not the one addressed first.
// In each half-warp the 16 first columns lie in 16 distinct 8-byte shared-memory
// banks (column mod 16), and so do the 16 second columns, so that every 8-byte
// access of a step's update takes the minimum of two wavefronts.  Such an order
// always exists: a step's pairs are the edges of a 4-regular multigraph on the 16
// residues; orienting it along closed trails gives each residue in- and
// out-degree 2, and the oriented edges split into two perfect matchings (tail
// residue -> head residue), one per half-warp.  Returns DMRG_OK or, if a check
// of the result fails, DMRG_E_STATE.
int build_pair_schedule(std::vector<uint32_t>& tab) {
    constexpr int kP = kPair / 2, kR = 16;
    tab.assign(kSteps * kP, 0);
    std::vector<int> met(kPair * kPair, 0);
    for (int r = 0; r < kSteps; ++r) {
        int pa[kP], pb[kP], first[kP], tail[kP], head[kP], side[kP];
        bool used[kP];
        std::vector<int> adj[kR];
        for (int k = 0; k < kP; ++k) {
            const int c0 = seat_column(k, r), c1 = seat_column(kPair - 1 - k, r);
            pa[k] = std::min(c0, c1);
            pb[k] = std::max(c0, c1);
            adj[pa[k] % kR].push_back(k);
            adj[pb[k] % kR].push_back(k);
            used[k] = false;
            side[k] = -1;
        }
        // closed trails: from v0, leave each residue along an unused edge; with
        // even degrees the walk can only stop back at v0
        for (int v0 = 0; v0 < kR; ++v0) {
            for (;;) {
                int cur = v0, len = 0;
                for (;;) {
                    int e = -1;
                    for (int x : adj[cur])
                        if (!used[x]) {
                            e = x;
                            break;
                        }
                    if (e < 0) break;
                    used[e] = true;
                    ++len;
                    const bool from_a = pa[e] % kR == cur;
                    first[e] = from_a ? pa[e] : pb[e];
                    tail[e] = cur;
                    head[e] = (from_a ? pb[e] : pa[e]) % kR;
                    cur = head[e];
                }
                if (len == 0) break;
                if (cur != v0) return set_error(DMRG_E_STATE, "pair schedule: open trail");
            }
        }
        // alternate the edges around each cycle of the 2-regular bipartite graph
        for (int e0 = 0; e0 < kP; ++e0) {
            for (int e = e0; side[e] < 0;) {
                side[e] = 0;
                int e2 = -1, e3 = -1;
                for (int k = 0; k < kP; ++k)
                    if (k != e && head[k] == head[e]) e2 = k;  // the other edge into head(e)
                if (e2 < 0 || side[e2] >= 0) break;
                side[e2] = 1;
                for (int k = 0; k < kP; ++k)
                    if (k != e2 && tail[k] == tail[e2]) e3 = k;  // the other edge out of tail(e2)
                if (e3 < 0) break;
                e = e3;
            }
        }
        int n[2] = {0, 0};
        for (int k = 0; k < kP; ++k) {
            if (side[k] < 0 || n[side[k]] >= kP / 2) return set_error(DMRG_E_STATE, "pair schedule: unbalanced split");
            const int slot = side[k] * (kP / 2) + n[side[k]]++;
            const int seated_first = seat_column(k, r);  // the column in seat k (seat lane k)
            tab[r * kP + slot] = (uint32_t)(pa[k] | pb[k] << 6 | (first[k] != pa[k] ? 1 : 0) << 12 | k << 13 |
                                            (seated_first != first[k] ? 1 : 0) << 18);
        }
        for (int h = 0; h < 2; ++h) {
            unsigned fm = 0, sm = 0;
            for (int l = 0; l < kP / 2; ++l) {
                const unsigned e = tab[r * kP + h * (kP / 2) + l];
                const int a = e & 63, b = (e >> 6) & 63, f = (e >> 12) & 1;
                fm |= 1u << ((f ? b : a) % kR);
                sm |= 1u << ((f ? a : b) % kR);
                ++met[a * kPair + b];
            }
            if (fm != 0xFFFFu || sm != 0xFFFFu) return set_error(DMRG_E_STATE, "pair schedule: bank collision");
        }
    }
    for (int a = 0; a < kPair; ++a)
        for (int b = a + 1; b < kPair; ++b)
            if (met[a * kPair + b] != 1) return set_error(DMRG_E_STATE, "pair schedule: pair (%d, %d) missed", a, b);
    return DMRG_OK;
}

const std::vector<uint32_t>* pair_schedule() {
    static std::vector<uint32_t> tab;
    static const int rc = build_pair_schedule(tab);
    return rc == DMRG_OK ? &tab : nullptr;
}

}  // namespace

int BatchedSvd::plan(const std::vector<int>& m, const std::vector<int>& n, cudaStream_t st) {
    probs.clear();
    xprobs.clear();
    t_size = 0;
    tiles.clear();
    tile_first.clear();
    index.assign(m.size(), -1);
    int64_t woff = 0, qoff = 0, soff = 0;
    for (size_t i = 0; i < m.size(); ++i) {
        if ((int64_t)m[i] * n[i] <= 0) continue;
        SvdProblem p{};
        p.m = m[i];
        p.n = n[i];
        p.transposed = n[i] > m[i];
        p.rows = p.transposed ? n[i] : m[i];
        p.cols = p.transposed ? m[i] : n[i];
        const int nb = (p.cols + kBlk - 1) / kBlk;
        p.nbe = std::max(2, nb + (nb & 1));
        p.w_off = woff;
        p.q_off = qoff;
        p.s_off = soff;
        p.perm_off = soff;
        p.t_off = t_size;
        t_size += (int64_t)((p.cols + kQrPanel - 1) / kQrPanel) * kQrPanel * kQrPanel;
        woff += (int64_t)p.rows * p.cols;
        qoff += (int64_t)p.cols * p.cols;
        soff += p.cols;
        index[i] = (int)probs.size();
        tile_first.push_back((int)tiles.size());
        for (int bi = 0; bi < nb; ++bi)
            for (int bj = bi; bj < nb; ++bj) tiles.push_back(SvdTile{(int)probs.size(), bi, bj, 0});
        probs.push_back(p);
        p.rows = p.cols;
        p.w_off = p.q_off;
        xprobs.push_back(p);
    }
    w_size = woff;
    q_size = qoff;
    tile_first.push_back((int)tiles.size());
    // Capacities.  A sweep holds at most every block pair of a problem plus one
    // pair per block for blocks unconverged only within themselves; a round at
    // most nbe / 2 pairs per problem.  Row ranges of the Gram items: at least
    // kGramMinRows rows each, fewer items than ~4 per SM in the widest round
    // (bounds the partial-Gram buffer).
    int64_t widest = 0, sweep_tasks = 0, sweep_gram = 0, sweep_rot = 0, round_tasks = 0;
    for (const SvdProblem& p : xprobs) {
        widest += (int64_t)p.rows * (p.nbe / 2);
        round_tasks += p.nbe / 2;
    }
    gram_rows = (int)std::max<int64_t>(kGramMinRows, ((widest / 600 + 31) / 32) * 32);
    int64_t round_gram = 0;
    for (const SvdProblem& p : xprobs) {
        const int64_t pairs = (int64_t)p.nbe * (p.nbe - 1) / 2 + p.nbe;
        const int64_t gi = (p.rows + gram_rows - 1) / gram_rows;
        const int64_t ri = (p.rows + kPair - 1) / kPair + (p.cols + kPair - 1) / kPair;
        sweep_tasks += pairs;
        sweep_gram += pairs * gi;
        sweep_rot += pairs * ri;
        round_gram += (int64_t)(p.nbe / 2) * gi;
    }
    max_tasks = (int)sweep_tasks;
    max_gram = (int)sweep_gram;
    max_rot = (int)sweep_rot;
    max_round_tasks = (int)round_tasks;
    max_round_gram = (int)round_gram;
    const auto some = [](int64_t n) { return (size_t)std::max<int64_t>(n, 1); };
    s_size = soff;
    DMRG_TRY(d_w.alloc(some(w_size) * sizeof(double)));
    DMRG_TRY(d_q.alloc(some(q_size) * sizeof(double)));
    DMRG_TRY(d_s.alloc(some(2 * soff) * sizeof(double)));
    DMRG_TRY(d_perm.alloc(some(soff) * sizeof(int)));
    DMRG_TRY(d_sign.alloc(some(soff) * sizeof(double)));
    Tables tab;
    tab.add(probs);  // at offset 0: d_probs is the problem table
    const size_t at_x = tab.add(xprobs), at_tiles = tab.add(tiles);
    DMRG_TRY(tab.to(d_probs, st));
    const unsigned char* tb = d_probs.as<unsigned char>();
    work.xprobs = reinterpret_cast<const SvdProblem*>(tb + at_x);
    work.tiles = reinterpret_cast<const SvdTile*>(tb + at_tiles);
    // the workspace: two passes over its pieces, sizes then addresses
    const int64_t np = (int64_t)probs.size();
    size_t bytes = 0;
    for (int pass = 0; pass < 2; ++pass) {
        if (pass) DMRG_TRY(d_work.alloc(some((int64_t)bytes)));
        unsigned char* base = d_work.as<unsigned char>();
        bytes = 0;
        const auto piece = [&](auto*& p, int64_t n) {
            if (pass) p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(base + bytes);
            bytes += (some(n) * sizeof(*p) + 255) & ~size_t(255);
        };
        piece(work.h, w_size);
        piece(work.h2, 2 * q_size);  // h2, then x: cleared together
        piece(work.qx, q_size);
        piece(work.t1, t_size);
        piece(work.t2, t_size);
        piece(work.fro2, np);
        piece(work.part, np * 2 * kSlices);
        piece(work.norm, soff);
        piece(work.bm, (int64_t)tiles.size());
        piece(work.gpart, (int64_t)max_round_gram * kPair * kPair);
        piece(work.rot, (int64_t)max_round_tasks * kPair * kPair);
        piece(work.tasks, max_tasks);
        piece(work.gram_items, max_gram);
        piece(work.rot_items, max_rot);
        piece(work.expo, np);
        piece(work.order, soff);
        piece(work.colmap, soff);
        piece(work.skip, max_round_tasks);
    }
    work.x = work.h2 + q_size;
    DMRG_CUDA_TRY(cudaFuncSetAttribute(solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(SvdSmem)));
    static_assert(sizeof(SvdSmem) <= 227 * 1024, "pair solve shared memory");
    DMRG_CUDA_TRY(cudaFuncSetAttribute(rotate_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRotSmem));
    return DMRG_OK;
}

void BatchedSvd::add_task(int problem, int bi, int bj) {
    const SvdProblem& p = xprobs[problem];
    const int t = (int)tasks.size();
    SvdTask task{problem, bi, bj, (int)gram_items.size() - round_gram_first.back(), 0};
    for (int r0 = 0; r0 < p.rows; r0 += gram_rows)
        gram_items.push_back(SvdItem{t, 0, r0, std::min(p.rows, r0 + gram_rows)});
    task.g_count = (int)gram_items.size() - round_gram_first.back() - task.g_first;
    tasks.push_back(task);
    for (int r0 = 0; r0 < p.rows; r0 += kPair) rot_items.push_back(SvdItem{t, 0, r0, std::min(p.rows, r0 + kPair)});
    for (int r0 = 0; r0 < p.cols; r0 += kPair) rot_items.push_back(SvdItem{t, 1, r0, std::min(p.cols, r0 + kPair)});
}

// Rounds of one problem's sweep: its unconverged block pairs (measure > tol) as
// a sequence of matchings, and every block unconverged within itself in some
// pair.  Two candidates, the fewer rounds kept: the round-robin order over nbe
// blocks restricted to those pairs, and a greedy matching by decreasing measure.
static std::vector<std::vector<std::pair<int, int>>> problem_rounds(const SvdProblem& p, const double* bm,
                                                                     double tol) {
    const int nb = (p.cols + kBlk - 1) / kBlk;
    auto at = [&](int i, int j) {  // tiles of a problem: bi <= bj, row-major over bi
        if (i > j) std::swap(i, j);
        return bm[i * nb - i * (i - 1) / 2 + (j - i)];
    };
    std::vector<std::pair<double, std::pair<int, int>>> cross;
    std::vector<int> internal;
    for (int i = 0; i < nb; ++i) {
        if (at(i, i) > tol) internal.push_back(i);
        for (int j = i + 1; j < nb; ++j)
            if (at(i, j) > tol) cross.push_back({at(i, j), {i, j}});
    }
    using Rounds = std::vector<std::vector<std::pair<int, int>>>;
    auto cover = [&](Rounds& rounds) {  // every internally unconverged block in some pair
        std::vector<char> seen(p.nbe, 0);
        for (const auto& rd : rounds)
            for (const auto& pr : rd) seen[pr.first] = seen[pr.second] = 1;
        for (int i : internal) {
            if (seen[i]) continue;
            bool placed = false;
            for (auto& rd : rounds) {
                std::vector<char> used(p.nbe, 0);
                for (const auto& pr : rd) used[pr.first] = used[pr.second] = 1;
                if (used[i]) continue;
                for (int j = 0; j < p.nbe && !placed; ++j)
                    if (j != i && !used[j]) {
                        rd.push_back({std::min(i, j), std::max(i, j)});
                        seen[j] = 1;
                        placed = true;
                    }
                if (placed) break;
            }
            if (!placed) {
                const int j = (i + 1) % p.nbe;
                rounds.push_back({{std::min(i, j), std::max(i, j)}});
                seen[j] = 1;
            }
            seen[i] = 1;
        }
    };
    Rounds rr;
    {
        std::vector<char> need((size_t)p.nbe * p.nbe, 0);
        for (const auto& c : cross) need[c.second.first * p.nbe + c.second.second] = 1;
        for (int r = 0; r < p.nbe - 1; ++r) {
            std::vector<std::pair<int, int>> rd;
            for (int k = 0; k < p.nbe / 2; ++k) {
                int i, j;
                rr_pair(r, k, p.nbe, i, j);
                if (need[i * p.nbe + j]) rd.push_back({i, j});
            }
            if (!rd.empty()) rr.push_back(rd);
        }
        cover(rr);
    }
    Rounds gr;
    {
        std::sort(cross.begin(), cross.end(), [](const auto& x, const auto& y) { return x.first > y.first; });
        std::vector<std::vector<char>> used;
        for (const auto& c : cross) {
            const int i = c.second.first, j = c.second.second;
            size_t r = 0;
            for (; r < gr.size(); ++r)
                if (!used[r][i] && !used[r][j]) break;
            if (r == gr.size()) {
                gr.emplace_back();
                used.emplace_back(p.nbe, 0);
            }
            gr[r].push_back({i, j});
            used[r][i] = used[r][j] = 1;
        }
        cover(gr);
    }
    return gr.size() < rr.size() ? gr : rr;
}

int BatchedSvd::schedule(const std::vector<double>& bm) {
    tasks.clear();
    gram_items.clear();
    rot_items.clear();
    round_first.clear();
    round_gram_first.clear();
    round_rot_first.clear();
    std::vector<std::vector<std::vector<std::pair<int, int>>>> per(probs.size());
    size_t rounds = 0;
    for (size_t pi = 0; pi < probs.size(); ++pi) {
        const double tol = 2.0 * DBL_EPSILON * std::sqrt((double)xprobs[pi].rows);
        per[pi] = problem_rounds(xprobs[pi], bm.data() + tile_first[pi], tol);
        rounds = std::max(rounds, per[pi].size());
    }
    for (size_t r = 0; r < rounds; ++r) {
        round_first.push_back((int)tasks.size());
        round_gram_first.push_back((int)gram_items.size());
        round_rot_first.push_back((int)rot_items.size());
        for (size_t pi = 0; pi < probs.size(); ++pi)
            if (r < per[pi].size())
                for (const auto& pr : per[pi][r]) add_task((int)pi, pr.first, pr.second);
    }
    round_first.push_back((int)tasks.size());
    round_gram_first.push_back((int)gram_items.size());
    round_rot_first.push_back((int)rot_items.size());
    return (int)rounds;
}

// Appends, for each problem whose last measure was above tol: m, n, rows,
// cols, transposed (int32), fro2 and the measure (float64), then its input and
// final working matrices (rows x cols float64, column-major).
void BatchedSvd::dump_unconverged(const char* path, const DeviceBuffer& w_in, const std::vector<double>& worst,
                                  cudaStream_t st) {
    std::FILE* f = std::fopen(path, "ab");
    if (!f) return;
    std::vector<double> fro2(probs.size());
    cudaMemcpyAsync(fro2.data(), work.fro2, fro2.size() * sizeof(double), cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    for (size_t i = 0; i < probs.size(); ++i) {
        const SvdProblem& p = probs[i];
        if (worst[i] <= 2.0 * DBL_EPSILON * std::sqrt((double)p.cols)) continue;
        const size_t cnt = (size_t)p.rows * p.cols;
        std::vector<double> a(cnt), b(cnt);
        cudaMemcpyAsync(a.data(), w_in.as<double>() + p.w_off, cnt * sizeof(double), cudaMemcpyDeviceToHost, st);
        cudaMemcpyAsync(b.data(), d_w.as<double>() + p.w_off, cnt * sizeof(double), cudaMemcpyDeviceToHost, st);
        cudaStreamSynchronize(st);
        const int hdr[5] = {p.m, p.n, p.rows, p.cols, p.transposed};
        const double val[2] = {fro2[i], worst[i]};
        std::fwrite(hdr, sizeof(int), 5, f);
        std::fwrite(val, sizeof(double), 2, f);
        std::fwrite(a.data(), sizeof(double), cnt, f);
        std::fwrite(b.data(), sizeof(double), cnt, f);
    }
    std::fclose(f);
}

int BatchedSvd::run(cudaStream_t st, int* sweeps_out) {
    if (probs.empty()) {
        if (sweeps_out) *sweeps_out = 0;
        return DMRG_OK;
    }
    const int np = (int)probs.size();
    // DMRG_SVD_FAIL_DUMP=path: keep the input, and if the sweeps do not converge
    // write every unconverged sector's input and final working matrix to path
    // (diagnostics only; see dump_unconverged)
    static const char* fail_dump = std::getenv("DMRG_SVD_FAIL_DUMP");
    DeviceBuffer w_in;
    if (fail_dump) {
        DMRG_TRY(w_in.alloc(d_w.bytes));
        DMRG_CUDA_TRY(cudaMemcpyAsync(w_in.ptr, d_w.ptr, d_w.bytes, cudaMemcpyDeviceToDevice, st));
    }
    const dim3 sliced(np, kSlices);
    DMRG_LAUNCH slice_max_kernel<<<sliced, 256, 0, st>>>(d_probs.as<SvdProblem>(), d_w.as<double>(), work.part);
    DMRG_LAUNCH prescale_kernel<<<sliced, 256, 0, st>>>(d_probs.as<SvdProblem>(), d_w.as<double>(), work.part,
                                                        work.expo, work.part + (int64_t)np * kSlices);
    DMRG_LAUNCH fro2_kernel<<<(np + 127) / 128, 128, 0, st>>>(work.part + (int64_t)np * kSlices, np, work.fro2);
    static const bool debug = std::getenv("DMRG_SVD_DEBUG") != nullptr;  // per-sweep convergence to stderr
    int max_cols = 0, max_blocks = 0;
    for (const SvdProblem& p : probs) {
        max_cols = std::max(max_cols, p.cols);
        max_blocks = std::max(max_blocks, p.nbe);
    }
    const int sweeps = inner_sweeps(max_blocks);
    const dim3 colgrid(np, (max_cols + 7) / 8);
    const dim3 rankgrid(np, (max_cols + 255) / 256);
    // Preconditioner: W P = Q1 R, R^T = Q2 R2, sweeps on X = R2^T (X J = Y), so that
    // U S = Q1 Y and V = P Q2 J.
    const SvdProblem* wp = d_probs.as<SvdProblem>();
    const SvdProblem* xp = work.xprobs;
    double *h = work.h, *h2 = work.h2, *x = work.x, *qx = work.qx, *t1 = work.t1, *t2 = work.t2;
    DMRG_CUDA_TRY(cudaMemsetAsync(h2, 0, 2 * q_size * sizeof(double), st));
    DMRG_LAUNCH colnorm_kernel<<<colgrid, 256, 0, st>>>(wp, d_w.as<double>(), work.norm);
    DMRG_LAUNCH rank_kernel<<<rankgrid, 256, 0, st>>>(wp, work.norm, work.order, nullptr);
    DMRG_LAUNCH order_columns_kernel<<<sliced, 256, 0, st>>>(wp, work.order, d_w.as<double>(), h);
    DMRG_TRY(qr_factor(wp, np, max_cols, h, h2, t1, st));
    DMRG_TRY(qr_factor(xp, np, max_cols, h2, x, t2, st));
    DMRG_TRY(qr_apply(xp, np, max_cols, h2, t2, nullptr, qx, st));
    std::vector<double> bm(tiles.size()), worst(np);
    const int max_sweeps = g_max_sweeps.load();
    auto t_sweep = std::chrono::steady_clock::now();
    int sweep = 0;
    bool converged = false;
    for (;; ++sweep) {
        // the sweep visits columns in descending norm order (blocks hold columns of
        // similar size); then every block pair is measured
        DMRG_LAUNCH colnorm_kernel<<<colgrid, 256, 0, st>>>(xp, x, work.norm);
        DMRG_LAUNCH rank_kernel<<<rankgrid, 256, 0, st>>>(xp, work.norm, work.colmap, nullptr);
        DMRG_LAUNCH measure_kernel<<<(int)tiles.size(), 128, 0, st>>>(
            xp, work.tiles, work.colmap, x, work.norm, work.fro2, work.bm);
        DMRG_CUDA_TRY(cudaGetLastError());
        DMRG_CUDA_TRY(cudaMemcpyAsync(bm.data(), work.bm, bm.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
        DMRG_CUDA_TRY(cudaStreamSynchronize(st));
        for (int i = 0; i < np; ++i) {
            worst[i] = 0.0;
            for (int k = tile_first[i]; k < tile_first[i + 1]; ++k) worst[i] = std::max(worst[i], bm[k]);
        }
        const int rounds = schedule(bm);
        if (debug) {
            int wi = 0;
            for (int i = 1; i < np; ++i)
                if (worst[i] > worst[wi]) wi = i;
            const auto now = std::chrono::steady_clock::now();
            std::fprintf(stderr, "svd sweep %d: %.2f ms, worst %.3e (sector %d x %d), %d rounds\n", sweep,
                         std::chrono::duration<double, std::milli>(now - t_sweep).count(), worst[wi], probs[wi].m,
                         probs[wi].n, rounds);
            t_sweep = now;
        }
        if (rounds == 0) {
            converged = true;
            break;
        }
        if (sweep >= max_sweeps) break;
        int widest_round = 0, widest_gram = 0;
        for (int r = 0; r < rounds; ++r) {
            widest_round = std::max(widest_round, round_first[r + 1] - round_first[r]);
            widest_gram = std::max(widest_gram, round_gram_first[r + 1] - round_gram_first[r]);
        }
        if ((int)tasks.size() > max_tasks || (int)gram_items.size() > max_gram || (int)rot_items.size() > max_rot ||
            widest_round > max_round_tasks || widest_gram > max_round_gram)
            return set_error(DMRG_E_STATE, "Jacobi SVD schedule exceeds its plan");
        DMRG_CUDA_TRY(cudaMemcpyAsync(work.tasks, tasks.data(), tasks.size() * sizeof(SvdTask), cudaMemcpyHostToDevice, st));
        DMRG_CUDA_TRY(cudaMemcpyAsync(work.gram_items, gram_items.data(), gram_items.size() * sizeof(SvdItem),
                                      cudaMemcpyHostToDevice, st));
        DMRG_CUDA_TRY(cudaMemcpyAsync(work.rot_items, rot_items.data(), rot_items.size() * sizeof(SvdItem),
                                      cudaMemcpyHostToDevice, st));
        for (int r = 0; r < rounds; ++r) {
            const int nt = round_first[r + 1] - round_first[r];
            const int ng = round_gram_first[r + 1] - round_gram_first[r];
            const int nr = round_rot_first[r + 1] - round_rot_first[r];
            if (nt == 0) continue;
            DMRG_LAUNCH gram_kernel<<<ng, 128, 0, st>>>(xp, work.tasks, work.gram_items + round_gram_first[r],
                                                        work.colmap, x, work.gpart);
            DMRG_LAUNCH solve_kernel<<<nt, kSolveThreads, sizeof(SvdSmem), st>>>(
                xp, work.tasks, round_first[r], sweeps, work.gpart, work.fro2, work.rot, work.skip);
            DMRG_LAUNCH rotate_kernel<<<nr, 128, kRotSmem, st>>>(xp, work.tasks, work.rot_items + round_rot_first[r],
                                                                 round_first[r], work.rot, work.skip, work.colmap, x,
                                                                 qx);
        }
        DMRG_CUDA_TRY(cudaGetLastError());
    }
    DMRG_TRY(qr_apply(wp, np, max_cols, h, t1, x, d_w.as<double>(), st));
    if (!converged) {
        if (fail_dump) dump_unconverged(fail_dump, w_in, worst, st);
        int wi = 0;
        for (int i = 1; i < np; ++i)
            if (worst[i] > worst[wi]) wi = i;
        return set_error(DMRG_E_NUMERIC, "Jacobi SVD did not converge in %d sweeps (sector %d x %d: off-diagonal %.3e)",
                         max_sweeps, probs[wi].m, probs[wi].n, worst[wi]);
    }
    DMRG_LAUNCH order_rows_kernel<<<sliced, 256, 0, st>>>(wp, work.order, qx, d_q.as<double>());
    // singular values = final column norms, sorted
    DMRG_LAUNCH colnorm_kernel<<<colgrid, 256, 0, st>>>(d_probs.as<SvdProblem>(), d_w.as<double>(), work.norm);
    DMRG_LAUNCH rank_kernel<<<rankgrid, 256, 0, st>>>(d_probs.as<SvdProblem>(), work.norm, d_perm.as<int>(), d_s.as<double>());
    DMRG_LAUNCH sign_kernel<<<colgrid, 256, 0, st>>>(d_probs.as<SvdProblem>(), d_w.as<double>(),
                                                               d_q.as<double>(), d_perm.as<int>(), d_sign.as<double>());
    DMRG_LAUNCH unscale_kernel<<<dim3(np, 32), 256, 0, st>>>(d_probs.as<SvdProblem>(), work.expo,
                                                             d_w.as<double>(), d_s.as<double>());
    DMRG_CUDA_TRY(cudaGetLastError());
    if (sweeps_out) *sweeps_out = sweep;  // sweeps that rotated
    return DMRG_OK;
}

int BatchedSvd::singular_values(std::vector<std::vector<double>>& out, cudaStream_t st) {
    out.assign(index.size(), std::vector<double>());
    if (probs.empty()) return DMRG_OK;
    int64_t total = 0;
    for (const auto& p : probs) total += p.cols;
    std::vector<double> all(total);
    DMRG_CUDA_TRY(cudaMemcpyAsync(all.data(), d_s.ptr, total * sizeof(double), cudaMemcpyDeviceToHost, st));
    DMRG_CUDA_TRY(cudaStreamSynchronize(st));
    for (size_t i = 0; i < index.size(); ++i) {
        if (index[i] < 0) continue;
        const SvdProblem& p = probs[index[i]];
        out[i].assign(all.begin() + p.s_off, all.begin() + p.s_off + p.cols);
    }
    return DMRG_OK;
}

}  // namespace dmrg

extern "C" int dmrg_svd_set_max_sweeps(int sweeps) {
    dmrg::g_max_sweeps.store(sweeps > 0 ? sweeps : dmrg::kMaxSweeps);
    return DMRG_OK;
}

extern "C" int dmrg_svd_plan_rounds(int cols, const double* bm, double tol, int cap, int* pairs, int* n_pairs,
                                    int* n_rounds) {
    if (cols <= 0 || !bm || !n_pairs || !n_rounds || (cap > 0 && !pairs))
        return dmrg::set_error(DMRG_E_ARG, "invalid argument");
    dmrg::SvdProblem p{};
    p.rows = p.cols = p.m = p.n = cols;
    const int nb = (cols + dmrg::kBlk - 1) / dmrg::kBlk;
    p.nbe = std::max(2, nb + (nb & 1));
    const auto rounds = dmrg::problem_rounds(p, bm, tol);
    int k = 0;
    for (size_t r = 0; r < rounds.size(); ++r)
        for (const auto& pr : rounds[r]) {
            if (k < cap) pairs[k] = (int)r << 16 | pr.first << 8 | pr.second;
            ++k;
        }
    *n_pairs = k;
    *n_rounds = (int)rounds.size();
    return k <= cap ? DMRG_OK : dmrg::set_error(DMRG_E_ARG, "%d pairs, room for %d", k, cap);
}

extern "C" int dmrg_svd_solve_groups(int* out) {
    if (!out) return dmrg::set_error(DMRG_E_ARG, "null argument");
    for (int c = 0; c < dmrg::kClasses; ++c) {
        const dmrg::QuadClass qc(c);
        for (int g = 0; g < dmrg::kQuads; ++g)
            for (int a = 0; a < 4; ++a) *out++ = qc.base(g) ^ qc.shift[a];
    }
    return DMRG_OK;
}

extern "C" int dmrg_svd_pair_schedule(unsigned int* out) {
    if (!out) return dmrg::set_error(DMRG_E_ARG, "null argument");
    const std::vector<uint32_t>* tab = dmrg::pair_schedule();
    if (!tab) return DMRG_E_STATE;
    std::memcpy(out, tab->data(), tab->size() * sizeof(uint32_t));
    return DMRG_OK;
}
