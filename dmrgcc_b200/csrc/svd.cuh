// Batched FP64 SVD of the sector matrices of one canonicalisation, on the device.
//
// Algorithm: one-sided (Hestenes) Jacobi with 32-column blocks, preconditioned by
// two QR factorisations.  Each sector matrix A (m x n) is held as a column-major
// working matrix W with c <= r columns: W = A when n <= m (right rotations
// accumulate V), W = A^T otherwise (they accumulate U).  With W P = Q1 R (P: columns
// by descending norm) and R^T = Q2 R2 (Householder, svd_qr.cu), the sweeps run on
// the c x c matrix X = R2^T, X J = Y, and U S = Q1 Y, V = P Q2 J.  A QR factor of
// a transposed QR factor is close to diagonal and graded, so few rotations remain:
// the tensors of a subspace expansion (spectra over nine decades and more) take 5
// sweeps instead of 19 at D = 1024 and 3 instead of 10 at D = 64, on r / c times
// fewer rows.  Two unpivoted factorisations did better than one with column
// pivoting (whose norms serialise the panels): 24 against 38 rounds on a
// 400 x 250 matrix.  Whole canonicalisation, D = 1024 cylinder tensor (17 sectors to
// 611 x 510): 47.2 ms without, 12.8 ms with; D = 64 chain tensor (33 columns):
// 2.03 and 0.92 ms (8.7 and 0.75 with the later pair solve and panels).  A sweep first orders the columns by descending norm
// (de Rijk's pivoting, applied block-wise), then measures every pair of column
// blocks at once (the 32x32 cross-Gram blocks, DMMA) and visits only the block
// pairs found unconverged, in as few rounds as a matching of them allows (the round-robin
// order restricted to them, or a greedy matching by measure if that needs
// fewer rounds).  In a round all pairs of all sectors are independent and each
// is split over CTAs by rows: (1) partial 64x64 Gram matrices of the pair over
// row ranges (DMMA), (2) one CTA per pair sums them and runs a few cyclic
// Jacobi sweeps on the Gram matrix in shared memory, (3) 64-row slices of the
// pair's columns of X and of the accumulated rotation are multiplied by the
// resulting 64x64 rotation (DMMA).  Converged when no pair has
// |g_ij| > tol ||A||_F max(|x_i|, |x_j|), tol = 2 eps sqrt(c): the
// remaining non-orthogonality is a backward perturbation of A below rounding
// level, the accuracy of a backward-stable SVD such as the reference's dgesvd
// (singular values to ~eps ||A||, enough for its canpre cut at 1e-12 of a
// normalised state); columns of a rank-deficient matrix
// whose norm falls to rounding level (4 eps sqrt(c) ||A||_F) are left out of
// rotations and of that test.  A matrix whose entries are all below 1/2 is
// first scaled by a power of two (exact) so that its largest entry lies in
// [0.5, 1), and scaled back at the end: the thresholds are relative, but their
// squared forms and the Gram entries of a sector with values near 1e-100 would
// underflow.  Singular values are the final column
// norms, sorted in descending order.  The free sign of each singular pair is
// fixed by a convention: the left singular vector's largest-magnitude component
// is positive (ties within a relative 1e-6: the first such component).
#pragma once

#include <vector>

#include "common.cuh"

namespace dmrg {

constexpr int kQrPanel = 16;  // columns of a QR panel

struct SvdProblem {
    int m, n;            // the sector matrix A is m x n
    int rows, cols;      // working matrix W: rows x cols, cols <= rows, column-major (ld = rows)
    int transposed;      // 1: W = A^T
    int nbe;             // number of 32-column blocks, rounded up to even (>= 2)
    int64_t w_off;       // offset of W in the W buffer (doubles)
    int64_t q_off;       // offset of the accumulated rotation (cols x cols, column-major)
    int64_t s_off;       // offset of the sorted singular values (cols doubles)
    int64_t perm_off;    // offset of the sort permutation (cols ints)
    int64_t t_off;       // offset of the QR panels' T (kQrPanel^2 doubles per panel)
};

struct SvdTask {
    int problem;
    int bi, bj;            // the pair's column blocks (sorted order), bi < bj; bj may be an empty block
    int g_first, g_count;  // its Gram items, as indices into the round's item list
};

struct SvdTile {           // a 32x32 block of a sector's cross-Gram matrix (convergence measure)
    int problem;
    int bi, bj;            // bi <= bj
    int pad;
};


struct SvdItem {   // a row range of one pair task's columns
    int task;      // index into the task list
    int seg;       // 0: rows of W, 1: rows of the accumulated rotation
    int r0, r1;
};

// Householder QR of every problem's matrix m (rows x cols at w_off): reflectors
// into m, R^T into rt (cols x cols at q_off, whose upper triangle must be zero),
// the panels' T into t.
int qr_factor(const SvdProblem* probs, int np, int max_cols, double* m, double* rt, double* t, cudaStream_t st);
// c (rows x cols at w_off) <- Q [src; 0] (src cols x cols at q_off), or the first
// cols columns of Q with src null, for the reflectors in m and t.
int qr_apply(const SvdProblem* probs, int np, int max_cols, const double* m, const double* t, const double* src,
             double* c, cudaStream_t st);

class BatchedSvd {
public:
    // Plans the batch for the given sector shapes (m[i] x n[i]; entries with
    // m*n == 0 are skipped and report no singular values).
    int plan(const std::vector<int>& m, const std::vector<int>& n, cudaStream_t st);
    // Device address of sector i's working matrix W (fill it before run()).
    double* w(int i) const { return d_w.as<double>() + probs[index[i]].w_off; }
    bool active(int i) const { return index[i] >= 0; }
    const SvdProblem& problem(int i) const { return probs[index[i]]; }
    // Runs the Jacobi sweeps to convergence (sync per sweep) and sorts.
    int run(cudaStream_t st, int* sweeps_out = nullptr);
    // Sorted singular values of every active sector, copied to the host.
    int singular_values(std::vector<std::vector<double>>& out, cudaStream_t st);
    void dump_unconverged(const char* path, const DeviceBuffer& w_in, const std::vector<double>& worst,
                          cudaStream_t st);

    // results: U S (the working matrices), the accumulated rotations, the sorted
    // singular values, their permutation, and +-1 per sorted triplet (sign convention)
    DeviceBuffer d_w, d_q, d_s, d_perm, d_sign;
    DeviceBuffer d_probs;               // probs, then the other tables (see Work)
    std::vector<SvdProblem> probs;
    std::vector<SvdProblem> xprobs;     // the square matrices that the sweeps run on: rows = cols, w_off = q_off
    int64_t w_size = 0, q_size = 0, s_size = 0, t_size = 0;
    std::vector<int> index;             // sector -> problem (-1 when empty)
    std::vector<SvdTile> tiles;         // all block pairs bi <= bj of every problem
    std::vector<int> tile_first;        // per problem: its first tile
    int gram_rows = 64;                 // rows of a Gram item
    // the current sweep's rounds (rebuilt every sweep from the measure)
    std::vector<int> round_first;       // task offset of each round
    std::vector<SvdTask> tasks;
    std::vector<SvdItem> gram_items, rot_items;    // per round, contiguous
    std::vector<int> round_gram_first, round_rot_first;
    int max_tasks = 0, max_gram = 0, max_rot = 0;  // capacities (per sweep)
    int max_round_tasks = 0, max_round_gram = 0;   // capacities (per round)

private:
    // Device addresses in d_probs (tables) and d_work (one allocation: a plan is
    // made for every site step, and an allocation costs more than a small kernel).
    struct Work {
        const SvdProblem* xprobs;
        const SvdTile* tiles;       // the convergence measure's tiles
        double *h, *t1;             // reflectors of W and their T
        double *h2, *t2;            // R^T, then its reflectors; their T
        double *x, *qx;             // the matrix of the sweeps and its accumulated rotation
        double *fro2, *part;        // per problem; per problem and slice: largest magnitude, then sum of squares
        double *norm, *bm;          // column norms; the tiles' measures
        double *gpart, *rot;        // partial Gram matrices and rotations of a round
        SvdTask* tasks;
        SvdItem *gram_items, *rot_items;
        int *expo;                  // per problem: the power of two W was scaled by (prescale_kernel)
        int *order, *colmap, *skip; // the columns of W, of x in descending norm order
    } work{};
    DeviceBuffer d_work;

    // Builds the sweep's rounds from the block measures bm (tiles order);
    // returns the number of rounds (0: converged).
    int schedule(const std::vector<double>& bm);
    void add_task(int problem, int bi, int bj);
};

}  // namespace dmrg
