// a2/a3: environment updates.
//
// Left (RealTensorContraction::LeftComputeTensorContraction,
// src/dmrg/realdmrg/real_tensor_contraction.cc:782-940):
//   L'[o2](i,j) += W[o1][o2](p(k,i), p(l,j)) * B(k,i)^T L[o1](k,l) K(l,j)
// stage 1: F = B(k,i)^T L[o1](k,l)      (transposed-A grouped GEMM)
// stage 2: L'[o2](i,j) += W * F K(l,j)   (one group per output block)
// Right (RightComputeTensorContraction, :959-1119):
//   R'[o1](j,i) += W[o1][o2](p(i,k), p(j,l)) * K(j,l) R[o2](l,k) B(i,k)^T
// stage 1: G = K(j,l) R[o2](l,k)
// stage 2: R'[o1](j,i) += W * G B(i,k)^T (transposed-B)
// The output block lists follow the reference's zero_flag pass (:797-883,
// :974-1060): per output bond index, blocks in row-major (first, second) sector
// order, present wherever some contribution has a nonzero W.
#include <algorithm>

#include "blocksparse.h"
#include "gemm.cuh"

using namespace dmrg;

namespace {

// The update's products, on either side.  Stage 1: a product of ket (or bra) block
// `ket` and an input block, m x n with inner extent k, for every pair that some term
// of stage 2 reads.  Stage 2: the terms of each output block, output blocks in order.
struct Stage1Task {
    int ket;
    int o, blk;   // input block
    int m, n, k;
    int64_t off;  // in the scratch of the products
};
struct Stage2Term {
    int task;
    int ket;
    double w;
};
struct EnvProducts {
    std::vector<Stage1Task> tasks;
    std::vector<Stage2Term> terms;  // by output block
    std::vector<int> first;         // terms before each output block, and in all
    int64_t scratch_size = 0;
};

}  // namespace

struct dmrg_env_s {
    dmrg_ctx_t ctx = nullptr;
    int side = 0;
    int precision = DMRG_PREC_FP64;
    SiteDesc site;
    EnvDesc in, out;
    EnvProducts products;  // of creation
    // FP64: images of the ket and of the input environment, stage 1 into images, stage 2 into blocks
    ImgPack img;
    ImgSchedule i1, i2;
    ImgWork work;
    SplitPlan p1, p2;  // split precisions: the same two stages on the tcgen05 path
    bool cplx = false;  // the complex path (dmrg_zenv_create): the same stages on complex blocks
    DeviceBuffer scratch;
    double flops_alg = 0, flops_exec = 0;
};

namespace {

// Output structure and products.  Left and right are mirror images: with (x, y) the
// sectors of an input block of bond index `o`, block u of the ket list with sector x
// (left: of its rows, right: of its columns) makes the stage 1 product, every block v
// with sector y a term, per output index with a nonzero weight; the output block has the
// other sectors of u and v.  One pass collects the terms, in the order of the reference's
// loops; they are then sorted, stably, by output block, and the blocks are those that occur.
int build_products(dmrg_env_s& e) {
    const SiteDesc& s = e.site;
    const BlockListDesc& ket = s.ket;
    const bool left = e.side == 0;
    const char* name = left ? "L" : "R";
    const int nx = left ? s.nl : s.nr, ny = left ? s.nr : s.nl;            // sectors of the input, of the output
    const int in_bond = left ? s.lb : s.rb, out_bond = left ? s.rb : s.lb;
    const std::vector<int>&inner = left ? ket.rows : ket.cols, &outer = left ? ket.cols : ket.rows;
    const std::vector<int>& osec = left ? ket.right : ket.left;
    const auto same = ket.by_sector(left ? 0 : 1, nx);
    std::vector<int> dim(ny, -1);  // outer extent of the ket blocks by output sector
    for (int k = 0; k < ket.count(); ++k) {
        int& d = dim[osec[k]];
        if (d == -1) d = outer[k];
        else if (d != outer[k])
            return left ? set_error(DMRG_E_ARG, "ket blocks of right sector %d have different widths", osec[k])
                        : set_error(DMRG_E_ARG, "ket blocks of left sector %d have different heights", osec[k]);
    }
    for (int o = 0; o < in_bond; ++o) {
        const BlockListDesc& in = e.in.o[o];
        for (int i = 0; i < in.count(); ++i)
            if (in.left[i] < 0 || in.left[i] >= nx || in.right[i] < 0 || in.right[i] >= nx)
                return set_error(DMRG_E_ARG, "%s[%d] block %d sectors out of range", name, o, i);
    }
    // by (o, pu): whether the reference takes the product; by (o, pu, pv): the output indexes
    // with a nonzero weight, ascending
    std::vector<char> taken((size_t)in_bond * s.d);
    std::vector<int> outs, outs_first(1, 0);
    for (int o = 0; o < in_bond; ++o)
        for (int pu = 0; pu < s.d; ++pu) {
            taken[(size_t)o * s.d + pu] = left ? s.left_nonzero(o, pu) : s.right_nonzero(o, pu);
            for (int pv = 0; pv < s.d; ++pv) {
                for (int q = 0; q < out_bond; ++q)
                    if ((left ? s.w(o, q, pu, pv) : s.w(q, o, pv, pu)) != 0.0) outs.push_back(q);
                outs_first.push_back((int)outs.size());
            }
        }
    struct Term {
        int row, j;  // output index and first sector, index * ny + sector; second sector
        Stage2Term t;
    };
    EnvProducts& pr = e.products;
    std::vector<Term> terms;
    std::vector<int> row_first((size_t)out_bond * ny + 1, 0);  // terms by row: counts, then first
    double f1_alg = 0, f2_alg = 0, f1_exec = 0, f2_exec = 0;
    for (int o = 0; o < in_bond; ++o) {
        const BlockListDesc& in = e.in.o[o];
        for (int i = 0; i < in.count(); ++i) {
            const int r = in.rows[i], c = in.cols[i];
            if (r == 0) continue;
            for (int u : same[in.left[i]]) {
                const int pu = s.pb(u);
                if (!taken[(size_t)o * s.d + pu]) continue;
                if (inner[u] != r)
                    return left ? set_error(DMRG_E_ARG, "ket block %d rows %d != L rows %d", u, inner[u], r)
                                : set_error(DMRG_E_ARG, "ket block %d cols %d != R rows %d", u, inner[u], r);
                f1_alg += 2.0 * outer[u] * r * c;
                const size_t before = terms.size();
                for (int v : same[in.right[i]]) {
                    const int pv = s.pb(v);
                    if (inner[v] != c)
                        return left ? set_error(DMRG_E_ARG, "ket block %d rows != L cols", v)
                                    : set_error(DMRG_E_ARG, "ket block %d cols != R cols", v);
                    const double f = 2.0 * outer[u] * c * outer[v];
                    f2_alg += f;
                    const size_t at = ((size_t)o * s.d + pu) * s.d + pv;
                    for (int x = outs_first[at]; x < outs_first[at + 1]; ++x) {
                        const int q = outs[x], row = q * ny + osec[u];
                        const double w = left ? s.w(o, q, pu, pv) : s.w(q, o, pv, pu);
                        terms.push_back(Term{row, osec[v], Stage2Term{(int)pr.tasks.size(), v, w}});
                        ++row_first[row + 1];
                        f2_exec += f;
                    }
                }
                if (terms.size() > before) {
                    pr.tasks.push_back(Stage1Task{u, o, i, outer[u], c, r, pr.scratch_size});
                    pr.scratch_size += (int64_t)outer[u] * c;
                    f1_exec += 2.0 * outer[u] * r * c;
                }
            }
        }
    }
    for (size_t r = 1; r < row_first.size(); ++r) row_first[r] += row_first[r - 1];
    std::vector<int> order(terms.size()), next(row_first.begin(), row_first.end() - 1);
    for (int i = 0; i < (int)terms.size(); ++i) order[next[terms[i].row]++] = i;
    e.out.o.assign(out_bond, BlockListDesc());
    pr.first.assign(1, 0);
    pr.terms.reserve(terms.size());
    for (int r = 0; r + 1 < (int)row_first.size(); ++r) {
        const auto b = order.begin() + row_first[r], end = order.begin() + row_first[r + 1];
        auto second = [&](int x, int y) { return terms[x].j < terms[y].j; };
        if (!std::is_sorted(b, end, second)) std::stable_sort(b, end, second);  // (one second sector, mostly)
        for (auto x = b; x != end; ++x) {
            const Term& t = terms[*x];
            if (x == b || t.j != terms[x[-1]].j) {
                if (x != b) pr.first.push_back((int)pr.terms.size());
                e.out.o[r / ny].push(r % ny, t.j, dim[r % ny], dim[t.j]);
            }
            pr.terms.push_back(t.t);
        }
        if (b != end) pr.first.push_back((int)pr.terms.size());
    }
    e.out.rebase();
    e.flops_alg = f1_alg + f2_alg;
    e.flops_exec = f1_exec + f2_exec;
    return DMRG_OK;
}

// Calls f(offset, rows, cols, first term, end of its terms) for every output block.
template <class F>
void for_output(const dmrg_env_s& e, F f) {
    int g = 0;
    for (size_t o = 0; o < e.out.o.size(); ++o) {
        const BlockListDesc& b = e.out.o[o];
        for (int q = 0; q < b.count(); ++q, ++g)
            f(e.out.base[o] + b.off[q], b.rows[q], b.cols[q], e.products.first[g], e.products.first[g + 1]);
    }
}

// The split precisions: the products on the operands where they lie.  Left: stage 1
// F = B^T L (transposed A), stage 2 out += w F K; right: G = K R, out += w G B^T
// (transposed B).
int build_split(dmrg_env_s& e, cudaStream_t st) {
    const BlockListDesc& ket = e.site.ket;
    const EnvProducts& pr = e.products;
    GemmSchedule s1, s2;
    s1.ta = e.side == 0;
    s2.tb = e.side == 1;
    for (const Stage1Task& t : pr.tasks) {
        s1.add_group(t.off, t.n, t.m, t.n);
        s1.add_term(ket.off[t.ket], ket.cols[t.ket], e.in.base[t.o] + e.in.o[t.o].off[t.blk], t.n, t.k, 1.0);
    }
    for_output(e, [&](int64_t off, int m, int n, int t0, int t1) {
        s2.add_group(off, n, m, n);
        for (int i = t0; i < t1; ++i) {
            const Stage2Term& t = pr.terms[i];
            const Stage1Task& f = pr.tasks[t.task];
            s2.add_term(f.off, f.n, ket.off[t.ket], ket.cols[t.ket], f.n, t.w);
        }
    });
    DMRG_TRY(s1.check_bounds(ket.size, e.in.size, pr.scratch_size));
    DMRG_TRY(s2.check_bounds(pr.scratch_size, ket.size, e.out.size));
    const int fmt = e.precision == DMRG_PREC_BF16X3 ? kFmtBF16 : kFmtTF32;
    DMRG_TRY(e.scratch.alloc((size_t)std::max<int64_t>(pr.scratch_size, 1) * sizeof(double)));
    DMRG_TRY(e.p1.build(s1, fmt, ket.size, e.in.size, pr.scratch_size, st, e.ctx->num_sms));
    return e.p2.build(s2, fmt, pr.scratch_size, ket.size, e.out.size, st, e.ctx->num_sms);
}

}  // namespace

namespace {

// FP64: the products on packed operands (gemm_image.cu).  Real: the
// ket's images serve stage 1 (its A operand) and stage 2 (its B operand): left, both
// read K^T; right, both read K.  Complex (W: the complex MPO, a term's weight is its
// 1-based position): real forms of the blocks (gemm.cuh, ImgKind), the
// bra conjugated (left: stage 1's A operand, right: stage 2's B operand); a term's
// complex weight w G B is Re w (G B) + Im w (G (i B)).
int build_images(dmrg_env_s& e, cudaStream_t st, const double* W) {
    const BlockListDesc& ket = e.site.ket;
    const EnvProducts& pr = e.products;
    const bool z = W != nullptr;
    const int f = z ? 2 : 1;  // doubles per element
    // images (-1: not made yet): the ket as stage 1's A operand, as stage 2's B operand (and
    // times i), the input environment, the products
    std::vector<int64_t> ket_a(ket.count(), -1), ket_b[2], mid(pr.tasks.size());
    for (auto& b : ket_b) b.assign(z ? ket.count() : 0, -1);
    std::vector<std::vector<int64_t>> env(e.in.o.size());
    for (size_t o = 0; o < env.size(); ++o) env[o].assign(e.in.o[o].count(), -1);
    auto ket_image = [&](std::vector<int64_t>& at, int k, ImgKind kind, bool conj, bool times_i) {
        if (at[k] >= 0) return at[k];
        const int r = ket.rows[k], c = ket.cols[k];
        const bool t = e.side == 0;
        return at[k] = z ? e.img.add_complex(0, ket.off[k], t ? c : r, t ? r : c, c, t, kind, conj, times_i)
                         : e.img.add(0, ket.off[k], t ? c : r, t ? r : c, c, t);
    };
    e.i1.panel = e.i2.panel = ImgSchedule::panel_for((z ? 4.0 : 1.0) * e.flops_exec);
    e.i1.out = kImgOutA;
    e.i1.groups.reserve(pr.tasks.size());
    e.i1.terms.reserve(pr.tasks.size());
    e.i2.groups.reserve(pr.first.size());
    e.i2.terms.reserve(f * pr.terms.size());
    int64_t blocks = 0;
    for (size_t i = 0; i < pr.tasks.size(); ++i) {
        const Stage1Task& t = pr.tasks[i];
        if (t.m <= 0 || t.n <= 0) continue;
        mid[i] = blocks;
        e.i1.add_group(blocks, 0, t.m, f * t.n);
        blocks += img_blocks(t.m, f * t.n);
        if (t.k <= 0) continue;
        int64_t& b = env[t.o][t.blk];
        const int64_t off = e.in.base[t.o] + e.in.o[t.o].off[t.blk];
        if (b < 0)
            b = z ? e.img.add_complex(1, off, t.n, t.k, t.n, true, kImgComplexB, false, false)
                  : e.img.add(1, off, t.n, t.k, t.n, true);
        e.i1.add_term(ket_image(ket_a, t.ket, kImgComplexA, e.side == 0, false), b, f * t.k, 1.0);
    }
    // (an output block without a live term is a group too: stage 2 overwrites everything)
    for_output(e, [&](int64_t off, int m, int n, int t0, int t1) {
        e.i2.add_group(f * off, f * n, m, f * n);
        if (m <= 0 || n <= 0) return;
        for (int i = t0; i < t1; ++i) {
            const Stage2Term& t = pr.terms[i];
            const int k = pr.tasks[t.task].n;
            if (k <= 0) continue;
            if (!z) {
                e.i2.add_term(mid[t.task], ket_image(ket_a, t.ket, kImgReal, false, false), k, t.w);
                continue;
            }
            const size_t pos = (size_t)t.w - 1;
            for (int im = 0; im < 2; ++im)
                if (W[2 * pos + im] != 0.0)
                    e.i2.add_term(mid[t.task], ket_image(ket_b[im], t.ket, kImgComplexB, e.side == 1, im != 0), 2 * k,
                                  W[2 * pos + im]);
        }
    });
    DMRG_TRY(e.img.check_bounds(f * ket.size, f * e.in.size, 0));
    DMRG_TRY(e.i1.check_bounds(e.img.blocks, e.img.blocks, blocks));
    DMRG_TRY(e.i2.check_bounds(blocks, e.img.blocks, f * e.out.size));
    DMRG_TRY(e.work.finalize(e.img, e.i1, e.i2, blocks, st, e.ctx->num_sms));
    return e.work.allocate(e.i1, e.i2);
}

int run_images(dmrg_env_s& e, const double* ket_dev, const double* env_in_dev, double* env_out_dev) {
    cudaStream_t st = e.ctx->stream;
    DMRG_TRY(launch_img_pack(e.img, e.work, e.i1.panel, 0, (int)e.img.chunks.size(), ket_dev, env_in_dev, nullptr, st));
    DMRG_TRY(launch_img_gemm(e.i1, e.work.img, e.work.img, e.work.mid, false, *e.ctx));
    return launch_img_gemm(e.i2, e.work.mid, e.work.img, env_out_dev, false, *e.ctx);
}

// The common part of both creators (Wc: a complex update's MPO).
int create(dmrg_ctx_t ctx, int side, int nl, int nr, const int* phys, const dmrg_blocks_t* ket, int d, int lb, int rb,
           const double* W, const dmrg_blocks_t* env_in, int precision, const double* Wc, dmrg_env_t* out) {
    if (!ctx || !out || !env_in) return set_error(DMRG_E_ARG, "null argument");
    if (side != 0 && side != 1) return set_error(DMRG_E_ARG, "side must be 0 (left) or 1 (right)");
    if (precision != DMRG_PREC_FP64 && precision != DMRG_PREC_TF32X3 && precision != DMRG_PREC_BF16X3)
        return set_error(DMRG_E_ARG, "unknown precision %d", precision);
    *out = nullptr;
    DMRG_CUDA_TRY(cudaSetDevice(ctx->device));
    auto* e = new dmrg_env_s();
    e->ctx = ctx;
    e->side = side;
    e->precision = precision;
    int rc = build_site_desc(e->site, nl, nr, phys, ket, d, lb, rb, W);
    if (rc == DMRG_OK && !e->in.assign(env_in, side == 0 ? lb : rb))
        rc = set_error(DMRG_E_ARG, "invalid input environment");
    if (rc == DMRG_OK) rc = build_products(*e);
    cudaStream_t st = ctx->stream;
    if (rc == DMRG_OK) rc = precision == DMRG_PREC_FP64 ? build_images(*e, st, Wc) : build_split(*e, st);
    e->products = EnvProducts();
    if (rc != DMRG_OK) {
        delete e;
        return rc;
    }
    *out = e;
    return DMRG_OK;
}

}  // namespace

extern "C" {

int dmrg_env_create(dmrg_ctx_t ctx, int side, int nl, int nr, const int* phys, const dmrg_blocks_t* ket, int d,
                    int lb, int rb, const double* W, const dmrg_blocks_t* env_in, int precision, dmrg_env_t* out) {
    return create(ctx, side, nl, nr, phys, ket, d, lb, rb, W, env_in, precision, nullptr, out);
}

int dmrg_env_destroy(dmrg_env_t e) {
    delete e;
    return DMRG_OK;
}

int dmrg_env_out_info(dmrg_env_t e, int* bond, int64_t* size) {
    if (!e) return set_error(DMRG_E_ARG, "null env");
    if (bond) *bond = (int)e->out.o.size();
    if (size) *size = e->out.size;
    return DMRG_OK;
}

int dmrg_env_out_blocks(dmrg_env_t e, int o, int cap, int* nblocks, int* left, int* right, int* rows, int* cols) {
    if (!e || !nblocks) return set_error(DMRG_E_ARG, "null argument");
    if (o < 0 || o >= (int)e->out.o.size()) return set_error(DMRG_E_ARG, "bond index %d out of range", o);
    const BlockListDesc& b = e->out.o[o];
    *nblocks = b.count();
    if (cap < b.count()) return cap == 0 ? DMRG_OK : set_error(DMRG_E_ARG, "capacity %d < %d", cap, b.count());
    for (int k = 0; k < b.count(); ++k) {
        if (left) left[k] = b.left[k];
        if (right) right[k] = b.right[k];
        if (rows) rows[k] = b.rows[k];
        if (cols) cols[k] = b.cols[k];
    }
    return DMRG_OK;
}

int dmrg_env_flops(dmrg_env_t e, double* alg, double* exec) {
    if (!e) return set_error(DMRG_E_ARG, "null env");
    if (alg) *alg = e->flops_alg;
    if (exec) *exec = e->flops_exec;
    return DMRG_OK;
}

int dmrg_env_apply(dmrg_env_t e, const double* ket_dev, const double* env_in_dev, double* env_out_dev) {
    if (!e) return set_error(DMRG_E_ARG, "null env");
    // Both sides: stage 1 reads (ket, env_in), stage 2 its products and the ket.
    if (e->cplx) return set_error(DMRG_E_STATE, "a complex environment update runs through dmrg_zenv_apply");
    if (e->precision != DMRG_PREC_FP64) {  // tcgen05 split products, FP64 sums and FP64 storage
        cudaStream_t st = e->ctx->stream;
        if (e->out.size) DMRG_CUDA_TRY(cudaMemsetAsync(env_out_dev, 0, (size_t)e->out.size * sizeof(double), st));
        DMRG_TRY(e->p1.run(ket_dev, env_in_dev, e->scratch.as<double>(), false, e->ctx->d_status, st));
        DMRG_TRY(e->p2.run(e->scratch.as<double>(), ket_dev, env_out_dev, true, e->ctx->d_status, st));
        return DMRG_OK;
    }
    return run_images(*e, ket_dev, env_in_dev, env_out_dev);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// The complex path: ComplexTensorContraction::Left/RightComputeTensorContraction
// (src/dmrg/complexdmrg/complex_tensor_contraction.cc:800-975, 977-1150) have
// the real structure with the bra block Hermitian-conjugated
// (HermitianConjugateMatrix, :929, :1113) and a complex MPO.  The real builder
// runs on a surrogate MPO whose nonzero entries are the (1-based) positions of
// the complex entries that are nonzero (|w| != 0 exactly where the complex
// reference takes the term), so the output block maps follow the same
// zero_flag pass; build_images then takes the complex entry at each term's
// position as its weight, with the conjugation on the bra operand.
// ---------------------------------------------------------------------------
extern "C" {

int dmrg_zenv_create(dmrg_ctx_t ctx, int side, int nl, int nr, const int* phys, const dmrg_blocks_t* ket, int d,
                     int lb, int rb, const double* W, const dmrg_blocks_t* env_in, dmrg_env_t* out) {
    if (!W || lb <= 0 || rb <= 0 || d <= 0 || !out) return set_error(DMRG_E_ARG, "null argument");
    const size_t nw = (size_t)lb * rb * d * d;
    std::vector<double> ids(nw, 0.0);
    for (size_t i = 0; i < nw; ++i)
        if (W[2 * i] != 0.0 || W[2 * i + 1] != 0.0) ids[i] = (double)(i + 1);
    DMRG_TRY(create(ctx, side, nl, nr, phys, ket, d, lb, rb, ids.data(), env_in, DMRG_PREC_FP64, W, out));
    dmrg_env_s* e = *out;
    e->cplx = true;
    e->flops_alg *= 4.0;  // a complex product is four real ones
    e->flops_exec *= 4.0;
    return DMRG_OK;
}

int dmrg_zenv_apply(dmrg_env_t e, const double* ket_dev, const double* env_in_dev, double* env_out_dev) {
    if (!e || !e->cplx) return set_error(DMRG_E_ARG, "not a complex environment update (dmrg_zenv_create)");
    return run_images(*e, ket_dev, env_in_dev, env_out_dev);
}

}  // extern "C"
