// FP64 grouped multi-term block GEMM on packed operand images (gemm.cuh), on the
// FP64 tensor path (DMMA, mma.sync.m8n8k4.f64; tcgen05 has no f64 kind).
//
// Why packed.  The raw blocks are ragged (1 to ~200 rows) with offsets and leading
// dimensions of any parity, so neither TMA tensor maps nor 16-byte loads fit them,
// and 8-byte cp.async, with their addresses, cost as much time as they leave for
// DMMAs (gemm_f64.cu: 77% DMMA pipe, but 1.5 times the algorithmic FLOPs in
// padding; with the padding trimmed the same loads hold the pipe at 64%).  Every
// operand tile is read by several tiles and terms, so the blocks are packed once
// per application, in the order in which a warp's lanes hold DMMA fragments: a
// k-step's operands are then two bulk copies (cp.async.bulk, up to 16 KB each), a
// fragment pair is one conflict-free 16-byte shared load, k needs no masks, and
// the first product of a chain leaves its result as the next one's image with
// fully coalesced 512-byte stores.
//
// Complex products run as real ones of twice the columns and k (ImgKind): same DMMAs
// as four real products per complex one, and the same kernel.
//
// GEMM CTA: four consumer warps (2 x 2 quarters of the tile, MI x NJ units of 8x8
// each) and a producer warp that issues the copies; steps are handed over by
// mbarriers, so warps and tiles overlap.  All waits are bounded (kWaitPolls, or the
// context's limit): a warp whose wait gives up sets the status word and leaves, before it
// uses anything that the wait was for; the others' waits on it then run out too.
//
// Split of the work: two persistent CTAs per SM take tiles, largest first, from a
// queue (equal shares dealt out beforehand left SMs idle for a fifth of a D=1024
// launch: the time of a step depends on what the SM's other CTA runs).  A long tile
// is cut into parts, summed in order by the last CTA to finish one.
//
// Measured, one H_eff*psi of the 8x4 cylinder's middle site: D=1024 216 -> 186 us
// (pack 10, first stage 70, second 105; its DMMAs alone 104 us at the 37 TFLOP/s of
// a register-only loop), D=300 59 -> 22.5 us, 16-site chain at D=64 21.5 -> 14.8 us.
// What bounds it now: at D=1024 the DMMA pipe (75% busy; the rest is the tiles'
// epilogues with one other CTA to cover them, and the last tiles); below D~300 three
// launches' latency and the k-step chain of one tile.
#include <algorithm>
#include <atomic>

#include "gemm.cuh"

namespace dmrg {
namespace {

constexpr int kConsumers = 128;            // threads of the four consumer warps
constexpr int kThreads = kConsumers + 32;  // and the producer warp

constexpr int kCtasPerSm = 2;
constexpr int kRegs = 168;                     // per thread: at most 3 of the 10 warps share a sub-core's registers
// Operand ring.  A step takes only the space of its own blocks, so that narrow
// tiles keep many steps in flight.
constexpr int kSlots = 16;                     // steps in flight, at most
constexpr int kRing = 106 * 1024;              // bytes
constexpr int kPad = kImgSlice * kImgBlock * 8;  // a quarter with an odd unit reads one unit further

struct Tile {  // a segment, as the consumers need it
    int64_t c_off, aux_off;
    int ldc, rows, cols, pm, pn, out_kb, steps, split;
};
struct StepMeta {  // of the step in a slot
    double scale;
    int kb;        // blocks of k
    int off;       // its operands in the ring (bytes): A's blocks, then B's
};
constexpr int kTiles = kSlots + 1;  // every tile has a step
struct Shared {
    StepMeta meta[kSlots];
    uint64_t full[kSlots], empty[kSlots], met;
    Tile tiles[kTiles];
    int last;
    int gave_up;  // a consumer has
    int issued;   // steps, once the producer is through
};
constexpr size_t kSmem = kRing + kPad + sizeof(Shared);

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, int count) {
    asm volatile("mbarrier.init.shared.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
// Waits for the barrier's phase `parity`; false when it gave up after `polls` tries
// (at least one).
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, int polls) {
    for (int n = 1;; ++n) {
        unsigned done;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if (n >= polls) return false;
    }
}
// The same for a whole warp, which agrees: false when any lane gave up.
__device__ __forceinline__ bool warp_wait(unsigned bar, unsigned parity, int polls) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, polls));
}
__device__ __forceinline__ void bulk_copy(unsigned dst, const double* src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// Launches are chained (launch_pdl): D=300 matvec 30 -> 22.5 us.  The pack kernel lets
// the next launch in early (launch_next); the GEMM kernel leaves it to its CTAs' exits
// (the next launch's waiting CTAs would take the shared memory of its own: Lanczos at
// D=512 1.27 -> 1.33 ms).

// The four consumer warps meet; false when one of them did not come (it gave up).  An
// mbarrier: bar.sync would wait for ever for a warp that has left.
__device__ __forceinline__ bool consumers_meet(unsigned bar, int& meetings, int polls) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
    return warp_wait(bar, meetings++ & 1, polls);
}

__device__ __forceinline__ void dmma_8x8x4(double& d0, double& d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

struct GemmArgs {
    const double *A, *B;
    double *C, *aux;
    const ImgTerm* terms;
    const ImgSegment* segments;
    int nsegments;
    int units;        // 8-row units of a full panel
    const GemmSplit* splits;
    unsigned* tickets;  // the queue's counter, then the split tiles'; zero at the start
    int* status;
    int polls;          // of a bounded wait
    int accumulate;
};

// Where a tile's units go in an image output: the image's rows are the tile's
// columns (B roles) or rows (A role), its k indices the other side's (twice, in the
// complex B role).
template <int OUT>
struct ImageOut {
    static constexpr bool kByColumn = OUT == kImgOutB || OUT == kImgOutZB;
    static constexpr int kPer = OUT == kImgOutZB ? 2 : 1;  // k units per unit of the tile
    double* base;   // the panel's first block
    int units, k0;  // row units of the panel; k unit of the tile's first unit
    int kb_all;
    __device__ __forceinline__ ImageOut(const GemmArgs& w, const Tile& g) {
        units = ((kByColumn ? g.cols : g.rows) + 7) >> 3;
        k0 = (kByColumn ? g.pm : g.pn) * w.units * kPer;
        kb_all = g.out_kb;
        base = w.C + (g.c_off + (int64_t)(kByColumn ? g.pn : g.pm) * w.units * g.out_kb) * kImgBlock;
    }
    // Block of k unit `k` (of the tile) and row unit 0; `pitch`: to the next row unit.
    __device__ __forceinline__ double* column(int k, int& pitch) const {
        const int s = (k0 + k) / kImgSlice;
        pitch = min(kImgSlice, kb_all - s * kImgSlice) * kImgBlock;
        return base + (units * s * kImgSlice + (k0 + k) % kImgSlice) * kImgBlock;
    }
    // Offset in a block of the lane's pair (row fr, columns 2 fc and 2 fc + 1 of a
    // unit; complex: in the block of k unit fr / 4 of the unit's two), and from the
    // first element of the pair to the second.
    static __device__ __forceinline__ int pair(int fr, int fc) {
        if (OUT == kImgOutB) return (4 * (2 * fc) + (fr & 3)) * 2 + (fr >> 2);
        if (OUT == kImgOutA) return (4 * fr + ((2 * fc) & 3)) * 2 + (fc >> 1);
        return (4 * (2 * fc) + 2 * (fr & 1)) * 2 + ((fr & 3) >> 1);
    }
    static constexpr int kStep = OUT == kImgOutA ? 2 : 8;
};

// The consumer warps' work on one tile or part.  The unit counts are template
// parameters of the whole loop (as run-time counts, or in a switch inside it, the
// accumulators move between registers at every step).  SCALED: terms have scales
// other than 1 (the products cost ~8% of the loop).  False when a wait gave up.
template <int OUT, bool SCALED, int MI, int NJ>
__device__ __forceinline__ bool run_tile(const GemmArgs& w, const Tile& g, const char* ring, Shared& sh, unsigned full,
                                         unsigned empty, int& step, int& meetings) {
    const StepMeta* meta = sh.meta;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int um0 = (warp >> 1) * MI, un0 = (warp & 1) * NJ, ua = (g.rows + 7) >> 3;
    double acc[MI][NJ][2];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    auto block = [&](const double2* As, const double2* Bs, int stride, double scale) {
        double2 a[MI], b[NJ];
#pragma unroll
        for (int i = 0; i < MI; ++i) {
            a[i] = As[i * stride];
            if (SCALED) {
                a[i].x *= scale;
                a[i].y *= scale;
            }
        }
#pragma unroll
        for (int j = 0; j < NJ; ++j) b[j] = Bs[j * stride];
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], a[i].x, b[j].x);
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], a[i].y, b[j].y);
    };
#pragma unroll 1
    for (int n = max(g.steps, 1); n > 0; --n) {  // (one empty step without terms)
        const int s = step % kSlots;
        const bool got = mbar_wait(full + 8 * s, (step / kSlots) & 1, w.polls);
        // Read ahead of the vote, used only after it.  (The vote stands in both branches: ahead
        // of them it costs an environment update at D=1024 3 us of 171.)
        const double scale = SCALED ? meta[s].scale : 1.0;
        const int kb = meta[s].kb, off = meta[s].off;
        const double2* As = reinterpret_cast<const double2*>(ring + off) + lane;
        const double2* Bs = As + ua * kb * 32;
        if (kb == kImgSlice) {
            if (!__all_sync(0xffffffffu, got)) return false;
#pragma unroll
            for (int q = 0; q < kImgSlice; ++q)
                block(As + (um0 * kImgSlice + q) * 32, Bs + (un0 * kImgSlice + q) * 32, kImgSlice * 32, scale);
        } else {
            if (!__all_sync(0xffffffffu, got)) return false;
#pragma unroll 1
            for (int q = 0; q < kb; ++q) block(As + (um0 * kb + q) * 32, Bs + (un0 * kb + q) * 32, kb * 32, scale);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty + 8 * s);
        ++step;
    }
    if (g.split >= 0) {
        // A part of a cut tile goes to the aux buffer as the threads hold it; the last CTA
        // to finish one of the tile's parts sums them, in order.
        const GemmSplit sp = w.splits[g.split];
        constexpr int kPart = MI * NJ * kConsumers;  // double2 per part
        double2* part = reinterpret_cast<double2*>(w.aux + g.aux_off) + threadIdx.x;
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) part[(i * NJ + j) * kConsumers] = make_double2(acc[i][j][0], acc[i][j][1]);
        const unsigned met = smem_u32(&sh.met);
        if (!consumers_meet(met, meetings, w.polls)) return false;  // every warp's part is written before the ticket is taken
        if (threadIdx.x == 0) {
            unsigned before;
            asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;\n"
                         : "=r"(before)
                         : "l"(w.tickets + 1 + sp.ticket)
                         : "memory");
            sh.last = before == (unsigned)sp.chunks - 1;
        }
        if (!consumers_meet(met, meetings, w.polls)) return false;
        if (!sh.last) return true;
#pragma unroll
        for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
        const double2* src = reinterpret_cast<const double2*>(w.aux + sp.aux_off) + threadIdx.x;
#pragma unroll 1
        for (int ch = 0; ch < sp.chunks; ++ch, src += kPart) {
            double2 v[MI][NJ];
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j) v[i][j] = __ldcg(src + (i * NJ + j) * kConsumers);
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    acc[i][j][0] += v[i][j].x;
                    acc[i][j][1] += v[i][j].y;
                }
        }
    }
    const int fr = lane >> 2, fc = lane & 3;
    if constexpr (OUT != kImgOutBlock) {  // whole units, zero outside the block
        using Image = ImageOut<OUT>;
        const Image image(w, g);
        const int el = Image::pair(fr, fc), rleft = g.rows - 8 * um0 - fr, cleft = g.cols - 8 * un0 - 2 * fc;
        constexpr bool kCol = Image::kByColumn;
        constexpr int KU = kCol ? MI : NJ, XU = kCol ? NJ : MI;  // k units, row units
#pragma unroll
        for (int k = 0; k < KU; ++k) {
            const int ku = ((kCol ? um0 : un0) + k) * Image::kPer + (OUT == kImgOutZB ? fr >> 2 : 0);
            if (image.k0 + ku >= image.kb_all) continue;
            int pitch;
            double* col = image.column(ku, pitch) + el;
#pragma unroll
            for (int x = 0; x < XU; ++x) {
                const int i = kCol ? k : x, j = kCol ? x : k;
                if (8 * (um0 + i) >= g.rows || 8 * (un0 + j) >= g.cols) continue;
                double* o = col + ((kCol ? un0 : um0) + x) * pitch;
                const double v0 = 8 * i < rleft && 8 * j < cleft ? acc[i][j][0] : 0.0;
                const double v1 = 8 * i < rleft && 8 * j + 1 < cleft ? acc[i][j][1] : 0.0;
                o[0] = v0;
                o[Image::kStep] = v1;
                if (OUT == kImgOutZB) {  // v0 + i v1: [[v0, -v1], [v1, v0]]
                    o[2] = -v1;
                    o[Image::kStep + 2] = v0;
                }
            }
        }
        return true;
    }
    const bool add = w.accumulate;
    double* crow = w.C + g.c_off + (int64_t)(8 * um0 + fr) * g.ldc + 8 * un0 + 2 * fc;
    const int rleft = g.rows - 8 * um0 - fr, cleft = g.cols - 8 * un0 - 2 * fc;
#pragma unroll
    for (int i = 0; i < MI; ++i, crow += 8 * (int64_t)g.ldc) {
        if (8 * i >= rleft) break;
        double old[NJ][2];
        if (add) {
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) old[j][e] = 8 * j + e < cleft ? crow[8 * j + e] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (8 * j + e < cleft) crow[8 * j + e] = add ? old[j][e] + acc[i][j][e] : acc[i][j][e];
    }
    return true;
}

// The producer warp: takes segments from the queue (its first is its CTA's own) and
// issues every step's copies in order.  The next segment's index, descriptor and
// first terms are requested after this segment's first, second and third step, so
// that each round trip passes behind a step (in one go, they held the first stage at
// D=1024 at 75 us).  A segment's terms are read 32 at a time, one per lane.
__device__ __forceinline__ void produce(const GemmArgs& w, char* ring, Shared& sh) {
    const int lane = threadIdx.x & 31;
    const unsigned full = smem_u32(sh.full), empty = smem_u32(sh.empty);
    bool ok = true;
    int n = 0, oldest = 0;   // steps issued; the oldest one not released yet
    int head = 0, tail = 0;  // ring: end of the newest step, start of the oldest
    // room for a step of `need` bytes: after the newest one, or at the ring's start; < 0: gave up
    auto room = [&](int need) {
        for (;;) {
            int at;
            if (oldest == n) at = 0;
            else if (n - oldest == kSlots) at = -1;
            else if (head > tail) at = head + need <= kRing ? head : need <= tail ? 0 : -1;
            else at = head + need <= tail ? head : -1;
            if (at >= 0) {
                if (oldest == n) tail = at;
                head = at + need;
                return at;
            }
            if (!warp_wait(empty + 8 * (oldest % kSlots), (oldest / kSlots) & 1, w.polls)) return -1;
            if (++oldest < n) tail = sh.meta[oldest % kSlots].off;
        }
    };
    auto term_of = [&](const ImgSegment& g, int t) { return w.terms[min(g.t0 + t, g.t1)]; };  // entry t1 is readable
    auto segment = [&](int i) { return w.segments[min(i, w.nsegments - 1)]; };
    int idx = blockIdx.x, claim = 0, tiles = 0;
    ImgSegment next = segment(idx);
    ImgTerm first = term_of(next, lane);
    wait_previous();  // the operands; before any step, so the consumers' writes are ordered as well
    for (; idx < w.nsegments && ok; ++tiles) {
        const ImgSegment g = next;
        ImgTerm mine = first;
        int ahead = 0;
        auto look_ahead = [&]() {
            if (ahead == 0) {
                if (lane == 0) claim = (int)(gridDim.x + atomicAdd(w.tickets, 1u));
            } else if (ahead == 1) {
                idx = __shfl_sync(0xffffffffu, claim, 0);
                next = segment(idx);
            } else if (ahead == 2) {
                first = term_of(next, lane);
            }
            ++ahead;
        };
        const int ua = (g.rows + 7) >> 3, ub = (g.cols + 7) >> 3;
        int ti = 0, slice = g.k0;
        for (int left = max(g.steps, 1); left > 0; --left) {  // a segment without terms: one empty step
            int64_t ta = 0, tb = 0;
            int tkb = 0;
            double scale = 1.0;
            if (g.steps > 0) {
                for (;;) {
                    tkb = __shfl_sync(0xffffffffu, mine.kb, ti & 31);
                    if (slice * kImgSlice < tkb) break;
                    slice = 0;
                    if ((++ti & 31) == 0) mine = term_of(g, ti + lane);
                }
                ta = __shfl_sync(0xffffffffu, mine.a, ti & 31);
                tb = __shfl_sync(0xffffffffu, mine.b, ti & 31);
                scale = __shfl_sync(0xffffffffu, mine.scale, ti & 31);
            }
            const int kb = min(kImgSlice, tkb - slice * kImgSlice), bytes = kb * kImgBlock * 8, need = (ua + ub) * bytes;
            const int at = room(need);
            ok = at >= 0;
            if (!ok) break;
            const int s = n % kSlots;
            if (lane == 0) {
                if (left == max(g.steps, 1))
                    sh.tiles[tiles % kTiles] = Tile{g.c_off, g.aux_off, g.ldc, g.rows, g.cols, g.pm, g.pn, g.out_kb, g.steps, g.split};
                sh.meta[s].scale = scale;
                sh.meta[s].kb = kb;
                sh.meta[s].off = at;
                const unsigned dst = smem_u32(ring) + at;
                const int64_t panel = (int64_t)w.units * tkb;
                mbar_expect(full + 8 * s, need);
                if (need) {
                    bulk_copy(dst, w.A + (ta + g.pm * panel + ua * slice * kImgSlice) * kImgBlock, ua * bytes, full + 8 * s);
                    bulk_copy(dst + ua * bytes, w.B + (tb + g.pn * panel + ub * slice * kImgSlice) * kImgBlock, ub * bytes,
                              full + 8 * s);
                }
            }
            __syncwarp();
            ++slice;
            ++n;
            look_ahead();
        }
        while (ahead < 3) look_ahead();
    }
    // the end: a step without a tile
    if (ok) ok = room(0) >= 0;
    if (lane == 0) {
        if (ok) {
            sh.tiles[tiles % kTiles].steps = -1;
            mbar_expect(full + 8 * (n % kSlots), 0);
        } else {  // gave up: the consumers have, or will
            if (w.status) *w.status = DMRG_E_NUMERIC;
        }
    }
    // No copy is in flight when the CTA leaves.  The consumers have waited for them all,
    // unless one gave up: one that does so later than this finds `issued`.
    if (lane == 0) *const_cast<volatile int*>(&sh.issued) = n;
    __threadfence_block();
    if (!ok || *const_cast<volatile int*>(&sh.gave_up))
        for (int i = oldest; i < n; ++i) warp_wait(full + 8 * (i % kSlots), (i / kSlots) & 1, kWaitPolls);
}

template <int OUT, bool SCALED>
__global__ void __maxnreg__(kRegs) img_gemm_kernel(const GemmArgs w) {
    extern __shared__ __align__(128) char ring[];
    Shared& sh = *reinterpret_cast<Shared*>(ring + kRing + kPad);
    const unsigned full = smem_u32(sh.full), empty = smem_u32(sh.empty);
    if (threadIdx.x == 0) {
        for (int s = 0; s < kSlots; ++s) {
            mbar_init(full + 8 * s, 1);
            mbar_init(empty + 8 * s, kConsumers / 32);
        }
        mbar_init(smem_u32(&sh.met), kConsumers / 32);
        sh.gave_up = sh.issued = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x >= kConsumers) {
        produce(w, ring, sh);
        return;
    }
    // A warp that gives up says so, and waits (with the full limit) for the copies that the
    // producer may have left in flight; one that is still issuing sees to them itself.
    auto give_up = [&](int step) {
        if (w.status) *w.status = DMRG_E_NUMERIC;
        *const_cast<volatile int*>(&sh.gave_up) = 1;
        __threadfence_block();
        const int issued = *const_cast<volatile int*>(&sh.issued);
        for (int i = step; i < issued; ++i) mbar_wait(full + 8 * (i % kSlots), (i / kSlots) & 1, kWaitPolls);
    };
    int step = 0, meetings = 0;  // steps computed (slot = step % kSlots, its phase = step / kSlots); of the warps
#pragma unroll 1
    for (int tile = 0;; ++tile) {
        // the tile's first step carries its descriptor (a lowered limit also caps the tiles,
        // so that a test can stop a launch part of the way)
        bool ok = tile < w.polls && warp_wait(full + 8 * (step % kSlots), (step / kSlots) & 1, w.polls);
        if (!ok) return give_up(step);
        const Tile g = sh.tiles[tile % kTiles];
        if (g.steps < 0) return;
        switch (((g.rows + 15) >> 4) * 4 + ((g.cols + 15) >> 4) - 5) {  // units per warp
#define DMRG_UNITS(MI, NJ)                                                                        \
    case (MI - 1) * 4 + NJ - 1:                                                                   \
        ok = run_tile<OUT, SCALED, MI, NJ>(w, g, ring, sh, full, empty, step, meetings);          \
        break;
#define DMRG_UNIT_ROW(MI) DMRG_UNITS(MI, 1) DMRG_UNITS(MI, 2) DMRG_UNITS(MI, 3) DMRG_UNITS(MI, 4)
            DMRG_UNIT_ROW(1)
            DMRG_UNIT_ROW(2)
            DMRG_UNIT_ROW(3)
            DMRG_UNIT_ROW(4)
#undef DMRG_UNIT_ROW
#undef DMRG_UNITS
            default: break;
        }
        if (!ok) return give_up(step);
    }
}

// Element (r, c) of a job's image (zero outside it).
template <bool COMPLEX>
__device__ __forceinline__ double image_element(const ImgJob& j, const double* __restrict__ src, int r, int c) {
    if (r >= j.image_rows() || c >= j.image_k()) return 0.0;
    if (!COMPLEX || j.kind == kImgReal) return src[j.trans ? (int64_t)c * j.ld + r : (int64_t)r * j.ld + c];
    const bool b = j.kind == kImgComplexB;
    const int zr = b ? r >> 1 : r, zc = c >> 1;
    // part 0: re z, 1: im z, with the B form's sign
    int part = b ? (r ^ c) & 1 : c & 1;
    double sign = b && (r & 1) == 0 && part ? -1.0 : 1.0;
    if (j.times_i) {  // re (i x) = -im x, im (i x) = re x
        if (part == 0) sign = -sign;
        part ^= 1;
    }
    if (j.conj && part) sign = -sign;
    return sign * src[2 * (j.trans ? (int64_t)zc * j.ld + zr : (int64_t)zr * j.ld + zc) + part];
}

// One (panel, slice) of a job per CTA; thread = lane of a block: two elements of the
// image (k indices 4 apart) to one 16-byte store.  Real: a warp reads 8 rows of 32 +
// 32 contiguous bytes (or, transposed, 4 + 4 rows of 64) and writes 512.  The first CTA
// also zeroes the counters of the products that follow: every application starts from
// zero, whatever became of the one before.
constexpr int kPackThreads = 256;
template <bool COMPLEX>
__global__ void __launch_bounds__(kPackThreads) img_pack_kernel(const ImgJob* __restrict__ jobs,
                                                                const ImgChunk* __restrict__ chunks, int nchunks,
                                                                unsigned* __restrict__ tickets, int ntickets, int panel,
                                                                const double* __restrict__ s0,
                                                                const double* __restrict__ s1,
                                                                const double* __restrict__ s2,
                                                                double* __restrict__ img) {
    const bool chunk = (int)blockIdx.x < nchunks;  // (a launch without chunks has one CTA)
    const ImgChunk ch = chunk ? chunks[blockIdx.x] : ImgChunk{};
    const ImgJob j = chunk ? jobs[ch.job] : ImgJob{};
    launch_next();
    wait_previous();  // the sources are written, and the images' last readers are done
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < ntickets; i += kPackThreads) tickets[i] = 0u;
    if (!chunk) return;
    const double* src = (j.src == 0 ? s0 : j.src == 1 ? s1 : s2) + j.src_off;
    const int kb_all = (j.image_k() + 7) >> 3, kb = min(kImgSlice, kb_all - ch.slice * kImgSlice);
    const int r0 = ch.panel * panel, units = (min(panel, j.image_rows() - r0) + 7) >> 3, k0 = ch.slice * kImgSlice * 8;
    double2* out = reinterpret_cast<double2*>(img) +
                   (j.img + (int64_t)ch.panel * (panel / 8) * kb_all + (int64_t)units * ch.slice * kImgSlice) * 32;
    const int lane = threadIdx.x & 31;
    for (int b = threadIdx.x >> 5; b < units * kb; b += kPackThreads / 32) {
        const int u = b / kb, q = b - u * kb;
        const int r = r0 + 8 * u + (lane >> 2), c = k0 + 8 * q + (lane & 3);
        out[(int64_t)b * 32 + lane] =
            make_double2(image_element<COMPLEX>(j, src, r, c), image_element<COMPLEX>(j, src, r, c + 4));
    }
}

// The kernels' dynamic shared memory is above the 48 KB default: raises their
// allowance, once per device.  Made when a product is planned, so that no launch inside
// a stream capture has to make it.
int allow_smem() {
    static std::atomic<bool> done[64] = {};
    int dev = 0;
    DMRG_CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && done[dev].load(std::memory_order_acquire)) return DMRG_OK;
    using Kernel = void (*)(const GemmArgs);
    for (Kernel k : {Kernel(img_gemm_kernel<kImgOutBlock, false>), Kernel(img_gemm_kernel<kImgOutBlock, true>),
                     Kernel(img_gemm_kernel<kImgOutB, false>), Kernel(img_gemm_kernel<kImgOutA, false>),
                     Kernel(img_gemm_kernel<kImgOutZB, false>)})
        DMRG_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
    if (dev >= 0 && dev < 64) done[dev].store(true, std::memory_order_release);
    return DMRG_OK;
}

template <int OUT, bool SCALED>
int launch(int n, const GemmArgs& w, cudaStream_t st) {
    return launch_pdl(img_gemm_kernel<OUT, SCALED>, dim3(n), kThreads, kSmem, st, w);
}

// The schedule's cost model (cycles of a step and of a tile's own work) and cuts.
constexpr int64_t kStepFixed = 400, kTileFixed = 2000;
// k-steps of a part of a cut tile, at least: a part costs a round trip through the aux
// buffer (D=300: 22.5 us; with parts of 4 steps 26.5, of 2 steps 40, uncut 28).
constexpr int kMinPart = 8;
// Products below use 32-wide tiles, see panel_for.
constexpr double kSmallFlops = 4e8;

// One k-step of a tile: 16 cycles per DMMA and sub-core.
int64_t step_cost(int rows, int cols) {
    return (int64_t)((rows + 15) / 16) * ((cols + 15) / 16) * kImgSlice * 2 * 16 + kStepFixed;
}
int steps_of(const ImgTerm& t) { return (t.kb + kImgSlice - 1) / kImgSlice; }

}  // namespace

int64_t ImgPack::add(int src, int64_t src_off, int rows, int k, int ld, bool trans) {
    const int64_t img = blocks;
    jobs.push_back(ImgJob{src_off, img, rows, k, ld, trans ? 1 : 0, src, kImgReal, 0, 0});
    blocks += img_blocks(rows, k);
    return img;
}

int64_t ImgPack::add_complex(int src, int64_t src_off, int rows, int k, int ld, bool trans, ImgKind kind, bool conj,
                             bool times_i) {
    const int64_t img = blocks;
    const ImgJob j{2 * src_off, img, rows, k, ld, trans ? 1 : 0, src, kind, conj ? 1 : 0, times_i ? 1 : 0};
    jobs.push_back(j);
    blocks += img_blocks(j.image_rows(), j.image_k());
    complex = true;
    return img;
}

int ImgPack::check_bounds(int64_t n0, int64_t n1, int64_t n2) const {
    const int64_t sizes[3] = {n0, n1, n2};
    for (const ImgJob& j : jobs) {
        if (j.rows <= 0 || j.k <= 0) continue;
        const int64_t count = j.trans ? (int64_t)(j.k - 1) * j.ld + j.rows : (int64_t)(j.rows - 1) * j.ld + j.k;
        const int64_t end = j.src_off + (j.kind == kImgReal ? count : 2 * count);
        if (j.src_off < 0 || end > sizes[j.src])
            return set_error(DMRG_E_ARG, "packed operand %lld (%dx%d, ld %d) outside %lld", (long long)j.src_off, j.rows, j.k,
                             j.ld, (long long)sizes[j.src]);
    }
    return DMRG_OK;
}

void ImgPack::plan(int panel, Tables& tab) {
    chunks.clear();
    first_chunk.assign(1, 0);
    for (int j = 0; j < (int)jobs.size(); ++j) {
        const int slices = (int)((img_units(jobs[j].image_k()) + kImgSlice - 1) / kImgSlice);
        for (int p = 0; p * panel < jobs[j].image_rows(); ++p)
            for (int s = 0; s < slices; ++s) chunks.push_back(ImgChunk{j, p, s, 0});
        first_chunk.push_back((int)chunks.size());
    }
    jobs_at = tab.add(jobs);
    chunks_at = tab.add(chunks);
}

int launch_img_pack(const ImgPack& p, const ImgWork& work, int panel, int c0, int c1, const double* s0, const double* s1,
                    const double* s2, cudaStream_t stream) {
    const int n = std::max(c1 - c0, 0);
    if (n == 0 && work.ntickets == 0) return DMRG_OK;
    return launch_pdl(p.complex ? img_pack_kernel<true> : img_pack_kernel<false>, dim3(std::max(n, 1)), kPackThreads, 0,
                      stream, reinterpret_cast<const ImgJob*>(p.tables + p.jobs_at),
                      reinterpret_cast<const ImgChunk*>(p.tables + p.chunks_at) + c0, n, work.tickets, work.ntickets, panel,
                      s0, s1, s2, work.img);
}

// A 64x64 tile's k-step takes a CTA about a microsecond: with few of them, whole
// blocks sit on few SMs.  Both widths measured: D=300 (0.1 GFLOP) 22.5 us in 32-wide
// tiles, 28 us in 64-wide ones; D=512 (0.5 GFLOP) the same to 2%; D=1024 64-wide,
// whose operand traffic is half.
int ImgSchedule::panel_for(double flops) { return flops < kSmallFlops ? 32 : 64; }

int ImgSchedule::check_bounds(int64_t a_blocks, int64_t b_blocks, int64_t out_size) const {
    for (const ImgGroup& g : groups) {
        if (g.m <= 0 || g.n <= 0) continue;
        const int64_t end = out == kImgOutBlock ? g.c_off + (int64_t)(g.m - 1) * g.ldc + g.n
                            : g.c_off + img_blocks(out == kImgOutZB ? g.n : g.m, out == kImgOutZB ? 2 * g.m : g.n);
        if (g.c_off < 0 || end > out_size || (out == kImgOutBlock && g.n > g.ldc))
            return set_error(DMRG_E_ARG, "packed GEMM output %lld (%dx%d) outside %lld", (long long)g.c_off, g.m, g.n,
                             (long long)out_size);
        for (int t = g.t0; t < g.t1; ++t) {
            const ImgTerm& x = terms[t];
            if (x.k <= 0) continue;
            if (x.a < 0 || x.b < 0 || x.a + img_blocks(g.m, x.k) > a_blocks || x.b + img_blocks(g.n, x.k) > b_blocks)
                return set_error(DMRG_E_ARG, "packed GEMM operand outside its images");
        }
    }
    return DMRG_OK;
}

void ImgSchedule::plan(int num_sms, Tables& tab) {
    segments.clear();
    splits.clear();
    aux_size = 0;
    ntickets = 0;
    scaled = false;
    if (num_sms <= 0) num_sms = 148;
    std::vector<ImgTerm> live;  // terms with k-steps, by group
    struct Tile {
        int group, t0, t1;      // its group's live terms
        int pm, pn, rows, cols;
        int64_t steps, cost;    // k-steps; cycles of one
        int64_t parts;
    };
    std::vector<Tile> tiles;
    live.reserve(terms.size() + 1);
    tiles.reserve(2 * groups.size());
    int64_t cost = 0;
    for (int gi = 0; gi < (int)groups.size(); ++gi) {
        const ImgGroup& g = groups[gi];
        if (g.m <= 0 || g.n <= 0) continue;
        const int t0 = (int)live.size();
        int64_t ks = 0;
        for (int t = g.t0; t < g.t1; ++t)
            if (terms[t].k > 0) {
                live.push_back(terms[t]);
                scaled = scaled || terms[t].scale != 1.0;
                ks += steps_of(terms[t]);
            }
        for (int pm = 0; pm * panel < g.m; ++pm)
            for (int pn = 0; pn * panel < g.n; ++pn) {
                Tile t{gi, t0, (int)live.size(), pm, pn, std::min(panel, g.m - pm * panel), std::min(panel, g.n - pn * panel),
                       ks, 0, 1};
                t.cost = step_cost(t.rows, t.cols);
                cost += ks * t.cost + kTileFixed;
                tiles.push_back(t);
            }
    }
    // a tile longer than a quarter of a CTA's share is cut into equal parts (a sixth or a
    // tenth: no gain at D=1024)
    const int64_t longest = std::max<int64_t>(1, cost / ((int64_t)num_sms * kCtasPerSm) / 4);
    // The queue: largest first, in classes of 1/1024 of the largest (as fast as exactly
    // sorted; planning is on a sweep's path, and there a sort counts).
    constexpr int kClasses = 1024;
    int64_t most = 1;
    for (Tile& t : tiles) {
        t.parts = std::max<int64_t>(1, std::min((t.steps * t.cost + longest - 1) / longest, t.steps / kMinPart));
        most = std::max(most, (t.steps + t.parts - 1) / t.parts * t.cost);
    }
    auto first_step = [](const Tile& t, int64_t part) { return t.steps * part / t.parts; };
    auto class_of = [&](int64_t c) { return (int)((kClasses - 1) - c * (kClasses - 1) / most); };
    std::vector<int> next(kClasses + 1, 0);  // where a class's next segment goes
    for (const Tile& t : tiles)
        for (int64_t k = 0; k < t.parts; ++k) ++next[class_of((first_step(t, k + 1) - first_step(t, k)) * t.cost) + 1];
    for (int c = 0; c < kClasses; ++c) next[c + 1] += next[c];
    segments.resize(next[kClasses]);
    for (const Tile& t : tiles) {
        const ImgGroup& g = groups[t.group];
        ImgSegment s{};
        s.c_off = out == kImgOutBlock ? g.c_off + (int64_t)t.pm * panel * g.ldc + t.pn * panel : g.c_off;
        s.ldc = g.ldc;
        s.rows = t.rows;
        s.cols = t.cols;
        s.pm = t.pm;
        s.pn = t.pn;
        s.t0 = t.t0;
        s.t1 = t.t1;
        s.split = -1;
        s.out_kb = (int)img_units(out == kImgOutZB ? 2 * g.m : out == kImgOutB ? g.m : g.n);
        if (t.parts > 1) {
            s.split = (int)splits.size();
            splits.push_back(GemmSplit{s.c_off, aux_size, g.ldc, t.rows, t.cols, (int)t.parts, ntickets++, 0});
        }
        for (int64_t k = 0; k < t.parts; ++k) {
            s.steps = (int)(first_step(t, k + 1) - first_step(t, k));
            if (t.parts > 1) {
                s.aux_off = aux_size;
                aux_size += (int64_t)((t.rows + 15) / 16) * ((t.cols + 15) / 16) * 2 * kConsumers;
            }
            segments[next[class_of(s.steps * t.cost)]++] = s;
            // the next part's first slice: its term, and the slice in it
            int64_t skip = s.k0 + (int64_t)s.steps;
            while (s.t0 < t.t1 && skip >= steps_of(live[s.t0])) skip -= steps_of(live[s.t0++]);
            s.k0 = (int)skip;
        }
    }
    ctas = (int)std::min<int64_t>((int64_t)num_sms * kCtasPerSm, (int64_t)segments.size());
    live.push_back(ImgTerm{});  // a group's t1 is readable
    terms_at = tab.add(live);
    segments_at = tab.add(segments);
    splits_at = tab.add(splits);
}

int ImgWork::finalize(ImgPack& p, ImgSchedule& a, ImgSchedule& b, int64_t mid_blocks, cudaStream_t stream, int num_sms) {
    DMRG_TRY(allow_smem());
    Tables tab;
    p.plan(a.panel, tab);
    a.plan(num_sms, tab);
    b.plan(num_sms, tab);
    // the counters of both stages, one after the other (none where there is no product)
    ntickets = a.segments.empty() && b.segments.empty() ? 0 : 2 + a.ntickets + b.ntickets;
    const size_t tickets_at = tab.add(std::vector<unsigned>(ntickets, 0u));
    DMRG_TRY(tab.to(d_tables, stream));
    p.tables = a.tables = b.tables = d_tables.as<char>();
    tickets = a.tickets = reinterpret_cast<unsigned*>(d_tables.as<char>() + tickets_at);
    b.tickets = a.tickets + 1 + a.ntickets;
    img_size = p.blocks * kImgBlock;
    mid_size = mid_blocks * kImgBlock;
    return DMRG_OK;
}

int ImgWork::allocate(ImgSchedule& a, ImgSchedule& b) {
    if (img) return DMRG_OK;
    const int64_t n = img_size + mid_size;
    DMRG_TRY(buf.alloc((size_t)std::max<int64_t>(n + a.aux_size + b.aux_size, 1) * sizeof(double)));
    img = buf.as<double>();
    mid = img + img_size;
    a.aux = img + n;
    b.aux = a.aux + a.aux_size;
    return DMRG_OK;
}

int launch_img_gemm(const ImgSchedule& s, const double* A, const double* B, double* C, bool accumulate,
                    const dmrg_ctx_s& ctx) {
    cudaStream_t stream = ctx.stream;
    if (s.segments.empty()) return DMRG_OK;
    const char* tab = s.tables;
    const GemmArgs w{A, B, C, s.aux, reinterpret_cast<const ImgTerm*>(tab + s.terms_at),
                     reinterpret_cast<const ImgSegment*>(tab + s.segments_at), (int)s.segments.size(), s.panel / 8,
                     reinterpret_cast<const GemmSplit*>(tab + s.splits_at), s.tickets,
                     ctx.d_status, ctx.wait_polls, accumulate ? 1 : 0};
    switch (s.out * 2 + (s.scaled ? 1 : 0)) {
        case kImgOutBlock * 2: return launch<kImgOutBlock, false>(s.ctas, w, stream);
        case kImgOutBlock * 2 + 1: return launch<kImgOutBlock, true>(s.ctas, w, stream);
        case kImgOutB * 2: return launch<kImgOutB, false>(s.ctas, w, stream);
        case kImgOutA * 2: return launch<kImgOutA, false>(s.ctas, w, stream);
        case kImgOutZB * 2: return launch<kImgOutZB, false>(s.ctas, w, stream);
        default: return set_error(DMRG_E_STATE, "image products take no scales");
    }
}

}  // namespace dmrg
