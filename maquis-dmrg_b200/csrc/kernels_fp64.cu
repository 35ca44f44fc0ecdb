// Native-FP64 execution of a lowered plan on sm_100a.
//
// Stage 1 (T tasks) and stage 3 (cohort contractions) run as grouped,
// persistent GEMM launches over precomputed tile lists; every output tile is
// owned by exactly one CTA, which loops over the tile's K segments (for H psi:
// every cohort that writes the output block), so the result is written once,
// without atomics, and is bitwise reproducible.  Stage 2 (S build) gathers
// alpha-weighted T columns (Cohort::create_s_r / create_s, tasks.cpp:425-494).
//
// The FP64 inner product uses the FP64 tensor-core instruction
// mma.sync.m8n8k4.f64 (DMMA) on 64x64x16 CTA tiles, 4 warps of 32x32.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <numeric>
#include <tuple>
#include <string>
#include <type_traits>
#include <unordered_map>

#include "../../include/dmrgb200.h"
#include "device.hpp"
#include "async_copy.cuh"

namespace dmrgb200 {

namespace {

// shared-memory row pitch of a tile of ROWS (m or n) columns: 8 words mod 32,
// which makes the fragment loads conflict-free
template <int ROWS>
__host__ __device__ constexpr int pitch() {
    return ROWS + 4;
}

__device__ __forceinline__ const double* op_base(Bases const& bs, DevOp const& op, uint32_t batch) {
    return reinterpret_cast<const double*>(base_of(bs, op.buf) + 8ull * (op.off + uint64_t(batch) * op.bstride));
}

// Kernels launched with programmatic stream serialisation (launch_pdl) may be
// scheduled while the previous kernel of the stream drains; each starts with this
// wait, so none touches memory before its predecessor has completed and its
// writes are visible.
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

// 16 x 8 x 8 and 16 x 8 x 4 forms (rows g and g + 8 of A and C in one lane; k = q, q + 4)
__device__ __forceinline__ void dmma16x8(double (&c)[4], const double (&a)[4], double b0, double b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b0), "d"(b1));
}
__device__ __forceinline__ void dmma16x4(double (&c)[4], double a0, double a1, double b) {
    asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
                 : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
                 : "d"(a0), "d"(a1), "d"(b));
}

// 8-byte asynchronous global->shared copy; src_bytes = 0 writes a zero (out-of-range element).
__device__ __forceinline__ void cp_async8(double* smem, const double* gmem, bool valid) {
    unsigned saddr = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    int n = valid ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(saddr), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void cp_async8_all(double* smem, const char* gmem) {
    unsigned saddr = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(saddr), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// Shared-memory column swizzle of the operand tiles: row k stores column c at
// c ^ ((k >> 2) & 3).  With row pitches of 8 words mod 32, copies in which
// consecutive threads take consecutive k (the coalesced order for K-contiguous
// operands) then hit distinct banks, and the fragment loads of one 4-deep K
// step (one XOR constant) stay conflict-free.
__device__ __forceinline__ int swz(int k) { return (k >> 2) & 3; }

// One thread's copies of one operand tile over the K steps of a segment.  The
// operand tile is ROWS (m or n) x BK_ (k), stored in shared memory as
// [k][ROWS + pad]; a thread issues NC = ROWS * BK_ / NTHREADS 8-byte copies per
// K step.  When the operand's contiguous global dimension is m or n
// ("row-major copies": A not transposed or read through the row table, B
// transposed), the thread's copies share one row r = tid % ROWS and take
// k = kt + j * (NTHREADS / ROWS); otherwise they share k = kt = tid % BK_ and
// take rows r + j * (NTHREADS / BK_).  Copy j reads base + j * jstride; every
// K step advances base by kstep.  All byte strides, fixed per segment.  Rows outside the
// problem are not copied: what the tile holds there only reaches outputs that are not
// stored.  A whole K step has no per-copy conditions (about five instructions per copy
// instead of ten: on blocks of 17 to 52 rows the copies' arithmetic is most of what the
// kernel executes); the last one of a segment zero-fills its K rows past the end, in the half
// or the whole stage that is multiplied.  Eight-deep stages have so few copies each that the
// two forms and the running address (each copy's waits for the one before) cost more than the
// conditions: there every copy has its own, in one loop for both layouts
// (tile16x64_k8_stages3_ctas6 on stage 3 of Heisenberg m = 230, 300, 400: H psi 19.8, 22.5, 28.0
// us in the two forms, 17.4, 19.5, 23.8 this way).
struct CopyStream {
    const char* base;
    const char* safe;  // a readable address for copies that fetch nothing
    uint64_t jstride, kstep;
    uint32_t mask;  // bit j: copy j's row lies inside the problem
    uint32_t r, kt;
    bool rowmajor;
};

template <int ROWS, int BK_, int NTHREADS, int LD, bool HALVES>
__device__ __forceinline__ void issue_copies(double* tile, CopyStream& cs, uint32_t krem) {
    constexpr int NC = ROWS * BK_ / NTHREADS;
    if (BK_ < 16) {
        constexpr int KJ = NTHREADS / ROWS, RJ = NTHREADS / BK_;
#pragma unroll
        for (int j = 0; j < NC; ++j) {
            const uint32_t k = cs.rowmajor ? cs.kt + j * KJ : cs.kt, r = cs.rowmajor ? cs.r : cs.r + j * RJ;
            const bool ok = ((cs.mask >> j) & 1u) && k < krem;
            cp_async8(&tile[k * LD + (r ^ swz(k))], reinterpret_cast<const double*>(ok ? cs.base + j * cs.jstride : cs.safe),
                      ok);
        }
    } else if (cs.rowmajor) {
        constexpr int KJ = NTHREADS / ROWS;
        static_assert(KJ <= 4 || NC == 1 || KJ % 4 == 0, "swizzle of copy j");
        if (cs.mask) {
            const char* p = cs.base;
            // swz(kt + j KJ): kt < KJ, so for KJ <= 4 it depends on j alone
            const uint32_t t0 = KJ <= 4 ? 0u : cs.kt >> 2;
            if (krem >= uint32_t(BK_)) {
#pragma unroll
                for (int j = 0; j < NC; ++j, p += cs.jstride)
                    cp_async8_all(&tile[(cs.kt + j * KJ) * LD + (cs.r ^ ((t0 + ((j * KJ) >> 2)) & 3u))], p);
            } else {
                const uint32_t kend = !HALVES || krem > uint32_t(BK_ / 2) ? BK_ : BK_ / 2;
#pragma unroll
                for (int j = 0; j < NC; ++j, p += cs.jstride) {
                    const uint32_t k = cs.kt + j * KJ;
                    if (k < kend)
                        cp_async8(&tile[k * LD + (cs.r ^ swz(k))], reinterpret_cast<const double*>(k < krem ? p : cs.safe),
                                  k < krem);
                }
            }
        }
    } else {
        constexpr int RJ = NTHREADS / BK_;
        static_assert(RJ % 4 == 0, "swizzle of copy j");
        double* dst = &tile[cs.kt * LD + (cs.r ^ swz(cs.kt))];  // (r + j RJ) ^ swz = (r ^ swz) + j RJ
        const char* p = cs.base;
        const bool kok = cs.kt < krem;
        if (krem >= uint32_t(BK_)) {
#pragma unroll
            for (int j = 0; j < NC; ++j, p += cs.jstride)
                if ((cs.mask >> j) & 1u) cp_async8_all(dst + j * RJ, p);
        } else if (!HALVES || cs.kt < (krem > uint32_t(BK_ / 2) ? BK_ : BK_ / 2)) {
#pragma unroll
            for (int j = 0; j < NC; ++j, p += cs.jstride)
                if ((cs.mask >> j) & 1u) cp_async8(dst + j * RJ, reinterpret_cast<const double*>(kok ? p : cs.safe), kok);
        }
    }
    cs.base += cs.kstep;
}

// Copy stream of an operand whose element (row, k) sits at elem + row * rs + k * ks
// (element strides; rows from row0, nrows of them inside the problem).
template <int ROWS, int BK_, int NTHREADS>
__device__ __forceinline__ void setup_copies(CopyStream& cs, const double* elem, uint64_t rs, uint64_t ks,
                                             uint32_t row0, uint32_t nrows, int tid) {
    constexpr int NC = ROWS * BK_ / NTHREADS;
    cs.safe = reinterpret_cast<const char*>(elem);
    cs.rowmajor = rs == 1;
    if (cs.rowmajor) {
        constexpr int KJ = NTHREADS / ROWS;
        cs.r = tid % ROWS;
        cs.kt = tid / ROWS;
        cs.base = reinterpret_cast<const char*>(elem + (row0 + cs.r) + cs.kt * ks);
        cs.jstride = 8ull * KJ * ks;
        cs.kstep = 8ull * BK_ * ks;
        cs.mask = row0 + cs.r < nrows ? (1u << NC) - 1u : 0u;
    } else {
        constexpr int RJ = NTHREADS / BK_;
        cs.kt = tid % BK_;
        cs.r = tid / BK_;
        cs.base = reinterpret_cast<const char*>(elem + (row0 + cs.r) * rs + cs.kt * ks);
        cs.jstride = 8ull * RJ * rs;
        cs.kstep = 8ull * BK_ * ks;
        cs.mask = 0;
#pragma unroll
        for (int j = 0; j < NC; ++j)
            if (row0 + cs.r + j * RJ < nrows) cs.mask |= 1u << j;
    }
}

// Grouped, persistent FP64 GEMM over a tile list.  Each CTA owns whole output
// tiles (BM_ x 64) and walks every K step (BK_ deep) of every segment of its
// problem; the CTA's K steps over all its tiles form one stream, so the
// cp.async pipeline (STAGES deep) keeps loading the next tile's operands while
// the current tile finishes and stores.  Warps: 2 x 2 of (BM_/2) x 32 (BM_ = 32,
// 64), or for BM_ = 16 a row of 16 x (64 / warps), DMMA m8n8k4.  A tile whose segments are all
// empty (one step, no copies) stores zeros.
struct LoadCursor {
    uint32_t ti, seg, seg_end, krem;
    bool valid;
};

template <int BM_, int BN_, int BK_, int STAGES, int MINB, int NTHREADS, int WARPS_M, bool HALVES = true,
          bool LEAN = false>
__global__ void __launch_bounds__(NTHREADS, MINB) gemm_f64_grouped(const DevProb* __restrict__ probs,
                                                                   const DevSeg* __restrict__ segs,
                                                                   const DevTile* __restrict__ tiles, uint32_t n_tiles,
                                                                   const DevRow* __restrict__ rowtab, SplitArgs split,
                                                                   Bases bases) {
    // warps: WARPS_M x (warps / WARPS_M), warp tiles WM x WN of 8 x 8 DMMA tiles
    constexpr int WM = BM_ / WARPS_M;
    constexpr int WN = BN_ / (NTHREADS / 32 / WARPS_M), NJ = WN / 8;
    constexpr int MI = WM / 8;  // 8 x 8 accumulator tiles (m8n8k4)
    constexpr int NCA = BM_ * BK_ / NTHREADS;
    static_assert(MI >= 1 && NJ >= 1 && NTHREADS % BM_ == 0 && NTHREADS % BN_ == 0 && NTHREADS % BK_ == 0,
                  "tile shape");
    __shared__ __align__(16) double As[STAGES][BK_][pitch<BM_>()];
    __shared__ __align__(16) double Bs[STAGES][BK_][pitch<BN_>()];
    __shared__ uint32_t st_last;  // this tile's part arrived last (K-split problems)
    wait_for_predecessor();

    const int tid = threadIdx.x;
    // one value per warp also to the compiler: branches on the warp's place need no reconvergence
    // (Heisenberg m = 230 to 400 19.2 to 26.8 us without, 18.8 to 26.4 with)
    const int lane = tid & 31, warp = LEAN ? tid >> 5 : __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int wm = (warp % WARPS_M) * WM, wn = (warp / WARPS_M) * WN;
    const int g = lane >> 2, q = lane & 3;

    // ---- producer: walks (tile, segment, K step) and issues one K step per call;
    // the copy streams are set up once per segment ----
    LoadCursor L{blockIdx.x, 0, 0, 0, false};
    CopyStream ca, cb;
    auto enter_segment = [&]() {
        while (L.seg < L.seg_end && segs[L.seg].K == 0) ++L.seg;
        if (L.seg >= L.seg_end) return;
        const DevTile tl = tiles[L.ti];
        const DevProb& pr = probs[tl.prob];
        const DevSeg sg = segs[L.seg];
        L.krem = sg.K;
        const double* A = op_base(bases, sg.A, tl.batch);
        const double* B = op_base(bases, sg.B, tl.batch);
        if (pr.rows != DevProb::NO_ROWS) {
            // row-table A: this thread's row (tid % BM_ in every copy) has its own start and stride
            const uint32_t gm = tl.m0 + uint32_t(tid % BM_);
            ca.safe = reinterpret_cast<const char*>(B);
            ca.rowmajor = true;
            ca.r = tid % BM_;
            ca.kt = tid / BM_;
            ca.mask = 0;
            ca.base = ca.safe;
            ca.jstride = ca.kstep = 0;
            if (gm < pr.M) {
                const DevRow rw = rowtab[pr.rows + gm];
                ca.base = reinterpret_cast<const char*>(base_of(bases, sg.A.buf) + 8ull * (rw.a_off + uint64_t(ca.kt) * rw.ld));
                ca.jstride = 8ull * (NTHREADS / BM_) * rw.ld;
                ca.kstep = 8ull * BK_ * rw.ld;
                ca.mask = (1u << NCA) - 1u;
            }
        } else if (!sg.A.trans) {
            setup_copies<BM_, BK_, NTHREADS>(ca, A, 1, sg.A.ld, tl.m0, pr.M, tid);
        } else {
            setup_copies<BM_, BK_, NTHREADS>(ca, A, sg.A.ld, 1, tl.m0, pr.M, tid);
        }
        if (!sg.B.trans)
            setup_copies<BN_, BK_, NTHREADS>(cb, B, sg.B.ld, 1, tl.n0, pr.N, tid);
        else
            setup_copies<BN_, BK_, NTHREADS>(cb, B, 1, sg.B.ld, tl.n0, pr.N, tid);
    };
    auto enter_tile = [&]() {
        L.valid = L.ti < n_tiles;
        if (!L.valid) return;
        const DevProb& pr = probs[tiles[L.ti].prob];
        L.seg = pr.seg_begin;
        L.seg_end = pr.seg_end;
        enter_segment();
    };
    // returns the K rows the stage holds
    auto issue = [&](int slot) -> uint32_t {
        if (!L.valid) return 0u;
        uint32_t rows = 0;
        if (L.seg < L.seg_end) {  // an empty tile issues no copies
            rows = min(L.krem, uint32_t(BK_));
            issue_copies<BM_, BK_, NTHREADS, pitch<BM_>(), HALVES>(&As[slot][0][0], ca, L.krem);
            issue_copies<BN_, BK_, NTHREADS, pitch<BN_>(), HALVES>(&Bs[slot][0][0], cb, L.krem);
            if (L.krem > uint32_t(BK_)) {
                L.krem -= BK_;
                return rows;
            }
            ++L.seg;
            enter_segment();
            if (L.seg < L.seg_end) return rows;
        }
        L.ti += gridDim.x;
        enter_tile();
        return rows;
    };

    // K rows of the stages in flight, the oldest first.  Every thread walks the same cursor, so
    // each keeps them in registers (a shared word would need a barrier between the prologue's
    // write and the first step's read).
    uint32_t held[STAGES];
    enter_tile();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        held[s] = issue(s);
        cp_async_commit();
    }

    double acc[MI][NJ][2];
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

    // ---- consumer: tiles in the same order, nsteps K steps each ----
    int slot = 0;
    for (uint32_t ti = blockIdx.x; ti < n_tiles; ti += gridDim.x) {
        const DevTile tl = tiles[ti];
        const DevProb& pr = probs[tl.prob];
        const uint32_t M = pr.M, N = pr.N;
        const bool inside = LEAN || (tl.m0 + wm < M && tl.n0 + wn < N);  // any of this warp's tile
        for (uint32_t st = 0; st < tl.nsteps; ++st) {
            const uint32_t kn = held[0];
            held[STAGES - 1] = issue((slot + STAGES - 1) % STAGES);
#pragma unroll
            for (int s = 0; s < STAGES - 1; ++s) held[s] = held[s + 1];
            cp_async_commit();
            cp_async_wait<STAGES - 1>();
            __syncthreads();
            // the second half of a stage that holds at most half its K rows is not multiplied
            // (HALVES), nor tiles of warps outside the problem; unrolled forms keep the fragment
            // reads ahead of the products (a condition per K step of four, or a form per count of
            // them, costs more than it saves where a CTA has its SM to itself)
            if (inside) {
                auto product = [&](auto steps) {
                    constexpr int KS = decltype(steps)::value;
#pragma unroll
                    for (int kk = 0; kk < 4 * KS; kk += 4) {
                        double a[MI], b[NJ];
#pragma unroll
                        for (int i = 0; i < MI; ++i) a[i] = As[slot][kk + q][(wm + i * 8 + g) ^ (kk >> 2)];
#pragma unroll
                        for (int j = 0; j < NJ; ++j) b[j] = Bs[slot][kk + q][(wn + j * 8 + g) ^ (kk >> 2)];
#pragma unroll
                        for (int i = 0; i < MI; ++i)
#pragma unroll
                            for (int j = 0; j < NJ; ++j) dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
                    }
                };
                if (LEAN || (HALVES ? kn > uint32_t(BK_ / 2) : kn > 0)) product(std::integral_constant<int, BK_ / 4>());
                else if (HALVES && kn) product(std::integral_constant<int, BK_ / 8>());
            }
            __syncthreads();
            slot = (slot + 1) % STAGES;
        }
        // epilogue (the next tile's first steps are already in flight); an empty tile multiplied
        // nothing (LEAN: what it found) and stores zeros
        bool empty = LEAN;
        for (uint32_t sg = pr.seg_begin; LEAN && sg < pr.seg_end; ++sg) empty = empty && segs[sg].K == 0;
        if (pr.split != DevProb::NO_SPLIT) {
            const DevSplit sp = split.tab[pr.split];
            const uint64_t mn = uint64_t(M) * N;
            double* part = split.ws + sp.ws + sp.part * mn;
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const uint32_t r = tl.m0 + wm + i * 8 + g, c = tl.n0 + wn + j * 8 + q * 2 + e;
                        if (r < M && c < N) __stcg(part + r + uint64_t(c) * M, acc[i][j][e]);
                    }
            // the last part to arrive sees every part's sums (release and acquire around the count)
            __threadfence();
            __syncthreads();
            if (tid == 0) {
                unsigned* ctr = split.ctr + sp.ctr + (tl.m0 / BM_) * ((N + BN_ - 1) / BN_) + tl.n0 / BN_;
                const bool last = atomicAdd(ctr, 1u) == sp.parts - 1;
                if (last) *ctr = 0;
                st_last = last ? 1u : 0u;
                __threadfence();
            }
            __syncthreads();
            const bool last = st_last != 0;
#pragma unroll
            for (int i = 0; i < MI; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
            // part by part, all of a thread's elements of one part in flight at once
            const double* ws = split.ws + sp.ws;
            for (uint32_t x = 0; last && x < sp.parts; ++x, ws += mn)
#pragma unroll
                for (int i = 0; i < MI; ++i)
#pragma unroll
                    for (int j = 0; j < NJ; ++j)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const uint32_t r = tl.m0 + wm + i * 8 + g, c = tl.n0 + wn + j * 8 + q * 2 + e;
                            if (r < M && c < N) acc[i][j][e] += __ldcg(ws + r + uint64_t(c) * M);
                        }
            if (!last) continue;
        }
        const bool rowmode = pr.rows != DevProb::NO_ROWS;
        double* C = const_cast<double*>(op_base(bases, pr.C, tl.batch));
        const uint64_t ldc = pr.C.ld;
#pragma unroll
        for (int i = 0; i < MI; ++i) {
            const uint32_t r = tl.m0 + wm + i * 8 + g;
            // the row's start and leading dimension: from the row table or the plain operand
            double* crow = C + r;
            uint64_t ld = ldc;
            if (rowmode && r < M) {
                const DevRow rw = rowtab[pr.rows + r];
                crow = reinterpret_cast<double*>(base_of(bases, pr.C.buf) + 8ull * (rw.c_off + tl.batch * rw.cbs));
                ld = rw.ld;
            }
#pragma unroll
            for (int j = 0; j < NJ; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    uint32_t c = tl.n0 + wn + j * 8 + q * 2 + e;
                    if (r < M && c < N) crow[c * ld] = empty ? 0.0 : acc[i][j][e];
                    acc[i][j][e] = 0.0;
                }
        }
    }
    cp_async_wait<0>();
}

// S build: S is tiled by cells (one per unit and MPO row block); a cell with a
// line writes the alpha-weighted sum of its T sources (summed in term order like
// the reference's axpy sequence), a cell without one writes zeros, so S needs
// no separate clearing.  One warp per work item (a line and a chunk of SB_CHUNK
// consecutive elements of its column-major walk): every lane owns SB_EPT elements
// (lane + 32 u).  A source is one run of T (leading dimension = rows), so the elements
// of a term are its start plus fixed offsets: a term costs one broadcast read and a load
// and a multiply-add per element, four terms in flight.  Only the store needs (i, c), by a
// multiplication with the reciprocal of the row count.  (The terms handed round by
// shuffles and a division per element took 71 instructions per element and warp on lines
// of two terms, 18.8 us at the Hubbard middle of m = 1024 with the issue slots 45% busy.)
constexpr int SB_EPT = 4, SB_CHUNK = 32 * SB_EPT;
__global__ void __launch_bounds__(256) sbuild_lines(const DevSLine* __restrict__ lines,
                                                    const DevSTerm* __restrict__ terms,
                                                    const DevSItem* __restrict__ items, uint32_t n_items,
                                                    double* __restrict__ S, const double* __restrict__ T, int more) {
    const uint32_t lane = threadIdx.x & 31, stride = gridDim.x * (blockDim.x >> 5);
    uint32_t it = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    // the tables are complete before the predecessor began; the next item's line is read
    // while this one's sources are
    DevSItem I{}, In{};
    DevSLine L{};
    if (it < n_items) I = items[it];
    if (it + stride < n_items) In = items[it + stride];
    if (it < n_items) L = lines[I.group];
    wait_for_predecessor();
    if (more) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // see sbuild_groups
    while (it < n_items) {
        const uint32_t e0 = I.e0 + lane, n = L.rows * L.cols;
        bool in[SB_EPT];
        double v[SB_EPT];
#pragma unroll
        for (int u = 0; u < SB_EPT; ++u) {
            in[u] = e0 + 32u * u < n;
            v[u] = 0.0;
        }
        const double* Te = T + e0;
#pragma unroll 4
        for (uint32_t t = L.term_begin; t < L.term_end; ++t) {
            const double2 raw = __ldg(reinterpret_cast<const double2*>(terms + t));
            const double* src = Te + __double_as_longlong(raw.y);
#pragma unroll
            for (int u = 0; u < SB_EPT; ++u)
                if (in[u]) v[u] = fma(raw.x, src[32 * u], v[u]);
        }
        const DevSLine Lc = L;
        it += stride;
        I = In;
        if (it < n_items) L = lines[I.group];
        if (it + stride < n_items) In = items[it + stride];
        // column of element e: e / rows as the high word of e * (2^32 / rows + 1), exact while
        // e * rows < 2^32
        const uint32_t magic = 0xFFFFFFFFu / Lc.rows + 1u;
        const bool small = uint64_t(n) * Lc.rows < (1ull << 32) && Lc.rows > 1;
        double* dst = S + Lc.s_base;
#pragma unroll
        for (int u = 0; u < SB_EPT; ++u)
            if (in[u]) {
                const uint32_t e = e0 + 32u * u, c = small ? __umulhi(e, magic) : e / Lc.rows;
                dst[(e - c * Lc.rows) + uint64_t(c) * Lc.ld_s] = v[u];
            }
    }
}

// S build of line groups (DevSGroup): one warp per work item (a group and a
// chunk of SG_CHUNK consecutive elements of its lines).  The chunk of every line is
// one product (elements x sources) * (sources x lines) on the FP64 tensor cores
// (DMMA m8n8k4: 8 elements x 8 lines x 4 sources per instruction, the warp holding
// SG_CHUNK x lines accumulators), so each source cell is read once for all lines of
// the group and one warp instruction does 256 multiply-adds.  The sources stream
// through the warp's own shared-memory ring with bulk copies (TMA engine, no
// multicast): a stage holds SGB_NC source rows of the chunk and their alpha
// columns; lanes 0 .. SGB_NC - 1 each copy one row and lane SGB_NC the alphas,
// every lane expecting its own bytes on the stage's mbarrier before lane 0
// arrives, SGB_STAGES - 1 stages ahead of the multiply-adds.  The copies bypass
// the L1 miss path, so a warp keeps kilobytes in flight without registers.  A
// bulk copy starts on a 16-byte boundary, so a row whose first element is odd is
// copied from one element earlier and read with that shift.  Every wait is
// bounded (2 s; the thread is suspended while it waits): on a timeout the warp
// records it in *err, lets its copies land (bounded) and stops.  Each line sums
// its sources in the group's entry order, four per DMMA.  The row pitch of a stage
// (SG_CHUNK + 4 doubles, 4 mod 16) puts the four sources of a K step in different
// banks for the fragment loads.
// Groups of up to 8 lines run as one launch (8 accumulated lines), larger groups as
// another (SG_LINES lines); both with 2 stages and 3 CTAs (12 warps) per SM, which caps
// the wide launch (its 128 x 16 accumulators included) at 168 registers.
constexpr int SGB_WARPS = 4, SGB_NC = 8, SGB_ROW = SG_CHUNK + 4;
template <int STAGES>
struct alignas(16) SgbRing {
    double rows[STAGES][SGB_NC][SGB_ROW];
    double alpha[STAGES][SGB_NC][SG_LINES];
    uint64_t full[STAGES];
    uint32_t shift[STAGES][SGB_NC];
};
static_assert(sizeof(double) * SGB_ROW % 16 == 0 && sizeof(SgbRing<2>) % 16 == 0 && sizeof(SgbRing<3>) % 16 == 0,
              "bulk copy alignment");
static_assert(SGB_NC < 32 && SGB_NC % 4 == 0, "one lane per row plus one for the alphas; whole DMMA K steps");
template <int NL>
struct SgbShape;
template <>
struct SgbShape<8> {
    static constexpr int STAGES = 2, MINB = 3;
};
template <>
struct SgbShape<SG_LINES> {
    static constexpr int STAGES = 2, MINB = 3;
};
template <int NL>
constexpr size_t sgb_smem() {
    return sizeof(SgbRing<SgbShape<NL>::STAGES>) * SGB_WARPS;
}

// One work item of the grouped S build with NL accumulated lines (NL = 8 for groups of
// at most 8 lines, SG_LINES otherwise; the alpha columns always hold SG_LINES entries).
// Returns false when a wait failed (the warp then stops).
template <int NL, int SGB_STAGES>
__device__ __forceinline__ bool sgb_item(SgbRing<SGB_STAGES>& R, DevSGroup const& G, uint32_t e0,
                                         const uint64_t* __restrict__ ent_t,
                                         const double* __restrict__ ent_a, double* __restrict__ S,
                                         const double* __restrict__ T, int* err, unsigned long long wait_ns,
                                         uint32_t lane, uint32_t& issued, uint32_t& consumed) {
    using namespace async;
    const uint32_t n = G.rows * G.cols, cnt = min(uint32_t(SG_CHUNK), n - e0);
    const uint32_t k0 = G.ent_begin, k1 = G.ent_end;
    constexpr int MT = SG_CHUNK / 16, NT = NL / 8;  // m16n8 tiles: elements x lines
    const uint32_t g = lane >> 2, q = lane & 3;
    double acc[MT][NT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.0;
    // every lane: the stage of sources kb .. kb + SGB_NC - 1 (those below k1)
    auto fill = [&](uint32_t kb) {
        const uint32_t slot = issued % SGB_STAGES, nc = min(uint32_t(SGB_NC), k1 - kb);
        if (lane < nc) {
            const uint64_t tb = ent_t[kb + lane];
            const uint32_t sh = uint32_t((tb + e0) & 1u), sz = ((cnt + sh) * 8u + 15u) & ~15u;
            R.shift[slot][lane] = sh;
            mbar_expect_tx_only(&R.full[slot], sz);
            bulk_load(R.rows[slot][lane], T + tb + e0 - sh, sz, &R.full[slot]);
        } else if (lane == uint32_t(SGB_NC)) {
            const uint32_t sz = nc * SG_LINES * uint32_t(sizeof(double));
            mbar_expect_tx_only(&R.full[slot], sz);
            bulk_load(R.alpha[slot], ent_a + uint64_t(kb) * SG_LINES, sz, &R.full[slot]);
        }
        __syncwarp();  // every expected byte count is in before the phase can complete
        if (lane == 0) mbar_arrive(&R.full[slot]);
        ++issued;
    };
    const uint32_t nst = (k1 - k0 + SGB_NC - 1) / SGB_NC;
    for (uint32_t st = 0; st < min(nst, uint32_t(SGB_STAGES - 1)); ++st) fill(k0 + st * SGB_NC);
    for (uint32_t st = 0; st < nst; ++st) {
        const uint32_t slot = consumed % SGB_STAGES, kb = k0 + st * SGB_NC;
        // the stage SGB_STAGES - 1 ahead goes into the slot freed in the previous step
        if (st + SGB_STAGES - 1 < nst) {
            fence_proxy_async_smem();
            fill(k0 + (st + SGB_STAGES - 1) * SGB_NC);
        }
        const bool ok = mbar_wait_suspend(&R.full[slot], (consumed / SGB_STAGES) & 1u, err, wait_ns);
        if (__any_sync(0xffffffffu, !ok)) return false;
        const uint32_t nc = min(uint32_t(SGB_NC), k1 - kb);
        // D (elements x lines) += T (elements x sources) * alpha (sources x lines): a whole
        // stage of eight sources per DMMA, or its first four (a group's sources are padded to
        // a multiple of four)
        const double* r0 = R.rows[slot][q] + R.shift[slot][q] + g;
        if (nc == uint32_t(SGB_NC)) {
            const double* r1 = R.rows[slot][q + 4] + R.shift[slot][q + 4] + g;
            double b0[NT], b1[NT];
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                b0[j] = R.alpha[slot][q][j * 8 + g];
                b1[j] = R.alpha[slot][q + 4][j * 8 + g];
            }
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                const double a[4] = {r0[i * 16], r0[i * 16 + 8], r1[i * 16], r1[i * 16 + 8]};
#pragma unroll
                for (int j = 0; j < NT; ++j) dmma16x8(acc[i][j], a, b0[j], b1[j]);
            }
        } else {
            double b0[NT];
#pragma unroll
            for (int j = 0; j < NT; ++j) b0[j] = R.alpha[slot][q][j * 8 + g];
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                const double a0 = r0[i * 16], a1 = r0[i * 16 + 8];
#pragma unroll
                for (int j = 0; j < NT; ++j) dmma16x4(acc[i][j], a0, a1, b0[j]);
            }
        }
        ++consumed;
        __syncwarp();  // every lane's reads of this slot are done before it is refilled
    }
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int r2 = 0; r2 < 2; ++r2) {
            const uint32_t e = e0 + uint32_t(i * 16 + r2 * 8) + g;
            if (e >= n) continue;
            const uint32_t col = e / G.rows, r = e - col * G.rows;
            double* dst = S + G.s_base + r + uint64_t(col) * G.ld_s;
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t line = uint32_t(j * 8) + 2u * q + uint32_t(h);
                    if (line < G.nlines)
                        dst[uint64_t(line) * G.line_stride] = ((G.mask >> line) & 1u) ? acc[i][j][2 * r2 + h] : 0.0;
                }
        }
    return true;
}

template <int NL>
__global__ void __launch_bounds__(32 * SGB_WARPS, SgbShape<NL>::MINB)
    sbuild_groups(const DevSGroup* __restrict__ groups, const DevSItem* __restrict__ items, uint32_t n_items,
                  const uint64_t* __restrict__ ent_t, const double* __restrict__ ent_a, double* __restrict__ S,
                  const double* __restrict__ T, int* err, unsigned long long wait_ns, int after_sbuild, int more) {
    using namespace async;
    constexpr int SGB_STAGES = SgbShape<NL>::STAGES;
    extern __shared__ __align__(16) unsigned char sgb_smem_raw[];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SgbRing<SGB_STAGES>& R = reinterpret_cast<SgbRing<SGB_STAGES>*>(sgb_smem_raw)[warp];
    // The launches of one S build write different parts of S from the same T.  The first waits
    // for stage 1 and only then lets the next start (launch_dependents, where more follow), so a
    // later one (after another of the S build) finds T complete and fills the SMs its
    // predecessor's last CTAs leave; its own wait, at its end, keeps completion in stream order.
    // At L = 12, m = 300 in quantum chemistry the three launches take 245 us instead of 330.  The
    // last one lets nothing start early: stage 3's CTAs would hold SMs and wait.
    if (!after_sbuild) wait_for_predecessor();
    if (more) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (lane == 0) {
        for (int i = 0; i < SGB_STAGES; ++i) mbar_init(&R.full[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    uint32_t issued = 0, consumed = 0;  // stage fills of this warp, in order (the same in every lane)
    bool failed = false;
    for (uint32_t it = blockIdx.x * SGB_WARPS + warp; it < n_items && !failed; it += gridDim.x * SGB_WARPS) {
        const DevSItem I = items[it];
        failed = !sgb_item<NL, SGB_STAGES>(R, groups[I.group], I.e0, ent_t, ent_a, S, T, err, wait_ns, lane, issued,
                                           consumed);
    }
    if (failed && lane == 0) {
        // let the copies still in flight land before the warp's shared memory is released (bounded)
        for (; consumed < issued; ++consumed) {
            const unsigned long long t0 = global_ns();
            while (!mbar_try(&R.full[consumed % SGB_STAGES], (consumed / SGB_STAGES) & 1u) &&
                   global_ns() - t0 < WAIT_LIMIT_NS) {
            }
        }
    }
    if (after_sbuild) wait_for_predecessor();
}

// Register-resident DMMA loop for the FP64 tensor-core rate (calibration).
__global__ void __launch_bounds__(128) dmma_rate_loop(int iters, double* sink) {
    double acc[8][2];
    double a = 1.0 + threadIdx.x * 1e-9, b = 1.0 - threadIdx.x * 1e-9;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = 0.0;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int i = 0; i < 8; ++i) dmma(acc[i][0], acc[i][1], a, b);
    }
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += acc[i][0] + acc[i][1];
    if (s == 1.2345) sink[threadIdx.x] = s;
}

// --- host-side lowering ---------------------------------------------------------

// tile classes (rows x columns, K step): 0 = 32 x 64 / 16, 1 = 16 x 64 / 8,
// 2 = 64 x 64 / 16, 3 = 16 x 64 / 16 (two warps), 4 = 128 x 32 / 16, 5 = 64 x 32 / 8
constexpr int CLASS_BM[N_TILE_CLASSES] = {32, 16, 64, 16, 128, 64};
constexpr int CLASS_BN[N_TILE_CLASSES] = {64, 64, 64, 64, 32, 32};
constexpr int CLASS_BK[N_TILE_CLASSES] = {16, 8, 16, 16, 16, 8};

void add_tiles(GemmList& gl, uint32_t prob, uint32_t nbatch) {
    DevProb const& p = gl.probs[prob];
    for (int c = 0; c < N_TILE_CLASSES; ++c) {
        const uint32_t bm = CLASS_BM[c], bn = CLASS_BN[c], bk = CLASS_BK[c];
        uint32_t nsteps = 0;
        for (uint32_t s = p.seg_begin; s < p.seg_end; ++s) nsteps += (gl.segs[s].K + bk - 1) / bk;
        nsteps = std::max<uint32_t>(nsteps, 1);  // an empty problem: one step that issues no copies
        auto& out = c == 0 ? gl.tiles : gl.tiles_cls[c];
        for (uint32_t b = 0; b < nbatch; ++b)
            for (uint32_t m0 = 0; m0 < std::max<uint32_t>(p.M, 1); m0 += bm)
                for (uint32_t n0 = 0; n0 < std::max<uint32_t>(p.N, 1); n0 += bn)
                    out.push_back(DevTile{prob, b, m0, n0, nsteps});
    }
}

// Order tiles by decreasing K work so that the static round-robin of the
// persistent grid starts with the longest tiles (LPT-style balance).
void sort_tiles(GemmList& gl) {
    std::vector<uint64_t> kwork(gl.probs.size(), 0);
    for (size_t p = 0; p < gl.probs.size(); ++p)
        for (uint32_t s = gl.probs[p].seg_begin; s < gl.probs[p].seg_end; ++s) kwork[p] += gl.segs[s].K;
    for (int c = 0; c < N_TILE_CLASSES; ++c) {
        auto& tl = c == 0 ? gl.tiles : gl.tiles_cls[c];
        std::stable_sort(tl.begin(), tl.end(),
                         [&](DevTile const& a, DevTile const& b) { return kwork[a.prob] > kwork[b.prob]; });
    }
}

DevOp op(uint16_t buf, uint64_t off, uint32_t ld, bool trans, uint64_t bstride = 0) {
    DevOp o;
    o.off = off;
    o.bstride = bstride;
    o.ld = ld;
    o.buf = buf;
    o.trans = trans ? 1 : 0;
    return o;
}

}  // namespace

DevOp dev_op(uint16_t buf, uint64_t off, uint32_t ld, bool trans, uint64_t bstride) {
    return op(buf, off, ld, trans, bstride);
}
void gemm_add_tiles(GemmList& gl, uint32_t prob, uint32_t nbatch) { add_tiles(gl, prob, nbatch); }
void gemm_sort_tiles(GemmList& gl) { sort_tiles(gl); }

std::vector<uint64_t> t_offsets(FlatPlan const& p, uint64_t* total) {
    std::vector<uint64_t> off(p.n_t());
    uint64_t sum = 0;
    for (uint32_t t = 0; t < p.n_t(); ++t) {
        off[t] = sum;
        sum += round_up(p.t_size(t), 32);
    }
    if (total) *total = sum;
    return off;
}

std::vector<uint64_t> s_offsets(FlatPlan const& p, uint64_t* total) {
    std::vector<uint64_t> off(p.n_cohorts());
    uint64_t sum = 0;
    for (uint32_t c = 0; c < p.n_cohorts(); ++c) {
        off[c] = sum;
        sum += round_up(uint64_t(p.c_nsrows[c]) * p.c_stripe[c] * (p.kind == KIND_LEFT ? p.c_rs[c] : p.c_ls[c]), 32);
    }
    if (total) *total = sum;
    return off;
}

namespace {
// Blocks of every T task that some term reads; the others are never used (at the middle
// of a Fermi-Hubbard chain the tasks hold 2312 blocks of which 1624 are read).
struct BlocksRead {
    std::vector<uint64_t> first;  // per task: its flags in `flag`
    std::vector<char> flag;
    const char* of(uint32_t t) const { return flag.data() + first[t]; }
};
BlocksRead t_blocks_read(FlatPlan const& p) {
    BlocksRead r;
    r.first.resize(p.n_t());
    uint64_t n = 0;
    for (uint32_t t = 0; t < p.n_t(); ++t) {
        r.first[t] = n;
        n += p.t_nb[t];
    }
    r.flag.assign(n, 0);
    for (uint32_t u = 0; u < p.n_units(); ++u) {
        const uint32_t ms = p.u_ms[u];
        if (!ms) continue;
        const uint32_t k1 = p.u_line[u] < p.u_line[u + 1] ? p.l_term[p.u_line[u + 1]] : 0;
        for (uint32_t k = k1 ? p.l_term[p.u_line[u]] : 0; k < k1; ++k) {
            // columns term_col .. + ms of the task's T, usually one whole block
            const uint32_t t = p.term_t[k], w = p.t_bcols[t], col = p.term_col[k];
            if (!w) continue;
            char* f = r.flag.data() + r.first[t];
            uint32_t b = col / w;
            for (uint32_t end = b * w; end < col + ms && b < p.t_nb[t]; end += w) f[b++] = 1;
        }
    }
    return r;
}

// Stage 1 of H psi / right step with the rows of all T tasks that share a
// boundary cohort (same cohort, transposition and shape) stacked into one
// row-table problem: A row r is row r' of task t's psi slice, C row r is row r'
// of T_t (leading dimension = the task's row count), so one tile covers several
// small psi blocks instead of padding each to a full tile.  T blocks that no term reads
// can be left out: the tasks are then stacked by the set of blocks they need, one problem
// per run of adjacent blocks (a run goes on over a gap where that takes no more tiles).  That
// undoes some of the stacking, so a cohort is cut up only where it saves a tenth of its tile
// K steps or more, on tiles of 32 rows and of 64 (the shapes of most variants).  Lattice
// chains save 19 to 34% (Hubbard L = 64, m = 1024, middle: 7352 steps to 5072, H psi 57.8 us to 52.4;
// Heisenberg m = 1024 84.5 to 77.4).  Quantum chemistry reads nearly all blocks at the middle
// and, left of it, slightly different sets per task: cut up by the share of blocks saved, L =
// 12, m = 300, sites 3 and 4 would go from 3017 and 13260 steps to 9693 and 22089.
void stack_stage1(FlatPlan const& p, std::vector<uint64_t> const& stage1_bnd, std::vector<uint64_t> const& t_off,
                  GemmList& g1, std::vector<char> const* keep = nullptr, bool skip_unread = false) {
    g1 = GemmList();
    std::map<std::tuple<uint32_t, uint8_t, uint32_t, uint32_t, uint32_t>, std::vector<uint32_t>> groups;
    for (uint32_t t = 0; t < p.n_t(); ++t)
        if (!keep || (*keep)[t]) groups[{p.t_ci[t], p.t_trans[t], p.t_brows[t], p.t_bcols[t], p.t_nb[t]}].push_back(t);
    BlocksRead read;
    if (skip_unread) read = t_blocks_read(p);
    auto problem = [&](std::vector<uint32_t> const& tasks, uint32_t b0, uint32_t nb) {
        const uint32_t t0 = tasks.front();
        const uint32_t K = p.t_brows[t0], Nf = p.t_bcols[t0];
        const bool tr = p.t_trans[t0] != 0;
        const uint64_t bnd = stage1_bnd.at(p.t_ci[t0]) / 8 + uint64_t(b0) * K * Nf;
        DevProb pr;
        pr.rows = uint32_t(g1.rowtab.size());
        uint32_t M = 0;
        for (uint32_t t : tasks) {
            const uint32_t Mt = p.in_rows[p.t_lb[t]];
            for (uint32_t r = 0; r < Mt; ++r)
                g1.rowtab.push_back(DevRow{p.in_off[p.t_lb[t]] + uint64_t(p.t_col[t]) * Mt + r,
                                           t_off[t] + uint64_t(b0) * Mt * Nf + r, tr ? uint64_t(Mt) * Nf : 0, Mt, 0});
            M += Mt;
        }
        pr.M = M;
        pr.C = op(BUF_T, 0, 0, false);
        DevSeg sg{};
        sg.A = op(BUF_IN, 0, 0, false);
        sg.K = K;
        uint32_t nbatch = 1;
        if (!tr) {
            // the nb stored blocks are adjacent K x Nf column blocks: one product of width nb * Nf
            pr.N = Nf * nb;
            sg.B = op(BUF_ABS, bnd, K, false, 0);
        } else {
            pr.N = Nf;
            sg.B = op(BUF_ABS, bnd, Nf, true, uint64_t(K) * Nf);
            nbatch = nb;
        }
        pr.seg_begin = uint32_t(g1.segs.size());
        g1.segs.push_back(sg);
        pr.seg_end = uint32_t(g1.segs.size());
        g1.probs.push_back(pr);
        add_tiles(g1, uint32_t(g1.probs.size() - 1), nbatch);
    };
    // K steps of one problem of M stacked rows and nb blocks on tiles of bm x 64
    auto steps = [&](uint32_t t0, uint64_t bm, uint64_t M, uint64_t nb) {
        const uint64_t Nf = p.t_bcols[t0], nt = p.t_trans[t0] ? nb * ((Nf + 63) / 64) : (nb * Nf + 63) / 64;
        return (M + bm - 1) / bm * nt * ((p.t_brows[t0] + 15) / 16);
    };
    struct Piece {
        std::vector<uint32_t> const* tasks;
        uint32_t b0, nb;
    };
    for (auto const& kv : groups) {
        const uint32_t t0 = kv.second.front(), nb = p.t_nb[t0];
        if (!skip_unread) {
            problem(kv.second, 0, nb);
            continue;
        }
        auto rows = [&](std::vector<uint32_t> const& tasks) {
            uint64_t M = 0;
            for (uint32_t t : tasks) M += p.in_rows[p.t_lb[t]];
            return M;
        };
        const uint64_t M = rows(kv.second), w32 = steps(t0, 32, M, nb), w64 = steps(t0, 64, M, nb);
        // the elements read fill so many tiles of 32 x 64 at least
        uint64_t used = 0;
        for (uint32_t t : kv.second)
            used += uint64_t(std::count(read.of(t), read.of(t) + nb, 1)) * p.in_rows[p.t_lb[t]];
        if (10 * used * p.t_bcols[t0] * ((p.t_brows[t0] + 15) / 16) > 9 * w32 * (32 * 64)) {
            problem(kv.second, 0, nb);
            continue;
        }
        std::map<std::string, std::vector<uint32_t>> by_set;
        for (uint32_t t : kv.second) by_set[std::string(read.of(t), nb)].push_back(t);
        std::vector<Piece> pieces;
        uint64_t c32 = 0, c64 = 0;
        for (auto const& sv : by_set) {
            const uint64_t Ms = rows(sv.second);
            for (uint32_t b = 0; b < nb;) {
                uint32_t e = b;
                while (e < nb && sv.first[e]) ++e;
                if (e > b) {
                    // over a gap to the run before, where the wider problem has no more tiles
                    if (!pieces.empty() && pieces.back().tasks == &sv.second &&
                        steps(t0, 32, Ms, e - pieces.back().b0) <=
                            steps(t0, 32, Ms, pieces.back().nb) + steps(t0, 32, Ms, e - b))
                        pieces.back().nb = e - pieces.back().b0;
                    else
                        pieces.push_back({&sv.second, b, e - b});
                }
                b = e + 1;
            }
        }
        for (auto const& x : pieces) {
            c32 += steps(t0, 32, rows(*x.tasks), x.nb);
            c64 += steps(t0, 64, rows(*x.tasks), x.nb);
        }
        if (10 * c32 > 9 * w32 || 10 * c64 > 9 * w64) {
            problem(kv.second, 0, nb);
            continue;
        }
        for (auto const& x : pieces) problem(*x.tasks, x.b0, x.nb);
    }
    sort_tiles(g1);
}
}  // namespace

namespace {
// S build of one unit as line groups: groups of `width` (8 or SG_LINES) consecutive
// MPO row blocks, each with the union of its lines' source cells in address order
// and the summed alphas per (cell, line) (SG_LINES alpha slots per entry either
// way).  Returns the multiply-adds per element this issues (entries x the lines the
// kernel accumulates); `terms` receives the per-line walk's count.
struct UnitGroups {
    std::vector<DevSGroup> groups;
    std::vector<uint64_t> ent_t;
    std::vector<double> ent_a;
    std::vector<uint32_t> term_k, term_slot;  // plan term -> entry * SG_LINES + line
};
uint64_t group_unit(FlatPlan const& p, uint32_t c, uint32_t u, std::vector<int64_t> const& line_of,
                    std::vector<uint64_t> const& t_off, std::vector<uint64_t> const& s_off, UnitGroups& out,
                    uint64_t* terms, uint32_t width) {
    const bool left = p.kind == KIND_LEFT;
    const uint32_t ns = p.c_nsrows[c], ls = p.c_ls[c], rs = p.c_rs[c];
    std::unordered_map<uint64_t, uint32_t> slot;
    uint64_t fmas = 0;
    *terms = 0;
    for (uint32_t g0 = 0; g0 < ns; g0 += width) {
        DevSGroup G{};
        G.nlines = std::min<uint32_t>(width, ns - g0);
        if (left) {
            G.rows = p.u_ms[u];
            G.cols = rs;
            G.ld_s = p.c_stripe[c];
            G.line_stride = rs * p.c_stripe[c];
            G.s_base = s_off[c] + p.u_offset[u] + uint64_t(g0) * rs * p.c_stripe[c];
        } else {
            G.rows = ls;
            G.cols = p.u_ms[u];
            G.ld_s = ns * ls;
            G.line_stride = ls;
            G.s_base = s_off[c] + uint64_t(g0) * ls + uint64_t(p.u_offset[u]) * G.ld_s;
        }
        G.ent_begin = uint32_t(out.ent_t.size());
        slot.clear();
        const size_t map0 = out.term_k.size();
        for (uint32_t j = 0; j < G.nlines; ++j) {
            const int64_t l = line_of[g0 + j];
            if (l < 0) continue;
            for (uint32_t k = p.l_term[l]; k < p.l_term[l + 1]; ++k) {
                const uint64_t src = t_off[p.term_t[k]] + uint64_t(p.term_col[k]) * (left ? rs : ls);
                auto it = slot.find(src);
                uint32_t e;
                if (it == slot.end()) {
                    e = uint32_t(out.ent_t.size());
                    slot.emplace(src, e);
                    out.ent_t.push_back(src);
                    out.ent_a.insert(out.ent_a.end(), SG_LINES, 0.0);
                } else {
                    e = it->second;
                }
                out.ent_a[uint64_t(e) * SG_LINES + j] += p.term_alpha[k];
                out.term_k.push_back(k);
                out.term_slot.push_back((e - G.ent_begin) * SG_LINES + j);  // group-local until sorted
                G.mask |= 1u << j;
                ++*terms;
            }
        }
        G.ent_end = uint32_t(out.ent_t.size());
        // sources in address order: the warps on the groups of one unit then sweep
        // the shared T slices together (L1 / L2 reuse)
        {
            const uint32_t n = G.ent_end - G.ent_begin;
            std::vector<uint32_t> ord(n);
            std::iota(ord.begin(), ord.end(), 0u);
            std::sort(ord.begin(), ord.end(), [&](uint32_t a, uint32_t b) {
                return out.ent_t[G.ent_begin + a] < out.ent_t[G.ent_begin + b];
            });
            std::vector<uint64_t> t(n);
            std::vector<double> al(uint64_t(n) * SG_LINES);
            for (uint32_t x = 0; x < n; ++x) {
                t[x] = out.ent_t[G.ent_begin + ord[x]];
                std::copy_n(&out.ent_a[uint64_t(G.ent_begin + ord[x]) * SG_LINES], SG_LINES, &al[uint64_t(x) * SG_LINES]);
            }
            std::copy(t.begin(), t.end(), out.ent_t.begin() + G.ent_begin);
            std::copy(al.begin(), al.end(), out.ent_a.begin() + uint64_t(G.ent_begin) * SG_LINES);
            // the terms' slots follow their entries to the sorted positions
            std::vector<uint32_t> pos(n);
            for (uint32_t x = 0; x < n; ++x) pos[ord[x]] = x;
            for (size_t q = map0; q < out.term_slot.size(); ++q) {
                const uint32_t le = out.term_slot[q] / SG_LINES, j = out.term_slot[q] % SG_LINES;
                out.term_slot[q] = (G.ent_begin + pos[le]) * SG_LINES + j;
            }
        }
        // the kernel accumulates 8 lines for groups of up to 8, SG_LINES otherwise
        fmas += uint64_t(G.ent_end - G.ent_begin) * (G.nlines <= 8 ? 8u : uint32_t(SG_LINES));
        // the kernel walks sources SG_UNROLL at a time: pad with zero-alpha copies of the
        // group's first source.  A padded source is multiplied by zero, so it must read
        // written T elements: T blocks are padded to 32 elements and stage 1 never writes
        // the gaps, which may hold non-finite leftovers (0 * NaN = NaN in every line)
        while ((out.ent_t.size() - G.ent_begin) % SG_UNROLL) {
            const uint64_t first = out.ent_t[G.ent_begin];
            out.ent_t.push_back(first);
            out.ent_a.insert(out.ent_a.end(), SG_LINES, 0.0);
        }
        G.ent_end = uint32_t(out.ent_t.size());
        out.groups.push_back(G);
    }
    return fmas;
}

// DMRGB200_SBUILD: "lines" or "groups" forces one S-build form; anything else chooses per unit
int sbuild_mode() {
    const char* v = std::getenv("DMRGB200_SBUILD");
    if (!v) return 0;
    if (!std::strcmp(v, "lines")) return 1;
    if (!std::strcmp(v, "groups")) return 2;
    return 0;
}
}  // namespace

namespace {
// Stage 3 of H psi: one problem per output block (every cohort writing the block is
// a K segment of it); keep (optional) selects output blocks.
void build_stage3_hpsi(FlatPlan const& p, std::vector<uint64_t> const& stage3_bnd, std::vector<uint64_t> const& s_off,
                       GemmList& g3, std::vector<char> const* keep) {
    const uint32_t nc = p.n_cohorts();
    std::vector<std::vector<uint32_t>> by_out(p.out_rows.size());
    for (uint32_t c = 0; c < nc; ++c) by_out[p.c_rb[c]].push_back(c);
    for (uint32_t ob = 0; ob < p.out_rows.size(); ++ob) {
        if (keep && !(*keep)[ob]) continue;
        DevProb pr;
        pr.M = p.out_rows[ob];
        pr.N = p.out_cols[ob];
        pr.C = op(BUF_OUT, p.out_off[ob], pr.M, false, 0);
        pr.seg_begin = uint32_t(g3.segs.size());
        for (uint32_t c : by_out[ob]) {
            uint32_t ls = p.c_ls[c], rs = p.c_rs[c], ns = p.c_nsrows[c];
            uint64_t lbase = stage3_bnd.at(p.c_ci[c]) / 8;
            if (!p.c_trans[c]) {
                DevSeg sg{};
                sg.A = op(BUF_ABS, lbase, rs, false);
                sg.B = op(BUF_S, s_off[c], ns * ls, false);
                sg.K = ns * ls;
                g3.segs.push_back(sg);
            } else {
                // each stored block (ls x rs) is read transposed: one segment per MPO row block
                for (uint32_t b = 0; b < ns; ++b) {
                    DevSeg sg{};
                    sg.A = op(BUF_ABS, lbase + uint64_t(b) * ls * rs, ls, true);
                    sg.B = op(BUF_S, s_off[c] + uint64_t(b) * ls, ns * ls, false);
                    sg.K = ls;
                    g3.segs.push_back(sg);
                }
            }
        }
        pr.seg_end = uint32_t(g3.segs.size());
        g3.probs.push_back(pr);
        add_tiles(g3, uint32_t(g3.probs.size() - 1), 1);
    }
}
}  // namespace

namespace {
// K steps (of 16) of a part when long problems are cut: half of what each of the CTAs that
// fill the chip (four per SM) would get if the list's work were spread evenly, so that the
// parts also balance.  At least 48: storing, counting and adding a tile's partial sums costs
// a CTA about 4 us, and shorter parts lose (at the Hubbard middle of m = 1024, 6 to 24 steps per
// tile, parts of 8 took 41 us where whole tiles take 27).  In quantum chemistry stage 3 has one
// problem per output block: at L = 12, m = 300 10 problems of 107 to 382 steps, whose 127 tiles
// of 16 x 64 took 220 us whole and take 104 us in parts.
uint32_t split_target(GemmList const& gl) {
    uint64_t total = 0;
    for (auto const& t : gl.tiles) total += t.nsteps;
    return uint32_t(std::max<uint64_t>(48, total / (2 * 4 * B200_SMS)));
}

// `gl` with K ranges of more than `target` steps cut into parts, a function of the problem and
// the target alone (the sums do not depend on the list a problem stands in nor on the kernel
// variant).  Returns false where nothing is cut: the tiles are many, or short.
bool split_list(GemmList const& gl, uint32_t target, GemmList& out) {
    out = GemmList();
    bool any = false;
    std::vector<uint32_t> nbatch(gl.probs.size(), 0);
    for (auto const& t : gl.tiles) nbatch[t.prob] = std::max(nbatch[t.prob], t.batch + 1);
    for (uint32_t i = 0; i < gl.probs.size(); ++i) {
        DevProb pr = gl.probs[i];
        uint64_t steps = 0;
        for (uint32_t s = pr.seg_begin; s < pr.seg_end; ++s) steps += (gl.segs[s].K + 15) / 16;
        // one part at least: a problem without segments stores zeros
        const uint32_t parts = nbatch[i] == 1 && pr.rows == DevProb::NO_ROWS && pr.M && pr.N
                                   ? uint32_t(std::max<uint64_t>(1, std::min<uint64_t>((steps + target - 1) / target, 16)))
                                   : 1;
        uint32_t sg = pr.seg_begin, koff = 0;  // next segment and the K rows of it already given out
        uint64_t given = 0;
        const uint64_t ws = out.split_ws;
        const uint32_t ctr = out.split_ctrs;
        for (uint32_t x = 0; x < parts; ++x) {
            DevProb q = pr;
            q.seg_begin = uint32_t(out.segs.size());
            // steps [given, upto) of the problem: whole segments, or pieces of 16 K rows
            const uint64_t upto = steps * (x + 1) / parts;
            while (sg < pr.seg_end && (given < upto || x + 1 == parts)) {
                DevSeg piece = gl.segs[sg];
                const uint32_t left = piece.K - koff, here = (left + 15) / 16;
                const uint32_t take = x + 1 == parts ? left : uint32_t(std::min<uint64_t>(left, (upto - given) * 16));
                piece.A.off += piece.A.trans ? koff : uint64_t(koff) * piece.A.ld;
                piece.B.off += piece.B.trans ? uint64_t(koff) * piece.B.ld : koff;
                piece.K = take;
                if (take) out.segs.push_back(piece);
                given += take == left ? here : (take + 15) / 16;
                koff += take;
                if (koff == gl.segs[sg].K) {
                    ++sg;
                    koff = 0;
                }
            }
            q.seg_end = uint32_t(out.segs.size());
            if (parts > 1) {
                any = true;
                q.split = uint32_t(out.splits.size());
                out.splits.push_back(DevSplit{ws, parts, x, ctr, 0});
            }
            out.probs.push_back(q);
            add_tiles(out, uint32_t(out.probs.size() - 1), nbatch[i]);
        }
        if (parts > 1) {
            out.split_ws += uint64_t(parts) * pr.M * pr.N;
            // counters for the smallest tiles of any class (16 rows, 32 columns)
            out.split_ctrs += ((pr.M + 15) / 16) * ((pr.N + 31) / 32);
        }
    }
    out.rowtab = gl.rowtab;
    if (!any) {
        out = GemmList();
        return false;
    }
    sort_tiles(out);
    return true;
}
}  // namespace

ProgramForm program_form(FlatPlan const& p) {
    // any addresses do: nothing is read
    auto ptrs = [](std::vector<uint32_t> const& ci) {
        uint32_t n = 0;
        for (uint32_t c : ci) n = std::max(n, c + 1);
        return std::vector<uint64_t>(n, 8);
    };
    const bool hpsi = p.kind == KIND_HPSI;
    const std::vector<uint64_t> s1 = ptrs(p.t_ci), s3 = hpsi ? ptrs(p.c_ci) : std::vector<uint64_t>(),
                                out = hpsi ? std::vector<uint64_t>() : ptrs(p.c_out_ci);
    DeviceProgram prog;
    compile_program(p, s3, s1, out, prog, true, true);
    ProgramForm f;
    f.chained = prog.chained;
    f.chain_tiles = uint32_t(prog.chain.tiles.size());
    f.chain_warps = prog.chained ? uint32_t(prog.chain.split) : 0;
    GemmList const& g3 = prog.own3 ? prog.stage3f : prog.stage3;
    for (auto const& s : prog.stage3f.splits) f.stage3_parts = std::max(f.stage3_parts, s.parts);
    for (auto const& pr : g3.probs)
        if (pr.seg_begin == pr.seg_end && pr.M && pr.N) ++f.stage3_zero_blocks;
    auto steps = [](GemmList const& gl) {
        uint64_t n = 0;
        for (auto const& t : gl.tiles) n += t.nsteps;
        return n;
    };
    f.stage1_steps = f.stage1_steps_whole = steps(prog.stage1);
    if (p.kind != KIND_LEFT && p.n_t()) {
        GemmList whole;
        stack_stage1(p, s1, t_offsets(p, nullptr), whole);
        f.stage1_steps_whole = steps(whole);
    }
    return f;
}

void compile_program(FlatPlan const& p, std::vector<uint64_t> const& stage3_bnd,
                     std::vector<uint64_t> const& stage1_bnd, std::vector<uint64_t> const& outptr,
                     DeviceProgram& prog, bool stack_rows, bool group_lines) {
    prog = DeviceProgram();
    prog.in_elems = p.in_size;
    prog.out_elems = p.out_size;
    const uint32_t nt = p.n_t(), nc = p.n_cohorts();
    std::vector<uint64_t> t_off = t_offsets(p, &prog.t_elems);
    // slack after the last T block: the grouped S build's bulk copies may read one
    // element past a source row
    prog.t_elems += 32;

    // ---- stage 1: rows stacked by boundary cohort, or one problem per T task ----
    GemmList& g1 = prog.stage1;
    const bool stacked = stack_rows && p.kind != KIND_LEFT && nt;
    if (stacked) stack_stage1(p, stage1_bnd, t_off, g1, nullptr, group_lines);
    for (uint32_t t = 0; !stacked && t < nt; ++t) {
        DevProb pr;
        DevSeg sg{};
        uint64_t bnd = stage1_bnd.at(p.t_ci[t]) / 8;
        if (p.kind == KIND_LEFT) {
            uint32_t M = p.t_brows[t], N = p.t_width[t], K = p.t_bcols[t];
            sg.A = op(BUF_ABS, bnd, p.t_trans[t] ? K : M, p.t_trans[t], uint64_t(M) * K);
            sg.B = op(BUF_IN, p.in_off[p.t_lb[t]] + uint64_t(p.t_col[t]) * K, K, false, 0);
            sg.K = K;
            pr.C = op(BUF_T, t_off[t], M, false, uint64_t(M) * N);
            pr.M = M;
            pr.N = N;
        } else {
            uint32_t M = p.in_rows[p.t_lb[t]], N = p.t_bcols[t], K = p.t_brows[t];
            sg.A = op(BUF_IN, p.in_off[p.t_lb[t]] + uint64_t(p.t_col[t]) * M, M, false, 0);
            sg.B = op(BUF_ABS, bnd, p.t_trans[t] ? N : K, p.t_trans[t], uint64_t(K) * N);
            sg.K = K;
            pr.C = op(BUF_T, t_off[t], M, false, uint64_t(M) * N);
            pr.M = M;
            pr.N = N;
            if (!p.t_trans[t]) {
                // the nb stored blocks are adjacent K x N column blocks: one GEMM of width nb * N
                pr.N = N * p.t_nb[t];
                pr.seg_begin = uint32_t(g1.segs.size());
                g1.segs.push_back(sg);
                pr.seg_end = uint32_t(g1.segs.size());
                g1.probs.push_back(pr);
                add_tiles(g1, uint32_t(g1.probs.size() - 1), 1);
                continue;
            }
        }
        pr.seg_begin = uint32_t(g1.segs.size());
        g1.segs.push_back(sg);
        pr.seg_end = uint32_t(g1.segs.size());
        g1.probs.push_back(pr);
        add_tiles(g1, uint32_t(g1.probs.size() - 1), p.t_nb[t]);
    }
    if (!stacked) sort_tiles(g1);

    // ---- stage 2 (S lines) ----
    std::vector<uint64_t> s_off = s_offsets(p, &prog.s_elems);
    // units tile the S columns (rows for the left step) and b1 its row blocks, so
    // the cells (unit, b1) cover S exactly once
    const int mode = group_lines ? sbuild_mode() : 1;
    UnitGroups ug;
    std::vector<std::pair<uint32_t, uint32_t>> ug_units;  // group range of every grouped unit
    for (uint32_t c = 0; c < nc; ++c) {
        for (uint32_t u = p.c_unit[c]; u < p.c_unit[c + 1]; ++u) {
            std::vector<int64_t> line_of(p.c_nsrows[c], -1);
            for (uint32_t l = p.u_line[u]; l < p.u_line[u + 1]; ++l) line_of[p.l_b1[l]] = l;
            const uint64_t w = uint64_t(p.u_ms[u]) * (p.kind == KIND_LEFT ? p.c_rs[c] : p.c_ls[c]);
            // the group construction is tried only where lines average 4 or more terms: sparser
            // units (Heisenberg, Hubbard: about two terms per line) keep the line walk without
            // paying for the trial, which would cost more host time than it could save
            const uint64_t unit_terms = p.l_term[p.u_line[u + 1]] - p.l_term[p.u_line[u]];
            const bool dense_enough = unit_terms >= 4ull * (p.u_line[u + 1] - p.u_line[u]);
            if (mode != 1 && w && (mode == 2 || dense_enough)) {
                // line groups when they issue at most twice the per-line walk's multiply-adds
                // (a unit without terms is zero-filled by the line walk)
                // wide groups read each shared source once for more lines; narrow ones waste
                // fewer multiply-adds on lines that do not read a source
                const size_t g0 = ug.groups.size(), e0 = ug.ent_t.size(), m0 = ug.term_k.size();
                bool grouped = false;
                for (uint32_t width : {uint32_t(SG_LINES), 8u}) {
                    uint64_t nterms = 0;
                    const uint64_t fmas = group_unit(p, c, u, line_of, t_off, s_off, ug, &nterms, width);
                    if (mode == 2 || (nterms && fmas <= 2 * nterms)) {
                        ug_units.emplace_back(uint32_t(g0), uint32_t(ug.groups.size()));
                        grouped = true;
                        break;
                    }
                    ug.groups.resize(g0);
                    ug.ent_t.resize(e0);
                    ug.ent_a.resize(e0 * SG_LINES);
                    ug.term_k.resize(m0);
                    ug.term_slot.resize(m0);
                }
                if (grouped) continue;
            }
            for (uint32_t b1 = 0; b1 < p.c_nsrows[c]; ++b1) {
                DevSLine L;
                L.term_begin = uint32_t(prog.terms.size());
                int64_t l = line_of[b1];
                if (p.kind == KIND_LEFT) {
                    L.ld_s = p.c_stripe[c];
                    L.rows = p.u_ms[u];
                    L.cols = p.c_rs[c];
                    L.ld_t = p.u_ms[u];
                    L.s_base = s_off[c] + p.u_offset[u] + uint64_t(b1) * p.c_rs[c] * p.c_stripe[c];
                    if (l >= 0)
                        for (uint32_t k = p.l_term[l]; k < p.l_term[l + 1]; ++k)
                            prog.terms.push_back(
                                DevSTerm{p.term_alpha[k], t_off[p.term_t[k]] + uint64_t(p.term_col[k]) * p.c_rs[c]});
                } else {
                    uint32_t ls = p.c_ls[c];
                    L.ld_s = p.c_nsrows[c] * ls;
                    L.rows = ls;
                    L.cols = p.u_ms[u];
                    L.ld_t = ls;
                    L.s_base = s_off[c] + uint64_t(b1) * ls + uint64_t(p.u_offset[u]) * L.ld_s;
                    if (l >= 0)
                        for (uint32_t k = p.l_term[l]; k < p.l_term[l + 1]; ++k)
                            prog.terms.push_back(
                                DevSTerm{p.term_alpha[k], t_off[p.term_t[k]] + uint64_t(p.term_col[k]) * ls});
                }
                L.term_end = uint32_t(prog.terms.size());
                if (uint64_t(L.rows) * L.cols) prog.lines.push_back(L);
            }
        }
    }
    // warp items of the lines: every line in chunks of SB_CHUNK elements, in line order
    for (uint32_t li = 0; li < prog.lines.size(); ++li) {
        const uint64_t n = uint64_t(prog.lines[li].rows) * prog.lines[li].cols;
        for (uint64_t e0 = 0; e0 < n; e0 += SB_CHUNK) prog.litems.push_back(DevSItem{li, uint32_t(e0)});
    }
    // warp items of the line groups: units by decreasing work, then group by
    // group, each group's element chunks consecutive (the warps of a CTA share the
    // group's source list and read its T slices in long contiguous runs; the
    // groups of a unit follow each other and reuse the unit's slices from L2)
    prog.groups = std::move(ug.groups);
    prog.gent_t = std::move(ug.ent_t);
    prog.gent_a = std::move(ug.ent_a);
    prog.gterm_k = std::move(ug.term_k);
    prog.gterm_slot = std::move(ug.term_slot);
    {
        std::vector<uint64_t> work(ug_units.size(), 0);
        for (size_t x = 0; x < ug_units.size(); ++x)
            for (uint32_t gi = ug_units[x].first; gi < ug_units[x].second; ++gi) {
                DevSGroup const& G = prog.groups[gi];
                work[x] += uint64_t(G.ent_end - G.ent_begin + 1) * G.rows * G.cols;
            }
        std::vector<uint32_t> order(ug_units.size());
        std::iota(order.begin(), order.end(), 0u);
        std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return work[a] > work[b]; });
        // groups of up to 8 lines first (their own launch), then the wide ones
        for (int wide = 0; wide < 2; ++wide) {
            for (uint32_t x : order) {
                const uint32_t g0 = ug_units[x].first, g1 = ug_units[x].second;
                if (g0 == g1) continue;
                const uint64_t n = uint64_t(prog.groups[g0].rows) * prog.groups[g0].cols;
                for (uint32_t gi = g0; gi < g1; ++gi) {
                    if ((prog.groups[gi].nlines > 8) != (wide == 1)) continue;
                    for (uint64_t e0 = 0; e0 < n; e0 += SG_CHUNK) prog.gitems.push_back(DevSItem{gi, uint32_t(e0)});
                }
            }
            if (!wide) prog.n_gitems8 = uint32_t(prog.gitems.size());
        }
    }

    // ---- stage 3 ----
    GemmList& g3 = prog.stage3;
    if (p.kind == KIND_HPSI) {
        build_stage3_hpsi(p, stage3_bnd, s_off, g3, nullptr);
    } else if (p.kind == KIND_RIGHT) {
        for (uint32_t c = 0; c < nc; ++c) {
            uint32_t ls = p.c_ls[c], rs = p.c_rs[c], ns = p.c_nsrows[c];
            DevProb pr;
            pr.M = ls;
            pr.N = rs;
            pr.C = op(BUF_ABS, outptr.at(p.c_out_ci[c]) / 8, ls, false, uint64_t(ls) * rs);
            DevSeg sg{};
            sg.A = op(BUF_S, s_off[c], ns * ls, false, ls);
            sg.B = op(BUF_OUT, p.out_off[p.c_rb[c]], rs, true, 0);
            sg.K = p.c_stripe[c];
            pr.seg_begin = uint32_t(g3.segs.size());
            g3.segs.push_back(sg);
            pr.seg_end = uint32_t(g3.segs.size());
            g3.probs.push_back(pr);
            add_tiles(g3, uint32_t(g3.probs.size() - 1), ns);
        }
    } else {
        for (uint32_t c = 0; c < nc; ++c) {
            uint32_t ls = p.c_ls[c], rs = p.c_rs[c], ns = p.c_nsrows[c], stripe = p.c_stripe[c];
            DevProb pr;
            pr.M = ls;
            pr.N = ns * rs;
            pr.C = op(BUF_ABS, outptr.at(p.c_out_ci[c]) / 8, ls, false, 0);
            DevSeg sg{};
            sg.A = op(BUF_OUT, p.out_off[p.c_lb[c]], stripe, true, 0);
            sg.B = op(BUF_S, s_off[c], stripe, false, 0);
            sg.K = stripe;
            pr.seg_begin = uint32_t(g3.segs.size());
            g3.segs.push_back(sg);
            pr.seg_end = uint32_t(g3.segs.size());
            g3.probs.push_back(pr);
            add_tiles(g3, uint32_t(g3.probs.size() - 1), 1);
        }
    }
    sort_tiles(g3);

    // ---- the whole plan as chained products (the general entry points; not where an S-build form
    // is forced) ----
    if (stack_rows && group_lines && mode == 0 && ug_units.empty())
        prog.chained = prog.chain_built = build_chain(p, stage3_bnd, stage1_bnd, outptr, prog.chain);
    // ---- stage 3 with long K ranges split ----
    if (stack_rows && group_lines && g3.tiles.size() < 4 * 4 * B200_SMS) {
        prog.split_steps = split_target(g3);
        prog.own3 = split_list(g3, prog.split_steps, prog.stage3f);
    }
}

namespace {
template <class T>
cudaError_t up(std::vector<T> const& v, T** d) {
    *d = nullptr;
    if (v.empty()) return cudaSuccess;
    cudaError_t e = cudaMalloc(d, v.size() * sizeof(T));
    if (e != cudaSuccess) return e;
    return cudaMemcpy(*d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
}
}  // namespace

namespace {
// All tables of a program in one device allocation: packed into one host buffer
// (each table 256-byte aligned), copied with one transfer, freed with one call.
struct TablePacker {
    std::vector<unsigned char> host;
    static constexpr size_t NONE = ~size_t(0);
    template <class T>
    size_t add(std::vector<T> const& v) {
        if (v.empty()) return NONE;
        const size_t off = (host.size() + 255) / 256 * 256;
        host.resize(off + v.size() * sizeof(T));
        std::memcpy(host.data() + off, v.data(), v.size() * sizeof(T));
        return off;
    }
    size_t zeros(size_t bytes) {
        const size_t off = (host.size() + 255) / 256 * 256;
        host.resize(off + bytes, 0);
        return off;
    }
};
template <class T>
T* at(unsigned char* base, size_t off) {
    return off == TablePacker::NONE ? nullptr : reinterpret_cast<T*>(base + off);
}
}  // namespace

cudaError_t upload_program(DeviceProgram& prog) {
    TablePacker pk;
    const size_t o_p1 = pk.add(prog.stage1.probs), o_s1 = pk.add(prog.stage1.segs), o_t1 = pk.add(prog.stage1.tiles);
    const size_t o_p3 = pk.add(prog.stage3.probs), o_s3 = pk.add(prog.stage3.segs), o_t3 = pk.add(prog.stage3.tiles);
    const size_t o_r1 = pk.add(prog.stage1.rowtab);
    size_t o_x1[N_TILE_CLASSES], o_x3[N_TILE_CLASSES];
    for (int c = 1; c < N_TILE_CLASSES; ++c) {
        o_x1[c] = pk.add(prog.stage1.tiles_cls[c]);
        o_x3[c] = pk.add(prog.stage3.tiles_cls[c]);
    }
    const size_t o_l = pk.add(prog.lines), o_k = pk.add(prog.terms), o_li = pk.add(prog.litems);
    const size_t o_pf = pk.add(prog.stage3f.probs), o_sf = pk.add(prog.stage3f.segs), o_tf = pk.add(prog.stage3f.tiles);
    const size_t o_sp = pk.add(prog.stage3f.splits);
    const size_t o_cn = prog.stage3f.split_ctrs ? pk.zeros(prog.stage3f.split_ctrs * sizeof(unsigned)) : TablePacker::NONE;
    size_t o_xf[N_TILE_CLASSES];
    for (int c = 1; c < N_TILE_CLASSES; ++c) o_xf[c] = pk.add(prog.stage3f.tiles_cls[c]);
    const size_t o_ct = pk.add(prog.chain.tiles), o_cs = pk.add(prog.chain.terms);
    const size_t o_g = pk.add(prog.groups), o_gt = pk.add(prog.gent_t), o_ga = pk.add(prog.gent_a);
    const size_t o_gi = pk.add(prog.gitems);
    const size_t o_err = prog.gitems.empty() ? TablePacker::NONE : pk.zeros(sizeof(int));
    prog.d_arena = nullptr;
    if (!pk.host.empty()) {
        cudaError_t e = cudaMalloc(&prog.d_arena, pk.host.size());
        if (e != cudaSuccess) return e;
        if ((e = cudaMemcpy(prog.d_arena, pk.host.data(), pk.host.size(), cudaMemcpyHostToDevice)) != cudaSuccess)
            return e;
    }
    unsigned char* b = prog.d_arena;
    prog.d_p1 = at<DevProb>(b, o_p1);
    prog.d_s1 = at<DevSeg>(b, o_s1);
    prog.d_t1 = at<DevTile>(b, o_t1);
    prog.d_p3 = at<DevProb>(b, o_p3);
    prog.d_s3 = at<DevSeg>(b, o_s3);
    prog.d_t3 = at<DevTile>(b, o_t3);
    prog.d_r1 = at<DevRow>(b, o_r1);
    for (int c = 1; c < N_TILE_CLASSES; ++c) {
        prog.x1.t[c] = at<DevTile>(b, o_x1[c]);
        prog.x3.t[c] = at<DevTile>(b, o_x3[c]);
        prog.x1.n[c] = uint32_t(prog.stage1.tiles_cls[c].size());
        prog.x3.n[c] = uint32_t(prog.stage3.tiles_cls[c].size());
    }
    prog.f3 = GemmDev();
    if (prog.own3) {
        const cudaError_t e = cudaMalloc(&prog.d_split_ws, prog.stage3f.split_ws * sizeof(double));
        if (e != cudaSuccess) return e;
        prog.f3.split = SplitArgs{at<DevSplit>(b, o_sp), prog.d_split_ws, at<unsigned>(b, o_cn)};
        prog.f3.p = at<DevProb>(b, o_pf);
        prog.f3.s = at<DevSeg>(b, o_sf);
        prog.f3.t = at<DevTile>(b, o_tf);
        prog.f3.n = uint32_t(prog.stage3f.tiles.size());
        for (int c = 1; c < N_TILE_CLASSES; ++c) {
            prog.f3.x.t[c] = at<DevTile>(b, o_xf[c]);
            prog.f3.x.n[c] = uint32_t(prog.stage3f.tiles_cls[c].size());
        }
    }
    static_cast<ChainShape&>(prog.d_chain) = prog.chain;
    prog.d_chain.tiles = at<DevChainTile>(b, o_ct);
    prog.d_chain.terms = at<DevChainTerm>(b, o_cs);
    prog.d_chain.n = uint32_t(prog.chain.tiles.size());
    prog.d_lines = at<DevSLine>(b, o_l);
    prog.d_terms = at<DevSTerm>(b, o_k);
    prog.d_litems = at<DevSItem>(b, o_li);
    prog.d_groups = at<DevSGroup>(b, o_g);
    prog.d_gent_t = at<uint64_t>(b, o_gt);
    prog.d_gent_a = at<double>(b, o_ga);
    prog.d_gitems = at<DevSItem>(b, o_gi);
    prog.d_err = at<int>(b, o_err);
    prog.n_t1 = uint32_t(prog.stage1.tiles.size());
    prog.n_t3 = uint32_t(prog.stage3.tiles.size());
    prog.n_lines = uint32_t(prog.lines.size());
    prog.n_litems = uint32_t(prog.litems.size());
    prog.n_gitems = uint32_t(prog.gitems.size());
    return cudaSuccess;
}

void free_program(DeviceProgram& prog) {
    cudaFree(prog.d_arena);
    prog.d_arena = nullptr;
    prog.d_p1 = nullptr;
    prog.d_s1 = nullptr;
    prog.d_t1 = nullptr;
    prog.d_p3 = nullptr;
    prog.d_s3 = nullptr;
    prog.d_t3 = nullptr;
    prog.d_r1 = nullptr;
    cudaFree(prog.d_split_ws);
    prog.d_split_ws = nullptr;
    prog.f3 = GemmDev();
    prog.d_chain = ChainDev();
    prog.x1 = TileLists();
    prog.x3 = TileLists();
    prog.d_lines = nullptr;
    prog.d_terms = nullptr;
    prog.d_litems = nullptr;
    prog.d_groups = nullptr;
    prog.d_gent_t = nullptr;
    prog.d_gent_a = nullptr;
    prog.d_gitems = nullptr;
    prog.d_err = nullptr;
}

namespace {
// cut points at block boundaries near equal shares of [0, total)
std::vector<uint64_t> cut_ranges(std::vector<uint64_t> const& block_off, uint64_t total, uint32_t nparts) {
    std::vector<uint64_t> starts(block_off);
    std::sort(starts.begin(), starts.end());
    std::vector<uint64_t> cut{0};
    for (uint32_t q = 1; q < nparts; ++q) {
        const uint64_t want = total * q / nparts;
        auto it = std::lower_bound(starts.begin(), starts.end(), want);
        uint64_t c = it == starts.end() ? total : *it;
        cut.push_back(std::max(c, cut.back()));
    }
    cut.push_back(total);
    return cut;
}
}  // namespace

cudaError_t compile_pipeline(FlatPlan const& p, std::vector<uint64_t> const& stage3_bnd,
                             std::vector<uint64_t> const& stage1_bnd, DeviceProgram const& prog, uint32_t nparts,
                             PipelineProgram& pp) {
    pp = PipelineProgram();
    pp.chained = prog.chained;
    if (pp.chained) return cudaSuccess;  // one launch, no ranges
    pp.nparts = nparts;
    std::vector<uint64_t> in_off(p.in_off.begin(), p.in_off.end()), out_off(p.out_off.begin(), p.out_off.end());
    pp.in_cut = cut_ranges(in_off, p.in_size, nparts);
    pp.out_cut = cut_ranges(out_off, p.out_size, nparts);
    const std::vector<uint64_t> t_off = t_offsets(p, nullptr), s_off = s_offsets(p, nullptr);
    pp.s1.resize(nparts);
    pp.s3.resize(nparts);
    for (uint32_t q = 0; q < nparts; ++q) {
        std::vector<char> keep_t(p.n_t()), keep_o(p.out_rows.size());
        for (uint32_t t = 0; t < p.n_t(); ++t) {
            const uint64_t o = p.in_off[p.t_lb[t]];
            keep_t[t] = o >= pp.in_cut[q] && o < pp.in_cut[q + 1];
        }
        for (uint32_t ob = 0; ob < p.out_rows.size(); ++ob)
            keep_o[ob] = p.out_off[ob] >= pp.out_cut[q] && p.out_off[ob] < pp.out_cut[q + 1];
        GemmList g1, g3;
        stack_stage1(p, stage1_bnd, t_off, g1, &keep_t, true);
        build_stage3_hpsi(p, stage3_bnd, s_off, g3, &keep_o);
        sort_tiles(g3);
        GemmList g3s;  // the whole plan's K parts, so that the sums are the same
        if (prog.own3 && split_list(g3, prog.split_steps, g3s)) g3 = std::move(g3s);
        cudaError_t e;
        if ((e = upload_gemm(g1, pp.s1[q])) != cudaSuccess) return e;
        if ((e = upload_gemm(g3, pp.s3[q])) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

void free_pipeline(PipelineProgram& pp) {
    for (auto& g : pp.s1) free_gemm(g);
    for (auto& g : pp.s3) free_gemm(g);
    pp = PipelineProgram();
}

cudaError_t run_pipeline(DeviceProgram const& prog, PipelineProgram const& pp, const double* x_host, double* y_host,
                         double* xd, double* yd, double* T, double* S, cudaStream_t s, cudaStream_t c,
                         cudaEvent_t const* ev) {
    const uint32_t np = pp.nparts;
    Bases bs{};
    bs.b[BUF_IN] = reinterpret_cast<uint64_t>(xd);
    bs.b[BUF_OUT] = reinterpret_cast<uint64_t>(yd);
    bs.b[BUF_T] = reinterpret_cast<uint64_t>(T);
    bs.b[BUF_S] = reinterpret_cast<uint64_t>(S);
    cudaError_t e;
    if (pp.chained) {
        // Chained products read all of x for every output, so nothing overlaps the copy in, and a
        // launch per output range to overlap the copy out costs more than it hides: the ranges
        // are too short to fill the chip (Hubbard L = 32, m = 480, 0.96 MB each way: 115 us by
        // four ranges, 107 by the stages in ranges, 70 in sequence).
        if ((e = cudaMemcpyAsync(xd, x_host, prog.in_elems * sizeof(double), cudaMemcpyHostToDevice, s)) != cudaSuccess)
            return e;
        if ((e = launch_chain(prog.d_chain, bs, s)) != cudaSuccess) return e;
        return cudaMemcpyAsync(y_host, yd, prog.out_elems * sizeof(double), cudaMemcpyDeviceToHost, s);
    }
    // the copies start after the work already queued on the caller's stream
    if ((e = cudaEventRecord(ev[0], s)) != cudaSuccess) return e;
    if ((e = cudaStreamWaitEvent(c, ev[0], 0)) != cudaSuccess) return e;
    for (uint32_t q = 0; q < np; ++q) {
        const uint64_t n = pp.in_cut[q + 1] - pp.in_cut[q];
        if (n && (e = cudaMemcpyAsync(xd + pp.in_cut[q], x_host + pp.in_cut[q], n * sizeof(double),
                                      cudaMemcpyHostToDevice, c)) != cudaSuccess)
            return e;
        if ((e = cudaEventRecord(ev[1 + q], c)) != cudaSuccess) return e;
    }
    for (uint32_t q = 0; q < np; ++q) {
        if ((e = cudaStreamWaitEvent(s, ev[1 + q], 0)) != cudaSuccess) return e;
        GemmDev g = pp.s1[q];
        g.var = prog.var1;
        if ((e = launch_gemm(g, bs, s)) != cudaSuccess) return e;
    }
    if ((e = run_sbuild(prog, T, S, s)) != cudaSuccess) return e;
    for (uint32_t q = 0; q < np; ++q) {
        GemmDev g = pp.s3[q];
        g.var = prog.var3;
        if ((e = launch_gemm(g, bs, s)) != cudaSuccess) return e;
        if ((e = cudaEventRecord(ev[1 + np + q], s)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(c, ev[1 + np + q], 0)) != cudaSuccess) return e;
        const uint64_t n = pp.out_cut[q + 1] - pp.out_cut[q];
        if (n && (e = cudaMemcpyAsync(y_host + pp.out_cut[q], yd + pp.out_cut[q], n * sizeof(double),
                                      cudaMemcpyDeviceToHost, c)) != cudaSuccess)
            return e;
    }
    if ((e = cudaEventRecord(ev[1 + 2 * np], c)) != cudaSuccess) return e;
    return cudaStreamWaitEvent(s, ev[1 + 2 * np], 0);
}

double calibrate_fp64_tflops() {
    const int sms = device_sm_count();
    double* sink = nullptr;
    cudaMalloc(&sink, 128 * sizeof(double));
    const int iters = 20000, blocks = sms * 8;
    dmma_rate_loop<<<blocks, 128>>>(1000, sink);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0);
    dmma_rate_loop<<<blocks, 128>>>(iters, sink);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(sink);
    // one m8n8k4 DMMA = 8*8*4 FMA = 512 flops per warp instruction
    double flops = double(blocks) * 4 /*warps*/ * iters * 8 * 512.0;
    return ms > 0 ? flops / (ms * 1e-3) / 1e12 : 0.0;
}

void gemm_split_long(GemmList& gl) {
    GemmList cut;
    if (gl.tiles.size() < 4 * 4 * B200_SMS && split_list(gl, split_target(gl), cut)) gl = std::move(cut);
}

cudaError_t upload_gemm(GemmList const& gl, GemmDev& d) {
    cudaError_t e;
    if ((e = up(gl.probs, &d.p)) != cudaSuccess) return e;
    if ((e = up(gl.segs, &d.s)) != cudaSuccess) return e;
    if ((e = up(gl.tiles, &d.t)) != cudaSuccess) return e;
    if ((e = up(gl.rowtab, &d.r)) != cudaSuccess) return e;
    for (int c = 1; c < N_TILE_CLASSES; ++c) {
        if ((e = up(gl.tiles_cls[c], &d.x.t[c])) != cudaSuccess) return e;
        d.x.n[c] = uint32_t(gl.tiles_cls[c].size());
    }
    d.n = uint32_t(gl.tiles.size());
    if (!gl.splits.empty()) {
        DevSplit* tab = nullptr;
        if ((e = up(gl.splits, &tab)) != cudaSuccess) return e;
        d.split.tab = tab;
        if ((e = cudaMalloc(&d.split.ws, gl.split_ws * sizeof(double))) != cudaSuccess) return e;
        if ((e = up(std::vector<unsigned>(gl.split_ctrs, 0u), &d.split.ctr)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

void free_gemm(GemmDev& d) {
    cudaFree(d.p);
    cudaFree(d.s);
    cudaFree(d.t);
    for (int c = 1; c < N_TILE_CLASSES; ++c) cudaFree(d.x.t[c]);
    cudaFree(d.r);
    cudaFree(const_cast<DevSplit*>(d.split.tab));
    cudaFree(d.split.ws);
    cudaFree(d.split.ctr);
    d = GemmDev();
}

namespace {
using GemmKernel = void (*)(const DevProb*, const DevSeg*, const DevTile*, uint32_t, const DevRow*, SplitArgs,
                            Bases);

// pipeline depth x CTAs per SM of the grouped GEMM, chosen per stage by the autotuner
struct GemmVariant {
    GemmKernel fn;
    const char* name;
    int tile_class;  // which tile list it runs on
    int threads;     // CTA size
};
// Variant 0 multiplies whole stages: it is the one of plans too small to tune, whose CTAs have an
// SM to themselves, and there the second form and its branch cost more than the skipped products
// (H psi of Heisenberg m = 240, 300 19.9, 21.5 us with halves, 19.6, 20.9 without; Hubbard m = 1600,
// full of short stages and tuned to others, 143 us with and 147 without).
// Variant 5 has 64 registers a thread for eight CTAs per SM: it goes without the counts of the
// stages in flight and the test of the warp's place (LEAN), which spilled 80 bytes into every K
// step (4096^3 6.1 TFLOP/s; Heisenberg m = 400 33.5 us on stage 3, 23.5 LEAN).
const GemmVariant kVariants[N_GEMM_VARIANTS] = {
    {gemm_f64_grouped<32, 64, 16, 2, 4, 128, 2, false>, "tile32x64_k16_stages2_ctas4", 0, 128},
    {gemm_f64_grouped<32, 64, 16, 3, 4, 128, 2>, "tile32x64_k16_stages3_ctas4", 0, 128},
    {gemm_f64_grouped<32, 64, 16, 2, 5, 128, 2>, "tile32x64_k16_stages2_ctas5", 0, 128},
    {gemm_f64_grouped<32, 64, 16, 3, 5, 128, 2>, "tile32x64_k16_stages3_ctas5", 0, 128},
    {gemm_f64_grouped<16, 64, 8, 3, 6, 128, 1>, "tile16x64_k8_stages3_ctas6", 1, 128},
    {gemm_f64_grouped<16, 64, 8, 4, 8, 128, 1, false, true>, "tile16x64_k8_stages4_ctas8", 1, 128},
    {gemm_f64_grouped<64, 64, 16, 2, 3, 128, 2>, "tile64x64_k16_stages2_ctas3", 2, 128},
    {gemm_f64_grouped<64, 64, 16, 2, 2, 128, 2>, "tile64x64_k16_stages2_ctas2", 2, 128},
    {gemm_f64_grouped<16, 64, 16, 2, 8, 64, 1>, "tile16x64_k16_warps2_stages2_ctas8", 3, 64},
    {gemm_f64_grouped<16, 64, 16, 3, 8, 64, 1>, "tile16x64_k16_warps2_stages3_ctas8", 3, 64},
    {gemm_f64_grouped<16, 64, 16, 2, 10, 64, 1>, "tile16x64_k16_warps2_stages2_ctas10", 3, 64},
    {gemm_f64_grouped<16, 64, 16, 3, 10, 64, 1>, "tile16x64_k16_warps2_stages3_ctas10", 3, 64},
    {gemm_f64_grouped<128, 32, 16, 2, 2, 128, 4>, "tile128x32_k16_stages2_ctas2", 4, 128},
    {gemm_f64_grouped<128, 32, 16, 2, 3, 128, 4>, "tile128x32_k16_stages2_ctas3", 4, 128},
    {gemm_f64_grouped<64, 32, 8, 3, 4, 128, 2>, "tile64x32_k8_stages3_ctas4", 5, 128},
    {gemm_f64_grouped<64, 32, 8, 4, 5, 128, 2>, "tile64x32_k8_stages4_ctas5", 5, 128},
};

int variant_occupancy(int v) {
    static int occ[N_GEMM_VARIANTS] = {0};
    if (!occ[v]) {
        int o = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kVariants[v].fn, kVariants[v].threads, 0);
        occ[v] = o > 0 ? o : 1;
    }
    return occ[v];
}

// t / n: the tile list of class 0; x: the other classes (a variant whose list is
// absent falls back to variant 0)
// Launch with programmatic stream serialisation (the kernel must begin with
// wait_for_predecessor): its CTAs can be scheduled while the previous kernel's last
// CTAs finish, which hides most of the launch gap between the H·psi stages.
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), uint32_t grid, uint32_t block, size_t smem, cudaStream_t stream,
                       Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

cudaError_t launch_variant(int v, const DevProb* p, const DevSeg* sg, const DevTile* t, uint32_t n,
                           TileLists const& x, const DevRow* rows, SplitArgs const& split, Bases const& bs,
                           cudaStream_t stream) {
    if (!n) return cudaSuccess;
    if (v < 0 || v >= N_GEMM_VARIANTS) v = 0;
    const int c = kVariants[v].tile_class;
    if (c > 0 && !x.t[c]) v = 0;
    if (kVariants[v].tile_class > 0) {
        t = x.t[c];
        n = x.n[c];
    }
    uint32_t grid = std::min<uint32_t>(n, uint32_t(device_sm_count()) * variant_occupancy(v));
    return launch_pdl(kVariants[v].fn, grid, uint32_t(kVariants[v].threads), 0, stream, p, sg, t, n, rows, split, bs);
}
}  // namespace

// 64 x 64 tiles at three CTAs per SM where they fill the chip twice (SU2U1 L=16 m=512 stage 1,
// 472 us against 536 for 32 x 64; on shorter lists the smaller tiles balance better)
int gemm_default_variant(GemmList const& gl) { return gl.tiles_cls[2].size() >= 2 * 3 * B200_SMS ? 6 : 0; }

const char* gemm_variant_name(int v) { return (v >= 0 && v < N_GEMM_VARIANTS) ? kVariants[v].name : "?"; }

cudaError_t launch_gemm(GemmDev const& d, Bases const& bs, cudaStream_t stream) {
    return launch_variant(d.var, d.p, d.s, d.t, d.n, d.x, d.r, d.split, bs, stream);
}

cudaError_t tune_program(DeviceProgram& prog, uint64_t in, uint64_t out, double* T, double* S, cudaStream_t stream) {
    Bases bs{};
    bs.b[BUF_IN] = in;
    bs.b[BUF_OUT] = out;
    bs.b[BUF_T] = reinterpret_cast<uint64_t>(T);
    bs.b[BUF_S] = reinterpret_cast<uint64_t>(S);
    cudaEvent_t e0, e1;
    cudaError_t e;
    if ((e = cudaEventCreate(&e0)) != cudaSuccess) return e;
    if ((e = cudaEventCreate(&e1)) != cudaSuccess) {
        cudaEventDestroy(e0);
        return e;
    }
    struct Stage {
        const DevProb* p;
        const DevSeg* s;
        const DevTile* t;
        uint32_t n;
        TileLists x;
        const DevRow* r;
        SplitArgs split;
        int* var;
    } stages[2] = {{prog.d_p1, prog.d_s1, prog.d_t1, prog.n_t1, prog.x1, prog.d_r1, {}, &prog.var1},
                   {prog.d_p3, prog.d_s3, prog.d_t3, prog.n_t3, prog.x3, nullptr, {}, &prog.var3}};
    if (prog.own3)
        stages[1] = Stage{prog.f3.p, prog.f3.s, prog.f3.t, prog.f3.n, prog.f3.x, nullptr, prog.f3.split, &prog.var3};
    // stage 1 writes T, read by nothing else here; stage 3 reads S: both are timed on the
    // plan's current scratch contents (the kernels' speed does not depend on the values)
    // the clocks settle on a short run of the default variant first; then every
    // variant is timed once per round, round-robin, and keeps its best round, so a
    // clock ramp or a stray slow launch favours no variant; a variant must beat the
    // default by 1.5% to replace it (at QC L=24 m=2000 the 64x64 stage-3 variants run 4%
    // faster than the default inside H psi, which a 3% margin missed in some runs)
    constexpr int ROUNDS = 4;
    for (auto& st : stages) {
        if (!st.n) continue;
        for (int w = 0; w < 8 && e == cudaSuccess; ++w) e = launch_variant(0, st.p, st.s, st.t, st.n, st.x, st.r, st.split, bs, stream);
        float best_v[N_GEMM_VARIANTS];
        for (int v = 0; v < N_GEMM_VARIANTS; ++v) best_v[v] = 1e30f;
        for (int round = 0; round < ROUNDS && e == cudaSuccess; ++round)
            for (int v = 0; v < N_GEMM_VARIANTS && e == cudaSuccess; ++v) {
                cudaEventRecord(e0, stream);
                e = launch_variant(v, st.p, st.s, st.t, st.n, st.x, st.r, st.split, bs, stream);
                cudaEventRecord(e1, stream);
                if (e == cudaSuccess) e = cudaEventSynchronize(e1);
                float ms = 0.f;
                cudaEventElapsedTime(&ms, e0, e1);
                if (round > 0 || v > 0) best_v[v] = std::min(best_v[v], ms);  // round 0 of v 0 is a warm-up
            }
        int bv = 0;
        for (int v = 1; v < N_GEMM_VARIANTS; ++v)
            if (best_v[v] < best_v[bv] * (bv == 0 ? 0.985f : 1.0f)) bv = v;
        *st.var = bv;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    prog.tuned = e == cudaSuccess;
    return e;
}

cudaError_t run_sbuild(DeviceProgram const& prog, double* T, double* S, cudaStream_t stream) {
    const uint32_t sms = uint32_t(device_sm_count());
    if (prog.n_litems) {
        // 8 warps per CTA, up to 8 CTAs per SM resident
        uint32_t grid = std::min<uint32_t>((prog.n_litems + 7) / 8, sms * 8);
        cudaError_t e = launch_pdl(sbuild_lines, grid, 256, 0, stream, static_cast<const DevSLine*>(prog.d_lines),
                                   static_cast<const DevSTerm*>(prog.d_terms),
                                   static_cast<const DevSItem*>(prog.d_litems), prog.n_litems, S,
                                   static_cast<const double*>(T), prog.n_gitems ? 1 : 0);
        if (e != cudaSuccess) return e;
    }
    // the items of groups of up to 8 lines come first (prog.n_gitems8 of them)
    int after = prog.n_litems ? 1 : 0;
    auto groups_launch = [&](auto kernel, size_t smem, int minb, const DevSItem* items, uint32_t n,
                             int more) -> cudaError_t {
        if (!n) return cudaSuccess;
        const int after_sbuild = after;
        after = 1;
        cudaError_t ea = ensure_smem_limit(reinterpret_cast<const void*>(kernel), int(smem));
        if (ea != cudaSuccess) return ea;
        // SGB_WARPS warps per CTA, minb CTAs per SM resident
        const uint32_t grid = std::min<uint32_t>((n + SGB_WARPS - 1) / SGB_WARPS, sms * uint32_t(minb));
        return launch_pdl(kernel, grid, 32 * SGB_WARPS, smem, stream, static_cast<const DevSGroup*>(prog.d_groups),
                          items, n, static_cast<const uint64_t*>(prog.d_gent_t),
                          static_cast<const double*>(prog.d_gent_a), S, static_cast<const double*>(T), prog.d_err,
                          wait_limit_ns(), after_sbuild, more);
    };
    if (prog.n_gitems) {
        const DevSItem* items = static_cast<const DevSItem*>(prog.d_gitems);
        cudaError_t e = groups_launch(sbuild_groups<8>, sgb_smem<8>(), SgbShape<8>::MINB, items, prog.n_gitems8,
                                      prog.n_gitems > prog.n_gitems8 ? 1 : 0);
        if (e != cudaSuccess) return e;
        e = groups_launch(sbuild_groups<SG_LINES>, sgb_smem<SG_LINES>(), SgbShape<SG_LINES>::MINB,
                          items + prog.n_gitems8, prog.n_gitems - prog.n_gitems8, 0);
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

bool sbuild_timed_out(DeviceProgram const& prog) {
    if (!prog.d_err) return false;
    int v = 0;
    if (cudaMemcpy(&v, prog.d_err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return false;
    if (v) cudaMemset(prog.d_err, 0, sizeof(int));
    return v != 0;
}

int device_sm_count() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : int(B200_SMS);
}

cudaError_t run_stages12(DeviceProgram const& prog, uint64_t in, uint64_t out, double* T, double* S,
                         cudaStream_t stream) {
    Bases bs{};
    bs.b[BUF_IN] = in;
    bs.b[BUF_OUT] = out;
    bs.b[BUF_T] = reinterpret_cast<uint64_t>(T);
    bs.b[BUF_S] = reinterpret_cast<uint64_t>(S);
    bs.b[BUF_ABS] = 0;
    launch_variant(prog.var1, prog.d_p1, prog.d_s1, prog.d_t1, prog.n_t1, prog.x1, prog.d_r1, SplitArgs{}, bs, stream);
    cudaError_t e = run_sbuild(prog, T, S, stream);
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

cudaError_t run_program(DeviceProgram const& prog, uint64_t in, uint64_t out, double* T, double* S,
                        cudaStream_t stream, cudaEvent_t const* ev, bool staged) {
    Bases bs{};
    bs.b[BUF_IN] = in;
    bs.b[BUF_OUT] = out;
    bs.b[BUF_T] = reinterpret_cast<uint64_t>(T);
    bs.b[BUF_S] = reinterpret_cast<uint64_t>(S);
    bs.b[BUF_ABS] = 0;
    if (ev) cudaEventRecord(ev[0], stream);
    if (prog.chained && !staged) {
        // timed as the contraction (stage 2)
        if (ev) cudaEventRecord(ev[1], stream);
        if (ev) cudaEventRecord(ev[2], stream);
        const cudaError_t e = launch_chain(prog.d_chain, bs, stream);
        if (ev) cudaEventRecord(ev[3], stream);
        return e != cudaSuccess ? e : cudaGetLastError();
    }
    launch_variant(prog.var1, prog.d_p1, prog.d_s1, prog.d_t1, prog.n_t1, prog.x1, prog.d_r1, SplitArgs{}, bs, stream);
    if (ev) cudaEventRecord(ev[1], stream);
    cudaError_t e = run_sbuild(prog, T, S, stream);
    if (e != cudaSuccess) return e;
    if (ev) cudaEventRecord(ev[2], stream);
    if (prog.own3) {
        GemmDev f3 = prog.f3;
        f3.var = prog.var3;
        if ((e = launch_gemm(f3, bs, stream)) != cudaSuccess) return e;
    } else {
        launch_variant(prog.var3, prog.d_p3, prog.d_s3, prog.d_t3, prog.n_t3, prog.x3, nullptr, SplitArgs{}, bs, stream);
    }
    if (ev) cudaEventRecord(ev[3], stream);
    return cudaGetLastError();
}

}  // namespace dmrgb200

using namespace dmrgb200;

namespace dmrgb200 {
dmrgb200_status noalloc_fail(dmrgb200_status s, std::string const& msg);
}

extern "C" dmrgb200_status dmrgb200_dgemm_f64(uint32_t M, uint32_t N, uint32_t K, const double* A, uint64_t lda,
                                              const double* B, uint64_t ldb, double* C, uint64_t ldc, int variant,
                                              void* cuda_stream) {
    if (!A || !B || !C) return noalloc_fail(DMRGB200_INVALID_ARGUMENT, "null argument");
    if (lda < M || ldb < K || ldc < M) return noalloc_fail(DMRGB200_INVALID_ARGUMENT, "leading dimension too small");
    if (variant < 0 || variant >= N_GEMM_VARIANTS) return noalloc_fail(DMRGB200_INVALID_ARGUMENT, "unknown variant");
    if (lda > UINT32_MAX || ldb > UINT32_MAX || ldc > UINT32_MAX)
        return noalloc_fail(DMRGB200_INVALID_ARGUMENT, "leading dimension above 2^32");
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    GemmList gl;
    DevProb pr{};
    pr.M = M;
    pr.N = N;
    pr.C = DevOp{reinterpret_cast<uint64_t>(C) / 8, 0, uint32_t(ldc), uint16_t(BUF_ABS), 0};
    pr.seg_begin = 0;
    pr.seg_end = 1;
    DevSeg sg{};
    sg.A = DevOp{reinterpret_cast<uint64_t>(A) / 8, 0, uint32_t(lda), uint16_t(BUF_ABS), 0};
    sg.B = DevOp{reinterpret_cast<uint64_t>(B) / 8, 0, uint32_t(ldb), uint16_t(BUF_ABS), 0};
    sg.K = K;
    gl.probs.push_back(pr);
    gl.segs.push_back(sg);
    add_tiles(gl, 0, 1);
    GemmDev d;
    cudaError_t e = upload_gemm(gl, d);
    if (e == cudaSuccess) {
        d.var = variant;
        e = launch_gemm(d, Bases{}, st);
    }
    cudaError_t e2 = cudaStreamSynchronize(st);
    free_gemm(d);
    if (e == cudaSuccess) e = e2;
    if (e != cudaSuccess)
        return noalloc_fail(e == cudaErrorMemoryAllocation ? DMRGB200_OUT_OF_MEMORY : DMRGB200_DEVICE_ERROR,
                            std::string("FP64 GEMM: ") + cudaGetErrorString(e));
    return DMRGB200_OK;
}
