// H psi and boundary steps of plans with few terms per line, in one launch.
//
// For lattice models (Hubbard, Heisenberg, Bose-Hubbard) a line of S is the sum of about
// two T blocks, and a T block is read by about two terms.  Forming T and S and contracting
// S takes three launches, each short of work, and writes and reads both matrices once.
// Here every output tile runs its terms as a chain of two products in registers,
//
//   C (M x N) = sum over lines  A (M x K1) * [ sum over terms  alpha P (K1 x K2) Q (K2 x N) ]
//
//   H psi:       A = L block           P = psi slice       Q = R block
//   left step:   A = bra^T slice       P = L block         Q = ket slice
//   right step:  A = bra slice         P = R block^T       Q = ket slice^T   (C transposed)
//
// (T = P Q per term, S = the bracket), on the FP64 tensor cores (DMMA m8n8k4).  T and S are
// never formed: a warp owns a tile of at most 32 rows and eight columns, accumulates its
// columns of the bracket transposed, 8 x K1, in registers, and multiplies them by A.  An
// accumulator of a DMMA holds row g, columns 2q and 2q + 1 in lane 4 g + q, and as the second
// product's B operand (k in the lane's q, column in its g) the even columns make one K step
// and the odd ones another, so no data moves between the two products; A is read at the same
// permuted k.  The terms' weights scale Q.
//
// What bounds plans of small blocks is instructions and latency, not the pipe: the three
// launches spend 14 to 16 instructions per DMMA on 17 to 52 wide blocks (copies, addresses,
// descriptors, epilogues).  So the fragments are read straight from L1 / L2 (the four warps of a CTA are
// column tiles of one problem and share P and A there), addressed by one add each; the reads
// of a K step are in flight while the step before multiplies, across terms; the term records
// go to shared memory before the wait for the previous kernel.  Where the tiles are too few
// to fill the SMs, a tile's lines are split over 2 or 4 warps, added in order at the end.
// Every output element is summed in an order fixed by the plan: bitwise reproducible.
#include <algorithm>

#include "device.hpp"

namespace dmrgb200 {

namespace {

constexpr int CH_WARPS = 4;    // per CTA
constexpr int CH_REC = 64;     // term records per tile held in shared memory
constexpr uint32_t CH_TILE = 32;  // rows and K1 of a tile at most

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ const double* operand(Bases const& bs, uint64_t ref) {
    return reinterpret_cast<const double*>(base_of(bs, uint32_t(ref >> 56)) + 8ull * (ref & ((1ull << 56) - 1)));
}

// B: blocks of eight in K1 and M held by a warp
template <int B, int MINB>
__global__ void __launch_bounds__(32 * CH_WARPS, MINB)
    chain_tiles(const DevChainTile* __restrict__ tiles, uint32_t n_tiles, const DevChainTerm* __restrict__ terms,
                Bases bases, int split) {
    __shared__ DevChainTerm recs[CH_WARPS][CH_REC];
    __shared__ double part[CH_WARPS][B][2][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    const int slot = warp / split, share = warp % split;  // tile of the CTA, this warp's part of its lines
    const uint32_t ti = blockIdx.x * (CH_WARPS / split) + slot;
    const bool live = ti < n_tiles;
    // the tables do not change between launches: read before the wait
    DevChainTile t{};
    if (live) t = tiles[ti];
    const uint32_t* bounds = tiles[live ? ti : 0].bounds;
    const uint32_t t0 = live ? bounds[share * (CH_WARPS / split)] : 0, t1 = live ? bounds[(share + 1) * (CH_WARPS / split)] : 0;
    const bool held = t1 - t0 <= uint32_t(CH_REC);
    if (held) {
        const uint4* src = reinterpret_cast<const uint4*>(terms + t0);
        uint4* dst = reinterpret_cast<uint4*>(recs[warp]);
        for (uint32_t i = lane; i < (t1 - t0) * (sizeof(DevChainTerm) / 16); i += 32) dst[i] = src[i];
    }
    __syncwarp();
    const DevChainTerm* rec = held ? recs[warp] : terms + t0;
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const int M = int(t.rows), N = int(t.cols), mb = (M + 7) / 8, n_terms = int(t1 - t0);
    // z: the product of the current term.  The terms of a line before it lie added up in shared
    // memory (`open`: there are any): each is summed by itself and then added, as T and S are in the
    // stages.  Adding a small term's products one by one to a large sum would round at the size of
    // the large one every time (errors against long double up to 1.3 times the stages' on boundary
    // steps, 0.75 to 0.95 times this way).
    bool open = false;
    double acc[B][2], z[B][2];
#pragma unroll
    for (int j = 0; j < B; ++j) acc[j][0] = acc[j][1] = z[j][0] = z[j][1] = 0.0;

    // cursor of the reads: term kt, K step s; this lane reads Q(k2 = 4 s + q, column g) and
    // P(k1 = 8 x + g, k2 = 4 s + q).  Rows and columns outside the tile repeat the last one
    // inside (their products are not used); K2 rows past the end read zero.
    int kt = 0, s = 0, k2 = 0, kb = 0;
    const double *qp = nullptr, *pp = nullptr;
    uint32_t qs = 0, ps = 0;
    uint32_t ro[B];
    double alpha = 0.0;
    auto enter = [&]() {
        if (kt >= n_terms) return;
        const DevChainTerm& T = rec[kt];
        const int k1 = int(T.k1);
        k2 = int(T.k2);
        kb = (k1 + 7) / 8;
        alpha = T.alpha;
        qp = operand(bases, T.q) + (uint64_t(q) * T.q2 + uint64_t(int(t.n0) + min(g, N - 1)) * T.qn);
        pp = operand(bases, T.p) + uint64_t(q) * T.p2;
        qs = 4u * T.q2;
        ps = 4u * T.p2;
#pragma unroll
        for (int x = 0; x < B; ++x) ro[x] = uint32_t(min(8 * x + g, k1 - 1)) * T.p1;
    };
    struct Step {
        double f, p[B];
        int code;  // blocks of K1, and above bit 3 one more than the term that ends with this step (0: none)
    };
    auto load = [&](Step& st) -> bool {
        if (kt >= n_terms) return false;
        st.code = kb;
        if (s + 4 <= k2) {
            st.f = alpha * *qp;
#pragma unroll
            for (int x = 0; x < B; ++x)
                if (x < kb) st.p[x] = pp[ro[x]];
        } else {
            const bool in = s + q < k2;
            st.f = in ? alpha * *qp : 0.0;
#pragma unroll
            for (int x = 0; x < B; ++x)
                if (x < kb) st.p[x] = in ? pp[ro[x]] : 0.0;
        }
        s += 4;
        qp += qs;
        pp += ps;
        if (s >= k2) {
            st.code |= ++kt << 3;
            s = 0;
            enter();
        }
        return true;
    };
    auto consume = [&](Step const& st) {
#pragma unroll
        for (int x = 0; x < B; ++x) {
            if (x >= (st.code & 7)) break;
            dmma(z[x], st.f, st.p[x]);
        }
        if (st.code < 8) return;
        const DevChainTerm& T = rec[(st.code >> 3) - 1];
        double(*before)[2][32] = part[warp];
        if (open) {
#pragma unroll
            for (int x = 0; x < B; ++x) {
                z[x][0] += before[x][0][lane];
                z[x][1] += before[x][1][lane];
            }
        }
        open = !T.last;
        if (open) {
#pragma unroll
            for (int x = 0; x < B; ++x) {
                before[x][0][lane] = z[x][0];
                before[x][1][lane] = z[x][1];
                z[x][0] = z[x][1] = 0.0;
            }
            return;
        }
        // acc (M x 8) += A z^T, the even and the odd k of every block of eight
        const int k1 = int(T.k1);
        const double* A = operand(bases, T.a);
        uint32_t ao[B];
#pragma unroll
        for (int j = 0; j < B; ++j) ao[j] = uint32_t(min(8 * j + g, M - 1)) * T.am;
        double a[2][B];
        auto fetch = [&](int i, double (&d)[B]) {  // K step i: k1 = 8 (i / 2) + 2 q + i % 2
            const int k = 8 * (i >> 1) + 2 * q + (i & 1);
            const double* ap = A + uint64_t(min(k, k1 - 1)) * T.ak;
#pragma unroll
            for (int j = 0; j < B; ++j)
                if (j < mb) d[j] = k < k1 ? ap[ao[j]] : 0.0;
        };
        fetch(0, a[0]);
#pragma unroll
        for (int i = 0; i < 2 * B; ++i) {
            if (8 * (i >> 1) >= k1) break;
            if (i + 1 < 2 * B && 8 * ((i + 1) >> 1) < k1) fetch(i + 1, a[(i + 1) & 1]);
            // columns of z past K1 repeat another one: not used
            const double b = 8 * (i >> 1) + 2 * q + (i & 1) < k1 ? z[i >> 1][i & 1] : 0.0;
#pragma unroll
            for (int j = 0; j < B; ++j) {
                if (j >= mb) break;
                dmma(acc[j], a[i & 1][j], b);
            }
        }
#pragma unroll
        for (int x = 0; x < B; ++x) z[x][0] = z[x][1] = 0.0;
    };
    enter();
    Step u, v;
    bool hu = load(u), hv;
    for (;;) {
        if (!hu) break;
        hv = load(v);
        consume(u);
        if (!hv) break;
        hu = load(u);
        consume(v);
    }

    if (split > 1) {
        if (share > 0) {
#pragma unroll
            for (int j = 0; j < B; ++j) {
                part[warp][j][0][lane] = acc[j][0];
                part[warp][j][1][lane] = acc[j][1];
            }
        }
        __syncthreads();
        if (share > 0) return;
        for (int w = warp + 1; w < warp + split; ++w)
#pragma unroll
            for (int j = 0; j < B; ++j) {
                acc[j][0] += part[w][j][0][lane];
                acc[j][1] += part[w][j][1][lane];
            }
    }
    if (!live) return;
    // the tile's output is read again here instead of being held in registers through the products
    uint32_t to = ti;
    asm volatile("" : "+r"(to));
    const DevChainTile& o = tiles[to];
    const uint32_t cm = o.cm, cn = o.cn;
    double* C = const_cast<double*>(operand(bases, o.c)) + uint64_t(o.n0) * cn;
#pragma unroll
    for (int j = 0; j < B; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int r = 8 * j + g, c = 2 * q + e;
            if (r < M && c < N) C[uint64_t(r) * cm + uint64_t(c) * cn] = acc[j][e];
        }
}

uint64_t ref(uint16_t buf, uint64_t off) { return (uint64_t(buf) << 56) | off; }

// one term and one line of a problem before they are cut into stages
struct Term {
    double alpha;
    uint64_t p, q;  // P(k1, k2) at p + k1 p1 + k2 p2, Q(k2, n) at q + k2 q2 + n qn
    uint32_t p1, p2, q2, qn, k2;
};
struct Line {
    uint64_t a;  // A(m, k1) at a + m am + k1 ak
    uint32_t am, ak, k1, term_begin, term_end;
};
// a problem before it is cut into tiles
struct ChainProblem {
    uint64_t c;  // output reference
    uint32_t M, N, cm, cn;
    uint32_t line_begin, line_end;
    uint64_t work;
};

// Where the chain is faster than the three launches, both measured, in us: Hubbard m = 100 6.9
// against 15.0, 200 7.7 / 17, 333 12.4 / 20.3, 480 19.5 / 28 (blocks of at most 25 rows), 700 45
// / 42 (36 rows), 1024 85 / 63; Heisenberg m = 64 6.7 / 12.2, 200 16.0 / 18 (30 rows).  Larger
// blocks keep the pipe busier through shared memory, and computing T anew for every term that
// reads it starts to cost.  Read off the plan's sizes before anything is built: most plans that
// are too large are so by these.
bool chain_sizes(FlatPlan const& p) {
    const bool left = p.kind == KIND_LEFT;
    uint64_t tiles = 0;
    auto problem = [&](uint32_t M, uint32_t N) {
        tiles += (N + 7) / 8;
        return M <= CH_TILE;
    };
    std::vector<char> written(p.out_rows.size(), 0);
    for (uint32_t c = 0; c < p.n_cohorts(); ++c) {
        const bool first = p.kind != KIND_HPSI || !written[p.c_rb[c]];
        if (p.kind == KIND_HPSI) {
            written[p.c_rb[c]] = 1;
        } else {
            for (uint32_t b = 0; b < p.c_nsrows[c]; ++b)
                if (!problem(left ? p.c_ls[c] : p.c_rs[c], left ? p.c_rs[c] : p.c_ls[c])) return false;
        }
        for (uint32_t u = p.c_unit[c]; u < p.c_unit[c + 1]; ++u) {
            if (!p.u_ms[u]) continue;
            if (p.kind == KIND_HPSI && first && !problem(p.out_rows[p.c_rb[c]], p.u_ms[u])) return false;
            const uint32_t K1 = p.kind == KIND_HPSI ? p.c_ls[c] : p.u_ms[u];
            if (K1 > CH_TILE)
                for (uint32_t l = p.u_line[u]; l < p.u_line[u + 1]; ++l)
                    if (p.l_term[l] < p.l_term[l + 1]) return false;
        }
    }
    for (uint32_t ob = 0; p.kind == KIND_HPSI && ob < p.out_rows.size(); ++ob)
        if (!written[ob] && !problem(p.out_rows[ob], p.out_cols[ob])) return false;
    return tiles <= 16 * B200_SMS;
}

}  // namespace

bool build_chain(FlatPlan const& p, std::vector<uint64_t> const& stage3_bnd, std::vector<uint64_t> const& stage1_bnd,
                 std::vector<uint64_t> const& outptr, ChainList& cl) {
    cl = ChainList();
    const uint32_t nc = p.n_cohorts();
    const bool left = p.kind == KIND_LEFT;
    // lines of few terms only: the chain computes a term's T anew for every line that reads it
    if (!nc || p.n_terms() > 4ull * p.n_lines() || !chain_sizes(p)) return false;
    // units of every cohort by offset; they must tile the cohort's S
    std::vector<std::vector<uint32_t>> units(nc);
    for (uint32_t c = 0; c < nc; ++c) {
        for (uint32_t u = p.c_unit[c]; u < p.c_unit[c + 1]; ++u)
            if (p.u_ms[u]) units[c].push_back(u);
        std::sort(units[c].begin(), units[c].end(), [&](uint32_t a, uint32_t b) { return p.u_offset[a] < p.u_offset[b]; });
        uint32_t at = 0;
        for (uint32_t u : units[c]) {
            if (p.u_offset[u] != at) return false;
            at += p.u_ms[u];
        }
        if (at != p.c_stripe[c]) return false;
    }
    std::vector<int64_t> line_of;
    auto lines = [&](uint32_t c, uint32_t u) {
        line_of.assign(p.c_nsrows[c], -1);
        for (uint32_t l = p.u_line[u]; l < p.u_line[u + 1]; ++l) line_of[p.l_b1[l]] = l;
    };
    std::vector<ChainProblem> probs;
    std::vector<Line> all_lines;
    std::vector<Term> all_terms;
    all_lines.reserve(2 * size_t(p.n_lines()));  // a line is read by one or two problems
    all_terms.reserve(2 * size_t(p.n_terms()));
    uint64_t macs = 0, staged = 0;
    bool whole = true;  // every term reads one whole T block
    auto add_line = [&](ChainProblem& pr, int64_t l, uint64_t a, uint32_t am, uint32_t ak, uint32_t K1) {
        if (l < 0 || !K1 || p.l_term[l] == p.l_term[l + 1]) return;
        Line L{};
        L.a = a;
        L.am = am;
        L.ak = ak;
        L.k1 = K1;
        L.term_begin = uint32_t(all_terms.size());
        for (uint32_t k = p.l_term[l]; k < p.l_term[l + 1]; ++k) {
            const uint32_t t = p.term_t[k], lb = p.t_lb[t], Mt = p.in_rows[lb], br = p.t_brows[t], bc = p.t_bcols[t];
            const uint32_t w = left ? br : bc;
            const bool tr = p.t_trans[t] != 0;
            // the T block the term reads: term_col counts columns of T (H psi, right step) or
            // rows of the stacked blocks (left step)
            if (!w || p.term_col[k] % w) {
                whole = false;
                return;
            }
            const uint32_t b = p.term_col[k] / w;
            Term T{};
            T.alpha = p.term_alpha[k];
            const uint64_t bnd = stage1_bnd.at(p.t_ci[t]) / 8 + uint64_t(b) * br * bc;
            if (left) {
                // T = B (br x bc) * ket (bc x width), K1 = br, N = width
                if (br != K1 || p.t_width[t] != pr.N) whole = false;
                T.p = ref(BUF_ABS, bnd);
                T.p1 = tr ? bc : 1;
                T.p2 = tr ? 1 : br;
                T.q = ref(BUF_IN, p.in_off[lb] + uint64_t(p.t_col[t]) * bc);
                T.q2 = 1;
                T.qn = bc;
                T.k2 = bc;
                if (Mt != bc) whole = false;  // ket slice columns are bc long
            } else if (p.kind == KIND_HPSI) {
                // T = x (Mt x br) * B (br x bc), K1 = Mt, N = bc
                if (Mt != K1 || bc != pr.N) whole = false;
                T.p = ref(BUF_IN, p.in_off[lb] + uint64_t(p.t_col[t]) * Mt);
                T.p1 = 1;
                T.p2 = Mt;
                T.q = ref(BUF_ABS, bnd);
                T.q2 = tr ? bc : 1;
                T.qn = tr ? 1 : br;
                T.k2 = br;
            } else {
                // T^T = B^T (bc x br) * x^T (br x Mt), K1 = bc, N = Mt
                if (bc != K1 || Mt != pr.N) whole = false;
                T.p = ref(BUF_ABS, bnd);
                T.p1 = tr ? 1 : br;
                T.p2 = tr ? bc : 1;
                T.q = ref(BUF_IN, p.in_off[lb] + uint64_t(p.t_col[t]) * Mt);
                T.q2 = Mt;
                T.qn = 1;
                T.k2 = br;
            }
            all_terms.push_back(T);
            pr.work += uint64_t((K1 + 7) / 8) * ((T.k2 + 3) / 4);
            macs += uint64_t(K1) * T.k2 * pr.N;
        }
        pr.work += uint64_t((K1 + 7) / 8) * 2 * ((pr.M + 7) / 8);
        macs += uint64_t(K1) * pr.M * pr.N;
        L.term_end = uint32_t(all_terms.size());
        all_lines.push_back(L);
    };
    if (p.kind == KIND_HPSI) {
        std::vector<std::vector<uint32_t>> by_out(p.out_rows.size());
        for (uint32_t c = 0; c < nc; ++c) by_out[p.c_rb[c]].push_back(c);
        for (uint32_t ob = 0; ob < p.out_rows.size(); ++ob) {
            auto const& cs = by_out[ob];
            const uint32_t M = p.out_rows[ob];
            if (cs.empty()) {  // no cohort writes the block: zeros
                probs.push_back({ref(BUF_OUT, p.out_off[ob]), M, p.out_cols[ob], 1, M, uint32_t(all_lines.size()),
                                 uint32_t(all_lines.size()), 0});
                continue;
            }
            auto const& first = units[cs[0]];
            for (uint32_t c : cs) {
                if (p.c_stripe[c] != p.out_cols[ob] || p.c_rs[c] != M || units[c].size() != first.size()) return false;
                for (size_t x = 0; x < first.size(); ++x)
                    if (p.u_offset[units[c][x]] != p.u_offset[first[x]]) return false;
            }
            for (size_t x = 0; x < first.size(); ++x) {
                ChainProblem pr{ref(BUF_OUT, p.out_off[ob] + uint64_t(p.u_offset[first[x]]) * M), M,
                                p.u_ms[first[x]], 1, M, uint32_t(all_lines.size()), 0, 0};
                for (uint32_t c : cs) {
                    const uint32_t ls = p.c_ls[c], rs = p.c_rs[c];
                    const uint64_t lbase = stage3_bnd.at(p.c_ci[c]) / 8;
                    lines(c, units[c][x]);
                    for (uint32_t b = 0; b < p.c_nsrows[c]; ++b)
                        add_line(pr, line_of[b], ref(BUF_ABS, lbase + uint64_t(b) * ls * rs), p.c_trans[c] ? ls : 1,
                                 p.c_trans[c] ? 1 : rs, ls);
                }
                pr.line_end = uint32_t(all_lines.size());
                probs.push_back(pr);
            }
        }
    } else {
        for (uint32_t c = 0; c < nc; ++c) {
            const uint32_t ls = p.c_ls[c], rs = p.c_rs[c], stripe = p.c_stripe[c];
            if (p.c_out_ci[c] >= outptr.size()) return false;
            std::vector<std::vector<int64_t>> unit_lines;
            for (uint32_t u : units[c]) {
                lines(c, u);
                unit_lines.push_back(line_of);
            }
            for (uint32_t b = 0; b < p.c_nsrows[c]; ++b) {
                ChainProblem pr{ref(BUF_ABS, outptr[p.c_out_ci[c]] / 8 + uint64_t(b) * ls * rs), left ? ls : rs,
                                left ? rs : ls, left ? 1 : ls, left ? ls : 1, uint32_t(all_lines.size()), 0, 0};
                for (size_t x = 0; x < units[c].size(); ++x) {
                    const uint32_t u = units[c][x], ms = p.u_ms[u];
                    if (left)
                        add_line(pr, unit_lines[x][b], ref(BUF_OUT, p.out_off[p.c_lb[c]] + p.u_offset[u]), stripe, 1, ms);
                    else
                        add_line(pr, unit_lines[x][b], ref(BUF_OUT, p.out_off[p.c_rb[c]] + uint64_t(p.u_offset[u]) * rs), 1, rs,
                                 ms);
                }
                pr.line_end = uint32_t(all_lines.size());
                probs.push_back(pr);
            }
        }
    }
    if (!whole) {
        cl = ChainList();
        return false;
    }
    for (uint32_t t = 0; t < p.n_t(); ++t) staged += p.t_size(t) * (left ? p.t_bcols[t] : p.t_brows[t]);
    for (uint32_t c = 0; c < nc; ++c) staged += uint64_t(p.c_ls[c]) * p.c_nsrows[c] * p.c_rs[c] * p.c_stripe[c];
    // T computed anew for every term that reads it must not outweigh the stages' work
    if (probs.empty() || macs > 2 * staged) {
        cl = ChainList();
        return false;
    }
    // the records of every problem: a line's terms, the last one closing the line; then tiles
    // of all rows and eight columns, the longest problems first
    std::stable_sort(probs.begin(), probs.end(), [](ChainProblem const& a, ChainProblem const& b) { return a.work > b.work; });
    uint32_t d1 = 1, dm = 1;
    std::vector<uint64_t> cost;  // work up to each line end of a problem
    std::vector<uint32_t> ends;  // record index there
    cl.terms.reserve(all_terms.size());
    uint64_t n_tiles = 0;
    for (auto const& pr : probs) n_tiles += (pr.N + 7) / 8;
    cl.tiles.reserve(n_tiles);
    for (auto const& pr : probs) {
        const uint32_t begin = uint32_t(cl.terms.size());
        cost.assign(1, 0);
        ends.assign(1, begin);
        for (uint32_t l = pr.line_begin; l < pr.line_end; ++l) {
            Line const& L = all_lines[l];
            d1 = std::max(d1, L.k1);
            uint64_t w = cost.back();
            for (uint32_t k = L.term_begin; k < L.term_end; ++k) {
                Term const& T = all_terms[k];
                DevChainTerm r{};
                r.alpha = T.alpha;
                r.p = T.p;
                r.q = T.q;
                r.a = L.a;
                r.p1 = T.p1;
                r.p2 = T.p2;
                r.q2 = T.q2;
                r.qn = T.qn;
                r.am = L.am;
                r.ak = L.ak;
                r.k1 = L.k1;
                r.k2 = T.k2;
                r.last = k + 1 == L.term_end;
                cl.terms.push_back(r);
                w += uint64_t((L.k1 + 7) / 8) * ((T.k2 + 3) / 4);
            }
            w += uint64_t((L.k1 + 7) / 8) * 2 * ((pr.M + 7) / 8);
            cost.push_back(w);
            ends.push_back(uint32_t(cl.terms.size()));
        }
        // the lines in CH_WARPS shares of about equal work
        uint32_t bounds[CH_WARPS + 1];
        for (int x = 0; x <= CH_WARPS; ++x) {
            const uint64_t want = cost.back() * x / CH_WARPS;
            size_t i = size_t(std::lower_bound(cost.begin(), cost.end(), want) - cost.begin());
            if (i > 0 && want - cost[i - 1] < cost[i] - want) --i;
            bounds[x] = x == 0 ? begin : x == CH_WARPS ? ends.back() : ends[i];
        }
        dm = std::max(dm, pr.M);
        for (uint32_t n0 = 0; pr.M && n0 < pr.N; n0 += 8) {
            DevChainTile t{};
            t.c = pr.c;
            t.n0 = n0;
            t.rows = pr.M;
            t.cols = std::min<uint32_t>(pr.N - n0, 8);
            t.cm = pr.cm;
            t.cn = pr.cn;
            std::copy(bounds, bounds + CH_WARPS + 1, t.bounds);
            cl.tiles.push_back(t);
        }
    }
    // Shares per tile: more warps in flight where the tiles are few (Heisenberg m = 64, 55 tiles:
    // 10.4 us whole, 6.9 in four; Hubbard m = 200: 11.4 and 7.7; m = 480: 26.4 whole, 20.5 in
    // two, 26.3 in four).
    cl.blocks = std::max(2, int((std::max(d1, dm) + 7) / 8));
    if (cl.blocks > int(CH_TILE / 8)) {  // chain_sizes has seen to it
        cl = ChainList();
        return false;
    }
    cl.split = cl.tiles.size() < 6 * B200_SMS ? 4 : cl.tiles.size() < 10 * B200_SMS ? 2 : 1;
    return true;
}

cudaError_t launch_chain(ChainDev const& d, Bases const& bs, cudaStream_t stream) {
    if (!d.n) return cudaSuccess;
    const uint32_t per = uint32_t(CH_WARPS / d.split);  // tiles per CTA
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((d.n + per - 1) / per);
    cfg.blockDim = dim3(32 * CH_WARPS);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto* kernel = d.blocks == 2 ? chain_tiles<2, 4> : d.blocks == 3 ? chain_tiles<3, 4> : chain_tiles<4, 3>;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<const DevChainTile*>(d.tiles), d.n,
                              static_cast<const DevChainTerm*>(d.terms), bs, d.split);
}

}  // namespace dmrgb200
