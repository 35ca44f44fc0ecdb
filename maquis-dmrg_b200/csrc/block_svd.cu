// Block-wise thin SVD and block copies for the two-site split on the device.
//
// The reference splits a two-site tensor by a thin SVD of every symmetry block
// of the matrix Theta (rows (l, s1), columns (s2, r) of one middle charge),
// keeps the largest singular values over all blocks and writes U and S V^T (or
// U S and V^T) back as site tensors (svd: block_matrix/block_matrix_algorithms.h:
// 95-113; svd_truncate: :185-298; TwoSiteTensor::split_mps_l2r / r2l:
// mp_tensors/twositetensor.hpp:153-200).
//
// svd_cluster: blocks of up to 256 x 256, one thread-block cluster per block, pivoted QR
// then one-sided Jacobi on R^T with the columns in registers (see the kernel).
//
// block_svd_jacobi: larger blocks, and the blocks svd_cluster hands back (a vanishing
// pivot, non-finite input); one CTA of 16 warps per block, one-sided (Hestenes) Jacobi.  The block is
// taken as m x n columns with n = min(rows, cols) (the transpose when rows < cols).
// Column pairs are orthogonalised in round-robin order, n/2 disjoint pairs per
// round spread over the warps; a pair rotates when |g_p . g_q| > tol |g_p| |g_q|
// (tol = sqrt(m) eps), on the block scaled exactly by a power of two to a
// largest element in [1, 2).  Sweeps repeat until one makes no rotation (at most
// SVD_MAX_SWEEPS; exhausting them sets the error flag).  Then sigma_j = |g_j|,
// U = G / sigma, V is the accumulated rotation, all sorted by descending sigma.
// The columns and V live in shared memory when they fit, else in a global
// scratch (L2-resident at these sizes).  There is no spin-wait: every loop is
// bounded.
//
// copy_blocks: dst block = src block (column-major, own leading dimensions),
// optionally scaled per row or per column; it gathers Theta from the two-site
// tensor and scatters U / V^T into the new site tensors.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/dmrgb200.h"
#include "device.hpp"

namespace dmrgb200 {

dmrgb200_status noalloc_fail(dmrgb200_status s, std::string const& msg);

namespace {

constexpr int SVD_THREADS = 512, SVD_WARPS = SVD_THREADS / 32, SVD_MAX_SWEEPS = 60;
constexpr int SVD_REG = 8;  // register path for columns of up to 32 * SVD_REG elements
constexpr size_t SVD_SMEM_LIMIT = 200 * 1024;

struct SvdBlock {
    const double* a;  // rows x cols, ld = rows
    double* u;        // rows x k, ld = rows
    double* s;        // k
    double* vt;       // k x cols, ld = k
    double* work;     // null: shared memory
    uint32_t rows, cols;
    // work of block_svd_jacobi: 1 to do; 0 done by svd_cluster, which sets it back to 1 for
    // a block it hands over
    int general;
    int pad;
};

// work elements of one block: G (m x n), V (n x n), sigma (n), rank table (n ints in n doubles);
// svd_cluster: reflectors (m x n), R (n x n), sigma (n), pivot columns and their taus
__host__ __device__ inline size_t svd_work_elems(uint32_t rows, uint32_t cols) {
    const size_t m = rows > cols ? rows : cols, n = rows < cols ? rows : cols;
    return m * n + n * n + 3 * n;
}

__device__ inline double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Rutishauser's rotation of columns p, q from their squared norms al, be and
// inner product ga: t the smaller root of t^2 + 2 zeta t - 1 = 0.  Returns false
// when the pair is already orthogonal to tol.
__device__ inline bool jacobi_cs(double al, double be, double ga, double tol, double& c, double& s) {
    if (ga == 0.0 || !(fabs(ga) > tol * sqrt(al) * sqrt(be))) return false;
    const double zeta = (be - al) / (2.0 * ga);
    const double az = fabs(zeta);
    const double t = (az > 1e150) ? 0.5 / zeta : copysign(1.0, zeta) / (az + sqrt(1.0 + zeta * zeta));
    c = 1.0 / sqrt(1.0 + t * t);
    s = c * t;
    return true;
}

// One pair, columns of up to 32 * SVD_REG elements: every lane loads its
// elements of both columns in one unrolled batch (one memory latency instead of
// one per element), and the same for V when the pair rotates.
__device__ inline bool pair_rotate_regs(double* gp, double* gq, uint32_t m, double* vp, double* vq, uint32_t n,
                                        double tol) {
    const uint32_t lane = threadIdx.x & 31u;
    double x[SVD_REG], y[SVD_REG];
#pragma unroll
    for (int r = 0; r < SVD_REG; ++r) {
        const uint32_t i = lane + 32u * r;
        x[r] = i < m ? gp[i] : 0.0;
        y[r] = i < m ? gq[i] : 0.0;
    }
    double al = 0.0, be = 0.0, ga = 0.0;
#pragma unroll
    for (int r = 0; r < SVD_REG; ++r) {
        al = fma(x[r], x[r], al);
        be = fma(y[r], y[r], be);
        ga = fma(x[r], y[r], ga);
    }
    al = warp_sum(al);
    be = warp_sum(be);
    ga = warp_sum(ga);
    double c, s;
    if (!jacobi_cs(al, be, ga, tol, c, s)) return false;
#pragma unroll
    for (int r = 0; r < SVD_REG; ++r) {
        const uint32_t i = lane + 32u * r;
        if (i < m) {
            gp[i] = c * x[r] - s * y[r];
            gq[i] = s * x[r] + c * y[r];
        }
    }
#pragma unroll
    for (int r = 0; r < SVD_REG; ++r) {
        const uint32_t i = lane + 32u * r;
        x[r] = i < n ? vp[i] : 0.0;
        y[r] = i < n ? vq[i] : 0.0;
    }
#pragma unroll
    for (int r = 0; r < SVD_REG; ++r) {
        const uint32_t i = lane + 32u * r;
        if (i < n) {
            vp[i] = c * x[r] - s * y[r];
            vq[i] = s * x[r] + c * y[r];
        }
    }
    return true;
}

// The same for longer columns, element by element.
__device__ inline bool pair_rotate_loop(double* gp, double* gq, uint32_t m, double* vp, double* vq, uint32_t n,
                                        double tol) {
    const uint32_t lane = threadIdx.x & 31u;
    double al = 0.0, be = 0.0, ga = 0.0;
    for (uint32_t i = lane; i < m; i += 32) {
        const double x = gp[i], y = gq[i];
        al = fma(x, x, al);
        be = fma(y, y, be);
        ga = fma(x, y, ga);
    }
    al = warp_sum(al);
    be = warp_sum(be);
    ga = warp_sum(ga);
    double c, s;
    if (!jacobi_cs(al, be, ga, tol, c, s)) return false;
    for (uint32_t i = lane; i < m; i += 32) {
        const double x = gp[i], y = gq[i];
        gp[i] = c * x - s * y;
        gq[i] = s * x + c * y;
    }
    for (uint32_t i = lane; i < n; i += 32) {
        const double x = vp[i], y = vq[i];
        vp[i] = c * x - s * y;
        vq[i] = s * x + c * y;
    }
    return true;
}

// Sum and maximum over the warp of several values at once (independent chains overlap).
template <int N>
__device__ __forceinline__ void warp_sums(double (&v)[N]) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
}

// The rotation of a pair as jacobi_cs gives it, with one square root, one division and
// one reciprocal square root instead of seven such operations in sequence:
// t = 2 ga / (d + sign(d) sqrt(d^2 + (2 ga)^2)), d = be - al.  Products of squared norms
// that could leave the normal range take jacobi_cs.
__device__ __forceinline__ bool jacobi_cs_fast(double al, double be, double ga, double tol, double& c, double& s) {
    const double pr = al * be;
    if (!(pr > 1e-280) || !(pr < 1e280)) return jacobi_cs(al, be, ga, tol, c, s);
    if (!(ga * ga > tol * tol * pr)) return false;
    const double d = be - al, g2 = 2.0 * ga;
    const double t = g2 / (d + copysign(sqrt(fma(d, d, g2 * g2)), d));
    // a Newton step on rsqrt's result: its last-bit error has a sign of its own, and c^2 + s^2
    // - 1 accumulates over the 2000 rotations a column takes part in
    const double w = fma(t, t, 1.0), c0 = rsqrt(w);
    c = fma(0.5 * c0, fma(-(w * c0), c0, 1.0), c0);
    s = c * t;
    return true;
}

// barrier of the cluster by converged warps
__device__ __forceinline__ void cluster_sync(cooperative_groups::cluster_group const& cl) {
    __syncwarp();
    cl.sync();
}

// Thin SVD of one block per thread-block cluster, EPL * 32 >= max(rows, cols).  The block
// is taken as A (m x n, n = min, the transpose when rows < cols).
//
// 1. QR with column pivoting, A P = Q R, by Householder reflections; one warp holds two
//    columns in registers (EPL elements per lane each), the remaining norms are
//    recomputed at every step, and a step's reflector reaches all CTAs of the cluster
//    through their shared memory.
// 2. One-sided Jacobi on the columns of L = R^T with the rotations accumulated in J:
//    L J = W Sigma, so A = (Q J) Sigma (P W)^T.  Pivoting orders and decouples the
//    columns: on a two-site block whose singular values fall by eight decades it takes
//    10 sweeps instead of 32, on a random one 11 instead of 13.  Householder QR is
//    accurate column by column and one-sided Jacobi is insensitive to column scaling, so
//    small singular values keep their relative accuracy.
//    The pairs follow the odd-even order: neighbours in a line of n positions meet and
//    exchange places, alternately at even and odd positions.  The window of two
//    positions a warp holds slides by one place per round, so a round moves one column
//    per warp (to the warp on its left, through that CTA's shared memory) and keeps the
//    other in registers; the pair across the ends of the line does not meet.
// 3. sigma = |column of L J| / |column of J| (what the rounding of the rotations has done to
//    their length it has done to both), descending order, U = Q J by the reflectors in
//    reverse, V = P W.
//
// What bounds it is the chain of a round (a cluster barrier, the inner products' shuffle
// trees, one rotation's square root, division and reciprocal square root), not bandwidth:
// so the columns of a block are spread over as many SMs as the cluster has (16 warps per
// CTA, up to 8 CTAs) and never leave the registers.  The 45 blocks (17 to 208 square) of a
// split at m = 1024 with singular values over eight decades: 4.9 ms, against 90 ms by
// block_svd_jacobi (one CTA per block, columns in L2, no pivoting).
// A block with a zero, vanishing (below 1e-140 of the largest element) or non-finite pivot,
// or that does not converge, is handed to block_svd_jacobi (general = 1), which keeps V
// orthonormal there.
template <int EPL>
struct SvdShared {
    double col[SVD_WARPS][2][2][EPL * 32];  // [warp][round parity][L, J][element]
    double v[2][EPL * 32];                  // reflector of a QR step
    double cand_val[2][SVD_WARPS * 8];      // largest remaining squared norm per warp
    int cand_id[2][SVD_WARPS * 8];
    int col_id[SVD_WARPS][2];
    double tau[2];
    double amax[8];
    int rotated[2];
};

template <int EPL>
__global__ void __launch_bounds__(SVD_THREADS) svd_cluster(SvdBlock* blocks) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char svd_smem_raw[];
    SvdShared<EPL>& sh = *reinterpret_cast<SvdShared<EPL>*>(svd_smem_raw);
    __shared__ double red[SVD_WARPS];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    cg::cluster_group cl = cg::this_cluster();
    const int C = int(cl.num_blocks()), rank = int(cl.block_rank());
    SvdBlock& blk = blocks[blockIdx.x / C];
    const SvdBlock b = blk;
    const bool tr = b.rows < b.cols;
    const int m = int(tr ? b.cols : b.rows), n = int(tr ? b.rows : b.cols);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // NP column pairs, WPC of them per CTA; warp slot `w` of the cluster
    const int NP = (n + 1) / 2, WPC = (NP + C - 1) / C;
    const int w = rank * WPC + warp;
    const bool active = warp < WPC && w < NP;
    double* Vh = b.work;                    // reflectors, m per step
    double* Lg = Vh + size_t(m) * n;        // R, row r at r * n (= column r of L)
    double* sig = Lg + size_t(n) * n;       // n
    double* taus = sig + n;                 // n
    int* perm = reinterpret_cast<int*>(taus + n);  // n

    double x[EPL], y[EPL], u[EPL], v[EPL];
    int idx = 2 * w, idy = 2 * w + 1;
    double amax = 0.0;
#pragma unroll
    for (int e = 0; e < EPL; ++e) {
        const int i = lane + 32 * e;
        x[e] = y[e] = 0.0;
        if (active && i < m) {
            x[e] = tr ? b.a[idx + size_t(i) * b.rows] : b.a[i + size_t(idx) * b.rows];
            if (idy < n) y[e] = tr ? b.a[idy + size_t(i) * b.rows] : b.a[i + size_t(idy) * b.rows];
        }
        amax = fmax(amax, fmax(fabs(x[e]), fabs(y[e])));
    }
    // largest element of the block; exact power-of-two scaling to [1, 2)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane == 0) red[warp] = amax;
    if (threadIdx.x == 0) sh.rotated[0] = sh.rotated[1] = 0;
    __syncthreads();
    if (threadIdx.x < unsigned(C)) {
        double a = 0.0;
        for (int i = 0; i < SVD_WARPS; ++i) a = fmax(a, red[i]);
        cl.map_shared_rank(sh.amax, threadIdx.x)[rank] = a;
    }
    cluster_sync(cl);
    for (int i = 0; i < C; ++i) amax = fmax(amax, sh.amax[i]);
    bool ok = amax > 0.0 && amax < 1.7976931348623157e308;  // the same in every thread of the cluster
    const int ex = ok ? ilogb(amax) : 0;
#pragma unroll
    for (int e = 0; e < EPL; ++e) {
        x[e] = ldexp(x[e], -ex);
        y[e] = ldexp(y[e], -ex);
    }

    // ---- 1. QR with column pivoting ----
    int kx = -1, ky = -1;  // the step that took the column (its position in R)
    double nrm[2] = {0.0, 0.0};
#pragma unroll
    for (int e = 0; e < EPL; ++e) {
        nrm[0] = fma(x[e], x[e], nrm[0]);
        nrm[1] = fma(y[e], y[e], nrm[1]);
    }
    warp_sums(nrm);
    for (int k = 0; ok && k < n; ++k) {
        const int par = k & 1;
        if (active && lane < C) {
            const double a0 = kx < 0 ? nrm[0] : -1.0, a1 = (ky < 0 && idy < n) ? nrm[1] : -1.0;
            cl.map_shared_rank(sh.cand_val[par], lane)[w] = a1 > a0 ? a1 : a0;
            cl.map_shared_rank(sh.cand_id[par], lane)[w] = a1 > a0 ? idy : idx;
        }
        cluster_sync(cl);
        // largest remaining column, ties to the lower index; every warp finds the same one
        double best = 0.0;
        int bid = n;
        for (int i = lane; i < NP; i += 32) {
            const double val = sh.cand_val[par][i];
            const int id = sh.cand_id[par][i];
            if (val > best || (val == best && id < bid)) {
                best = val;
                bid = id;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double val = __shfl_xor_sync(0xffffffffu, best, o);
            const int id = __shfl_xor_sync(0xffffffffu, bid, o);
            if (val > best || (val == best && id < bid)) {
                best = val;
                bid = id;
            }
        }
        // (a squared norm near the subnormal range has lost digits, and a reflector made from it
        // is not orthogonal: such columns, 1e-140 of the largest element, are handed over too)
        ok = best > 1e-280 && best < 1.7976931348623157e308;
        if (!ok) break;
        if (active && (bid == idx || bid == idy)) {
            const bool first = bid == idx;
            double al = 0.0;
#pragma unroll
            for (int e = 0; e < EPL; ++e)
                al += lane + 32 * e == k ? (first ? x[e] : y[e]) : 0.0;
            al = __shfl_sync(0xffffffffu, al, k & 31);
            const double beta = -copysign(sqrt(best), al), inv = 1.0 / (al - beta), tau = (beta - al) / beta;
            double h[EPL];
#pragma unroll
            for (int e = 0; e < EPL; ++e) {
                const int i = lane + 32 * e;
                const double z = first ? x[e] : y[e];
                h[e] = i > k ? z * inv : (i == k ? 1.0 : 0.0);
                if (i < m) Vh[size_t(k) * m + i] = h[e];
                const double f = i < k ? z : (i == k ? beta : 0.0);
                x[e] = first ? f : x[e];
                y[e] = first ? y[e] : f;
            }
            for (int r = 0; r < C; ++r) {
                double* dst = cl.map_shared_rank(sh.v[par], r);
#pragma unroll
                for (int e = 0; e < EPL; ++e) dst[lane + 32 * e] = h[e];
                if (lane == 0) cl.map_shared_rank(sh.tau, r)[par] = tau;
            }
            if (lane == 0) {
                taus[k] = tau;
                perm[k] = bid;
            }
            kx = first ? k : kx;
            ky = first ? ky : k;
        }
        cluster_sync(cl);
        double d[2] = {0.0, 0.0}, h[EPL];
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
            h[e] = sh.v[par][lane + 32 * e];
            d[0] = fma(h[e], x[e], d[0]);
            d[1] = fma(h[e], y[e], d[1]);
        }
        warp_sums(d);
        const double tau = sh.tau[par];
        const double dx = kx < 0 ? tau * d[0] : 0.0, dy = ky < 0 ? tau * d[1] : 0.0;
        nrm[0] = nrm[1] = 0.0;
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
            x[e] = fma(-dx, h[e], x[e]);
            y[e] = fma(-dy, h[e], y[e]);
            if (lane + 32 * e > k) {
                nrm[0] = fma(x[e], x[e], nrm[0]);
                nrm[1] = fma(y[e], y[e], nrm[1]);
            }
        }
        warp_sums(nrm);
    }

    // ---- 2. one-sided Jacobi on L = R^T ----
    if (ok) {
        if (active) {
#pragma unroll
            for (int e = 0; e < EPL; ++e) {
                const int i = lane + 32 * e;
                if (i < n) {
                    Lg[size_t(i) * n + kx] = x[e];
                    if (idy < n) Lg[size_t(i) * n + ky] = y[e];
                }
            }
        }
        cluster_sync(cl);
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
            const int i = lane + 32 * e;
            const bool in = active && i < n;
            x[e] = in ? __ldcg(Lg + size_t(idx) * n + i) : 0.0;
            y[e] = in && idy < n ? __ldcg(Lg + size_t(idy) * n + i) : 0.0;
            u[e] = in && i == idx ? 1.0 : 0.0;
            v[e] = in && i == idy ? 1.0 : 0.0;
        }
        const double tol = sqrt(double(m)) * 2.220446049250313e-16;
        const int N = 2 * NP;
        const int left = w > 0 ? w - 1 : NP - 1;  // the warp that takes this warp's first column
        SvdShared<EPL>* to = active ? cl.map_shared_rank(&sh, left / WPC) : &sh;
        const int tw = left % WPC;
        bool converged = n < 2;
        for (int sweep = 0; sweep < SVD_MAX_SWEEPS && !converged; ++sweep) {
            bool rotated = false;
            for (int r = 0; r < N; ++r) {
                const int par = r & 1;
                if (active) {
                    const int pos = (2 * w + r) % N;
                    double c = 0.0, s = 1.0;  // columns change places: first = c x + .., see below
                    bool swap = pos != N - 1, rot = false;
                    if (swap) {
                        double g[3] = {0.0, 0.0, 0.0};
#pragma unroll
                        for (int e = 0; e < EPL; ++e) {
                            g[0] = fma(x[e], x[e], g[0]);
                            g[1] = fma(y[e], y[e], g[1]);
                            g[2] = fma(x[e], y[e], g[2]);
                        }
                        warp_sums(g);
                        rot = jacobi_cs_fast(g[0], g[1], g[2], tol, c, s);
                    }
                    double* bl = to->col[tw][par][0];
                    double* bj = to->col[tw][par][1];
                    if (rot) {
                        rotated = true;
                        // x -> c x - s y goes one place right (stays), y -> s x + c y one place left (leaves)
#pragma unroll
                        for (int e = 0; e < EPL; ++e) {
                            bl[lane + 32 * e] = fma(s, x[e], c * y[e]);
                            x[e] = fma(c, x[e], -(s * y[e]));
                            bj[lane + 32 * e] = fma(s, u[e], c * v[e]);
                            u[e] = fma(c, u[e], -(s * v[e]));
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < EPL; ++e) {
                            bl[lane + 32 * e] = swap ? y[e] : x[e];
                            bj[lane + 32 * e] = swap ? v[e] : u[e];
                            if (!swap) {
                                x[e] = y[e];
                                u[e] = v[e];
                            }
                        }
                    }
                    if (lane == 0) to->col_id[tw][par] = swap ? idy : idx;
                    if (!swap) idx = idy;
                }
                cluster_sync(cl);
                if (active) {
#pragma unroll
                    for (int e = 0; e < EPL; ++e) {
                        y[e] = sh.col[warp][par][0][lane + 32 * e];
                        v[e] = sh.col[warp][par][1][lane + 32 * e];
                    }
                    idy = sh.col_id[warp][par];
                }
            }
            // any rotation anywhere in the cluster (the flag words alternate between sweeps; the
            // other word is cleared while nobody writes it)
            const int fp = sweep & 1;
            if (rotated && lane < C) atomicOr(&cl.map_shared_rank(sh.rotated, lane)[fp], 1);
            cluster_sync(cl);
            converged = sh.rotated[fp] == 0;
            if (threadIdx.x == 0) sh.rotated[fp ^ 1] = 0;
            cluster_sync(cl);
        }
        ok = converged;
    }

    // ---- 3. singular values, order, U and V ----
    bool live0 = false, live1 = false;
    double sx = 0.0, sy = 0.0, lx = 0.0, ly = 0.0;
    if (ok) {
        double g[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
            g[0] = fma(x[e], x[e], g[0]);
            g[1] = fma(y[e], y[e], g[1]);
            g[2] = fma(u[e], u[e], g[2]);
            g[3] = fma(v[e], v[e], g[3]);
        }
        warp_sums(g);
        // lengths of the columns, and J's to one
        lx = sqrt(g[0]);
        ly = sqrt(g[1]);
        const double ju = sqrt(g[2]), jv = sqrt(g[3]);
        sx = lx / ju;
        sy = ly / jv;
#pragma unroll
        for (int e = 0; e < EPL; ++e) {
            u[e] /= ju;
            v[e] /= jv;
        }
        live0 = active && idx < n;
        live1 = active && idy < n;
        if (lane == 0 && live0) sig[idx] = sx;
        if (lane == 0 && live1) sig[idy] = sy;
        cluster_sync(cl);
        int rk[2] = {0, 0};
        bool zero = false;
        for (int i = lane; i < n; i += 32) {
            const double si = __ldcg(sig + i);
            zero = zero || !(si > 0.0);
            rk[0] += (si > sx || (si == sx && i < idx)) ? 1 : 0;
            rk[1] += (si > sy || (si == sy && i < idy)) ? 1 : 0;
        }
        ok = !__any_sync(0xffffffffu, zero);
        if (ok && active) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                rk[0] += __shfl_xor_sync(0xffffffffu, rk[0], o);
                rk[1] += __shfl_xor_sync(0xffffffffu, rk[1], o);
            }
            if (lane == 0 && live0) b.s[rk[0]] = ldexp(sx, ex);
            if (lane == 0 && live1) b.s[rk[1]] = ldexp(sy, ex);
            // V = P W: element i of W belongs to column perm[i] of A
#pragma unroll
            for (int e = 0; e < EPL; ++e) {
                const int i = lane + 32 * e;
                if (i < n) {
                    const size_t pi = size_t(__ldcg(perm + i));
                    if (live0) (tr ? b.u[pi + size_t(rk[0]) * b.rows] : b.vt[rk[0] + pi * n]) = x[e] / lx;
                    if (live1) (tr ? b.u[pi + size_t(rk[1]) * b.rows] : b.vt[rk[1] + pi * n]) = y[e] / ly;
                }
            }
            // Q J: the reflectors in reverse on both columns, the next one loaded ahead
            double h[EPL], hn[EPL];
#pragma unroll
            for (int e = 0; e < EPL; ++e) {
                const int i = lane + 32 * e;
                hn[e] = i < m ? __ldcg(Vh + size_t(n - 1) * m + i) : 0.0;
            }
            for (int k = n - 1; k >= 0; --k) {
                const double tau = __ldcg(taus + k);
                double d[2] = {0.0, 0.0};
#pragma unroll
                for (int e = 0; e < EPL; ++e) {
                    h[e] = hn[e];
                    const int i = lane + 32 * e;
                    hn[e] = (k > 0 && i < m) ? __ldcg(Vh + size_t(k - 1) * m + i) : 0.0;
                }
#pragma unroll
                for (int e = 0; e < EPL; ++e) {
                    d[0] = fma(h[e], u[e], d[0]);
                    d[1] = fma(h[e], v[e], d[1]);
                }
                warp_sums(d);
                d[0] *= tau;
                d[1] *= tau;
#pragma unroll
                for (int e = 0; e < EPL; ++e) {
                    u[e] = fma(-d[0], h[e], u[e]);
                    v[e] = fma(-d[1], h[e], v[e]);
                }
            }
#pragma unroll
            for (int e = 0; e < EPL; ++e) {
                const int i = lane + 32 * e;
                if (i < m) {
                    if (live0) (tr ? b.vt[rk[0] + size_t(i) * n] : b.u[i + size_t(rk[0]) * b.rows]) = u[e];
                    if (live1) (tr ? b.vt[rk[1] + size_t(i) * n] : b.u[i + size_t(rk[1]) * b.rows]) = v[e];
                }
            }
        }
    }
    if (rank == 0 && threadIdx.x == 0) blk.general = ok ? 0 : 1;
    // no CTA leaves while another may still write into its shared memory
    cluster_sync(cl);
    // completion in stream order although the next launch may have started early
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// One CTA per SM at least is all it needs: without saying so the compiler stayed at 64 registers and
// spilled into every column pair.
__global__ void __launch_bounds__(SVD_THREADS, 1) block_svd_jacobi(const SvdBlock* blocks, int* err) {
    extern __shared__ double smem[];
    const SvdBlock b = blocks[blockIdx.x];
    if (!b.general) return;
    const bool tr = b.rows < b.cols;
    const uint32_t m = tr ? b.cols : b.rows, n = tr ? b.rows : b.cols;
    if (n == 0) return;
    double* G = b.work ? b.work : smem;
    double* V = G + size_t(m) * n;
    double* sig = V + size_t(n) * n;
    int* rank_col = reinterpret_cast<int*>(sig + n);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    __shared__ double red[SVD_WARPS];
    double amax = 0.0;
    for (size_t e = threadIdx.x; e < size_t(m) * n; e += blockDim.x) {
        const uint32_t j = uint32_t(e / m), i = uint32_t(e % m);
        const double v = tr ? b.a[j + size_t(i) * b.rows] : b.a[i + size_t(j) * b.rows];
        G[e] = v;
        amax = fmax(amax, fabs(v));
    }
    for (size_t e = threadIdx.x; e < size_t(n) * n; e += blockDim.x) V[e] = (e / n == e % n) ? 1.0 : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane == 0) red[warp] = amax;
    __syncthreads();
    for (int w = 0; w < SVD_WARPS; ++w) amax = fmax(amax, red[w]);
    // exact power-of-two scaling to a largest element in [1, 2): the squared
    // norms neither underflow nor overflow; sigma is scaled back at the end
    const int ex = amax > 0.0 ? ilogb(amax) : 0;
    if (ex != 0) {
        for (size_t e = threadIdx.x; e < size_t(m) * n; e += blockDim.x) G[e] = ldexp(G[e], -ex);
    }
    __syncthreads();

    const double tol = sqrt(double(m)) * 2.220446049250313e-16;
    const uint32_t n2 = n + (n & 1u);  // even player count; index n is the bye when n is odd
    bool converged = n < 2;
    for (int sweep = 0; sweep < SVD_MAX_SWEEPS && !converged; ++sweep) {
        int rotated = 0;
        for (uint32_t r = 0; r + 1 < n2; ++r) {
            // circle method: player n2-1 meets r, player (r+k) meets (r-k) (mod n2-1)
            for (uint32_t k = warp; k < n2 / 2; k += SVD_WARPS) {
                uint32_t p, q;
                if (k == 0) {
                    p = n2 - 1;
                    q = r;
                } else {
                    p = (r + k) % (n2 - 1);
                    q = (r + (n2 - 1) - k) % (n2 - 1);
                }
                if (p >= n || q >= n) continue;
                if (p > q) {
                    const uint32_t t = p;
                    p = q;
                    q = t;
                }
                double* gp = G + size_t(p) * m;
                double* gq = G + size_t(q) * m;
                double* vp = V + size_t(p) * n;
                double* vq = V + size_t(q) * n;
                const bool rot = (m <= 32u * SVD_REG) ? pair_rotate_regs(gp, gq, m, vp, vq, n, tol)
                                                     : pair_rotate_loop(gp, gq, m, vp, vq, n, tol);
                if (rot) rotated = 1;
            }
            __syncthreads();
        }
        converged = __syncthreads_or(rotated) == 0;
    }
    if (!converged && threadIdx.x == 0) atomicOr(err, 1);

    for (uint32_t j = warp; j < n; j += SVD_WARPS) {
        const double* g = G + size_t(j) * m;
        double ss = 0.0;
        for (uint32_t i = lane; i < m; i += 32) ss = fma(g[i], g[i], ss);
        ss = warp_sum(ss);
        if (lane == 0) sig[j] = sqrt(ss);
    }
    __syncthreads();
    // descending order, ties by column index, NaN (from a non-finite block) first: a total
    // order, so that every entry of rank_col is written
    for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) {
        const double sj = sig[j];
        uint32_t rk = 0;
        for (uint32_t i = 0; i < n; ++i) {
            const double si = sig[i];
            const bool same = si == sj || (isnan(si) && isnan(sj));
            rk += (si > sj || (isnan(si) && !isnan(sj)) || (same && i < j)) ? 1u : 0u;
        }
        rank_col[rk] = int(j);
    }
    __syncthreads();
    for (uint32_t r = threadIdx.x; r < n; r += blockDim.x) b.s[r] = ldexp(sig[rank_col[r]], ex);
    // U (rows x n) and V^T (n x cols)
    for (size_t e = threadIdx.x; e < size_t(b.rows) * n; e += blockDim.x) {
        const uint32_t r = uint32_t(e / b.rows), i = uint32_t(e % b.rows);
        const uint32_t j = uint32_t(rank_col[r]);
        double v;
        if (tr) {
            v = V[size_t(j) * n + i];
        } else {
            const double sj = sig[j];
            v = sj > 0.0 ? G[size_t(j) * m + i] / sj : 0.0;
        }
        b.u[e] = v;
    }
    for (size_t e = threadIdx.x; e < size_t(n) * b.cols; e += blockDim.x) {
        const uint32_t c = uint32_t(e / n), r = uint32_t(e % n);
        const uint32_t j = uint32_t(rank_col[r]);
        double v;
        if (tr) {
            const double sj = sig[j];
            v = sj > 0.0 ? G[size_t(j) * m + c] / sj : 0.0;
        } else {
            v = V[size_t(j) * n + c];
        }
        b.vt[e] = v;
    }
}

// Launch class of a block: 4 * log2(cluster size) + element class (64, 128 or 256 rows),
// -1 for blocks above 256.  A cluster has 16 column pairs per CTA at most, so that a
// CTA's columns fit its registers; fewer CTAs than that would leave SMs idle when the
// blocks of a split are few (a split at m = 1024 has 45 blocks, 13 of them above 128).
int svd_class(uint32_t rows, uint32_t cols) {
    const uint32_t m = std::max(rows, cols), n = std::min(rows, cols);
    if (m > 256) return -1;
    const int epl = m <= 64 ? 0 : m <= 128 ? 1 : 2;
    const uint32_t np = (n + 1) / 2;
    const int c = np <= 16 ? 0 : np <= 32 ? 1 : np <= 64 ? 2 : 3;
    return 4 * c + epl;
}

// `chained`: an earlier svd_cluster launch of this call precedes it on the stream; the two
// touch different blocks, so this one may start as soon as the other's CTAs have.
template <int EPL>
cudaError_t launch_svd_cluster_epl(int cl, SvdBlock* blocks, uint32_t n, bool chained, cudaStream_t st) {
    cudaError_t e = ensure_smem_limit(reinterpret_cast<const void*>(svd_cluster<EPL>), int(sizeof(SvdShared<EPL>)));
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(n << cl);
    cfg.blockDim = dim3(SVD_THREADS);
    cfg.dynamicSmemBytes = sizeof(SvdShared<EPL>);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1u << cl;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = chained ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, svd_cluster<EPL>, blocks);
}
cudaError_t launch_svd_cluster(int cls, SvdBlock* blocks, uint32_t n, bool chained, cudaStream_t st) {
    const int cl = cls >> 2;
    switch (cls & 3) {
        case 0: return launch_svd_cluster_epl<2>(cl, blocks, n, chained, st);
        case 1: return launch_svd_cluster_epl<4>(cl, blocks, n, chained, st);
        default: return launch_svd_cluster_epl<8>(cl, blocks, n, chained, st);
    }
}

__global__ void copy_blocks(const dmrgb200_block_copy* cp, uint32_t n, const double* src, double* dst,
                            const double* scale) {
    for (uint32_t k = blockIdx.x; k < n; k += gridDim.x) {
        const dmrgb200_block_copy c = cp[k];
        const size_t total = size_t(c.rows) * c.cols;
        for (size_t e = threadIdx.x; e < total; e += blockDim.x) {
            const uint32_t j = uint32_t(e / c.rows), i = uint32_t(e % c.rows);
            double v = src[c.src_off + i + size_t(j) * c.src_ld];
            if (c.scale_mode == DMRGB200_SCALE_ROWS) v *= scale[c.scale_off + i];
            else if (c.scale_mode == DMRGB200_SCALE_COLS) v *= scale[c.scale_off + j];
            dst[c.dst_off + i + size_t(j) * c.dst_ld] = v;
        }
    }
}

}  // namespace
}  // namespace dmrgb200

using namespace dmrgb200;

extern "C" dmrgb200_status dmrgb200_block_svd(uint32_t n_blocks, const uint32_t* rows, const uint32_t* cols,
                                              const double* const* a, double* const* u, double* const* s,
                                              double* const* vt, void* cuda_stream) {
    if (n_blocks && (!rows || !cols || !a || !u || !s || !vt))
        return noalloc_fail(DMRGB200_INVALID_ARGUMENT, "block SVD: null argument");
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    std::vector<SvdBlock> bl;
    std::vector<int> cls;          // svd_cluster launch of the block, -1: block_svd_jacobi
    std::vector<size_t> work_off;  // per block: offset in the global scratch, or SIZE_MAX for shared memory
    size_t work = 0, smem = 0;
    for (uint32_t i = 0; i < n_blocks; ++i) {
        if (!rows[i] || !cols[i]) continue;
        if (!a[i] || !u[i] || !s[i] || !vt[i]) return noalloc_fail(DMRGB200_INVALID_ARGUMENT, "block SVD: null block");
        bl.push_back(SvdBlock{a[i], u[i], s[i], vt[i], nullptr, rows[i], cols[i], 1, 0});
        cls.push_back(svd_class(rows[i], cols[i]));
        const size_t w = svd_work_elems(rows[i], cols[i]);
        if (cls.back() < 0 && w * sizeof(double) <= SVD_SMEM_LIMIT) {
            smem = std::max(smem, w * sizeof(double));
            work_off.push_back(SIZE_MAX);
        } else {
            // 256-byte starts: columns that begin inside a 32-byte sector cost block_svd_jacobi a
            // quarter of its time (9 blocks of 268 to 324 rows 617 ms, 480 aligned)
            work_off.push_back(work);
            work += (w + 31) / 32 * 32;
        }
    }
    if (bl.empty()) return DMRGB200_OK;
    const size_t tab = (bl.size() * sizeof(SvdBlock) + 255) / 256 * 256;
    unsigned char* mem = nullptr;
    cudaError_t e = cudaMallocAsync(reinterpret_cast<void**>(&mem), tab + 256 + work * sizeof(double), st);
    if (e != cudaSuccess) return noalloc_fail(DMRGB200_OUT_OF_MEMORY, std::string("block SVD: ") + cudaGetErrorString(e));
    int* d_err = reinterpret_cast<int*>(mem + tab);
    double* scratch = reinterpret_cast<double*>(mem + tab + 256);
    for (size_t i = 0; i < bl.size(); ++i)
        if (work_off[i] != SIZE_MAX) bl[i].work = scratch + work_off[i];
    // blocks by svd_cluster launch, the largest first
    std::vector<size_t> order(bl.size());
    for (size_t i = 0; i < order.size(); ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](size_t x, size_t y) {
        if (cls[x] != cls[y]) return cls[x] > cls[y];
        return uint64_t(bl[x].rows) * bl[x].cols > uint64_t(bl[y].rows) * bl[y].cols;
    });
    std::vector<SvdBlock> tabl;
    for (size_t i : order) tabl.push_back(bl[i]);
    e = ensure_smem_limit(reinterpret_cast<const void*>(block_svd_jacobi), int(SVD_SMEM_LIMIT));
    if (e != cudaSuccess) {
        cudaFreeAsync(mem, st);
        return noalloc_fail(DMRGB200_DEVICE_ERROR, std::string("block SVD shared memory: ") + cudaGetErrorString(e));
    }
    SvdBlock* d_bl = reinterpret_cast<SvdBlock*>(mem);
    cudaMemcpyAsync(mem, tabl.data(), tabl.size() * sizeof(SvdBlock), cudaMemcpyHostToDevice, st);
    cudaMemsetAsync(d_err, 0, sizeof(int), st);
    bool chained = false;
    for (size_t i = 0; i < order.size() && e == cudaSuccess;) {
        const int c = cls[order[i]];
        if (c < 0) break;
        size_t j = i;
        while (j < order.size() && cls[order[j]] == c) ++j;
        e = launch_svd_cluster(c, d_bl + i, uint32_t(j - i), chained, st);
        chained = true;
        i = j;
    }
    // the other blocks, and those svd_cluster handed back
    if (e == cudaSuccess) {
        block_svd_jacobi<<<uint32_t(bl.size()), SVD_THREADS, smem, st>>>(d_bl, d_err);
        e = cudaGetLastError();
    }
    int h_err = 0;
    cudaMemcpyAsync(&h_err, d_err, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaError_t e2 = cudaStreamSynchronize(st);
    cudaFreeAsync(mem, st);
    if (e != cudaSuccess) return noalloc_fail(DMRGB200_DEVICE_ERROR, std::string("block SVD launch: ") + cudaGetErrorString(e));
    if (e2 != cudaSuccess) return noalloc_fail(DMRGB200_DEVICE_ERROR, std::string("block SVD: ") + cudaGetErrorString(e2));
    if (h_err) return noalloc_fail(DMRGB200_NUMERIC, "block SVD: Jacobi sweeps did not converge");
    return DMRGB200_OK;
}

extern "C" dmrgb200_status dmrgb200_copy_blocks(uint32_t n, const dmrgb200_block_copy* copies, const double* src,
                                                double* dst, const double* scale, void* cuda_stream) {
    if (!n) return DMRGB200_OK;
    if (!copies || !src || !dst) return noalloc_fail(DMRGB200_INVALID_ARGUMENT, "block copy: null argument");
    for (uint32_t k = 0; k < n; ++k) {
        dmrgb200_block_copy const& c = copies[k];
        if (c.scale_mode > DMRGB200_SCALE_COLS) return noalloc_fail(DMRGB200_INVALID_ARGUMENT, "block copy: scale mode");
        if (c.scale_mode != DMRGB200_SCALE_NONE && !scale)
            return noalloc_fail(DMRGB200_INVALID_ARGUMENT, "block copy: scaling without factors");
        if (c.cols > 1 && (c.src_ld < c.rows || c.dst_ld < c.rows))
            return noalloc_fail(DMRGB200_INVALID_ARGUMENT, "block copy: leading dimension below the row count");
    }
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    void* d = nullptr;
    cudaError_t e = cudaMallocAsync(&d, size_t(n) * sizeof(dmrgb200_block_copy), st);
    if (e != cudaSuccess) return noalloc_fail(DMRGB200_OUT_OF_MEMORY, std::string("block copy: ") + cudaGetErrorString(e));
    // upload from a pageable copy: a pageable source is staged before cudaMemcpyAsync
    // returns, so the caller's array (pinned or not) may be released on return
    std::vector<dmrgb200_block_copy> staged(copies, copies + n);
    cudaMemcpyAsync(d, staged.data(), size_t(n) * sizeof(dmrgb200_block_copy), cudaMemcpyHostToDevice, st);
    copy_blocks<<<std::min<uint32_t>(n, 148u * 8u), 256, 0, st>>>(static_cast<const dmrgb200_block_copy*>(d), n, src,
                                                                   dst, scale);
    e = cudaGetLastError();
    cudaFreeAsync(d, st);
    if (e != cudaSuccess) return noalloc_fail(DMRGB200_DEVICE_ERROR, std::string("block copy: ") + cudaGetErrorString(e));
    return DMRGB200_OK;
}
