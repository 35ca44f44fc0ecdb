// Jacobi-Davidson as one CUDA graph: every scalar of the iteration lives on the
// device, one iteration is the body of a conditional WHILE node (one H psi and one
// jd_step launch), and the step decides whether the body runs again.  The steps are
// those of the stepwise solver in jd.cu (ietl/jacobi.h:386-474,
// ietl_jacobi_davidson.h:35-76): MGS with one refinement pass below kappa = 0.25,
// projection of the orthogonal vectors, Rayleigh-Ritz (cyclic Jacobi on the k x k
// projected matrix), convergence |r| <= tol |theta| or |r| < tol, and the correction
// t = -r + (r.u / u.u) u.
//
// jd_step is one cooperative launch of one CTA per SM.  Every thread owns the same
// elements of all vectors throughout and keeps the target (t, u, uA) in registers; what
// the CTAs exchange are the inner products: each CTA publishes its partial sums, every CTA
// waits for all of them and adds them in the same order, so all hold the same coefficients
// without a second exchange, and a solve is bitwise reproducible.  What bounds it are those
// exchanges (k + 4 of them with k + 1 basis vectors, 2k + 6 with refinement) and the chain of
// rotations of the k x k eigenproblem, which every CTA solves for itself; as separate
// launches, one per inner product and vector operation (about 30 per iteration), it was
// the launches and their drains.
//
// Each body sets the WHILE condition to 0 first and sets it back to 1 only at its end,
// after incrementing the iteration count, so the loop ends after at most max_iter bodies
// whatever the data.  The wait for the other CTAs' sums is bounded (2 s): a CTA that gives up
// records it, every later step returns at once and the solve reports DMRGB200_TIMEOUT.
#include <cuda_runtime.h>

#include <cmath>
#include <string>
#include <vector>

#include "../../include/dmrgb200.h"
#include "async_copy.cuh"
#include "device.hpp"

namespace dmrgb200 {

dmrgb200_status noalloc_fail(dmrgb200_status s, std::string const& msg);
cudaError_t plan_hpsi_launch(dmrgb200_plan_t plan, const double* x, double* y, cudaStream_t stream);
cudaError_t plan_ensure_tuned(dmrgb200_plan_t plan, const double* x, double* y, cudaStream_t stream);

namespace {

constexpr int JT = 1024;       // threads per CTA of the step kernels (one CTA per SM)
constexpr int MAXK = 32;       // max_iter bound (and the warps of a CTA)
constexpr int MAXO = 8;        // orthogonal vectors bound
constexpr int EPT = 4;         // elements per thread kept in registers

struct JdState {
    unsigned phase;              // exchanges since the solve began
    int iter, done, status, converged;  // status: 1 vanished direction, 2 a wait ran out
    double theta, rnorm;
    double oo[MAXO];       // <o_i, o_i>
    double M[MAXK * MAXK]; // projected matrix, column-major, leading dimension MAXK
};

struct JdArgs {
    double* vec;          // vector slots, n doubles each
    uint64_t n;
    int max_iter, n_ortho;
    double tol;
    JdState* st;
    double* partial;      // [2][MAXK][grid] places of the CTAs' partial sums, 16 bytes each
    cudaGraphConditionalHandle cond;
};

// slots: V(0..max_iter), VA(0..max_iter), u, uA, t, y, O(0..n_ortho)
__device__ __forceinline__ double* V(JdArgs const& a, int i) { return a.vec + a.n * uint64_t(i); }
__device__ __forceinline__ double* VA(JdArgs const& a, int i) { return a.vec + a.n * uint64_t(a.max_iter + i); }
__device__ __forceinline__ double* U(JdArgs const& a) { return a.vec + a.n * uint64_t(2 * a.max_iter); }
__device__ __forceinline__ double* UA(JdArgs const& a) { return a.vec + a.n * uint64_t(2 * a.max_iter + 1); }
__device__ __forceinline__ double* Tv(JdArgs const& a) { return a.vec + a.n * uint64_t(2 * a.max_iter + 2); }
__device__ __forceinline__ double* Yv(JdArgs const& a) { return a.vec + a.n * uint64_t(2 * a.max_iter + 3); }
__device__ __forceinline__ double* Ov(JdArgs const& a, int i) { return a.vec + a.n * uint64_t(2 * a.max_iter + 4 + i); }

// This thread's elements of one vector: registers (REG) or its own elements of a global
// slot, which no other thread touches.
template <bool REG>
struct Own {
    double r[REG ? EPT : 1];
    double* g;
    __device__ __forceinline__ double get(int e, uint64_t i) const { return REG ? r[e] : g[i]; }
    __device__ __forceinline__ void set(int e, uint64_t i, double v) {
        if (REG) r[e] = v;
        else g[i] = v;
    }
};

// f(e, i) for every element i this thread owns
template <bool REG, class F>
__device__ __forceinline__ void each(JdArgs const& a, F&& f) {
    const uint64_t i0 = uint64_t(blockIdx.x) * JT + threadIdx.x, stride = uint64_t(gridDim.x) * JT;
    if (REG) {
#pragma unroll
        for (int e = 0; e < EPT; ++e) {
            const uint64_t i = i0 + e * stride;
            if (i < a.n) f(e, i);
        }
    } else {
        for (uint64_t i = i0; i < a.n; i += stride) f(0, i);
    }
}

struct StepShared {
    double red[JT / 32][MAXK];  // [warp][value]
    double sum[MAXK];
    double A[MAXK][MAXK + 1], Z[MAXK][MAXK + 1];
    double s[MAXK];
    double cs[MAXK / 2][2];
    double theta;
    int failed;
};

// A place of an exchange: a CTA's partial sum and the number of the exchange it belongs to,
// stored and read as one 128-bit word.
__device__ __forceinline__ void place_store(double* at, double v, unsigned long long tag) {
    asm volatile(
        "{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(at),
        "l"(__double_as_longlong(v)), "l"(tag)
        : "memory");
}
__device__ __forceinline__ void place_load(const double* at, unsigned long long& v, unsigned long long& tag) {
    asm volatile("{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}"
                 : "=l"(v), "=l"(tag)
                 : "l"(at)
                 : "memory");
}

// Sums of nv per-thread values over the grid: warp trees, the CTA's partial sums to global
// memory, then warp w of every CTA reads value w of all CTAs (waiting for those of an earlier
// exchange) and adds them, in the same order everywhere.  Results in sh.sum[0, nv).
// `val(k, v)` gives the thread's values k .. k + 3 (those below nv count), four at a time so
// that their loads overlap.  False when a wait ran out.
//
// The sum and its tag travel in one word, so it is its own flag: no counter, no fence, one trip
// through L2 (6 us per exchange with fences or a counted barrier).  Exchange `phase` uses the
// places phase % 2: a CTA stores there again two exchanges later, when it has seen every other
// CTA's sum of the exchange between, which each of them stored after it had read this one.
template <class F>
__device__ bool grid_sums(JdArgs const& a, StepShared& sh, int nv, unsigned& phase, F&& val) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* part = a.partial + uint64_t(phase & 1u) * 2 * MAXK * gridDim.x;
    const unsigned long long tag = ++phase;
    for (int k = 0; k < nv; k += 4) {
        double v[4] = {0.0, 0.0, 0.0, 0.0};
        val(k, v);
        if (nv - k == 1) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        } else {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
        }
        if (lane == 0)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (k + j < nv) sh.red[warp][k + j] = v[j];
    }
    if (threadIdx.x == 0) sh.failed = 0;
    __syncthreads();
    if (warp < nv) {
        double v = sh.red[lane][warp];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        double* row = part + 2 * uint64_t(warp) * gridDim.x;
        if (lane == 0) place_store(row + 2 * blockIdx.x, v, tag);
        const unsigned long long t0 = async::global_ns();
        v = 0.0;
        bool ok = true;
        for (unsigned b0 = lane; b0 < gridDim.x; b0 += 32 * 5) {
            // this lane's places, all read at once until each carries the tag
            unsigned long long x[5], y[5];
            for (;;) {
                bool all = true;
#pragma unroll
                for (int j = 0; j < 5; ++j) {
                    x[j] = 0ull;
                    y[j] = tag;
                    if (b0 + 32 * j < gridDim.x) place_load(row + 2 * (b0 + 32 * j), x[j], y[j]);
                }
#pragma unroll
                for (int j = 0; j < 5; ++j) all = all && y[j] == tag;
                if (all) break;
                if (async::global_ns() - t0 > async::WAIT_LIMIT_NS) {
                    ok = false;
                    break;
                }
            }
#pragma unroll
            for (int j = 0; j < 5; ++j) v += __longlong_as_double(x[j]);  // 0 past the last CTA
        }
        if (!ok) {
            sh.failed = 1;
            atomicExch(&a.st->status, 2);
        }
        __syncwarp();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) sh.sum[warp] = v;
    }
    __syncthreads();
    return !sh.failed;
}

// Project the orthogonal vectors out of x: x -= <o_i, x> / <o_i, o_i> o_i in turn.
template <bool REG>
__device__ bool project(JdArgs const& a, StepShared& sh, unsigned& phase, Own<REG>& x, int no) {
    for (int i = 0; i < no; ++i) {
        const double* o = Ov(a, i);
        double p = 0.0;
        each<REG>(a, [&](int e, uint64_t k) { p += o[k] * x.get(e, k); });
        if (!grid_sums(a, sh, 1, phase, [&](int, double* v) { v[0] = p; })) return false;
        const double c = sh.sum[0] / a.st->oo[i];
        each<REG>(a, [&](int e, uint64_t k) { x.set(e, k, x.get(e, k) - c * o[k]); });
    }
    return true;
}

// Basis vector V(it) from the target t: MGS against V(0..it), refinement, projection,
// normalisation; also left in the H psi input.
template <bool REG>
__device__ bool basis_vector(JdArgs const& a, StepShared& sh, unsigned& phase, Own<REG>& t, int it) {
    // v: the basis vector whose coefficient comes next, w: the one after it (read ahead of the
    // exchange that gives the coefficient)
    double v[REG ? EPT : 1], w[REG ? EPT : 1];
    auto fetch = [&](double(&d)[REG ? EPT : 1], int j) {
        if (REG && j < it) each<REG>(a, [&](int e, uint64_t k) { d[e] = V(a, j)[k]; });
    };
    auto basis = [&](double(&d)[REG ? EPT : 1], int j, int e, uint64_t k) { return REG ? d[e] : V(a, j)[k]; };
    fetch(v, 0);
    fetch(w, 1);
    // tau^2 = <t, t> and the first coefficient in one exchange
    double tt = 0.0, p = 0.0;
    each<REG>(a, [&](int e, uint64_t k) {
        const double x = t.get(e, k);
        tt += x * x;
        if (it > 0) p += basis(v, 0, e, k) * x;
    });
    if (!grid_sums(a, sh, it > 0 ? 2 : 1, phase, [&](int, double* s) {
            s[0] = tt;
            s[1] = p;
        }))
        return false;
    const double tau = sqrt(sh.sum[0]);
    double nn = sh.sum[0], c = it > 0 ? sh.sum[1] : 0.0;
    for (int pass = 0; it > 0 && pass < 2; ++pass) {
        if (pass == 1) {
            if (!(sqrt(nn) < 0.25 * tau)) break;
            fetch(v, 0);
            fetch(w, 1);
            p = 0.0;
            each<REG>(a, [&](int e, uint64_t k) { p += basis(v, 0, e, k) * t.get(e, k); });
            if (!grid_sums(a, sh, 1, phase, [&](int, double* s) { s[0] = p; })) return false;
            c = sh.sum[0];
        }
        // t -= c V(j) and, in the same pass over t, the next coefficient (or |t|^2 at the end)
        for (int j = 0; j < it; ++j) {
            const bool more = j + 1 < it;
            p = 0.0;
            each<REG>(a, [&](int e, uint64_t k) {
                const double x = t.get(e, k) - c * basis(v, j, e, k);
                t.set(e, k, x);
                p += (more ? basis(w, j + 1, e, k) : x) * x;
            });
            if (REG)
#pragma unroll
                for (int e = 0; e < (REG ? EPT : 1); ++e) v[e] = w[e];
            fetch(w, j + 2);
            if (!grid_sums(a, sh, 1, phase, [&](int, double* s) { s[0] = p; })) return false;
            c = nn = sh.sum[0];
        }
    }
    if (a.n_ortho > 0) {
        if (!project<REG>(a, sh, phase, t, a.n_ortho)) return false;
        p = 0.0;
        each<REG>(a, [&](int e, uint64_t k) { p += t.get(e, k) * t.get(e, k); });
        if (!grid_sums(a, sh, 1, phase, [&](int, double* v) { v[0] = p; })) return false;
        nn = sh.sum[0];
    }
    const double tn = sqrt(nn);
    const bool vanished = !(tn > 0.0);
    if (vanished && blockIdx.x == 0 && threadIdx.x == 0) {
        a.st->status = 1;
        a.st->done = 1;
    }
    const double inv = vanished ? 0.0 : 1.0 / tn;
    double *in = Tv(a), *out = V(a, it);
    each<REG>(a, [&](int e, uint64_t k) {
        const double x = t.get(e, k) * inv;
        in[k] = x;
        out[k] = x;
    });
    return !vanished;
}

// 1 / sqrt(w) to rounding: rsqrt and a Newton step
__device__ __forceinline__ double recip_sqrt(double w) {
    const double r = rsqrt(w);
    return fma(0.5 * r, fma(-(w * r), r, 1.0), r);
}

// Rotation of a pair, tan(2x) = h / d (h = 2 a_pq, d = a_qq - a_pp), the smaller angle:
// cos(2x) = |d| / sqrt(d^2 + h^2), c^2 = (1 + cos(2x)) / 2 and s = sin(2x) / (2 c), two reciprocal
// square roots in sequence instead of two square roots and three divisions.  (The tangent in
// single precision and two Newton steps is shorter still, but takes two sweeps more.)
__device__ __forceinline__ void rotation(double d, double h, double& c, double& s) {
    const double w = fma(d, d, h * h);
    if (d != 0.0 && w > 1e-280 && w < 1e280) {
        const double r = recip_sqrt(w), c2 = fma(0.5 * fabs(d), r, 0.5), ic = recip_sqrt(c2);
        c = c2 * ic;
        s = copysign(0.5, d) * h * r * ic;
    } else {
        const double tau = d / h, t = (tau >= 0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
        c = 1.0 / sqrt(1.0 + t * t);
        s = t * c;
    }
}

// Smallest eigenpair of the leading k x k block of M by cyclic Jacobi, one warp, from the
// upper triangle in sh.A (filled symmetric); theta and the vector into sh.  The rotations
// of a sweep are the row-cyclic ones, (0,1), (0,2) .. (0,k-1), (1,2) .., taken in
// wavefronts p + q = const: those of one wavefront touch different rows and columns and
// every other pair of rotations keeps its order, so 2k - 3 wavefronts do what k (k - 1) / 2
// rotations in sequence did (each a chain of a square root, a division and a reciprocal
// square root).
__device__ void ritz(StepShared& sh, int k) {
    const int lane = threadIdx.x & 31;
    const int inv = 65535 / k + 1;  // e / k = (e * inv) >> 16 for e < 512, k <= 32
    for (int e = lane; e < k * k; e += 32) sh.Z[e / k][e % k] = e / k == e % k ? 1.0 : 0.0;
    __syncwarp();
    for (int sweep = 0; sweep < 100; ++sweep) {
        double off = 0.0, tot = 0.0;
        if (lane < k)
            for (int j = 0; j < k; ++j) {
                const double v = sh.A[lane][j] * sh.A[lane][j];
                tot += v;
                if (j != lane) off += v;
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            off += __shfl_xor_sync(0xffffffffu, off, o);
            tot += __shfl_xor_sync(0xffffffffu, tot, o);
        }
        if (off <= 1e-34 * tot || off == 0.0) break;
        for (int sum = 1; sum <= 2 * k - 3; ++sum) {
            // pairs (p, sum - p), p0 <= p < (sum + 1) / 2
            const int p0 = sum > k - 1 ? sum - (k - 1) : 0, np = (sum + 1) / 2 - p0;
            bool any = false;
            if (lane < np) {
                const int p = p0 + lane, q = sum - p;
                const double apq = sh.A[p][q], app = sh.A[p][p], aqq = sh.A[q][q];
                double c = 1.0, s = 0.0;
                // negligible against both diagonal entries: dropped
                const bool drop = fabs(app) + 100.0 * fabs(apq) == fabs(app) && fabs(aqq) + 100.0 * fabs(apq) == fabs(aqq);
                if (drop) {
                    sh.A[p][q] = sh.A[q][p] = 0.0;
                } else if (apq != 0.0) {
                    rotation(aqq - app, 2.0 * apq, c, s);
                    any = true;
                }
                sh.cs[lane][0] = c;
                sh.cs[lane][1] = s;
            }
            // the vote orders no memory: without it a lane that sums A at the next sweep could miss a
            // dropped pair that another lane cleared
            __syncwarp();
            if (!__any_sync(0xffffffffu, any)) continue;
            // A <- A J and Z <- Z J, then A <- J^T A: one row (column) of one pair per lane at a
            // time, so that the lanes' reads do not wait for each other's writes
            for (int e = lane; e < np * k; e += 32) {
                const int x = (e * inv) >> 16, r = e - x * k, p = p0 + x, q = sum - p;
                const double c = sh.cs[x][0], s = sh.cs[x][1];
                const double ap = sh.A[r][p], aq = sh.A[r][q], zp = sh.Z[r][p], zq = sh.Z[r][q];
                sh.A[r][p] = c * ap - s * aq;
                sh.A[r][q] = s * ap + c * aq;
                sh.Z[r][p] = c * zp - s * zq;
                sh.Z[r][q] = s * zp + c * zq;
            }
            __syncwarp();
            for (int e = lane; e < np * k; e += 32) {
                const int x = (e * inv) >> 16, r = e - x * k, p = p0 + x, q = sum - p;
                const double c = sh.cs[x][0], s = sh.cs[x][1];
                const double ap = sh.A[p][r], aq = sh.A[q][r];
                sh.A[p][r] = c * ap - s * aq;
                sh.A[q][r] = s * ap + c * aq;
            }
            __syncwarp();
        }
    }
    __syncwarp();
    int best = 0;
    for (int i = 1; i < k; ++i)
        if (sh.A[i][i] < sh.A[best][best]) best = i;
    if (lane == 0) sh.theta = sh.A[best][best];
    if (lane < k) sh.s[lane] = sh.Z[lane][best];
}

// Orthogonal vectors among themselves (ietl_jacobi_davidson.h:44-48), projection of the
// start vector (t holds x0), first basis vector.
template <bool REG>
__global__ void __launch_bounds__(JT) jd_start(JdArgs a) {
    __shared__ StepShared sh;
    JdState* st = a.st;
    unsigned phase = st->phase;
    for (int i = 0; i < a.n_ortho; ++i) {
        Own<false> o;
        o.g = Ov(a, i);
        if (i > 0 && !project<false>(a, sh, phase, o, i)) return;
        double p = 0.0;
        each<false>(a, [&](int e, uint64_t k) { p += o.get(e, k) * o.get(e, k); });
        if (!grid_sums(a, sh, 1, phase, [&](int, double* v) { v[0] = p; })) return;
        // every CTA writes the same value before it reads it in project
        if (threadIdx.x == 0) st->oo[i] = sh.sum[0];
        __syncthreads();
    }
    Own<REG> t;
    t.g = Tv(a);
    each<REG>(a, [&](int e, uint64_t k) { t.set(e, k, Tv(a)[k]); });
    if (a.n_ortho > 0 && !project<REG>(a, sh, phase, t, a.n_ortho)) return;
    const bool ok = basis_vector<REG>(a, sh, phase, t, 0);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->phase = phase;
        if (!ok) cudaGraphSetConditional(a.cond, 0u);
    }
}

// The part of an iteration after its H psi (y): projected matrix, Ritz pair, residual and
// convergence, and, for the next iteration, the correction and the next basis vector.
template <bool REG>
__global__ void __launch_bounds__(JT) jd_step(JdArgs a) {
    __shared__ StepShared sh;
    JdState* st = a.st;
    const int it = st->iter, k = it + 1;
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    if (lead) cudaGraphSetConditional(a.cond, 0u);
    if (st->status) return;
    unsigned phase = st->phase;
    // VA(it) = y; M(j, it) = <V(j), y>, j <= it
    Own<REG> y;
    y.g = VA(a, it);
    each<REG>(a, [&](int e, uint64_t i) {
        const double x = Yv(a)[i];
        y.set(e, i, x);
        if (REG) VA(a, it)[i] = x;
    });
    if (!grid_sums(a, sh, k, phase, [&](int j, double* p) {
            const double *v0 = V(a, j), *v1 = V(a, min(j + 1, it)), *v2 = V(a, min(j + 2, it)), *v3 = V(a, min(j + 3, it));
            each<REG>(a, [&](int e, uint64_t i) {
                const double x = y.get(e, i);
                p[0] += v0[i] * x;
                p[1] += v1[i] * x;
                p[2] += v2[i] * x;
                p[3] += v3[i] * x;
            });
        }))
        return;
    if (blockIdx.x == 0 && int(threadIdx.x) < k) st->M[threadIdx.x + it * MAXK] = sh.sum[threadIdx.x];
    if (threadIdx.x < 32) {
        for (int e = threadIdx.x; e < k * k; e += 32) {
            const int r = e % k, c = e / k, lo = r < c ? r : c, hi = r < c ? c : r;
            sh.A[r][c] = hi == it ? sh.sum[lo] : __ldcg(&st->M[lo + hi * MAXK]);
        }
        __syncwarp();
        ritz(sh, k);
    }
    __syncthreads();
    const double theta = sh.theta;
    // u = sum_j s_j V(j), uA = sum_j s_j VA(j)
    Own<REG> u, ua;
    u.g = U(a);
    ua.g = UA(a);
    each<REG>(a, [&](int e, uint64_t i) {
        double x = V(a, 0)[i] * sh.s[0], z = VA(a, 0)[i] * sh.s[0];
#pragma unroll 4
        for (int j = 1; j < k; ++j) {
            x += V(a, j)[i] * sh.s[j];
            z += VA(a, j)[i] * sh.s[j];
        }
        u.set(e, i, x);
        ua.set(e, i, z);
    });
    if (a.n_ortho > 0 && !project<REG>(a, sh, phase, ua, a.n_ortho)) return;
    // r = uA - theta u
    double rr = 0.0, ru = 0.0, uu = 0.0;
    each<REG>(a, [&](int e, uint64_t i) {
        const double x = u.get(e, i), r = ua.get(e, i) - theta * x;
        ua.set(e, i, r);
        rr += r * r;
        ru += r * x;
        uu += x * x;
    });
    if (!grid_sums(a, sh, 3, phase, [&](int, double* v) {
            v[0] = rr;
            v[1] = ru;
            v[2] = uu;
        })) return;
    const double rnorm = sqrt(sh.sum[0]), corr = sh.sum[1] / sh.sum[2];
    const bool conv = rnorm <= a.tol * fabs(theta) || rnorm < a.tol, done = conv || it + 1 >= a.max_iter;
    // every CTA's sums have arrived, so none still reads st->iter
    if (lead) {
        st->theta = theta;
        st->rnorm = rnorm;
        st->iter = it + 1;
        st->converged = conv ? 1 : 0;
        if (done) st->done = 1;
    }
    if (done) {
        if (REG) each<REG>(a, [&](int e, uint64_t i) { U(a)[i] = u.get(e, i); });
        return;
    }
    // t = -r + corr u (in place of r)
    each<REG>(a, [&](int e, uint64_t i) { ua.set(e, i, -ua.get(e, i) + corr * u.get(e, i)); });
    const bool ok = basis_vector<REG>(a, sh, phase, ua, it + 1);
    if (lead) {
        st->phase = phase;
        if (ok) cudaGraphSetConditional(a.cond, 1u);
    }
}

}  // namespace

// Per-plan solver graph, rebuilt when the sizes, tolerance or stream change.
struct JdGraph {
    uint64_t n = 0;
    uint32_t max_iter = 0, n_ortho = 0;
    double tol = 0.0;
    double* vec = nullptr;
    JdState* st = nullptr;
    double* partial = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    ~JdGraph() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        cudaFree(vec);
        cudaFree(st);
        cudaFree(partial);
    }
};

void jd_graph_free(void* g) { delete static_cast<JdGraph*>(g); }

namespace {

cudaError_t launch_cooperative(void (*kernel)(JdArgs), int grid, JdArgs const& a, cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(grid));
    cfg.blockDim = dim3(JT);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

cudaError_t build_graph(JdGraph& g, dmrgb200_plan_t plan, cudaStream_t s) {
    // s: a private non-blocking stream (the legacy default stream cannot capture)
    cudaError_t e;
    const uint64_t n = g.n;
    const int nslots = int(2 * g.max_iter + 4 + g.n_ortho);
    const int nb = device_sm_count();  // one CTA per SM: all resident, as a cooperative launch needs
    if ((e = cudaMalloc(&g.vec, sizeof(double) * n * nslots)) != cudaSuccess) return e;
    if ((e = cudaMalloc(&g.st, sizeof(JdState))) != cudaSuccess) return e;
    if ((e = cudaMalloc(&g.partial, sizeof(double) * 4 * nb * MAXK)) != cudaSuccess) return e;
    // H psi writes only block elements: the padding of every slot stays zero
    if ((e = cudaMemset(g.vec, 0, sizeof(double) * n * nslots)) != cudaSuccess) return e;
    if ((e = cudaMemset(g.st, 0, sizeof(JdState))) != cudaSuccess) return e;
    if ((e = cudaEventCreate(&g.e0)) != cudaSuccess) return e;
    if ((e = cudaEventCreate(&g.e1)) != cudaSuccess) return e;

    JdArgs a{};
    a.vec = g.vec;
    a.n = n;
    a.max_iter = int(g.max_iter);
    a.n_ortho = int(g.n_ortho);
    a.tol = g.tol;
    a.st = g.st;
    a.partial = g.partial;

    // the grouped GEMMs are tuned before capture (on the zeroed t and y slots)
    if ((e = plan_ensure_tuned(plan, g.vec + n * (2 * g.max_iter + 2), g.vec + n * (2 * g.max_iter + 3), s)) !=
        cudaSuccess)
        return e;
    if ((e = cudaGraphCreate(&g.graph, 0)) != cudaSuccess) return e;
    if ((e = cudaGraphConditionalHandleCreate(&a.cond, g.graph, 1, cudaGraphCondAssignDefault)) != cudaSuccess)
        return e;

    // prologue: state, orthogonal vectors among themselves (ietl_jacobi_davidson.h:44-48),
    // projection of the start vector (t holds x0)
    if ((e = cudaStreamBeginCaptureToGraph(s, g.graph, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed)) !=
        cudaSuccess)
        return e;
    // vectors of up to EPT elements per thread stay in registers between the passes
    const bool reg = n <= uint64_t(EPT) * JT * nb;
    if ((e = cudaMemsetAsync(g.st, 0, sizeof(JdState), s)) == cudaSuccess)
        e = cudaMemsetAsync(g.partial, 0, sizeof(double) * 4 * nb * MAXK, s);  // tags start at 1
    if (e == cudaSuccess)
        e = launch_cooperative(reg ? jd_start<true> : jd_start<false>, nb, a, s);
    cudaGraph_t captured = nullptr;
    const cudaError_t le = e;
    e = cudaStreamEndCapture(s, &captured);
    if (e != cudaSuccess) return e;
    if (le != cudaSuccess) return le;

    // the WHILE node after the prologue
    std::vector<cudaGraphNode_t> leaves;
    size_t nn = 0;
    if ((e = cudaGraphGetNodes(g.graph, nullptr, &nn)) != cudaSuccess) return e;
    std::vector<cudaGraphNode_t> nodes(nn);
    if (nn && (e = cudaGraphGetNodes(g.graph, nodes.data(), &nn)) != cudaSuccess) return e;
    for (auto nd : nodes) {
        size_t ndep = 0;
        if ((e = cudaGraphNodeGetDependentNodes(nd, nullptr, &ndep)) != cudaSuccess) return e;
        if (ndep == 0) leaves.push_back(nd);
    }
    cudaGraphNodeParams cp{};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = a.cond;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t wnode;
    if ((e = cudaGraphAddNode(&wnode, g.graph, leaves.data(), leaves.size(), &cp)) != cudaSuccess) return e;
    cudaGraph_t body = cp.conditional.phGraph_out[0];

    // one iteration (jacobi.h:386-474)
    if ((e = cudaStreamBeginCaptureToGraph(s, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed)) !=
        cudaSuccess)
        return e;
    cudaError_t he = plan_hpsi_launch(plan, g.vec + n * (2 * g.max_iter + 2), g.vec + n * (2 * g.max_iter + 3), s);
    if (he == cudaSuccess) he = launch_cooperative(reg ? jd_step<true> : jd_step<false>, nb, a, s);
    cudaGraph_t body_out = nullptr;
    e = cudaStreamEndCapture(s, &body_out);
    if (e != cudaSuccess) return e;
    if (he != cudaSuccess) return he;
    return cudaGraphInstantiate(&g.exec, g.graph, 0);
}

}  // namespace

dmrgb200_status solve_graph(dmrgb200_plan_t plan, void** cache, uint64_t n, const double* x0,
                            const double* const* ortho, uint32_t n_ortho, double tol, uint32_t max_iter,
                            double* energy, double* x_out, dmrgb200_solve_stats* stats, cudaStream_t s) {
    JdGraph* g = static_cast<JdGraph*>(*cache);
    if (!g || g->n != n || g->max_iter != max_iter || g->n_ortho != n_ortho || g->tol != tol) {
        delete g;
        *cache = nullptr;
        g = new JdGraph;
        g->n = n;
        g->max_iter = max_iter;
        g->n_ortho = n_ortho;
        g->tol = tol;
        cudaStream_t cs = nullptr;
        cudaError_t e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);  // inputs of earlier work on s are complete
        if (e == cudaSuccess) e = build_graph(*g, plan, cs);
        if (cs) {
            cudaStreamCaptureStatus st;
            if (cudaStreamIsCapturing(cs, &st) == cudaSuccess && st != cudaStreamCaptureStatusNone) {
                cudaGraph_t junk = nullptr;
                cudaStreamEndCapture(cs, &junk);
                if (junk) cudaGraphDestroy(junk);
            }
            cudaStreamDestroy(cs);
        }
        if (e != cudaSuccess) {
            delete g;
            cudaGetLastError();
            // no cooperative kernels in graphs (a device under MPS): the caller steps on the host
            if (e == cudaErrorNotSupported || e == cudaErrorCooperativeLaunchTooLarge)
                return noalloc_fail(DMRGB200_NOT_SUPPORTED, "solver graph: no cooperative launch");
            return noalloc_fail(e == cudaErrorMemoryAllocation ? DMRGB200_OUT_OF_MEMORY : DMRGB200_DEVICE_ERROR,
                                std::string("solver graph: ") + cudaGetErrorString(e));
        }
        *cache = g;
    }
    const uint64_t T = n * (2 * max_iter + 2);
    cudaError_t e;
#define CK(x)                                                                                                \
    do {                                                                                                     \
        if ((e = (x)) != cudaSuccess)                                                                        \
            return noalloc_fail(DMRGB200_DEVICE_ERROR, std::string("solver: ") + cudaGetErrorString(e));     \
    } while (0)
    CK(cudaMemcpyAsync(g->vec + T, x0, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
    for (uint32_t i = 0; i < n_ortho; ++i)
        CK(cudaMemcpyAsync(g->vec + n * (2 * max_iter + 4 + i), ortho[i], n * sizeof(double), cudaMemcpyDeviceToDevice,
                           s));
    CK(cudaEventRecord(g->e0, s));
    CK(cudaGraphLaunch(g->exec, s));
    CK(cudaEventRecord(g->e1, s));
    CK(cudaMemcpyAsync(x_out, g->vec + n * (2 * max_iter), n * sizeof(double), cudaMemcpyDeviceToDevice, s));
    JdState hs;
    CK(cudaMemcpyAsync(&hs, g->st, sizeof(JdState), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
#undef CK
    float ms = 0.f;
    cudaEventElapsedTime(&ms, g->e0, g->e1);
    if (hs.status == 2) return noalloc_fail(DMRGB200_TIMEOUT, "solver: the wait for an inner product ran out");
    if (hs.status) return noalloc_fail(DMRGB200_NUMERIC, "Davidson direction vanished");
    *energy = hs.theta;
    if (stats) {
        stats->iterations = uint32_t(hs.iter);
        stats->converged = hs.converged;
        stats->residual = hs.rnorm;
        stats->hpsi_ms = 0.0;
        stats->solve_ms = ms;
    }
    return DMRGB200_OK;
}

}  // namespace dmrgb200
