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
// the CTAs exchange are the inner products: each CTA publishes its partial sums, a grid
// barrier follows, and every CTA adds all partials in the same order, so all hold the
// same coefficients without a second exchange, and a solve is bitwise reproducible.
// What bounds it are those barriers (iteration k has k + 4 of them, 2k + 5 with
// refinement) and the chain of rotations of the k x k eigenproblem, which every CTA
// solves for itself; as separate launches, one per inner product and vector operation
// (about 30 per iteration), it was the launches and their drains.
//
// Each body sets the WHILE condition to 0 first and sets it back to 1 only at its end,
// after incrementing the iteration count, so the loop ends after at most max_iter bodies
// whatever the data.  The wait at a grid barrier is bounded (2 s): a CTA that gives up
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
    unsigned long long barrier;  // arrivals at grid barriers since the solve began
    int iter, done, status, converged;  // status: 1 vanished direction, 2 barrier wait ran out
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
    double* partial;      // [2][MAXK][grid] partial sums of the CTAs
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

// Sums of nv per-thread values over the grid: warp trees, the CTA's partial sums to
// global memory, a grid barrier, then warp w of every CTA adds value w over all CTAs (the
// same order everywhere).  Results in sh.sum[0, nv).  `val(k, v)` gives the thread's values
// k .. k + 3 (those below nv count), four at a time so that their loads overlap.  False when
// the barrier's wait ran out.
template <class F>
__device__ bool grid_sums(JdArgs const& a, StepShared& sh, int nv, unsigned& phase, F&& val) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* part = a.partial + uint64_t(phase & 1u) * MAXK * gridDim.x;
    ++phase;
    for (int k = 0; k < nv; k += 4) {
        double v[4] = {0.0, 0.0, 0.0, 0.0};
        val(k, v);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
        if (lane == 0)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (k + j < nv) sh.red[warp][k + j] = v[j];
    }
    __syncthreads();
    if (warp < nv) {
        double v = sh.red[lane][warp];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) __stcg(part + uint64_t(warp) * gridDim.x + blockIdx.x, v);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // arrive, then wait until every CTA of this generation has (each CTA arrives once per
        // generation, so the arrival's number tells the generation)
        __threadfence();
        const unsigned long long target = (atomicAdd(&a.st->barrier, 1ull) / gridDim.x + 1ull) * gridDim.x;
        const unsigned long long t0 = async::global_ns();
        unsigned long long seen;
        sh.failed = 0;
        for (;;) {
            asm volatile("ld.acquire.gpu.u64 %0, [%1];" : "=l"(seen) : "l"(&a.st->barrier) : "memory");
            if (seen >= target) break;
            if (async::global_ns() - t0 > async::WAIT_LIMIT_NS) {
                sh.failed = 1;
                atomicExch(&a.st->status, 2);
                break;
            }
        }
    }
    __syncthreads();
    if (sh.failed) return false;
    if (warp < nv) {
        double v = 0.0;
        for (unsigned b = lane; b < gridDim.x; b += 32) v += __ldcg(part + uint64_t(warp) * gridDim.x + b);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) sh.sum[warp] = v;
    }
    __syncthreads();
    return true;
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
    // tau^2 = <t, t> and the first coefficient in one exchange
    double tt = 0.0, p = 0.0;
    each<REG>(a, [&](int e, uint64_t k) {
        const double x = t.get(e, k);
        tt += x * x;
        if (it > 0) p += V(a, 0)[k] * x;
    });
    if (!grid_sums(a, sh, it > 0 ? 2 : 1, phase, [&](int, double* v) {
            v[0] = tt;
            v[1] = p;
        })) return false;
    const double tau = sqrt(sh.sum[0]);
    double nn = sh.sum[0], c = it > 0 ? sh.sum[1] : 0.0;
    for (int pass = 0; it > 0 && pass < 2; ++pass) {
        if (pass == 1) {
            if (!(sqrt(nn) < 0.25 * tau)) break;
            p = 0.0;
            each<REG>(a, [&](int e, uint64_t k) { p += V(a, 0)[k] * t.get(e, k); });
            if (!grid_sums(a, sh, 1, phase, [&](int, double* v) { v[0] = p; })) return false;
            c = sh.sum[0];
        }
        // t -= c V(j) and, in the same pass over t, the next coefficient (or |t|^2 at the end)
        for (int j = 0; j < it; ++j) {
            const double* v = V(a, j);
            const double* w = j + 1 < it ? V(a, j + 1) : nullptr;
            p = 0.0;
            each<REG>(a, [&](int e, uint64_t k) {
                const double x = t.get(e, k) - c * v[k];
                t.set(e, k, x);
                p += (w ? w[k] : x) * x;
            });
            if (!grid_sums(a, sh, 1, phase, [&](int, double* v) { v[0] = p; })) return false;
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
    double *in = Tv(a), *v = V(a, it);
    each<REG>(a, [&](int e, uint64_t k) {
        const double x = t.get(e, k) * inv;
        in[k] = x;
        v[k] = x;
    });
    return !vanished;
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
                    const double d = aqq - app, h = 2.0 * apq;
                    const double t = d == 0.0 ? 1.0 : h / (d + copysign(sqrt(fma(d, d, h * h)), d));
                    const double w = fma(t, t, 1.0), c0 = rsqrt(w);
                    c = fma(0.5 * c0, fma(-(w * c0), c0, 1.0), c0);  // to rounding
                    s = t * c;
                    any = true;
                }
                sh.cs[lane][0] = c;
                sh.cs[lane][1] = s;
            }
            if (!__any_sync(0xffffffffu, any)) continue;
            __syncwarp();
            // A <- A J and Z <- Z J, then A <- J^T A
            for (int e = lane; e < np * k; e += 32) {
                const int r = e % k, x = e / k, p = p0 + x, q = sum - p;
                const double c = sh.cs[x][0], s = sh.cs[x][1];
                const double ap = sh.A[r][p], aq = sh.A[r][q], zp = sh.Z[r][p], zq = sh.Z[r][q];
                sh.A[r][p] = c * ap - s * aq;
                sh.A[r][q] = s * ap + c * aq;
                sh.Z[r][p] = c * zp - s * zq;
                sh.Z[r][q] = s * zp + c * zq;
            }
            __syncwarp();
            for (int e = lane; e < np * k; e += 32) {
                const int r = e % k, x = e / k, p = p0 + x, q = sum - p;
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
    unsigned phase = 0;
    JdState* st = a.st;
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
    if (!ok && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(a.cond, 0u);
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
    unsigned phase = 0;
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
    // every CTA is past the barrier above, so none still reads st->iter
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
    if (basis_vector<REG>(a, sh, phase, ua, it + 1) && lead) cudaGraphSetConditional(a.cond, 1u);
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
    if ((e = cudaMalloc(&g.partial, sizeof(double) * 2 * nb * MAXK)) != cudaSuccess) return e;
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
    if (hs.status == 2) return noalloc_fail(DMRGB200_TIMEOUT, "solver: the wait at a grid barrier ran out");
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
