// Float64 linear solves of the reference's linearised model and of its
// previous (Anderson) solver, as library kernels:
//   * the operator (diag M + alpha K) q with identity rows on fixed sites;
//   * one cooperative launch of block-Jacobi PCG with either stopping test
//     (the linear model's, or the previous solver's "balanced" test with the
//     local pose defect and a true-residual exit check);
//   * the vector updates of the linear implicit-midpoint step and its energy;
//   * the small reductions of Anderson mixing over device history buffers;
//   * a self-test of the time-limited grid barrier.
// Every reduction is per block then in a fixed order: results are bitwise
// reproducible run to run.
#include "common.cuh"

namespace dpf {
namespace lin {

constexpr int kMaxBlocks = 4096;
constexpr int kMaxHistory = 8;  // Anderson slots (the reference keeps 6 iterates)
constexpr int64_t kCounter = 8;  // doubles reserved for "last block" counters at the head of partials

inline int blocks_for(int64_t n, int threads) { return (int)((n + threads - 1) / threads); }
inline int reduce_grid(int64_t n) {
    int g = blocks_for(n, kThreads);
    if (g > 1024) g = 1024;
    return g < 1 ? 1 : g;
}

struct Operator {
    int64_t n, m;
    const int32_t *ptr, *inc;
    const int64_t *edges;
    dpf_stiffness k;
    dpf_tangent t;
    const double *mass;
    const uint8_t *fixed;
    double alpha;
    double *wrench;
};

// Wrenches of K v on the warp's bonds b0 .. b0 + 31, through its 288 doubles of shared memory.
__device__ __forceinline__ void operator_wrenches(const Operator &A, const double *v, int64_t b0, double *stage) {
    const int64_t b = b0 + (threadIdx.x & 31);
    Wrench f{};
    if (b < A.m) {
        int64_t i, j;
        edge(A.edges, b, i, j);
        f = stiffness_wrench(ld3(A.t.n, b), ld3(A.t.ri, b), ld3(A.t.rj, b), A.k.kn[b], A.k.ks[b], A.k.kb[b],
                             A.k.kt[b], v + 6 * i, v + 6 * j);
    }
    store_wrenches(A.wrench, b0, (int)(A.m - b0 < 32 ? A.m - b0 : 32), f, stage);
}

// Rows 3 half .. 3 half + 2 of (diag M + alpha K) v at site s from the bond
// wrenches of v; v on fixed sites.  kConst: another launch wrote the wrenches.
template <bool kConst>
__device__ __forceinline__ d3 operator_rows(const Operator &A, const double *v, int64_t s, int half) {
    const int64_t at = 6 * s + 3 * half;
    const d3 acc = gather_half<kConst>(A.ptr, A.inc, A.wrench, s, half), u = ld3(v + at), m = ld3(A.mass + at);
    return A.fixed[s] ? u
                      : mk(m.x * u.x + A.alpha * acc.x, m.y * u.y + A.alpha * acc.y, m.z * u.z + A.alpha * acc.z);
}

__global__ void __launch_bounds__(kThreads) operator_bonds(Operator A, const double *v) {
    __shared__ double stage[9 * kThreads];
    const int64_t b0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31);
    if (b0 < A.m) operator_wrenches(A, v, b0, stage + 9 * (threadIdx.x & ~31));
}

// Two lanes a site: its force rows and its torque rows.
__global__ void __launch_bounds__(kThreads) operator_sites(Operator A, const double *v, double *out) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, s = t / 2;
    if (s < A.n) st3(out, t, operator_rows<true>(A, v, s, (int)(t & 1)));
}

// ---------------------------------------------------------------------------
// Block-Jacobi PCG on (diag M + alpha K) x = b, identity rows on fixed sites
// and b's fixed rows read as zero, in one cooperative launch.
//
// kLinear (LinearBondsGPU.solve_increment, bonded_dem_linear_gpu.py:79-112):
//   start from the guess (fixed rows zeroed); every 10th iteration stop when
//   |r| / |b| < tol; afterwards the true residual |b - A x| / |b| is returned.
// kBalanced (FiniteBondsGPU.solve_increment, bonded_dem_finite_gpu.py:133-167):
//   start from zero; every 10th iteration, when |r| / |b| < tol and the pose
//   defect max |P r / scale| < 2e-8, check the true residual a = b - A x:
//   stop when |a| / |b| < 5 tol and max |P a / scale| < 1e-7.
// Both flag a non-finite residual at a test.  info = [iterations, relative
// residual (kLinear: true residual; kBalanced: the accepted true residual or
// the last tested one), state (0 converged, 1 iteration cap, 2 non-finite), |b|].
//
// The phases are those of csrc/solver.cu's elastic PCG (A applied to u = P r,
// p = u + beta p and s = w + beta s in the site pass of w): three grid
// barriers an iteration instead of four, two lanes a site, wrenches stored
// through shared memory.  30k sites / 218k bonds: 1.49 -> 0.90 ms a solve.

enum { kLinear = 0, kBalanced = 1 };

struct BlockPcgArgs {
    Operator A;
    const double *P, *scale, *rhs;
    double tol, zero_norm;
    int max_it, mode, use_guess;
    double *x, *info;
    double *r, *u, *p, *s, *part;  // part: 2 x 3 x kMaxBlocks
    unsigned *barrier;
    int *status;
};

struct Reducer {
    double *part;
    int buf;
    // Block partials (sum, sum, max) -> grid barrier -> the same totals in every block.
    __device__ __forceinline__ bool operator()(double s0, double s1, double m2, unsigned *barrier, int *status,
                                               double out[3]) {
        double v[3] = {s0, s1, m2};
        block_reduce<3, 4u>(v);
        double *p = part + (int64_t)buf * 3 * kMaxBlocks;
        if (threadIdx.x == 0) {
            p[3 * blockIdx.x] = v[0];
            p[3 * blockIdx.x + 1] = v[1];
            p[3 * blockIdx.x + 2] = v[2];
        }
        if (!grid_barrier(barrier, status)) return false;
        block_arrays<3, 4u>(p, gridDim.x, v);
#pragma unroll
        for (int k = 0; k < 3; ++k) out[k] = v[k];
        buf ^= 1;  // the other buffer: no block still reads it after the next barrier
        return true;
    }
    // the first sum alone
    __device__ __forceinline__ bool one(double s0, unsigned *barrier, int *status, double out[3]) {
        s0 = block_sum(s0);
        double *p = part + (int64_t)buf * 3 * kMaxBlocks;
        if (threadIdx.x == 0) p[blockIdx.x] = s0;
        if (!grid_barrier(barrier, status)) return false;
        out[0] = block_sum_array(p, gridDim.x);
        buf ^= 1;
        return true;
    }
};

__device__ __forceinline__ bool sweep_bonds(const BlockPcgArgs &a, const double *v, double *stage) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t b0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); b0 < a.A.m; b0 += stride)
        operator_wrenches(a.A, v, b0, stage + 9 * (threadIdx.x & ~31));
    return grid_barrier(a.barrier, a.status);
}

__device__ __forceinline__ d3 rhs_half(const BlockPcgArgs &a, int64_t s, int half) {
    return a.A.fixed[s] ? mk(0.0, 0.0, 0.0) : ld3(a.rhs + 6 * s + 3 * half);
}

__device__ __forceinline__ double scaled_max(const BlockPcgArgs &a, int64_t at, d3 z, double m) {
    if (!a.scale) return m;
    const d3 v = over_units(z, ld3(a.scale + at));
    return fmax(m, fmax(fabs(v.x), fmax(fabs(v.y), fabs(v.z))));
}

__global__ void __launch_bounds__(kThreads) block_pcg_kernel(BlockPcgArgs a) {
    __shared__ double stage[9 * kThreads];
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t n = a.A.n;
    const int half = threadIdx.x & 1;
    // site loops: lanes 2k and 2k + 1 of a warp share site s and run the same rounds
    const int64_t first = tid / 2, step = stride / 2, rounds = (n + step - 1) / step;
    Reducer reduce{a.part, 0};
    double tot[3];
    // x0: the guess with fixed rows zeroed, or zero
    for (int64_t s = first; s < n; s += step) {
        const int64_t at = 6 * s + 3 * half;
        if (!a.use_guess || a.A.fixed[s]) st3(a.x + at, mk(0.0, 0.0, 0.0));
    }
    if (a.use_guess) {
        if (!grid_barrier(a.barrier, a.status)) return;
        if (!sweep_bonds(a, a.x, stage)) return;
    }
    // r = b - A x0, u = P r
    double ru = 0.0, bb = 0.0;
    int64_t s = first;
    for (int64_t k = 0; k < rounds; ++k, s += step) {
        const bool live = s < n;
        const int64_t at = 6 * s + 3 * half;
        d3 r = mk(0.0, 0.0, 0.0);
        if (live) {
            r = rhs_half(a, s, half);
            bb = dot_add(bb, r, r);
            if (a.use_guess) r = r - operator_rows<false>(a.A, a.x, s, half);
        }
        const d3 ro = other_half(r);
        if (live) {
            const d3 u = half_rows(a.P + 36 * s, half, r, ro);
            st3(a.r + at, r);
            st3(a.u + at, u);
            ru = dot_add(ru, r, u);
        }
    }
    if (!reduce(ru, bb, 0.0, a.barrier, a.status, tot)) return;
    double gamma = tot[0];
    const double norm = sqrt(tot[1]);
    if (norm < a.zero_norm) {
        for (int64_t e = tid; e < 6 * n; e += stride) a.x[e] = 0.0;
        if (tid == 0) {
            a.info[0] = 0.0;
            a.info[1] = 0.0;
            a.info[2] = 0.0;
            a.info[3] = norm;
        }
        return;
    }
    int it = 0, state = 1;
    double relative = 0.0, beta = 0.0;
    for (; it < a.max_it; ++it) {
        // w = A u; p = u + beta p, s = w + beta s, (p, s)
        if (!sweep_bonds(a, a.u, stage)) return;
        double ps = 0.0;
        for (s = first; s < n; s += step) {
            const int64_t at = 6 * s + 3 * half;
            d3 q = operator_rows<false>(a.A, a.u, s, half), p = ld3(a.u + at);
            if (it) {
                p = axpy(beta, ld3(a.p + at), p);
                q = axpy(beta, ld3(a.s + at), q);
            }
            st3(a.p + at, p);
            st3(a.s + at, q);
            ps = dot_add(ps, p, q);
        }
        if (!reduce.one(ps, a.barrier, a.status, tot)) return;
        const double alpha = block_divide(gamma, tot[0]);
        // x += alpha p, r -= alpha s, u = P r; (r, u), and where they are tested |r|^2, max |u / scale|
        const bool tested = it % 10 == 0;
        double rr2 = 0.0, umax = 0.0;
        ru = 0.0;
        s = first;
        for (int64_t k = 0; k < rounds; ++k, s += step) {
            const bool live = s < n;
            const int64_t at = 6 * s + 3 * half;
            d3 r = mk(0.0, 0.0, 0.0);
            if (live) {
                r = axpy(-alpha, ld3(a.s + at), ld3(a.r + at));
                st3(a.x + at, axpy(alpha, ld3(a.p + at), ld3(a.x + at)));
                st3(a.r + at, r);
                if (tested) rr2 = dot_add(rr2, r, r);
            }
            const d3 ro = other_half(r);
            if (live) {
                const d3 u = half_rows(a.P + 36 * s, half, r, ro);
                st3(a.u + at, u);
                ru = dot_add(ru, r, u);
                if (tested) umax = scaled_max(a, at, u, umax);
            }
        }
        if (!(tested ? reduce(ru, rr2, umax, a.barrier, a.status, tot) : reduce.one(ru, a.barrier, a.status, tot)))
            return;
        ru = tot[0];
        if (tested) {
            relative = sqrt(tot[1]) / norm;
            if (a.mode == kLinear) {
                if (relative < a.tol) {
                    state = 0;
                    break;
                }
            } else if (relative < a.tol && tot[2] < 2e-8) {
                // true residual of the balanced test (x is complete after the last barrier)
                if (!sweep_bonds(a, a.x, stage)) return;
                double e2 = 0.0, emax = 0.0;
                s = first;
                for (int64_t k = 0; k < rounds; ++k, s += step) {
                    const bool live = s < n;
                    const d3 res = live ? rhs_half(a, s, half) - operator_rows<false>(a.A, a.x, s, half)
                                        : mk(0.0, 0.0, 0.0);
                    e2 = dot_add(e2, res, res);
                    const d3 other = other_half(res);
                    if (live) emax = scaled_max(a, 6 * s + 3 * half, half_rows(a.P + 36 * s, half, res, other), emax);
                }
                double tr[3];
                if (!reduce(e2, 0.0, emax, a.barrier, a.status, tr)) return;
                const double actual = sqrt(tr[0]) / norm;
                if (actual < 5.0 * a.tol && tr[2] < 1e-7) {
                    relative = actual;
                    state = 0;
                    break;
                }
            }
            if (!isfinite(relative)) {
                state = 2;
                break;
            }
        }
        beta = block_divide(ru, gamma);
        gamma = ru;
    }
    const int iterations = it < a.max_it ? it + 1 : a.max_it;
    if (a.mode == kLinear && state != 2) {
        if (!sweep_bonds(a, a.x, stage)) return;
        double e2 = 0.0;
        for (s = first; s < n; s += step) {
            const d3 res = rhs_half(a, s, half) - operator_rows<false>(a.A, a.x, s, half);
            e2 = dot_add(e2, res, res);
        }
        if (!reduce.one(e2, a.barrier, a.status, tot)) return;
        relative = sqrt(tot[0]) / norm;
    }
    if (tid == 0) {
        a.info[0] = (double)iterations;
        a.info[1] = relative;
        a.info[2] = (double)state;
        a.info[3] = norm;
    }
}

// ---------------------------------------------------------------------------
// Block preconditioner of the linear solves: B = diag M + alpha D per site
// (the identity on fixed sites) and P = B^-1 by the register Cholesky
// inverse (bonded_dem_linear_gpu.py:82-86, bonded_dem_finite_gpu.py:141-143).
__global__ void __launch_bounds__(128) block_inverse_kernel(int64_t n, const double *mass, const uint8_t *fixed,
                                                            const double *diagonal, double alpha, double *block,
                                                            double *P) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= n) return;
    double B[36], Pi[36];
    const bool fx = fixed[s] != 0;
#pragma unroll
    for (int e = 0; e < 36; ++e) {
        const int row = e / 6, col = e % 6;
        const double eye = row == col ? 1.0 : 0.0;
        B[e] = fx ? eye : eye * mass[6 * s + row] + alpha * diagonal[36 * s + e];
    }
    spd_inverse6(B, Pi);
#pragma unroll
    for (int e = 0; e < 36; ++e) {
        if (block) block[36 * s + e] = B[e];
        P[36 * s + e] = Pi[e];
    }
}

// ---------------------------------------------------------------------------
// Linear implicit midpoint (bonded_dem_linear_gpu.py:114-121):
//   rhs = dt M v + dt^2/2 (external - K q),  guess = dt v;
//   after the solve: v <- 2 dq / dt - v,  q <- q + dq.

__global__ void __launch_bounds__(kThreads) linear_rhs_kernel(int64_t len, const double *mass, const double *v,
                                                              const double *external, const double *kq, double dt,
                                                              double *rhs, double *guess) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const double h = 0.5 * dt * dt;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < len; e += stride) {
        rhs[e] = dt * mass[e] * v[e] + h * (external[e] - kq[e]);
        guess[e] = dt * v[e];
    }
}

__global__ void __launch_bounds__(kThreads) linear_advance_kernel(int64_t len, const double *dq, double dt, double *v,
                                                                  double *q) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < len; e += stride) {
        v[e] = 2.0 * dq[e] / dt - v[e];
        q[e] += dq[e];
    }
}

// [sum a.b, 1/2 (sum m v^2 + sum q kq)] with the "last block" protocol.
__global__ void __launch_bounds__(kThreads) pair_sums_kernel(int64_t len, const double *a, const double *b,
                                                             const double *mass, const double *v, const double *q,
                                                             const double *kq, double *out, double *partials) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    double ab = 0.0, en = 0.0;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < len; e += stride) {
        if (a) ab += a[e] * b[e];
        if (mass) en += mass[e] * v[e] * v[e] + q[e] * kq[e];
    }
    ab = block_sum(ab);
    en = block_sum(en);
    double *part = partials + kCounter;
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = ab;
        part[2 * blockIdx.x + 1] = en;
    }
    if (last_block(reinterpret_cast<unsigned *>(partials))) {
        double totals[2];
        block_arrays<2, 0u>(part, gridDim.x, totals);
        const double s_ab = totals[0], s_en = totals[1];
        if (threadIdx.x == 0) {
            out[0] = s_ab;
            out[1] = 0.5 * s_en;
        }
    }
}

// ---------------------------------------------------------------------------
// Anderson mixing over device history slots (bonded_dem_finite_gpu.py:215-229).
// Slots hold iterates y_k and corrections c_k as (N, 6) rows of two
// (slots, N, 6) arrays; order[0..count) lists the slots oldest first.  With
// dc_h = c_{h+1} - c_h and the weights u = [1, 1, 1, r, r, r]:
//   gram[h][l] = sum (u dc_h)(u dc_l),  proj[h] = sum (u dc_h)(u c_last).

struct History {
    const double *y, *c;
    int64_t ld;  // doubles per slot (6 N)
    int order[kMaxHistory];
    int count;
};

__global__ void __launch_bounds__(kThreads) anderson_gram_kernel(int64_t n, History H, const double *radii,
                                                                 double *out, double *partials) {
    constexpr int kPairs = (kMaxHistory - 1) * kMaxHistory / 2;
    const int dh = H.count - 1;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    double acc[kPairs + kMaxHistory - 1];
    const int terms = dh * (dh + 1) / 2 + dh;
    for (int k = 0; k < terms; ++k) acc[k] = 0.0;
    const double *last = H.c + (int64_t)H.order[H.count - 1] * H.ld;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < 6 * n; e += stride) {
        const double u = (e % 6) < 3 ? 1.0 : radii[e / 6];
        double w[kMaxHistory - 1];
        for (int h = 0; h < dh; ++h)
            w[h] = u * (H.c[(int64_t)H.order[h + 1] * H.ld + e] - H.c[(int64_t)H.order[h] * H.ld + e]);
        const double cl = u * last[e];
        int k = 0;
        for (int h = 0; h < dh; ++h)
            for (int l = h; l < dh; ++l) acc[k++] += w[h] * w[l];
        for (int h = 0; h < dh; ++h) acc[k++] += w[h] * cl;
    }
    double *part = partials + kCounter;
    for (int k = 0; k < terms; ++k) {
        const double v = block_sum(acc[k]);
        if (threadIdx.x == 0) part[(int64_t)k * gridDim.x + blockIdx.x] = v;
    }
    if (last_block(reinterpret_cast<unsigned *>(partials) + 1)) {
        for (int k = 0; k < terms; ++k) {
            const double v = block_sum_array(part + (int64_t)k * gridDim.x, gridDim.x);
            if (threadIdx.x == 0) out[k] = v;
        }
    }
}

struct Coefficients {
    double c[kMaxHistory];
};

// out = c_last - sum_h coef_h (dy_h + dc_h); flag[0] = 1 if any entry is not finite.
__global__ void __launch_bounds__(kThreads) anderson_mix_kernel(int64_t len, History H, Coefficients coef,
                                                                double *out, int *flag) {
    const int dh = H.count - 1;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const double *last = H.c + (int64_t)H.order[H.count - 1] * H.ld;
    bool bad = false;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < len; e += stride) {
        double v = last[e];
        for (int h = 0; h < dh; ++h) {
            const int64_t a = (int64_t)H.order[h] * H.ld + e, b = (int64_t)H.order[h + 1] * H.ld + e;
            v -= coef.c[h] * ((H.y[b] + H.c[b]) - (H.y[a] + H.c[a]));
        }
        out[e] = v;
        bad |= !isfinite(v);
    }
    if (bad) atomicOr(flag, 1);
}

// ---------------------------------------------------------------------------
// Self-test of the bounded grid barrier: every block waits for `parties`
// arrivals; with parties above the grid size nobody releases the barrier and
// each wait gives up after timeout_ns, setting DPF_ERR_BARRIER_TIMEOUT.
__global__ void barrier_selftest_kernel(unsigned *barrier, int *status, unsigned long long timeout_ns,
                                        unsigned parties, int *passed) {
    if (grid_barrier(barrier, status, timeout_ns, parties) && threadIdx.x == 0) atomicAdd(passed, 1);
}

struct DeviceInfo {
    int sms = 0, per_sm = 0;
};

DeviceInfo &device_info() {
    static DeviceInfo info[64];
    int dev = 0;
    cudaGetDevice(&dev);
    DeviceInfo &d = info[dev & 63];
    if (d.sms == 0) {
        cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.per_sm, block_pcg_kernel, kThreads, 0);
    }
    return d;
}

bool graph_ok(const dpf_graph *g) {
    return g && g->n_sites > 0 && g->n_bonds >= 0 && g->n_bonds < (int64_t(1) << 31) && g->inc_ptr &&
           (g->n_bonds == 0 || (g->edges && g->inc_bond));
}

Operator make_operator(const dpf_graph *g, const dpf_stiffness *k, const dpf_tangent *t, const double *mass,
                       const uint8_t *fixed, double alpha, double *wrench) {
    return Operator{g->n_sites, g->n_bonds, g->inc_ptr, g->inc_bond, g->edges, *k, *t, mass, fixed, alpha, wrench};
}

bool history_ok(const double *y, const double *c, int64_t n, int slots, const int32_t *order, int count) {
    if (!y || !c || !order || n <= 0 || slots < 1 || slots > kMaxHistory || count < 2 || count > slots) return false;
    for (int h = 0; h < count; ++h)
        if (order[h] < 0 || order[h] >= slots) return false;
    return true;
}

History make_history(const double *y, const double *c, int64_t n, const int32_t *order, int count) {
    History H{};
    H.y = y;
    H.c = c;
    H.ld = 6 * n;
    H.count = count;
    for (int h = 0; h < count; ++h) H.order[h] = order[h];
    return H;
}

}  // namespace lin
}  // namespace dpf

using namespace dpf;
using namespace dpf::lin;

extern "C" {

int dpf_operator_apply(const dpf_graph *g, const dpf_stiffness *k, const dpf_tangent *t, const double *mass,
                       const uint8_t *fixed, double alpha, const double *q, double *out, double *wrench,
                       void *stream) {
    if (!graph_ok(g) || !k || !t || !mass || !fixed || !q || !out || (g->n_bonds && !wrench))
        return DPF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    const Operator A = make_operator(g, k, t, mass, fixed, alpha, wrench);
    if (g->n_bonds) operator_bonds<<<blocks_for(g->n_bonds, kThreads), kThreads, 0, st>>>(A, q);
    operator_sites<<<blocks_for(2 * g->n_sites, kThreads), kThreads, 0, st>>>(A, q, out);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_block_inverse(int64_t n_sites, const double *mass, const uint8_t *fixed, const double *diagonal, double alpha,
                      double *block, double *preconditioner, void *stream) {
    if (n_sites <= 0 || !mass || !fixed || !diagonal || !preconditioner) return DPF_ERR_ARGUMENT;
    block_inverse_kernel<<<blocks_for(n_sites, 128), 128, 0, (cudaStream_t)stream>>>(n_sites, mass, fixed, diagonal,
                                                                                     alpha, block, preconditioner);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int64_t dpf_block_pcg_workspace_doubles(int64_t n_sites) { return 24 * n_sites + 6 * (int64_t)kMaxBlocks; }

int dpf_block_pcg(const dpf_graph *g, const dpf_stiffness *k, const dpf_tangent *t, const double *mass,
                  const uint8_t *fixed, const double *preconditioner, const double *scale, const double *rhs,
                  double alpha, double tolerance, int max_iterations, int mode, int use_guess, double *x,
                  double *info, double *wrench, double *workspace, unsigned *barrier, int *status, void *stream) {
    if (!graph_ok(g) || !k || !t || !mass || !fixed || !preconditioner || !rhs || !x || !info || !workspace ||
        !barrier || !status || (g->n_bonds && !wrench) || max_iterations < 1 || (mode != kLinear && mode != kBalanced) ||
        (mode == kBalanced && !scale) || !(tolerance >= 0.0))
        return DPF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    DeviceInfo &info_d = device_info();
    if (info_d.sms <= 0 || info_d.per_sm <= 0) return DPF_ERR_CUDA;
    // the grid of csrc/solver.cu's elastic PCG, and why
    const int64_t items = 2 * g->n_sites > g->n_bonds ? 2 * g->n_sites : g->n_bonds;
    const bool few = items <= 512 * (int64_t)info_d.sms;
    const int threads = few ? 128 : kThreads;
    int64_t cap = (int64_t)info_d.sms * (few ? 1 : info_d.per_sm < 2 ? info_d.per_sm : 2);
    if (cap > kMaxBlocks) cap = kMaxBlocks;
    const int64_t want = blocks_for(items, threads);
    const int grid = (int)(want < cap ? (want < 1 ? 1 : want) : cap);
    const int64_t n6 = 6 * g->n_sites;
    BlockPcgArgs a{};
    a.A = make_operator(g, k, t, mass, fixed, alpha, wrench);
    a.P = preconditioner;
    a.scale = scale;
    a.rhs = rhs;
    a.tol = tolerance;
    a.zero_norm = mode == kLinear ? 1e-30 : 1e-40;
    a.max_it = max_iterations;
    a.mode = mode;
    a.use_guess = use_guess ? 1 : 0;
    a.x = x;
    a.info = info;
    a.r = workspace;
    a.u = workspace + n6;
    a.p = workspace + 2 * n6;
    a.s = workspace + 3 * n6;
    a.part = workspace + 4 * n6;
    a.barrier = barrier;
    a.status = status;
    if (cudaMemsetAsync(barrier, 0, 2 * sizeof(unsigned), st) != cudaSuccess) {
        cudaGetLastError();
        return DPF_ERR_CUDA;
    }
    void *args[] = {&a};
    if (cudaLaunchCooperativeKernel((const void *)block_pcg_kernel, grid, threads, args, 0, st) != cudaSuccess) {
        cudaGetLastError();
        return DPF_ERR_CUDA;
    }
    return DPF_OK;
}

int dpf_linear_midpoint_rhs(int64_t n_sites, const double *mass, const double *v, const double *external,
                            const double *kq, double dt, double *rhs, double *guess, void *stream) {
    if (n_sites <= 0 || !mass || !v || !external || !kq || !rhs || !guess || !(dt > 0.0)) return DPF_ERR_ARGUMENT;
    linear_rhs_kernel<<<reduce_grid(6 * n_sites), kThreads, 0, (cudaStream_t)stream>>>(6 * n_sites, mass, v, external,
                                                                                       kq, dt, rhs, guess);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_linear_midpoint_advance(int64_t n_sites, const double *dq, double dt, double *v, double *q, void *stream) {
    if (n_sites <= 0 || !dq || !v || !q || !(dt > 0.0)) return DPF_ERR_ARGUMENT;
    linear_advance_kernel<<<reduce_grid(6 * n_sites), kThreads, 0, (cudaStream_t)stream>>>(6 * n_sites, dq, dt, v,
                                                                                           q);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int64_t dpf_small_partials_doubles(void) { return kCounter + 64 * 1024; }

int dpf_linear_sums(int64_t n_sites, const double *a, const double *b, const double *mass, const double *v,
                    const double *q, const double *kq, double *out, double *partials, void *stream) {
    if (n_sites <= 0 || !out || !partials || (a && !b) || (mass && (!v || !q || !kq)) || (!a && !mass))
        return DPF_ERR_ARGUMENT;
    pair_sums_kernel<<<reduce_grid(6 * n_sites), kThreads, 0, (cudaStream_t)stream>>>(6 * n_sites, a, b, mass, v, q,
                                                                                      kq, out, partials);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_anderson_gram(int64_t n_sites, const double *iterates, const double *corrections, int slots,
                      const int32_t *order, int count, const double *radii, double *out, double *partials,
                      void *stream) {
    if (!history_ok(iterates, corrections, n_sites, slots, order, count) || !radii || !out || !partials)
        return DPF_ERR_ARGUMENT;
    // one reduction term per block row: keep the grid within the partials' rows
    const int dh = count - 1, terms = dh * (dh + 1) / 2 + dh;
    int grid = reduce_grid(6 * n_sites);
    if ((int64_t)terms * grid > 64 * 1024) grid = (64 * 1024) / terms;
    anderson_gram_kernel<<<grid, kThreads, 0, (cudaStream_t)stream>>>(
        n_sites, make_history(iterates, corrections, n_sites, order, count), radii, out, partials);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_anderson_mix(int64_t n_sites, const double *iterates, const double *corrections, int slots,
                     const int32_t *order, int count, const double *coefficients, double *out, int *flag,
                     void *stream) {
    if (!history_ok(iterates, corrections, n_sites, slots, order, count) || !coefficients || !out || !flag)
        return DPF_ERR_ARGUMENT;
    Coefficients c{};
    for (int h = 0; h < count - 1; ++h) c.c[h] = coefficients[h];
    anderson_mix_kernel<<<reduce_grid(6 * n_sites), kThreads, 0, (cudaStream_t)stream>>>(
        6 * n_sites, make_history(iterates, corrections, n_sites, order, count), c, out, flag);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_barrier_selftest(int blocks, int64_t timeout_ns, int missing, unsigned *barrier, int *status, int *passed,
                         void *stream) {
    if (blocks < 1 || blocks > 64 || timeout_ns <= 0 || timeout_ns > 2000000000LL || missing < 0 || missing > 64 ||
        !barrier || !status || !passed)
        return DPF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaMemsetAsync(barrier, 0, 2 * sizeof(unsigned), st) != cudaSuccess) {
        cudaGetLastError();
        return DPF_ERR_CUDA;
    }
    void *args[5];
    unsigned long long t = (unsigned long long)timeout_ns;
    unsigned parties = (unsigned)(blocks + missing);
    args[0] = &barrier;
    args[1] = &status;
    args[2] = &t;
    args[3] = &parties;
    args[4] = &passed;
    if (cudaLaunchCooperativeKernel((const void *)barrier_selftest_kernel, blocks, 32, args, 0, st) != cudaSuccess) {
        cudaGetLastError();
        return DPF_ERR_CUDA;
    }
    return DPF_OK;
}

}  // extern "C"
