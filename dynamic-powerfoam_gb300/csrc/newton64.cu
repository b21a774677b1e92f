// Native step driver of the float64 Newton solver: the control flow of
// NewtonBonds.step and fgmres (experiments/bonded_dem_newton.py:13-60,
// 132-201) as host code that launches this library's passes directly, with the
// small vector kernels that only such a step needs.
//
// A step takes the decisions of the Python control path (newton.py) in the same
// order from the same float64 numbers.  What it leaves out:
//   * the residual and tangent of an accepted line-search candidate start the
//     next iteration (the same trial at the same increment would give them
//     again);
//   * the true residual of an FGMRES cycle comes from the Arnoldi relation,
//     b - J x = V (g0 e_1 - H c) with orthonormal V (CGS2): its norm is that of
//     the host's coefficient vector, and no J x is formed;
//   * the accepted increment's end state needs no force;
//   * the blocks, inverses and scaled norms of a line-search candidate are formed
//     behind its residual, before it is accepted, so that the next iteration starts
//     without a wait of its own (a rejected candidate costs the iterate's again);
//   * what the host decides on is written to pinned memory by the kernels.
// What the host does between launches (about a hundred library calls a step from
// Python) is a few microseconds here; at 512 sites that was most of a step.
// A step of two Newton iterations, Python control path and here: 512 sites 3.07
// and 1.04 ms, 37k sites 5.86 and 3.33 ms, 262k sites 33.2 and 23.2 ms (with the
// products formed from the state instead of a stored linearisation 1.09, 3.72 and
// 27.0 ms).
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "internal.cuh"

namespace dpf {
namespace newton64 {

constexpr int kMaxColumns = 64;
constexpr int kRows = 8;       // basis rows whose dot products a pass keeps in registers
constexpr int kMaxBlocks = 1024;

// ---- one Arnoldi step, CGS2 (bonded_dem_newton.py:35-43) -----------------------

struct ArnoldiArgs {
    int64_t len, ld;
    const double *basis;
    double *w, *next, *h, *part;
    int count;
    unsigned *barrier, *clear;
    int *status;
};

// Sums over the grid of each row's block partials (part[k * grid + block]), one
// warp a row, into shared memory: the same in every block.
__device__ __forceinline__ void row_totals(const double *part, int count, double *values) {
    __syncthreads();
    for (int k = threadIdx.x >> 5; k < count; k += blockDim.x >> 5) {
        double v = 0.0;
        for (int b = threadIdx.x & 31; b < (int)gridDim.x; b += 32) v += part[(int64_t)k * gridDim.x + b];
        v = warp_sum(v);
        if ((threadIdx.x & 31) == 0) values[k] = v;
    }
    __syncthreads();
}

// One cooperative launch with three grid barriers: dot products; projection and
// the second pass's dot products (a thread reads back only its own elements, so
// no barrier between them); second projection with |w|^2; normalisation.  One, two
// and three rows, as four launches of one pass each (dpf_arnoldi_cgs2) and fused: 37k
// sites 47, 66, 83 us and 34, 37, 40 us; 262k sites 87, 128, 164 us and 86, 94, 100 us.
__global__ void __launch_bounds__(kThreads) arnoldi_kernel(ArnoldiArgs a) {
    __shared__ double values[kMaxColumns];
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    double *part2 = a.part + (int64_t)kMaxColumns * kMaxBlocks, *part3 = part2 + (int64_t)kMaxColumns * kMaxBlocks;
    if (a.clear && tid == 0) *a.clear = 0u;
    double first = 0.0;      // thread k of block 0: column entry k of the first pass (h is only written)
    for (int pass = 0; pass < 2; ++pass) {
        double *part = pass ? part2 : a.part;
        if (pass) {
            row_totals(a.part, a.count, values);
            if (threadIdx.x < a.count) first = values[threadIdx.x];
        }
        for (int k0 = 0; k0 < a.count; k0 += kRows) {
            double p[kRows];
#pragma unroll
            for (int c = 0; c < kRows; ++c) p[c] = 0.0;
            for (int64_t e = tid; e < a.len; e += stride) {
                double wv = a.w[e];
                if (pass && k0 == 0) {
                    for (int k = 0; k < a.count; ++k) wv -= a.basis[k * a.ld + e] * values[k];
                    a.w[e] = wv;
                }
#pragma unroll
                for (int c = 0; c < kRows; ++c)
                    if (k0 + c < a.count) p[c] += a.basis[(k0 + c) * a.ld + e] * wv;
            }
#pragma unroll
            for (int c = 0; c < kRows; ++c)
                if (k0 + c < a.count) {
                    const double v = block_sum(p[c]);
                    if (threadIdx.x == 0) part[(int64_t)(k0 + c) * gridDim.x + blockIdx.x] = v;
                }
        }
        if (!grid_barrier(a.barrier, a.status)) {
            if (tid == 0) a.h[a.count] = NAN;    // no column: the solve ends without convergence
            return;
        }
    }
    row_totals(part2, a.count, values);
    if (blockIdx.x == 0 && threadIdx.x < a.count) a.h[threadIdx.x] = first + values[threadIdx.x];
    double sq = 0.0;
    for (int64_t e = tid; e < a.len; e += stride) {
        double wv = a.w[e];
        for (int k = 0; k < a.count; ++k) wv -= a.basis[k * a.ld + e] * values[k];
        a.w[e] = wv;
        sq += wv * wv;
    }
    sq = block_sum(sq);
    if (threadIdx.x == 0) part3[blockIdx.x] = sq;
    if (!grid_barrier(a.barrier, a.status)) {
        if (tid == 0) a.h[a.count] = NAN;
        return;
    }
    row_totals(part3, 1, values);
    const double length = sqrt(values[0]);
    if (tid == 0) a.h[a.count] = length;
    if (!(length >= 1e-14)) return;
    const double inv = block_divide(1.0, length);
    for (int64_t e = tid; e < a.len; e += stride) a.next[e] = a.w[e] * inv;
}

struct Coefficients {
    double c[kMaxColumns];
};

// x (+)= sum c_k rows_k, then the Newton correction (units x where the rows are in
// the scaled coordinates; zero rows on fixed sites) and the full-step candidate
// y + correction; clears the status word.
__global__ void __launch_bounds__(kThreads) candidate_kernel(int64_t len, const double *rows, int64_t ld, int count,
                                                             Coefficients coef, int add, double *x,
                                                             const double *units, const uint8_t *fixed,
                                                             const double *y, double *correction, double *candidate,
                                                             int *status) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    if (blockIdx.x == 0 && threadIdx.x == 0) *status = 0;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < len; e += stride) {
        double v = 0.0;
        for (int k = 0; k < count; ++k) v += rows[k * ld + e] * coef.c[k];
        if (add) v += x[e];
        x[e] = v;
        const double c = fixed[e / 6] ? 0.0 : units ? units[e] * v : v;
        correction[e] = c;
        candidate[e] = y[e] + c;
    }
}

// The accepted step of one site: x_end = x + u, v_end = 2 y / dt - v, R_end =
// exp(y_w) R; and external . y and max |y_w| over the sites (sums per block,
// then in a fixed order by the last block).
struct AcceptArgs {
    int64_t n;
    const double *x, *y, *v, *rotation, *external;
    double two_over_dt;
    double *x_end, *v_end, *rotation_end, *out, *partials;
    const int *inner;
    int *inner_to;
};

__global__ void __launch_bounds__(kThreads) accept_state_kernel(AcceptArgs a) {
    double work = 0.0, turn = 0.0;
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < a.n; s += (int64_t)gridDim.x * blockDim.x) {
        const d3 u = ld3(a.y + 6 * s), w = ld3(a.y + 6 * s + 3);
        st3(a.x_end, s, ld3(a.x, s) + u);
        st3(a.v_end + 6 * s, end_velocity(a.two_over_dt, u, ld3(a.v + 6 * s)));
        st3(a.v_end + 6 * s + 3, end_velocity(a.two_over_dt, w, ld3(a.v + 6 * s + 3)));
        rotate_site(w, a.rotation + 9 * s, a.rotation_end + 9 * s);
        work = dot_add(dot_add(work, ld3(a.external + 6 * s), u), ld3(a.external + 6 * s + 3), w);
        turn = fmax(turn, dot(w, w));
    }
    work = block_sum(work);
    turn = block_max(turn);
    double *part = a.partials + 8;
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = work;
        part[2 * blockIdx.x + 1] = turn;
    }
    if (last_block(reinterpret_cast<unsigned *>(a.partials) + 1)) {
        double totals[2];
        block_arrays<2, 2u>(part, gridDim.x, totals);
        const double sum = totals[0], most = totals[1];
        if (threadIdx.x == 0) {
            a.out[0] = sum;
            a.out[1] = sqrt(most);
            *a.inner_to = *a.inner;
        }
    }
}

// The start of a step: its scale [|dt M v + dt^2/2 ext|, |loads on free sites|]
// (bonded_dem_newton.py:138-139) with the sites' loads summed here from the bonds'
// wrenches, y = 0 and the cleared words.  Two lanes a site.
struct StartArgs {
    int64_t n;
    const int32_t *ptr, *inc;
    const double *wrench, *mass, *v, *external;
    const uint8_t *fixed;
    double dt, half_dt2;
    double *y, *scales, *partials, *general;
    int *status, *inner;
    unsigned *barrier;
};

__global__ void __launch_bounds__(kThreads) start_kernel(StartArgs a) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.status = *a.inner = a.barrier[0] = a.barrier[1] = 0;
        *a.general = 0.0;
    }
    double sums[2] = {0.0, 0.0};
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < 2 * a.n; t += stride) {
        const int64_t s = t / 2;
        const d3 m = ld3(a.mass, t), v = ld3(a.v, t), ext = ld3(a.external, t);
        const d3 rhs = mk(a.dt * m.x * v.x + a.half_dt2 * ext.x, a.dt * m.y * v.y + a.half_dt2 * ext.y,
                          a.dt * m.z * v.z + a.half_dt2 * ext.z);
        sums[0] = dot_add(sums[0], rhs, rhs);
        if (!a.fixed[s]) {
            const d3 loads = gather_half(a.ptr, a.inc, a.wrench, s, (int)(t & 1));
            sums[1] = dot_add(sums[1], loads, loads);
        }
        st3(a.y, t, mk(0.0, 0.0, 0.0));
    }
    block_reduce<2, 0u>(sums);
    double *part = a.partials + 8;
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = sums[0];
        part[2 * blockIdx.x + 1] = sums[1];
    }
    if (last_block(reinterpret_cast<unsigned *>(a.partials) + 1)) {
        block_arrays<2, 0u>(part, gridDim.x, sums);
        if (threadIdx.x == 0) {
            a.scales[0] = sqrt(sums[0]);
            a.scales[1] = sqrt(sums[1]);
        }
    }
}

inline int reduce_grid(int64_t count) {
    const int64_t g = (count + kThreads - 1) / kThreads;
    return (int)(g < 1 ? 1 : g > kMaxBlocks ? kMaxBlocks : g);
}

struct Step {
    const dpf_newton64 *s;
    const dpf_newton_step *a;
    dpf_newton_info *info;
    cudaStream_t st;
    int64_t n, n6, m;
    double *y, *cand, *r, *r_cand, *scaled, *x, *corr;
    double *host;     // pinned, written by the kernels: [0..3) a residual's norms, [4..6) scales, [6] normals without
                      // unit length, [8..11) the scaled residual's norms, [12..14) a restart's, [16..80) h column
    int *host_int;    // [0] status, [1] inner
    double rhs_scale = -1.0;
    dpf_tangent tangent;
    // elastic preconditioning with a stored linearisation: the preconditioner's rows
    // are in the coordinates of y (x instead of x / units), as the product wants them
    bool raw = false;

    int ran(int kernels, int rc) {
        if (!rc) info->launches += kernels;
        return rc;
    }

    // wait for the stream, after copying the status word when no kernel reported it
    int wait(bool status = false) {
        if (status && cudaMemcpyAsync(host_int, s->status, sizeof(int), cudaMemcpyDeviceToHost, st))
            return DPF_ERR_CUDA;
        return cudaStreamSynchronize(st) == cudaSuccess ? DPF_OK : DPF_ERR_CUDA;
    }

    // residual of yy with every trial guard and the tangent there; use_p: also
    // the norms of P r / units; cleared: the status word is
    int residual(const double *yy, double *out, bool use_p, bool cleared) {
        if (!cleared && cudaMemsetAsync(s->status, 0, sizeof(int), st)) return DPF_ERR_CUDA;
        dpf_trial_out t{};
        t.n = s->n;
        t.ri = s->ri;
        t.rj = s->rj;
        return ran(m ? 2 : 1, dpf::residual_pass(s->graph, &s->stiffness, &a->history, yy, a->v_in, a->external,
                                                 s->mass, s->fixed, a->dt, &t, use_p ? s->preconditioner : nullptr,
                                                 use_p ? s->units : nullptr, out, use_p ? host : nullptr,
                                                 s->wrench, s->partials, s->status, s->elastic ? s->linear : nullptr,
                                                 s->scalars + 6, st));
    }

    // blocks and scaling of the tangent, then P r / units and its norms (host[8..11)),
    // with the status word and the flag of the normals
    int scaling(const double *rr) {
        int rc = ran(1, dpf_prepare_scaling(s->graph, &s->stiffness, &tangent, s->mass, s->fixed, s->radii, a->dt,
                                            s->diagonal, s->block, s->preconditioner, s->units, st));
        if (rc) return rc;
        return ran(1, dpf::scale_residual64_pass(n, s->preconditioner, s->units, rr, scaled, host + 8, s->partials,
                                                 dpf::Report{s->scalars + 6, host + 6, 1, s->status, host_int}, st));
    }

    // the elastic PCG and the Arnoldi step clear each other's barrier word
    int arnoldi(int j) {
        return ran(1, dpf::arnoldi_pass(n6, s->basis, n6, j, s->w, host + 16, s->krylov_partials, s->barrier + 1,
                                        s->elastic ? s->barrier : nullptr, s->status, st));
    }

    // Right-preconditioned FGMRES on the scaled system from rhs = -scaled, |rhs| =
    // norm; leaves x, the correction and the full-step candidate.  *relative:
    // |b - J x| / |b| of the last cycle.
    int fgmres(double norm, int *krylov, double *relative, bool *singular) {
        *krylov = 0;
        *relative = 0.0;
        *singular = false;
        if (norm == 0.0) return candidate(nullptr, nullptr, 0, false);
        double H[65 * 64], entries[65 * 64], cs[64], sn[64], g[65], coef[64], left[65];
        const double *start = scaled;
        double sign = -1.0, g0 = norm;
        bool add = false;
        while (*krylov < 256) {
            const int width = 256 - *krylov < s->krylov_width ? 256 - *krylov : s->krylov_width;
            std::memset(H, 0, sizeof H);
            std::memset(entries, 0, sizeof entries);
            std::memset(g, 0, sizeof g);
            g[0] = g0;
            int rc = ran(1, dpf_axpby(n6, sign / g0, start, 0.0, start, s->basis, st));
            if (rc) return rc;
            int k = 0;
            for (int j = 0; j < width; ++j) {
                double *v = s->basis + (int64_t)j * n6, *z = s->transformed + (int64_t)j * n6;
                if (s->elastic) {
                    rc = ran(1, dpf::elastic_pass(s->graph, &s->stiffness, &tangent, s->mass, s->fixed, s->block,
                                                  s->preconditioner, s->units, v, a->dt, 0.03, 80, z, s->inner,
                                                  s->wrench, s->workspace, s->barrier, s->barrier + 1, s->status,
                                                  raw ? dpf::kElasticRaw : dpf::kElastic, st));
                    if (rc) return rc;
                } else {
                    z = v;
                }
                rc = ran(m ? 2 : 1,
                         raw ? dpf::jacobian_pass(s->graph, s->linear, z, s->mass, s->fixed, a->dt, s->units,
                                                  s->preconditioner, s->w, s->wrench, st)
                             : dpf_jacobian_vector(s->graph, &s->stiffness, &a->history, y, z, s->mass, s->fixed,
                                                   a->dt, s->units, s->preconditioner, s->w, s->wrench, st));
                if (rc) return rc;
                rc = arnoldi(j);
                if (rc) return rc;
                rc = wait();
                if (rc) return rc;
                const double *column = host + 16;
                for (int i = 0; i <= j + 1; ++i) H[i * 64 + j] = entries[i * 64 + j] = column[i];
                const bool breakdown = column[j + 1] < 1e-14;
                for (int i = 0; i < j; ++i) {
                    const double hi = H[i * 64 + j], hj = H[(i + 1) * 64 + j];
                    H[i * 64 + j] = cs[i] * hi + sn[i] * hj;
                    H[(i + 1) * 64 + j] = -sn[i] * hi + cs[i] * hj;
                }
                const double denominator = std::hypot(H[j * 64 + j], H[(j + 1) * 64 + j]);
                if (denominator == 0.0) {
                    *singular = true;
                    return DPF_OK;
                }
                cs[j] = H[j * 64 + j] / denominator;
                sn[j] = H[(j + 1) * 64 + j] / denominator;
                H[j * 64 + j] = denominator;
                H[(j + 1) * 64 + j] = 0.0;
                g[j + 1] = -sn[j] * g[j];
                g[j] = cs[j] * g[j];
                *krylov += 1;
                k = j + 1;
                if (std::fabs(g[k]) <= a->linear_tolerance * norm || breakdown || k == width) break;
            }
            for (int i = k - 1; i >= 0; --i) {
                double acc = g[i];
                for (int c = i + 1; c < k; ++c) acc -= H[i * 64 + c] * coef[c];
                coef[i] = acc / H[i * 64 + i];
            }
            rc = candidate(s->elastic ? s->transformed : s->basis, coef, k, add);
            if (rc) return rc;
            // b - J x = V left, left = g0 e_1 - H c
            double sum = 0.0;
            for (int i = 0; i <= k; ++i) {
                double acc = i == 0 ? g0 : 0.0;
                for (int c = 0; c < k; ++c) acc -= entries[i * 64 + c] * coef[c];
                left[i] = acc;
                sum += acc * acc;
            }
            *relative = std::sqrt(sum) / norm;
            if (*relative <= 1.05 * a->linear_tolerance) return DPF_OK;
            if (*krylov >= 256) break;
            // restart from V left (a breakdown leaves no last row, whose share is below 1e-14)
            const bool last = entries[k * 64 + k - 1] >= 1e-14;
            if (cudaMemsetAsync(s->residual, 0, n6 * sizeof(double), st)) return DPF_ERR_CUDA;
            rc = ran(1, dpf_combine_rows(n6, s->basis, n6, last ? k + 1 : k, left, s->residual, st));
            if (rc) return rc;
            rc = ran(1, dpf_dot_norm(n6, s->residual, nullptr, host + 12, s->partials, st));
            if (rc) return rc;
            rc = wait();
            if (rc) return rc;
            start = s->residual;
            sign = 1.0;
            g0 = host[13];
            add = true;
        }
        return DPF_OK;
    }

    int candidate(const double *rows, const double *coef, int count, bool add) {
        Coefficients c{};
        for (int k = 0; k < count; ++k) c.c[k] = coef[k];
        candidate_kernel<<<reduce_grid(n6), kThreads, 0, st>>>(n6, rows, n6, count, c, add ? 1 : 0, x,
                                                               raw ? nullptr : s->units, s->fixed, y, corr, cand,
                                                               s->status);
        return ran(1, cudaGetLastError() == cudaSuccess ? DPF_OK : DPF_ERR_CUDA);
    }

    int accept() {
        dpf_trial_out t{};
        t.normal_end = a->normal_end;
        t.offset_end = a->offset_end;
        t.fs_end = a->fs_end;
        t.mb_end = a->mb_end;
        t.fn_end = a->fn_end;
        t.mt_end = a->mt_end;
        int rc = ran(m ? 1 : 0, dpf_commit_state(s->graph, &s->stiffness, &a->history, y, &t, s->status, st));
        if (rc) return rc;
        AcceptArgs k{n, a->history.x, y, a->v_in, a->rotation_in, a->external, 2.0 / a->dt,
                     a->x_end, a->v, a->rotation, host, s->partials, s->inner, host_int + 1};
        accept_state_kernel<<<reduce_grid(n), kThreads, 0, st>>>(k);
        rc = ran(1, cudaGetLastError() == cudaSuccess ? DPF_OK : DPF_ERR_CUDA);
        if (rc) return rc;
        rc = wait();
        if (rc) return rc;
        info->work = host[0];
        info->max_rotation = host[1];
        info->cg_iterations = host_int[1];
        return DPF_OK;
    }

    int run() {
        const double dt = a->dt;
        tangent = {s->n, s->ri, s->rj};
        int rc = ran(m ? 1 : 0, dpf::loads_bonds_pass(s->graph, &a->history, s->wrench, st));
        if (rc) return rc;
        {
            StartArgs k{n, s->graph->inc_ptr, s->graph->inc_bond, s->wrench, s->mass, a->v_in, a->external, s->fixed,
                        dt, 0.5 * dt * dt, y, host + 4, s->partials, s->scalars + 6, s->status, s->inner, s->barrier};
            const int threads = reduce_threads(2 * n);
            const int64_t want = (2 * n + threads - 1) / threads;
            start_kernel<<<(int)(want < kMaxBlocks ? want : kMaxBlocks), threads, 0, st>>>(k);
            rc = ran(1, cudaGetLastError() == cudaSuccess ? DPF_OK : DPF_ERR_CUDA);
            if (rc) return rc;
        }
        rc = residual(y, r, false, true);
        if (rc) return rc;
        bool prefetched = false;
        for (int iteration = 0; iteration <= a->max_iterations; ++iteration) {
            const bool first = rhs_scale < 0.0;
            if (!prefetched) {
                rc = scaling(r);
                if (rc) return rc;
                rc = wait();
                if (rc) return rc;
            }
            prefetched = false;
            if (first && host_int[0]) {
                info->outcome = DPF_NEWTON_GUARD;
                info->guard = host_int[0];
                return DPF_OK;
            }
            if (first) {
                rhs_scale = host[4];
                if (0.5 * dt * dt * host[5] > rhs_scale) rhs_scale = 0.5 * dt * dt * host[5];
                if (1e-30 > rhs_scale) rhs_scale = 1e-30;
                raw = s->elastic && s->linear && host[6] == 0.0;
            }
            const double relative = host[8] / rhs_scale, local = host[9], merit = host[10];
            info->relative = relative;
            info->local = local;
            info->nonlinear_iterations = iteration;
            if (!std::isfinite(relative) || !std::isfinite(local)) {
                info->outcome = DPF_NEWTON_NONFINITE;
                return DPF_OK;
            }
            if (info->trace_len < DPF_NEWTON_TRACE) {
                info->trace[2 * info->trace_len] = relative;
                info->trace[2 * info->trace_len + 1] = local;
                info->trace_len += 1;
            }
            if (relative < a->tolerance && local < a->pose_tolerance) {
                rc = accept();
                if (rc) return rc;
                info->outcome = DPF_NEWTON_CONVERGED;
                return DPF_OK;
            }
            if (iteration == a->max_iterations) break;
            int krylov;
            bool singular;
            double linear;
            rc = fgmres(merit, &krylov, &linear, &singular);
            if (rc) return rc;
            if (singular) {
                info->outcome = DPF_NEWTON_SINGULAR;
                return DPF_OK;
            }
            if (!(linear <= 1.05 * a->linear_tolerance)) {
                info->outcome = DPF_NEWTON_KRYLOV;
                info->krylov_relative = linear;
                return DPF_OK;
            }
            info->krylov_iterations += krylov;
            bool accepted = false;
            for (int power = 0; power < 10 && !accepted; ++power) {
                const double factor = std::ldexp(1.0, -power);
                if (power) {
                    rc = ran(1, dpf_axpby(n6, 1.0, y, factor, corr, cand, st));
                    if (rc) return rc;
                }
                rc = residual(cand, r_cand, true, power == 0);
                if (rc) return rc;
                if (power == 0) {
                    rc = scaling(r_cand);
                    if (rc) return rc;
                }
                rc = wait(power > 0);
                if (rc) return rc;
                if (!host_int[0] && host[2] < (1.0 - 1e-4 * factor) * merit) {
                    double *t = y;
                    y = cand;
                    cand = t;
                    t = r;
                    r = r_cand;
                    r_cand = t;
                    accepted = true;
                    prefetched = power == 0;
                } else if (power == 0) {
                    // the iterate's tangent, blocks and inverses again for the other candidates
                    rc = residual(y, r, false, false);
                    if (rc) return rc;
                    rc = scaling(r);
                    if (rc) return rc;
                }
            }
            if (!accepted) {
                info->outcome = DPF_NEWTON_LINE_SEARCH;
                return DPF_OK;
            }
        }
        info->outcome = DPF_NEWTON_DIVERGED;
        return DPF_OK;
    }
};

}  // namespace newton64

int arnoldi_pass(int64_t length, double *basis, int64_t ld, int j, double *w, double *h, double *partials,
                 unsigned *barrier, unsigned *clear, int *status, cudaStream_t st) {
    using namespace newton64;
    static int per_device[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    int blocks = per_device[dev & 63];
    if (!blocks) {
        int sms = 0, per_sm = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, arnoldi_kernel, kThreads, 0);
        if (sms < 1 || per_sm < 1) return DPF_ERR_CUDA;
        blocks = sms * (per_sm < 4 ? per_sm : 4);
        if (blocks > kMaxBlocks) blocks = kMaxBlocks;
        per_device[dev & 63] = blocks;
    }
    const int64_t need = (length + kThreads - 1) / kThreads;
    if (blocks > need) blocks = (int)need;
    ArnoldiArgs k{length, ld, basis, w, basis + (int64_t)(j + 1) * ld, h, partials, j + 1, barrier, clear, status};
    if (!clear && cudaMemsetAsync(barrier, 0, sizeof(unsigned), st)) return DPF_ERR_CUDA;
    void *args[] = {&k};
    if (cudaLaunchCooperativeKernel((const void *)arnoldi_kernel, blocks, kThreads, args, 0, st) != cudaSuccess) {
        cudaGetLastError();
        return DPF_ERR_CUDA;
    }
    return DPF_OK;
}

}  // namespace dpf

extern "C" {

int dpf_pinned_writable(const void *host) {
    void *mapped = nullptr;
    if (host && cudaHostGetDevicePointer(&mapped, const_cast<void *>(host), 0) == cudaSuccess) return mapped == host;
    cudaGetLastError();
    return 0;
}

int64_t dpf_newton64_partials_doubles(void) {
    using namespace dpf::newton64;
    return (2 * (int64_t)kMaxColumns + 1) * kMaxBlocks;
}

int dpf_arnoldi_cgs2_fused(int64_t length, double *basis, int64_t ld, int j, double *w, double *h, double *partials,
                           unsigned *barrier, int *status, void *stream) {
    if (length <= 0 || !basis || !w || !h || !partials || !barrier || !status || j < 0 ||
        j + 1 >= dpf::newton64::kMaxColumns || ld < length)
        return DPF_ERR_ARGUMENT;
    return dpf::arnoldi_pass(length, basis, ld, j, w, h, partials, barrier, nullptr, status, (cudaStream_t)stream);
}

int64_t dpf_newton64_linear_doubles(int64_t n_bonds) { return n_bonds < 0 ? 0 : dpf::kLinear * n_bonds; }

int64_t dpf_newton64_struct_size(void) { return (int64_t)sizeof(dpf_newton64); }

int dpf_newton64_step(const dpf_newton64 *solver, const dpf_newton_step *step, dpf_newton_info *info, void *stream) {
    using dpf::newton64::Step;
    if (!solver || !step || !info || !solver->graph || solver->graph->n_sites <= 0 || !solver->vectors ||
        !solver->host || !solver->basis || !solver->transformed || !solver->w || !solver->residual || !solver->h ||
        !solver->krylov_partials || !solver->scalars || !solver->status || !solver->barrier || !solver->inner ||
        !solver->partials || solver->krylov_width < 1 || solver->krylov_width > 62 || !step->external || !step->v ||
        !step->rotation || !step->v_in || !step->rotation_in || !step->x_end || !(step->dt > 0.0) ||
        step->max_iterations < 0 || (solver->elastic && !solver->workspace))
        return DPF_ERR_ARGUMENT;
    std::memset(info, 0, sizeof(*info));
    Step run;
    run.s = solver;
    run.a = step;
    run.info = info;
    run.st = (cudaStream_t)stream;
    run.n = solver->graph->n_sites;
    run.n6 = 6 * run.n;
    run.m = solver->graph->n_bonds;
    double **slots[DPF_NEWTON64_VECTORS] = {&run.y, &run.cand, &run.r, &run.r_cand, &run.scaled, &run.x, &run.corr};
    for (int k = 0; k < DPF_NEWTON64_VECTORS; ++k) *slots[k] = solver->vectors + (int64_t)k * run.n6;
    if (!dpf_pinned_writable(solver->host)) return DPF_ERR_ARGUMENT;
    run.host = solver->host;
    run.host_int = reinterpret_cast<int *>(solver->host + 96);
    const int rc = run.run();
    if (rc) cudaStreamSynchronize(run.st);   // no launch writes the pinned block after the call
    info->scaling_alternate = run.y == solver->vectors ? 0 : 1;
    return rc;
}

}  // extern "C"
