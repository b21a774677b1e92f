// Native step driver of the mixed-precision Newton solver: the control flow of
// NewtonBonds.step and fgmres (experiments/bonded_dem_newton.py:13-60,
// 132-201) as host code that launches this library's entry points directly.
//
// The Python control path (MixedNewtonBonds.step) and this driver do the same
// arithmetic on every entry in the same order and take the same host decisions
// in float64 (Givens rotations with hypot, back substitution, convergence
// tests, Armijo line search), so a step gives bit-identical results either way.
// What changes is what lies between: the host's C++ instead of Python, passes
// over whole vectors joined into one (the start of a step, the end of a Krylov
// cycle, the end state), and results written to pinned host memory by the
// kernels instead of copied.  A 4k-site step is bound by the launches and by the
// waits: 62 launches, copies and memsets took 735 us, 22 launches take 578 us; at
// 262k sites the joined passes save the traffic of whole vectors (5186 us a step,
// now 4874).
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "internal.cuh"

namespace dpf {
namespace driver {

// The end of an accepted step: x_end = x + u, v_end = 2 y / dt - v, R_end = exp(y_w) R
// (each as dpf_mixed_commit and dpf_accept_step form it), and the largest |y_w|,
// with the PCG's iteration count, to the host.
struct AcceptArgs {
    int64_t n;
    const double *x, *y, *v, *rotation;
    double two_over_dt;
    double *x_end, *v_end, *rotation_end, *partials, *turn;
    const int *inner;
    int *inner_to;
};

__global__ void __launch_bounds__(kThreads) accept_kernel(AcceptArgs a) {
    double turn = 0.0;
    for (int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; s < a.n; s += (int64_t)gridDim.x * blockDim.x) {
        const double2 *yp = reinterpret_cast<const double2 *>(a.y + 6 * s);
        const double2 y0 = yp[0], y1 = yp[1], y2 = yp[2];
        const double y[6] = {y0.x, y0.y, y1.x, y1.y, y2.x, y2.y};
        const d3 u = mk(y[0], y[1], y[2]), w = mk(y[3], y[4], y[5]);
        double v[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) v[c] = end_velocity(a.two_over_dt, y[c], a.v[6 * s + c]);
        st3(a.x_end, s, ld3(a.x, s) + u);
#pragma unroll
        for (int c = 0; c < 6; ++c) a.v_end[6 * s + c] = v[c];
        rotate_site(w, a.rotation + 9 * s, a.rotation_end + 9 * s);
        turn = fmax(turn, dot(w, w));
    }
    turn = block_max(turn);
    double *part = a.partials + 8;
    if (threadIdx.x == 0) part[blockIdx.x] = turn;
    if (last_block(reinterpret_cast<unsigned *>(a.partials) + 1)) {
        const double most = block_max_array(part, gridDim.x, 1);
        if (threadIdx.x == 0) {
            *a.turn = sqrt(most);
            *a.inner_to = *a.inner;
        }
    }
}

// launch categories timed with step->timing (the order of DPF_NEWTON_TIMERS)
enum Timer {
    kSetup = 0,  // float64 setup or the per-step begin
    kResidual,   // residual bond and site passes
    kScaling,    // 6x6 blocks and their inverses
    kPcg,        // the elastic PCG
    kJvp,        // J d
    kCommit,     // end state of the accepted increment
    kPack,       // bond-end records of a tangent
    kKrylov,     // Arnoldi, row combination, Krylov norms and scaling
    kNorms,      // scaled residual and its norms
    kVector,     // float64 vector updates (rhs, correction, candidates, float32 copies)
    kAccept      // velocity, rotation, work and step statistics
};
static_assert(kAccept + 1 == DPF_NEWTON_TIMERS, "one timer per category");

// CUDA events around the launches (only with step->timing), created for the
// call and destroyed before it returns.
struct Timing {
    bool on = false;
    cudaStream_t stream = nullptr;
    std::vector<int> keys;
    std::vector<cudaEvent_t> events;
    void record(bool opening, int key) {
        if (!on) return;
        cudaEvent_t e = nullptr;
        if (cudaEventCreate(&e) != cudaSuccess) {
            on = false;  // no timing rather than a failed step
            return;
        }
        if (opening) keys.push_back(key);
        events.push_back(e);
        cudaEventRecord(e, stream);
    }
    // after the stream has been synchronised
    void collect(dpf_newton_info *info) {
        for (size_t k = 0; k < keys.size() && 2 * k + 1 < events.size(); ++k) {
            float ms = 0.0f;
            if (cudaEventElapsedTime(&ms, events[2 * k], events[2 * k + 1]) == cudaSuccess) {
                info->time_ms[keys[k]] += ms;
                info->timed_launches[keys[k]] += 1;
            }
        }
    }
    ~Timing() {
        for (cudaEvent_t e : events) cudaEventDestroy(e);
    }
};

struct Step {
    const dpf_mixed_newton *s;
    const dpf_newton_step *a;
    dpf_newton_info *info;
    cudaStream_t st;
    int64_t n, n6, m;
    double *y, *cand, *r, *r_cand, *scaled, *rhs, *x, *res, *corr;
    double *host;     // pinned, written by the kernels: [0..3) a residual's norms, [4..7) the scaled residual's,
                      // [8..10) scales, [12..14) the true Krylov residual's, [14..16) work, [16..80) h column
    int *host_int;    // pinned ints after the doubles: [0] status, [1] inner
    const double *v0, *rotation0;   // the step's start
    Timing timing;
    bool packed = false;
    double rhs_scale = -1.0;
    // the iterate's 6x6 blocks, their inverses and units, and the other set,
    // which the speculative scaling of a line-search candidate writes
    struct Scaling {
        float *block32, *p32, *units32;
        double *units;
    } cur, alt;

    // one library call of `kernels` launches, timed under `key`
    template <class F>
    int call(int key, int kernels, F &&f) {
        timing.record(true, key);
        const int rc = f();
        timing.record(false, key);
        if (!rc) info->launches += kernels;
        return rc;
    }

    // wait for the stream, after copying the status word when no kernel reported it
    int wait(bool status = false) {
        if (status && cudaMemcpyAsync(host_int, s->status, sizeof(int), cudaMemcpyDeviceToHost, st))
            return DPF_ERR_CUDA;
        return cudaStreamSynchronize(st) == cudaSuccess ? DPF_OK : DPF_ERR_CUDA;
    }

    // prepared: y32 = (float)yy and the cleared status word are there already
    int residual(const double *yy, double *out, bool use_p, bool prepared) {
        if (!prepared) {
            const int rc = call(kVector, 1, [&] { return dpf_to_float(n6, yy, s->y32, st); });
            if (rc) return rc;
            if (cudaMemsetAsync(s->status, 0, sizeof(int), st)) return DPF_ERR_CUDA;
        }
        return call(kResidual, m ? 2 : 1, [&] {
            return dpf_mixed_residual(s->graph, s->bond_data, yy, s->y32, s->mass, s->fixed, a->dt, s->r0, 1,
                                      use_p ? cur.p32 : nullptr, use_p ? cur.units32 : nullptr, out, nullptr,
                                      use_p ? host : nullptr, s->wrench32, s->partials, s->status, st);
        });
    }

    // blocks and scaling of the tangent in bond_data into `into`, then the
    // scaled residual of rr and its norms [|r|, max |s|, |s|] into norms, with
    // the report and the status word
    int scaling_norms(const Scaling &into, const double *rr, double *norms, Report report) {
        int rc = call(kScaling, 1, [&] {
            return dpf_mixed_scaling(s->graph, s->bond_data, s->mass32, s->fixed, s->radii, a->dt, into.block32,
                                     into.p32, into.units, into.units32, st);
        });
        if (rc) return rc;
        report.status = s->status;
        report.status_to = host_int;
        return call(kNorms, 1, [&] {
            return scale_residual_pass(n, into.p32, into.units32, rr, scaled, norms, s->partials, report, st);
        });
    }

    // the elastic PCG on a float32 Krylov vector; d32 = units * out for the JVP
    int precondition(const float *vector, float *out) {
        if (!packed) {
            const int rc = call(kPack, 1, [&] {
                return dpf_end_pack(s->graph, s->bond_data, 0.25 * a->dt * a->dt, cur.p32, s->mass32, s->fixed,
                                    s->ends, s->p24, s->site4, st);
            });
            if (rc) return rc;
            packed = true;
        }
        return call(kPcg, 1, [&] {
            return end_precondition32_pass(s->graph, s->ends, s->site4, s->fixed, cur.block32, s->p24, cur.units32,
                                           vector, 0.03, 80, out, s->d32, s->inner, s->end_workspace,
                                           s->end_partials, s->barrier, s->barrier + 1, s->status, s->end_variant,
                                           st);
        });
    }

    // J d on d32
    int jvp32(float *out) {
        return call(kJvp, m ? 2 : 1, [&] {
            return jvp32_pass(s->graph, s->bond_data, s->y32, s->mass32, s->fixed, a->dt, cur.units32, cur.p32, out,
                              s->d32, s->wrench32, st);
        });
    }

    // One restart cycle of the right-preconditioned FGMRES with CGS2 Arnoldi
    // (MixedNewtonBonds._fgmres32 in newton.py)
    // from sign * `start` with |start| = g0; the caller forms the correction, the
    // true residual (from the kept products J z_k) and its norm from the `columns`
    // coefficients.  The Krylov vectors are float32 (the PCG and JVP outputs carry
    // float32 precision), their sums exact float32 pairs; x and the true residual
    // are float64.  *krylov counts the Arnoldi steps; *singular reports a zero
    // Givens denominator.
    int fgmres_cycle(const double *start, double sign, double g0, double norm, double tolerance, int width,
                     int *krylov, bool *singular, double *coef, int *columns) {
        *singular = false;
        if (width > s->krylov_width) return DPF_ERR_ARGUMENT;
        const int ldh = width;  // H is (width + 1) x width, row-major
        double H[64 * 63];
        double cs[64], sn[64], g[65];
        std::memset(H, 0, sizeof(double) * (width + 1) * width);
        std::memset(cs, 0, sizeof(double) * width);
        std::memset(sn, 0, sizeof(double) * width);
        std::memset(g, 0, sizeof(double) * (width + 1));
        g[0] = g0;
        int rc = call(kKrylov, 1, [&] { return dpf_scale_to_float(n6, sign / g[0], start, s->basis, st); });
        if (rc) return rc;
        for (int j = 0; j < width; ++j) {
            float *bj = s->basis + (int64_t)j * n6;
            float *tj = s->transformed + (int64_t)j * n6;
            float *pj = s->products + (int64_t)j * n6;
            rc = precondition(bj, tj);
            if (rc) return rc;
            rc = jvp32(pj);
            if (rc) return rc;
            rc = call(kKrylov, 1, [&] {
                return arnoldi32_pass(n6, s->basis, n6, j, pj, s->w32, host + 16, s->krylov_partials,
                                      s->barrier + 1, s->barrier, s->status, st);
            });
            if (rc) return rc;
            rc = wait();
            if (rc) return rc;
            const double *column = host + 16;
            for (int k = 0; k <= j + 1; ++k) H[k * ldh + j] = column[k];
            const bool breakdown = H[(j + 1) * ldh + j] < 1e-14;
            for (int k = 0; k < j; ++k) {
                const double hk = H[k * ldh + j], hk1 = H[(k + 1) * ldh + j];
                H[k * ldh + j] = cs[k] * hk + sn[k] * hk1;
                H[(k + 1) * ldh + j] = -sn[k] * hk + cs[k] * hk1;
            }
            const double denominator = std::hypot(H[j * ldh + j], H[(j + 1) * ldh + j]);
            if (denominator == 0.0) {
                *singular = true;
                return DPF_OK;
            }
            cs[j] = H[j * ldh + j] / denominator;
            sn[j] = H[(j + 1) * ldh + j] / denominator;
            H[j * ldh + j] = denominator;
            H[(j + 1) * ldh + j] = 0.0;
            const double gj = g[j];
            g[j + 1] = -sn[j] * gj;
            g[j] = cs[j] * gj;
            *krylov += 1;
            if (std::fabs(g[j + 1]) <= tolerance * norm || breakdown || j + 1 == width) {
                // back substitution of the (j+1) x (j+1) upper triangle
                const int k = j + 1;
                for (int i = k - 1; i >= 0; --i) {
                    double acc = g[i];
                    for (int c = i + 1; c < k; ++c) acc -= H[i * ldh + c] * coef[c];
                    coef[i] = acc / H[i * ldh + i];
                }
                *columns = k;
                return DPF_OK;
            }
        }
        return DPF_OK;
    }

    // the end state (y32 is the accepted increment's already)
    int accept() {
        const dpf_history &h = a->history;
        int rc = call(kAccept, 1, [&] {
            const int threads = reduce_threads(n);
            const int64_t want = (n + threads - 1) / threads;
            AcceptArgs k{n, h.x, y, v0, rotation0, 2.0 / a->dt, a->x_end, a->v, a->rotation, s->partials, host + 2,
                         s->inner, host_int + 1};
            accept_kernel<<<(int)(want < 1024 ? want : 1024), threads, 0, st>>>(k);
            return cudaGetLastError() == cudaSuccess ? DPF_OK : DPF_ERR_CUDA;
        });
        if (rc) return rc;
        if (m) {
            rc = call(kCommit, 2, [&] {
                return mixed_commit_pass(s->graph, s->bond_data, &h, s->y32, a->x_end, a->normal_end, a->offset_end,
                                         a->fn_end, a->fs_end, a->mt_end, a->mb_end, s->history_corrections,
                                         s->wrench32, s->loads, st);
            });
            if (rc) return rc;
        }
        rc = call(kAccept, 1, [&] { return dpf_dot_norm(n6, a->external, y, host + 14, s->partials, st); });
        if (rc) return rc;
        rc = wait();
        if (rc) return rc;
        info->work = host[14];
        info->max_rotation = host[2];
        info->cg_iterations = host_int[1];
        return DPF_OK;
    }

    int run() {
        const bool committed = a->committed_start && !a->refresh;
        int rc;
        if (committed) {
            rc = call(kSetup, 1, [&] {
                return mixed_start_pass(n, s->loads, s->mass, v0, a->external, s->fixed, a->dt, s->r0, s->scales,
                                        s->partials, y, s->y32, r, s->status, s->inner, s->barrier, st);
            });
        } else {
            if (cudaMemsetAsync(s->inner, 0, sizeof(int), st) || cudaMemsetAsync(s->status, 0, sizeof(int), st) ||
                cudaMemsetAsync(s->barrier, 0, 2 * sizeof(unsigned), st) ||
                cudaMemsetAsync(y, 0, n6 * sizeof(double), st))
                return DPF_ERR_CUDA;
            rc = call(kSetup, !a->refresh ? 1 : m ? 2 : 1, [&] {
                if (!a->refresh)
                    return dpf_mixed_begin(n, s->loads, s->mass, v0, a->external, s->fixed, a->dt, s->r0, s->scales,
                                           s->partials, st);
                const dpf_history &h = a->history;
                return dpf_mixed_setup(s->graph, &s->stiffness, &h, s->mass, v0, a->external, s->fixed, a->dt,
                                       s->bond_data, s->r0, s->loads, s->scales, s->wrench64,
                                       s->history_corrections, s->partials, s->status, st);
            });
        }
        if (rc) return rc;
        bool cached = false, prefetched = false;
        double pre[3] = {0.0, 0.0, 0.0};
        const double dt = a->dt;
        for (int iteration = 0; iteration <= a->max_iterations; ++iteration) {
            double rnorm, local, merit;
            const bool first = rhs_scale < 0.0;
            if (prefetched) {
                // the accepted candidate's norms came with the line-search fetch
                rnorm = pre[0];
                local = pre[1];
                merit = pre[2];
            } else {
                if (!cached && !(iteration == 0 && committed)) {
                    rc = residual(y, r, false, false);
                    if (rc) return rc;
                }
                Report report;
                if (first) report = {s->scales, host + 8, 2};
                rc = scaling_norms(cur, r, host, report);
                if (rc) return rc;
                rc = wait();
                if (rc) return rc;
                const int status = cached ? 0 : host_int[0];
                if (status) {
                    info->outcome = DPF_NEWTON_GUARD;
                    info->guard = status;
                    return DPF_OK;
                }
                rnorm = host[0];
                local = host[1];
                merit = host[2];
            }
            cached = false;
            prefetched = false;
            packed = false;
            if (first) {
                const double sa = host[8], sl = host[9];
                double v = sa;
                if (0.5 * dt * dt * sl > v) v = 0.5 * dt * dt * sl;
                if (1e-30 > v) v = 1e-30;
                rhs_scale = v;
            }
            const double relative = rnorm / rhs_scale;
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
            // the right-hand side is -rhs (the scaled residual of the iterate); the
            // candidate's goes to the other vector
            {
                double *t = rhs;
                rhs = scaled;
                scaled = t;
            }
            // FGMRES cycles (restart 32, at most 256 Arnoldi steps).  Each cycle's
            // true-residual norm is fetched together with a speculative first
            // line-search step (factor 1) and the scaling and norms of that
            // candidate, which the next iteration starts from if it is accepted:
            // one wait instead of three.  A failed guess costs work, not results:
            // the iterate's scaling stays in `cur`, and y32 is restored before a
            // restart's JVPs.
            int krylov = 0;
            const double *start = rhs;
            double g0 = merit, sign = -1.0;
            bool speculated = false, again = false;
            for (;;) {
                double coef[64];
                int columns = 0;
                if (merit != 0.0) {
                    const int width = 256 - krylov < 32 ? 256 - krylov : 32;
                    bool singular;
                    rc = fgmres_cycle(start, sign, g0, merit, a->linear_tolerance, width, &krylov, &singular, coef,
                                      &columns);
                    if (rc) return rc;
                    if (singular) {
                        info->outcome = DPF_NEWTON_SINGULAR;
                        return DPF_OK;
                    }
                }
                rc = call(kVector, 1, [&] {
                    return mixed_correction_pass(n, s->transformed, s->products, columns, coef, again, rhs, cur.units,
                                                 s->fixed, y, x, res, corr, cand, s->y32, s->krylov_scalars,
                                                 s->krylov_partials, s->status, st);
                });
                if (rc) return rc;
                rc = residual(cand, r_cand, true, true);
                if (rc) return rc;
                rc = scaling_norms(alt, r_cand, host + 4, {s->krylov_scalars, host + 12, 2});
                if (rc) return rc;
                rc = wait();
                if (rc) return rc;
                const double krylov_relative = merit != 0.0 ? host[13] / merit : 0.0;
                info->krylov_relative = krylov_relative;
                if (krylov_relative <= 1.05 * a->linear_tolerance) {
                    speculated = true;
                    break;
                }
                if (krylov >= 256) {
                    info->outcome = DPF_NEWTON_KRYLOV;
                    return DPF_OK;
                }
                // restart from the true residual; the JVPs need the iterate's y32 again
                rc = call(kVector, 1, [&] { return dpf_to_float(n6, y, s->y32, st); });
                if (rc) return rc;
                start = res;
                sign = 1.0;
                again = true;
                g0 = host[13];
            }
            info->krylov_iterations += krylov;
            bool accepted = false;
            for (int power = 0; power < 10; ++power) {
                const double factor = std::ldexp(1.0, -power);
                if (power > 0 || !speculated) {
                    rc = call(kVector, 1, [&] { return dpf_axpby(n6, 1.0, y, factor, corr, cand, st); });
                    if (rc) return rc;
                    rc = residual(cand, r_cand, true, false);
                    if (rc) return rc;
                    rc = wait(true);
                    if (rc) return rc;
                }
                if (host_int[0]) continue;
                if (host[2] < (1.0 - 1e-4 * factor) * merit) {
                    double *t = y;
                    y = cand;
                    cand = t;
                    t = r;
                    r = r_cand;
                    r_cand = t;
                    if (power == 0) {
                        // the next iteration's scaling is the candidate's: swap the sets
                        const Scaling keep = cur;
                        cur = alt;
                        alt = keep;
                        info->scaling_alternate ^= 1;
                        prefetched = true;
                        pre[0] = host[4];
                        pre[1] = host[5];
                        pre[2] = host[6];
                    } else {
                        cached = true;
                    }
                    accepted = true;
                    break;
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

}  // namespace driver
}  // namespace dpf

extern "C" int dpf_mixed_newton_step(const dpf_mixed_newton *solver, const dpf_newton_step *step,
                                     dpf_newton_info *info, void *stream) {
    using dpf::driver::Step;
    if (!solver || !step || !info || !solver->graph || solver->graph->n_sites <= 0 || !solver->vectors ||
        !solver->host || !solver->basis || !solver->transformed || !solver->products || !solver->w32 || !solver->h ||
        !solver->block32_b || !solver->p32_b || !solver->units_b || !solver->units32_b ||
        solver->krylov_width < 1 ||
        solver->krylov_width > 62 || !step->external || !step->v || !step->rotation || !(step->dt > 0.0) ||
        step->max_iterations < 0 || ((uintptr_t)solver->vectors & 15u))
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
    double *v = solver->vectors;
    double **slots[] = {&run.y, &run.cand, &run.r, &run.r_cand, &run.scaled, &run.rhs, &run.x, &run.res, &run.corr};
    static_assert(sizeof(slots) / sizeof(slots[0]) <= DPF_NEWTON_VECTORS, "vectors of a step");
    for (size_t k = 0; k < sizeof(slots) / sizeof(slots[0]); ++k) *slots[k] = v + (int64_t)k * run.n6;
    if (!dpf_pinned_writable(solver->host)) return DPF_ERR_ARGUMENT;
    run.host = solver->host;
    run.host_int = reinterpret_cast<int *>(solver->host + 96);
    run.cur = {solver->block32, solver->p32, solver->units32, solver->units};
    run.alt = {solver->block32_b, solver->p32_b, solver->units32_b, solver->units_b};
    run.timing.on = step->timing != 0;
    run.timing.stream = run.st;
    run.v0 = step->v_in ? step->v_in : step->v;
    run.rotation0 = step->rotation_in ? step->rotation_in : step->rotation;
    int rc = run.run();
    if (rc) cudaStreamSynchronize(run.st);   // no launch writes the pinned block after the call
    // a step that did not commit leaves the start values
    if (!rc && info->outcome != DPF_NEWTON_CONVERGED &&
        ((step->v_in && cudaMemcpyAsync(step->v, step->v_in, run.n6 * sizeof(double), cudaMemcpyDeviceToDevice,
                                        run.st)) ||
         (step->rotation_in && cudaMemcpyAsync(step->rotation, step->rotation_in, 9 * run.n * sizeof(double),
                                               cudaMemcpyDeviceToDevice, run.st))))
        rc = DPF_ERR_CUDA;
    if (!run.timing.events.empty() && cudaStreamSynchronize(run.st) == cudaSuccess) run.timing.collect(info);
    return rc;
}

extern "C" int dpf_newton_struct_sizes(int64_t *out) {
    if (!out) return DPF_ERR_ARGUMENT;
    out[0] = (int64_t)sizeof(dpf_mixed_newton);
    out[1] = (int64_t)sizeof(dpf_newton_step);
    out[2] = (int64_t)sizeof(dpf_newton_info);
    return DPF_OK;
}
