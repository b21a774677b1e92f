// Solver kernels of the Newton path (float64): the elastic block-Jacobi PCG
// as one cooperative launch, the FGMRES Arnoldi building blocks, reductions,
// the accepted-step update and the energy.
#include "common.cuh"
#include "internal.cuh"

namespace dpf {

constexpr int kMaxReduceBlocks = 1024;
constexpr int64_t kPartialsOffset = 8;
constexpr int kMaxArnoldi = 64;
constexpr int kMaxPcgBlocks = 4096;

inline int blocks_for(int64_t n, int threads) { return (int)((n + threads - 1) / threads); }
constexpr int kNormResident = 5;   // dot_norm_kernel and correction_kernel: the same grid, the same sums
inline int reduce_grid(int64_t n) {
    int g = blocks_for(n, kThreads);
    if (g > kMaxReduceBlocks) g = kMaxReduceBlocks;
    if (g < 1) g = 1;
    return g;
}

__device__ __forceinline__ unsigned *counter_slot(double *partials, int slot) {
    return reinterpret_cast<unsigned *>(partials) + slot;
}

__device__ __forceinline__ void matvec6(const double *P, const double x[6], double y[6]) {
#pragma unroll
    for (int row = 0; row < 6; ++row) {
        double v = 0.0;
#pragma unroll
        for (int c = 0; c < 6; ++c) v += P[6 * row + c] * x[c];
        y[row] = v;
    }
}

// ---------------------------------------------------------------------------
// Elastic PCG (experiments/bonded_dem_newton.py:107-130) in one cooperative
// launch.  Every block reduces the per-block partials in the same order, so
// all blocks take the same (deterministic) stopping decision without a flag.

//
// The operator is applied to u = P r instead of the direction: with w = A u,
// p = u + beta p and s = w + beta s = A p are formed in the same site pass
// (beta is known by then) together with (p, s), so an iteration has three
// phases and three grid barriers (the bonds' wrenches of u; p, s and (p, s);
// x, r, u and (r, u)) where applying A to p needs a fourth phase that forms p
// before the bonds read it.  (p, s) is summed, not carried by a recurrence, so
// iterations past convergence stay harmless.  A site has two neighbouring
// lanes (force rows and torque rows), the wrenches leave a warp through shared
// memory in consecutive addresses.  x lives in `out` until the end.
// Measured per iteration, before and after: 118 -> 62 us at 37k sites / 267k
// bonds, 470 -> 339 us at 262k sites / 1.9M bonds.

struct PcgArgs {
    int64_t n, m;
    const int32_t *ptr, *inc;
    const int64_t *edges;
    dpf_stiffness k;
    dpf_tangent t;
    const double *mass, *block, *P, *units, *vector;
    const uint8_t *fixed;
    double alpha_op, tol2;
    int max_it, form;   // ElasticForm
    double *out;
    int *iterations;
    double *wrench, *r, *u, *p, *s, *part_a, *part_b;
    unsigned *barrier, *clear;   // clear: the next cooperative launch's word, or NULL
    int *status;
};

__global__ void __launch_bounds__(kThreads) pcg_kernel(PcgArgs a) {
    __shared__ double stage[9 * kThreads], over_gamma;
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int half = threadIdx.x & 1;
    if (a.clear && tid == 0) *a.clear = 0u;
    // site loops: lanes 2k and 2k + 1 of a warp share site s and run the same rounds
    const int64_t first = tid / 2, step = stride / 2, rounds = (a.n + step - 1) / step;
    double *mine = stage + 9 * (threadIdx.x & ~31);
    double part = 0.0;
    int64_t s = first;
    for (int64_t k = 0; k < rounds; ++k, s += step) {
        const bool live = s < a.n;
        const int64_t at = 6 * s + 3 * half;
        d3 v = mk(0.0, 0.0, 0.0), r = v;
        if (live) {
            const d3 un = ld3(a.units + at), in = ld3(a.vector + at);
            v = a.form == kElasticT ? over_units(in, un) : mk(un.x * in.x, un.y * in.y, un.z * in.z);
        }
        const d3 vo = other_half(v);
        if (live && !a.fixed[s]) r = a.form == kElasticT ? v : half_rows(a.block + 36 * s, half, v, vo);
        const d3 ro = other_half(r);
        if (live) {
            const d3 u = half_rows(a.P + 36 * s, half, r, ro);
            st3(a.r + at, r);
            st3(a.u + at, u);
            part = dot_add(part, r, u);
        }
    }
    part = block_sum(part);
    if (threadIdx.x == 0) a.part_b[blockIdx.x] = part;
    if (!grid_barrier(a.barrier, a.status)) return;
    double gamma = block_sum_array(a.part_b, gridDim.x);
    const double initial = gamma;
    if (initial == 0.0) {
        for (int64_t e = tid; e < 6 * a.n; e += stride) a.out[e] = 0.0;
        return;
    }
    double beta = 0.0;
    int it = 0;
    for (; it < a.max_it; ++it) {
        // wrenches of u
        for (int64_t b0 = tid - (threadIdx.x & 31); b0 < a.m; b0 += stride) {
            const int64_t b = b0 + (threadIdx.x & 31);
            Wrench f{};
            if (b < a.m) {
                int64_t i, j;
                edge(a.edges, b, i, j);
                f = stiffness_wrench(ld3(a.t.n, b), ld3(a.t.ri, b), ld3(a.t.rj, b), a.k.kn[b], a.k.ks[b], a.k.kb[b],
                                     a.k.kt[b], a.u + 6 * i, a.u + 6 * j);
            }
            store_wrenches(a.wrench, b0, (int)(a.m - b0 < 32 ? a.m - b0 : 32), f, mine);
        }
        if (!grid_barrier(a.barrier, a.status)) return;
        // w = (diag M + alpha K) u with identity rows on fixed sites; p = u + beta p, s = w + beta s, (p, s)
        part = 0.0;
        for (s = first; s < a.n; s += step) {
            const int64_t at = 6 * s + 3 * half;
            const d3 acc = gather_half<false>(a.ptr, a.inc, a.wrench, s, half), m = ld3(a.mass + at);
            d3 p = ld3(a.u + at);
            d3 q = a.fixed[s] ? p
                              : mk(m.x * p.x + a.alpha_op * acc.x, m.y * p.y + a.alpha_op * acc.y,
                                   m.z * p.z + a.alpha_op * acc.z);
            if (it) {
                p = axpy(beta, ld3(a.p + at), p);
                q = axpy(beta, ld3(a.s + at), q);
            }
            st3(a.p + at, p);
            st3(a.s + at, q);
            part = dot_add(part, p, q);
        }
        part = block_sum(part);
        if (threadIdx.x == 0) a.part_a[blockIdx.x] = part;
        if (!grid_barrier(a.barrier, a.status)) return;
        const double alpha = block_divide(gamma, block_sum_array(a.part_a, gridDim.x));
        // x += alpha p, r -= alpha s, u = P r; (r, u)
        part = 0.0;
        s = first;
        for (int64_t k = 0; k < rounds; ++k, s += step) {
            const bool live = s < a.n;
            const int64_t at = 6 * s + 3 * half;
            d3 r = mk(0.0, 0.0, 0.0);
            if (live) {
                const d3 p = ld3(a.p + at);
                r = axpy(-alpha, ld3(a.s + at), ld3(a.r + at));
                st3(a.out + at, it ? axpy(alpha, p, ld3(a.out + at)) : alpha * p);
                st3(a.r + at, r);
            }
            const d3 ro = other_half(r);
            if (live) {
                const d3 u = half_rows(a.P + 36 * s, half, r, ro);
                st3(a.u + at, u);
                part = dot_add(part, r, u);
            }
        }
        part = block_sum(part);
        if (threadIdx.x == 0) a.part_b[blockIdx.x] = part;
        const unsigned old = grid_arrive(a.barrier);
        if (threadIdx.x == 0) over_gamma = 1.0 / gamma;     // while the other blocks arrive
        if (!grid_wait(a.barrier, old, a.status)) return;
        const double following = block_sum_array(a.part_b, gridDim.x);
        if (it % 5 == 0 && following <= a.tol2 * initial) break;
        beta = following * over_gamma;
        gamma = following;
    }
    // a thread's own x: no barrier
    s = first;
    for (int64_t k = 0; k < rounds && a.form != kElasticRaw; ++k, s += step) {
        const bool live = s < a.n;
        const int64_t at = 6 * s + 3 * half;
        const d3 x = live ? ld3(a.out + at) : mk(0.0, 0.0, 0.0), un = live ? ld3(a.units + at) : x;
        if (a.form == kElasticT) {
            const d3 xo = other_half(x);
            if (live) {
                const d3 v = half_rows(a.block + 36 * s, half, x, xo);
                st3(a.out + at, mk(un.x * v.x, un.y * v.y, un.z * v.z));
            }
        } else if (live) {
            st3(a.out + at, over_units(x, un));
        }
    }
    if (tid == 0) atomicAdd(a.iterations, it < a.max_it ? it + 1 : a.max_it);
}

// ---------------------------------------------------------------------------
// Arnoldi CGS2 (experiments/bonded_dem_newton.py:35-43).

__global__ void __launch_bounds__(kThreads) arnoldi_dots(int64_t len, const double *basis, int64_t ld, int count,
                                                         const double *w, double *part) {
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int k = 0; k < count; ++k) {
        const double *row = basis + k * ld;
        double p = 0.0;
        for (int64_t e = tid; e < len; e += stride) p += row[e] * w[e];
        p = block_sum(p);
        if (threadIdx.x == 0) part[k * gridDim.x + blockIdx.x] = p;
    }
}

// values_k = sum of part_in; h[k] (=|+=) values_k; w -= sum_k values_k basis_k;
// then optionally the next pass's partial dots (part_out) or |w|^2 (part_out[blk]).
__global__ void __launch_bounds__(kThreads) arnoldi_update(int64_t len, const double *basis, int64_t ld, int count,
                                                           double *w, const double *part_in, double *h,
                                                           int accumulate, double *part_out, int want_dots) {
    __shared__ double values[kMaxArnoldi];
    for (int k = 0; k < count; ++k) {
        const double v = block_sum_array(part_in + k * gridDim.x, gridDim.x);
        if (threadIdx.x == 0) values[k] = v;
    }
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0)
        for (int k = 0; k < count; ++k) h[k] = accumulate ? h[k] + values[k] : values[k];
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    double sq = 0.0;
    for (int64_t e = tid; e < len; e += stride) {
        double proj = 0.0;
        for (int k = 0; k < count; ++k) proj += basis[k * ld + e] * values[k];
        const double wv = w[e] - proj;
        w[e] = wv;
        sq += wv * wv;
    }
    if (want_dots) {
        for (int k = 0; k < count; ++k) {
            const double *row = basis + k * ld;
            double p = 0.0;
            for (int64_t e = tid; e < len; e += stride) p += row[e] * w[e];
            p = block_sum(p);
            if (threadIdx.x == 0) part_out[k * gridDim.x + blockIdx.x] = p;
        }
    } else {
        sq = block_sum(sq);
        if (threadIdx.x == 0) part_out[blockIdx.x] = sq;
    }
}

__global__ void __launch_bounds__(kThreads) arnoldi_normalize(int64_t len, double *basis, int64_t ld, int j,
                                                              const double *w, const double *part, double *h) {
    const double nrm = sqrt(block_sum_array(part, gridDim.x));
    if (blockIdx.x == 0 && threadIdx.x == 0) h[j + 1] = nrm;
    if (!(nrm >= 1e-14)) return;
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    double *row = basis + (int64_t)(j + 1) * ld;
    // one float64 division per block, then products (float64 divides are slow on this part)
    const double inv = 1.0 / nrm;
    for (int64_t e = tid; e < len; e += stride) row[e] = w[e] * inv;
}

struct Coefficients {
    double c[kMaxArnoldi];
};

__global__ void __launch_bounds__(kThreads) combine_rows_kernel(int64_t len, const double *rows, int64_t ld, int count,
                                                                Coefficients coef, double *x) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < len; e += stride) {
        double acc = 0.0;
        for (int k = 0; k < count; ++k) acc += rows[k * ld + e] * coef.c[k];
        x[e] += acc;
    }
}

__global__ void __launch_bounds__(kThreads, kNormResident) dot_norm_kernel(int64_t len, const double *a, const double *b,
                                                            double *result, double *partials) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    double ab = 0.0, aa = 0.0;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < len; e += stride) {
        const double av = a[e];
        ab += av * (b ? b[e] : av);
        aa += av * av;
    }
    ab = block_sum(ab);
    aa = block_sum(aa);
    double *part = partials + kPartialsOffset;
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = ab;
        part[2 * blockIdx.x + 1] = aa;
    }
    if (last_block(counter_slot(partials, 1))) {
        double totals[2];
        block_arrays<2, 0u>(part, gridDim.x, totals);
        const double s_ab = totals[0], s_aa = totals[1];
        if (threadIdx.x == 0) {
            result[0] = s_ab;
            result[1] = sqrt(s_aa);
        }
    }
}

__global__ void __launch_bounds__(kThreads) axpby_kernel(int64_t len, double alpha, const double *a, double beta,
                                                         const double *b, double *out) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < len; e += stride)
        out[e] = alpha * a[e] + beta * b[e];
}

// Scaled residual s = P r / units and [|r|, max|s|, |s|] (bonded_dem_newton.py:104-105, 147).
__global__ void __launch_bounds__(kThreads) scale_kernel(int64_t n, const double *P, const double *units,
                                                         const double *r, double *scaled, double *norms,
                                                         double *partials, Report report) {
    double sum_r = 0.0, max_s = 0.0, sum_s = 0.0;
    const int half = threadIdx.x & 1;    // two neighbouring lanes a site: its force rows and its torque rows
    const int64_t step = (int64_t)gridDim.x * (blockDim.x / 2), rounds = (n + step - 1) / step;
    int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / 2;
    for (int64_t k = 0; k < rounds; ++k, s += step) {
        const bool live = s < n;
        const int64_t at = 6 * s + 3 * half;
        const d3 own = live ? ld3(r + at) : mk(0.0, 0.0, 0.0);
        sum_r = dot_add(sum_r, own, own);
        const d3 other = other_half(own);
        if (live) {
            const d3 v = over_units(half_rows(P + 36 * s, half, own, other), ld3(units + at));
            if (scaled) st3(scaled + at, v);
            max_s = fmax(max_s, fmax(fabs(v.x), fmax(fabs(v.y), fabs(v.z))));
            sum_s = dot_add(sum_s, v, v);
        }
    }
    if (!norms) return;
    double v[3] = {sum_r, max_s, sum_s};
    block_reduce<3, 2u>(v);
    double *part = partials + kPartialsOffset;
    if (threadIdx.x == 0) {
        part[3 * blockIdx.x] = v[0];
        part[3 * blockIdx.x + 1] = v[1];
        part[3 * blockIdx.x + 2] = v[2];
    }
    if (last_block(counter_slot(partials, 2))) {
        block_arrays<3, 2u>(part, gridDim.x, v);
        if (threadIdx.x == 0) {
            norms[0] = sqrt(v[0]);
            norms[1] = v[1];
            norms[2] = sqrt(v[2]);
            report.send();
        }
    }
}

// v <- 2 y / dt - v;  R <- exp(y_w) R   (bonded_dem_newton.py:150-153, bonded_dem_finite_gpu.py:35-43)
__global__ void __launch_bounds__(kThreads) accept_kernel(int64_t n, const double *y, double dt, double *v,
                                                          double *rotation) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= n) return;
    const double two_over_dt = 2.0 / dt;  // one float64 division per site, not six
#pragma unroll
    for (int c = 0; c < 6; ++c) v[6 * s + c] = end_velocity(two_over_dt, y[6 * s + c], v[6 * s + c]);
    rotate_site(ld3(y + 6 * s + 3), rotation + 9 * s, rotation + 9 * s);
}

// Elastic + kinetic energy (bonded_dem_finite_gpu.py:122-125).
__global__ void __launch_bounds__(kThreads) energy_kernel(int64_t m, int64_t n, dpf_stiffness k, dpf_history h,
                                                          const double *mass, const double *v, double *energy,
                                                          double *partials) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    double el = 0.0, kin = 0.0;
    for (int64_t b = tid; b < m; b += stride) {
        const d3 fs = ld3(h.fs, b), mb = ld3(h.mb, b);
        const double fn = h.fn[b], mt = h.mt[b];
        el += fn * fn / k.kn[b] + dot(fs, fs) / k.ks[b] + mt * mt / k.kt[b] + dot(mb, mb) / k.kb[b];
    }
    for (int64_t e = tid; e < 6 * n; e += stride) kin += mass[e] * v[e] * v[e];
    el = block_sum(el);
    kin = block_sum(kin);
    double *part = partials + kPartialsOffset;
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = el;
        part[2 * blockIdx.x + 1] = kin;
    }
    if (last_block(counter_slot(partials, 3))) {
        double totals[2];
        block_arrays<2, 0u>(part, gridDim.x, totals);
        const double se = totals[0], sk = totals[1];
        if (threadIdx.x == 0) *energy = 0.5 * se + 0.5 * sk;
    }
}

// [|dt M v + dt^2/2 ext|, |loads on free sites|] (bonded_dem_newton.py:138-139).
__global__ void __launch_bounds__(kThreads) rhs_scale_kernel(int64_t n, const double *mass, const double *v,
                                                             const double *external, const double *loads,
                                                             const uint8_t *fixed, double dt, double half_dt2,
                                                             double *out, double *partials) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    double a2 = 0.0, l2 = 0.0;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < 6 * n; e += stride) {
        const double a = dt * mass[e] * v[e] + half_dt2 * external[e];
        a2 += a * a;
        if (!fixed[e / 6]) l2 += loads[e] * loads[e];
    }
    a2 = block_sum(a2);
    l2 = block_sum(l2);
    double *part = partials + kPartialsOffset;
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = a2;
        part[2 * blockIdx.x + 1] = l2;
    }
    if (last_block(counter_slot(partials, 4))) {
        double totals[2];
        block_arrays<2, 0u>(part, gridDim.x, totals);
        const double sa = totals[0], sl = totals[1];
        if (threadIdx.x == 0) {
            out[0] = sqrt(sa);
            out[1] = sqrt(sl);
        }
    }
}

// out = units * a with zero rows on fixed sites (bonded_dem_newton.py:186-187).
__global__ void __launch_bounds__(kThreads) masked_scale_kernel(int64_t n, const double *a, const double *units,
                                                                const uint8_t *fixed, double *out) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < 6 * n; e += stride)
        out[e] = fixed[e / 6] ? 0.0 : units[e] * a[e];
}

struct DeviceInfo {
    int sms = 0;
    int pcg_blocks_per_sm = 0;
};

static DeviceInfo &device_info() {
    static DeviceInfo info[64];
    int dev = 0;
    cudaGetDevice(&dev);
    DeviceInfo &d = info[dev & 63];
    if (d.sms == 0) {
        cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.pcg_blocks_per_sm, pcg_kernel, kThreads, 0);
    }
    return d;
}

}  // namespace dpf

using namespace dpf;

namespace dpf {

// ---------------------------------------------------------------------------
// Krylov vectors in float32 with exactly accumulated float32 pairs.  The
// mixed Newton path's Krylov inputs (PCG and JVP outputs, the scaled residual)
// carry float32 precision; storing the basis in float32 and forming dot
// products and updates as float32 pairs (TwoProd by FMA, TwoSum) gives
// float64-quality sums without float64 arithmetic per entry, which is scarce
// on this part (the float64 form of these kernels ran at 77-82% of the FP64
// pipe).  Block partials and the Hessenberg entries stay float64.

__device__ __forceinline__ void ff_two_sum(float &s, float &e, float b) {
    const float t = s + b;
    const float bp = t - s;
    e += (s - (t - bp)) + (b - bp);
    s = t;
}

// (hi, lo) += a b exactly up to the pair's precision
__device__ __forceinline__ void ff_add_product(float &hi, float &lo, float a, float b) {
    const float p = a * b;
    const float e = fmaf(a, b, -p);
    ff_two_sum(hi, lo, p);
    lo += e;
}

__device__ __forceinline__ double ff_value(float hi, float lo) { return (double)hi + (double)lo; }

// float64 value v as hi + lo float32 (lo the rounded remainder)
__device__ __forceinline__ void ff_split(double v, float &hi, float &lo) {
    hi = (float)v;
    lo = (float)(v - (double)hi);
}

// x += sum_k c_k rows_k, the sum as a float32 pair, added to float64 x
__global__ void __launch_bounds__(kThreads) combine32_kernel(int64_t len, const float *rows, int64_t ld, int count,
                                                             Coefficients coef, double *x) {
    __shared__ float chi[kMaxArnoldi], clo[kMaxArnoldi];
    if (threadIdx.x < count) ff_split(coef.c[threadIdx.x], chi[threadIdx.x], clo[threadIdx.x]);
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < len; e += stride) {
        float hi = 0.0f, lo = 0.0f;
        for (int k = 0; k < count; ++k) {
            const float r = rows[k * ld + e];
            ff_add_product(hi, lo, chi[k], r);
            lo = fmaf(clo[k], r, lo);
        }
        x[e] += ff_value(hi, lo);
    }
}

// The end of a restart cycle in one pass over the entries (mixed_correction_pass):
// as eight launches (two row combinations into cleared vectors, the residual and its
// norm, the masked scaling, the candidate, its float32 copy) that each read and
// write whole float64 vectors it took 97 us at 262k sites, as one 49 us.  The sums
// over entries run in dot_norm_kernel's order.  The residual is -scaled - J z of the
// first cycle and from then on the kept residual minus the cycle's own J z.
struct CorrectionArgs {
    int64_t len;
    const float *z, *jz;
    int count, add;
    Coefficients coef;
    const double *scaled, *units;
    const uint8_t *fixed;
    const double *y;
    double *x, *res, *correction, *candidate;
    float *y32;
    double *norm, *partials;
    int *status;
};

__global__ void __launch_bounds__(kThreads, kNormResident) correction_kernel(CorrectionArgs a) {
    __shared__ float chi[kMaxArnoldi], clo[kMaxArnoldi];
    if (threadIdx.x < a.count) ff_split(a.coef.c[threadIdx.x], chi[threadIdx.x], clo[threadIdx.x]);
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.status = 0;
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    // what the cycle started from: -scaled or the kept residual (the sign off the float64 pipe)
    const double *start = a.add ? a.res : a.scaled;
    const long long flip = a.add ? 0ll : (long long)(1ull << 63);
    double aa = 0.0;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < a.len; e += stride) {
        const double kept = start[e], un = a.units[e], yv = a.y[e];
        const bool fx = a.fixed[e / 6] != 0;
        float zh = 0.0f, zl = 0.0f, jh = 0.0f, jl = 0.0f;
        for (int k = 0; k < a.count; ++k) {
            const float z = a.z[k * a.len + e], j = a.jz[k * a.len + e];
            ff_add_product(zh, zl, chi[k], z);
            zl = fmaf(clo[k], z, zl);
            ff_add_product(jh, jl, chi[k], j);
            jl = fmaf(clo[k], j, jl);
        }
        double xv = widen(zh) + widen(zl);
        if (a.add) xv += a.x[e];
        const double rv = __longlong_as_double(__double_as_longlong(kept) ^ flip) - (widen(jh) + widen(jl));
        const double c = fx ? 0.0 : __dmul_rn(un, xv), y1 = yv + c;   // rounded as masked_scale_kernel does
        a.x[e] = xv;
        a.res[e] = rv;
        a.correction[e] = c;
        a.candidate[e] = y1;
        a.y32[e] = narrow(y1);
        aa += rv * rv;
    }
    aa = block_sum(aa);
    double *part = a.partials + kPartialsOffset;
    if (threadIdx.x == 0) part[blockIdx.x] = aa;
    if (last_block(counter_slot(a.partials, 1))) {
        const double total = block_sum_array(part, gridDim.x, 1);
        if (threadIdx.x == 0) {
            a.norm[0] = total;
            a.norm[1] = sqrt(total);
        }
    }
}

// CGS2 of one Arnoldi step in one cooperative launch with three grid barriers:
// dots; projection with the second pass's dots (a thread reads back only its own
// elements); second projection with the norm; normalisation.  Pairs of floats per
// access, two of them in flight a thread.  Block partials are float32 pairs; every
// block sums them in the same order, so all take the same values.  Partials:
// part1 = count x grid, part2 = count x grid, part3 = grid pairs.  262k sites, rows
// of 1.6M floats, one to three rows: 40 us on average with four barriers and two
// passes over w more, now 33.5; 160 and 110 us at 1.4M sites.
struct Arnoldi32Args {
    int64_t half;        // length / 2 (the length is even: 6 per site)
    const float2 *basis;  // rows of ld2 float2
    float2 *next;         // row count (written)
    int64_t ld2;
    int count;
    const float2 *v;
    float2 *w;
    double *h, *part1, *part2, *part3;
    unsigned *barrier, *clear;   // clear: the next launch's barrier word, or NULL
    int *status;
};

constexpr int kArnoldiRows = 4;   // rows whose dots a pass keeps in registers

// this thread's pairs of rows k0.. reduced per block into part[k * gridDim.x + blockIdx.x]
__device__ __forceinline__ void store_row_partials(const float hi[kArnoldiRows], const float lo[kArnoldiRows], int k0,
                                                   int count, double *part) {
#pragma unroll
    for (int q = 0; q < kArnoldiRows; ++q)
        if (k0 + q < count) {
            const float2 p = block_pair_sum(hi[q], lo[q]);
            if (threadIdx.x == 0) reinterpret_cast<float2 *>(part)[(k0 + q) * gridDim.x + blockIdx.x] = p;
        }
}

// Column values of a pass from its partials, split into floats, in shared memory.
struct ArnoldiColumn {
    float hi[kMaxArnoldi], lo[kMaxArnoldi];
    double total[kMaxArnoldi];   // both passes' (h may be host memory, which is only written)
};

__device__ __forceinline__ void read_column(const Arnoldi32Args &a, const double *part, bool second,
                                            ArnoldiColumn &col) {
    __syncthreads();
    // a warp a row (one warp for all of them: 5 us a row more at 262k sites)
    for (int k = threadIdx.x >> 5; k < a.count; k += kThreads / 32) {
        const double v = warp_pair_array(reinterpret_cast<const float2 *>(part) + k * gridDim.x, gridDim.x);
        if ((threadIdx.x & 31) == 0) {
            ff_split(v, col.hi[k], col.lo[k]);
            col.total[k] = second ? col.total[k] + v : v;
            if (second && blockIdx.x == 0) a.h[k] = col.total[k];
        }
    }
    __syncthreads();
}

// in - sum_k column_k basis_k at pair e, the projection as float32 pairs
struct Projection {
    float2 ph, pl;
    __device__ __forceinline__ void add(const ArnoldiColumn &col, int k, float2 b) {
        ff_add_product(ph.x, pl.x, col.hi[k], b.x);
        ff_add_product(ph.y, pl.y, col.hi[k], b.y);
        pl.x = fmaf(col.lo[k], b.x, pl.x);
        pl.y = fmaf(col.lo[k], b.y, pl.y);
    }
    __device__ __forceinline__ float2 from(float2 iv) const {
        float dx = iv.x, ex = 0.0f, dy = iv.y, ey = 0.0f;
        ff_two_sum(dx, ex, -ph.x);
        ff_two_sum(dy, ey, -ph.y);
        return make_float2(dx + (ex - pl.x), dy + (ey - pl.y));
    }
};

__global__ void __launch_bounds__(kThreads, 4) arnoldi32_fused_kernel(Arnoldi32Args a) {
    __shared__ ArnoldiColumn col;
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    if (a.clear && tid == 0) *a.clear = 0u;
    // dots of the rows with v
    for (int k0 = 0; k0 < a.count; k0 += kArnoldiRows) {
        float hi[kArnoldiRows] = {}, lo[kArnoldiRows] = {};
        const int kn = a.count - k0;
        for (int64_t e = tid; e < a.half; e += 2 * stride) {
            const int64_t f = e + stride;
            const bool two = f < a.half;
            const float2 x0 = __ldg(a.v + e), x1 = two ? __ldg(a.v + f) : make_float2(0.0f, 0.0f);
            float2 b0[kArnoldiRows], b1[kArnoldiRows];
#pragma unroll
            for (int q = 0; q < kArnoldiRows; ++q)
                if (q < kn) {
                    b0[q] = __ldg(a.basis + (k0 + q) * a.ld2 + e);
                    b1[q] = two ? __ldg(a.basis + (k0 + q) * a.ld2 + f) : make_float2(0.0f, 0.0f);
                }
#pragma unroll
            for (int q = 0; q < kArnoldiRows; ++q)
                if (q < kn) {
                    ff_add_product(hi[q], lo[q], b0[q].x, x0.x);
                    ff_add_product(hi[q], lo[q], b0[q].y, x0.y);
                    ff_add_product(hi[q], lo[q], b1[q].x, x1.x);
                    ff_add_product(hi[q], lo[q], b1[q].y, x1.y);
                }
        }
        store_row_partials(hi, lo, k0, a.count, a.part1);
    }
    if (!grid_barrier(a.barrier, a.status)) return;
    // projection, and the dots of the rows with what it leaves
    read_column(a, a.part1, false, col);
    for (int k0 = 0; k0 < a.count; k0 += kArnoldiRows) {
        float hi[kArnoldiRows] = {}, lo[kArnoldiRows] = {};
        const int kn = a.count - k0;
        for (int64_t e = tid; e < a.half; e += stride) {
            float2 b[kArnoldiRows], w;
#pragma unroll
            for (int q = 0; q < kArnoldiRows; ++q)
                if (q < kn) b[q] = __ldg(a.basis + (k0 + q) * a.ld2 + e);
            if (k0 == 0) {
                const float2 iv = __ldg(a.v + e);
                Projection p{};
#pragma unroll
                for (int q = 0; q < kArnoldiRows; ++q)
                    if (q < kn) p.add(col, q, b[q]);
                for (int k = kArnoldiRows; k < a.count; ++k) p.add(col, k, __ldg(a.basis + k * a.ld2 + e));
                w = p.from(iv);
                a.w[e] = w;
            } else {
                w = a.w[e];
            }
#pragma unroll
            for (int q = 0; q < kArnoldiRows; ++q)
                if (q < kn) {
                    ff_add_product(hi[q], lo[q], b[q].x, w.x);
                    ff_add_product(hi[q], lo[q], b[q].y, w.y);
                }
        }
        store_row_partials(hi, lo, k0, a.count, a.part2);
    }
    if (!grid_barrier(a.barrier, a.status)) return;
    // second projection and the norm of what it leaves
    read_column(a, a.part2, true, col);
    float sh = 0.0f, sl = 0.0f;
    for (int64_t e = tid; e < a.half; e += stride) {
        const float2 iv = a.w[e];
        Projection p{};
#pragma unroll 4
        for (int k = 0; k < a.count; ++k) p.add(col, k, __ldg(a.basis + k * a.ld2 + e));
        const float2 w = p.from(iv);
        a.w[e] = w;
        ff_add_product(sh, sl, w.x, w.x);
        ff_add_product(sh, sl, w.y, w.y);
    }
    const float2 sq = block_pair_sum(sh, sl);
    if (threadIdx.x == 0) reinterpret_cast<float2 *>(a.part3)[blockIdx.x] = sq;
    if (!grid_barrier(a.barrier, a.status)) return;
    const double nrm = sqrt(pair_total(reinterpret_cast<const float2 *>(a.part3), gridDim.x));
    if (blockIdx.x == 0 && threadIdx.x == 0) a.h[a.count] = nrm;
    if (!(nrm >= 1e-14)) return;
    const float inv = (float)(1.0 / nrm);
    for (int64_t e = tid; e < a.half; e += stride) {
        const float2 wv = a.w[e];
        a.next[e] = make_float2(wv.x * inv, wv.y * inv);
    }
}

__global__ void __launch_bounds__(kThreads) scale_to_float_kernel(int64_t len, double alpha, const double *a,
                                                                  float *out) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < len; e += stride)
        out[e] = narrow(alpha * a[e]);
}

}  // namespace dpf

extern "C" {

int64_t dpf_elastic_workspace_doubles(int64_t n_sites) { return 30 * n_sites + 2 * (int64_t)kMaxPcgBlocks; }

}  // extern "C"

int dpf::elastic_pass(const dpf_graph *g, const dpf_stiffness *k, const dpf_tangent *t, const double *mass,
                      const uint8_t *fixed, const double *block, const double *preconditioner, const double *units,
                      const double *vector, double dt, double tolerance, int max_iterations, double *out,
                      int *iterations, double *wrench, double *workspace, unsigned *barrier, unsigned *clear,
                      int *status, ElasticForm form, cudaStream_t st) {
    if (!g || g->n_sites <= 0 || !g->inc_ptr || (g->n_bonds && !g->inc_bond) || !k || !t || !mass || !fixed ||
        !block ||
        !preconditioner || !units || !vector || !out || !iterations || !workspace || !barrier || !status ||
        max_iterations < 1 || (g->n_bonds && (!wrench || !g->edges)))
        return DPF_ERR_ARGUMENT;
    DeviceInfo &info = device_info();
    if (info.sms <= 0 || info.pcg_blocks_per_sm <= 0) return DPF_ERR_CUDA;
    // Few items: one block of 128 an SM, many: two of 256 (us an iteration: 54k
    // bonds 24.6 with one block of 128, 32.7 with four of 256; 254k bonds 58.1 with
    // two of 128, 58.7 with one to four of 256; 1.9M bonds 332 with four of 128,
    // 326 with two of 256).  A grid of more warps than that only waits longer at
    // the barriers.
    const int64_t items = 2 * g->n_sites > g->n_bonds ? 2 * g->n_sites : g->n_bonds;
    const bool few = items <= 512 * (int64_t)info.sms;
    const int threads = few ? 128 : kThreads;
    const int64_t want = blocks_for(items, threads);
    int64_t cap = (int64_t)info.sms * (few ? 1 : info.pcg_blocks_per_sm < 2 ? info.pcg_blocks_per_sm : 2);
    if (cap > kMaxPcgBlocks) cap = kMaxPcgBlocks;
    const int grid = (int)(want < cap ? (want < 1 ? 1 : want) : cap);
    const int64_t n6 = 6 * g->n_sites;
    PcgArgs a{};
    a.n = g->n_sites;
    a.m = g->n_bonds;
    a.ptr = g->inc_ptr;
    a.inc = g->inc_bond;
    a.edges = g->edges;
    a.k = *k;
    a.t = *t;
    a.mass = mass;
    a.block = block;
    a.P = preconditioner;
    a.units = units;
    a.vector = vector;
    a.fixed = fixed;
    a.alpha_op = 0.25 * dt * dt;
    a.tol2 = tolerance * tolerance;
    a.max_it = max_iterations;
    a.form = form;
    a.clear = clear;
    a.out = out;
    a.iterations = iterations;
    a.wrench = wrench;
    a.r = workspace;
    a.u = workspace + n6;
    a.p = workspace + 2 * n6;
    a.s = workspace + 3 * n6;
    a.part_a = workspace + 5 * n6;
    a.part_b = workspace + 5 * n6 + kMaxPcgBlocks;
    a.barrier = barrier;
    a.status = status;
    if (!clear && cudaMemsetAsync(barrier, 0, 2 * sizeof(unsigned), st) != cudaSuccess) return DPF_ERR_CUDA;
    void *args[] = {&a};
    if (cudaLaunchCooperativeKernel((const void *)pcg_kernel, grid, threads, args, 0, st) != cudaSuccess) {
        cudaGetLastError();
        return DPF_ERR_CUDA;
    }
    return DPF_OK;
}

extern "C" {

int dpf_elastic_precondition(const dpf_graph *g, const dpf_stiffness *k, const dpf_tangent *t, const double *mass,
                             const uint8_t *fixed, const double *block, const double *preconditioner,
                             const double *units, const double *vector, double dt, double tolerance,
                             int max_iterations, double *out, int *iterations, double *wrench, double *workspace,
                             unsigned *barrier, int *status, void *stream) {
    return dpf::elastic_pass(g, k, t, mass, fixed, block, preconditioner, units, vector, dt, tolerance, max_iterations,
                             out, iterations, wrench, workspace, barrier, nullptr, status, kElastic,
                             (cudaStream_t)stream);
}

int dpf_arnoldi_cgs2(int64_t length, double *basis, int64_t ld, int j, double *w, double *h, double *partials,
                     void *stream) {
    if (length <= 0 || !basis || !w || !h || !partials || j < 0 || j + 1 >= kMaxArnoldi || ld < length)
        return DPF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    const int grid = reduce_grid(length);
    const int count = j + 1;
    double *pa = partials + kPartialsOffset;
    double *pb = pa + (int64_t)kMaxArnoldi * kMaxReduceBlocks;
    arnoldi_dots<<<grid, kThreads, 0, st>>>(length, basis, ld, count, w, pa);
    arnoldi_update<<<grid, kThreads, 0, st>>>(length, basis, ld, count, w, pa, h, 0, pb, 1);
    arnoldi_update<<<grid, kThreads, 0, st>>>(length, basis, ld, count, w, pb, h, 1, pa, 0);
    arnoldi_normalize<<<grid, kThreads, 0, st>>>(length, basis, ld, j, w, pa, h);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_arnoldi_cgs2_f32(int64_t length, float *basis, int64_t ld, int j, const float *v, float *w, double *h,
                         double *partials, unsigned *barrier, int *status, void *stream) {
    return dpf::arnoldi32_pass(length, basis, ld, j, v, w, h, partials, barrier, nullptr, status,
                               (cudaStream_t)stream);
}

}  // extern "C"

int dpf::arnoldi32_pass(int64_t length, float *basis, int64_t ld, int j, const float *v, float *w, double *h,
                        double *partials, unsigned *barrier, unsigned *clear, int *status, cudaStream_t st) {
    if (length <= 0 || (length & 1) || (ld & 1) || !basis || !v || !w || !h || !partials || !barrier || !status ||
        j < 0 || j + 1 >= kMaxArnoldi || ld < length || (((uintptr_t)basis | (uintptr_t)v | (uintptr_t)w) & 7u))
        return DPF_ERR_ARGUMENT;
    static int per_sm[64] = {0}, sms[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (per_sm[dev & 63] == 0) {
        cudaDeviceGetAttribute(&sms[dev & 63], cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm[dev & 63], arnoldi32_fused_kernel, kThreads, 0);
    }
    int grid = sms[dev & 63] * (per_sm[dev & 63] < 4 ? per_sm[dev & 63] : 4);
    const int64_t need = (length / 2 + kThreads - 1) / kThreads;
    if (grid > need) grid = (int)need;
    if (grid > kMaxReduceBlocks) grid = kMaxReduceBlocks;
    if (grid < 1) return DPF_ERR_CUDA;
    Arnoldi32Args a;
    a.half = length / 2;
    a.basis = reinterpret_cast<const float2 *>(basis);
    a.ld2 = ld / 2;
    a.next = reinterpret_cast<float2 *>(basis + (int64_t)(j + 1) * ld);
    a.count = j + 1;
    a.v = reinterpret_cast<const float2 *>(v);
    a.w = reinterpret_cast<float2 *>(w);
    a.h = h;
    a.part1 = partials + kPartialsOffset;
    a.part2 = a.part1 + (int64_t)kMaxArnoldi * kMaxReduceBlocks;
    a.part3 = a.part2 + (int64_t)(kMaxArnoldi - 1) * kMaxReduceBlocks;
    a.barrier = barrier;
    a.clear = clear;
    a.status = status;
    // a wait that timed out in an earlier launch leaves a partial arrival count
    if (!clear && cudaMemsetAsync(barrier, 0, 2 * sizeof(unsigned), st) != cudaSuccess) {
        cudaGetLastError();
        return DPF_ERR_CUDA;
    }
    void *args[] = {&a};
    if (cudaLaunchCooperativeKernel((const void *)arnoldi32_fused_kernel, grid, kThreads, args, 0, st) !=
        cudaSuccess) {
        cudaGetLastError();
        return DPF_ERR_CUDA;
    }
    return DPF_OK;
}

int dpf::mixed_correction_pass(int64_t n_sites, const float *transformed, const float *products, int count,
                               const double *coefficients, bool add, const double *scaled, const double *units,
                               const uint8_t *fixed, const double *y, double *x, double *res, double *correction,
                               double *candidate, float *y32, double *norm, double *partials, int *status,
                               cudaStream_t st) {
    if (n_sites <= 0 || count < 0 || count > kMaxArnoldi || (count && (!transformed || !products || !coefficients)) ||
        !scaled || !units || !fixed || !y || !x || !res || !correction || !candidate || !y32 || !norm || !partials ||
        !status)
        return DPF_ERR_ARGUMENT;
    CorrectionArgs a{};
    a.len = 6 * n_sites;
    a.z = transformed;
    a.jz = products;
    a.count = count;
    for (int k = 0; k < count; ++k) a.coef.c[k] = coefficients[k];
    a.add = add ? 1 : 0;
    a.scaled = scaled;
    a.units = units;
    a.fixed = fixed;
    a.y = y;
    a.x = x;
    a.res = res;
    a.correction = correction;
    a.candidate = candidate;
    a.y32 = y32;
    a.norm = norm;
    a.partials = partials;
    a.status = status;
    correction_kernel<<<wave_grid(a.len, kNormResident), kThreads, 0, st>>>(a);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

extern "C" {

int dpf_combine_rows_f32(int64_t length, const float *rows, int64_t ld, int count, const double *coefficients,
                         double *x, void *stream) {
    if (length <= 0 || !rows || !x || count < 0 || count > kMaxArnoldi || (count && !coefficients))
        return DPF_ERR_ARGUMENT;
    Coefficients c{};
    for (int k = 0; k < count; ++k) c.c[k] = coefficients[k];
    combine32_kernel<<<reduce_grid(length), kThreads, 0, (cudaStream_t)stream>>>(length, rows, ld, count, c, x);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_scale_to_float(int64_t length, double alpha, const double *a, float *out, void *stream) {
    if (length <= 0 || !a || !out) return DPF_ERR_ARGUMENT;
    scale_to_float_kernel<<<reduce_grid(length), kThreads, 0, (cudaStream_t)stream>>>(length, alpha, a, out);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_combine_rows(int64_t length, const double *rows, int64_t ld, int count, const double *coefficients, double *x,
                     void *stream) {
    if (length <= 0 || !rows || !x || count < 0 || count > kMaxArnoldi || (count && !coefficients))
        return DPF_ERR_ARGUMENT;
    Coefficients c{};
    for (int k = 0; k < count; ++k) c.c[k] = coefficients[k];
    combine_rows_kernel<<<reduce_grid(length), kThreads, 0, (cudaStream_t)stream>>>(length, rows, ld, count, c, x);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_dot_norm(int64_t length, const double *a, const double *b, double *result, double *partials, void *stream) {
    if (length <= 0 || !a || !result || !partials) return DPF_ERR_ARGUMENT;
    dot_norm_kernel<<<wave_grid(length, kNormResident), kThreads, 0, (cudaStream_t)stream>>>(length, a, b, result, partials);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_axpby(int64_t length, double alpha, const double *a, double beta, const double *b, double *out,
              void *stream) {
    if (length <= 0 || !a || !b || !out) return DPF_ERR_ARGUMENT;
    axpby_kernel<<<reduce_grid(length), kThreads, 0, (cudaStream_t)stream>>>(length, alpha, a, beta, b, out);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_scale_residual(int64_t n_sites, const double *preconditioner, const double *units, const double *residual,
                       double *scaled, double *norms, double *partials, void *stream) {
    return dpf::scale_residual64_pass(n_sites, preconditioner, units, residual, scaled, norms, partials, Report(),
                                      (cudaStream_t)stream);
}

}  // extern "C"

int dpf::scale_residual64_pass(int64_t n_sites, const double *preconditioner, const double *units,
                               const double *residual, double *scaled, double *norms, double *partials,
                               const Report &report, cudaStream_t st) {
    if (n_sites <= 0 || !preconditioner || !units || !residual || (norms && !partials)) return DPF_ERR_ARGUMENT;
    const int threads = reduce_threads(2 * n_sites);
    const int64_t blocks = blocks_for(2 * n_sites, threads);
    scale_kernel<<<(int)(blocks < kMaxReduceBlocks ? blocks : kMaxReduceBlocks), threads, 0, st>>>(
        n_sites, preconditioner, units, residual, scaled, norms, partials, report);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

extern "C" {

int dpf_accept_step(int64_t n_sites, const double *y, double dt, double *v, double *rotation, void *stream) {
    if (n_sites <= 0 || !y || !v || !rotation) return DPF_ERR_ARGUMENT;
    accept_kernel<<<blocks_for(n_sites, kThreads), kThreads, 0, (cudaStream_t)stream>>>(n_sites, y, dt, v, rotation);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_energy(const dpf_graph *g, const dpf_stiffness *k, const dpf_history *h, const double *mass, const double *v,
               double *energy, double *partials, void *stream) {
    if (!g || g->n_sites <= 0 || !k || !h || !mass || !v || !energy || !partials) return DPF_ERR_ARGUMENT;
    const int64_t work = g->n_bonds > 6 * g->n_sites ? g->n_bonds : 6 * g->n_sites;
    energy_kernel<<<reduce_grid(work), kThreads, 0, (cudaStream_t)stream>>>(g->n_bonds, g->n_sites, *k, *h, mass, v,
                                                                            energy, partials);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_rhs_scale(int64_t n_sites, const double *mass, const double *v, const double *external, const double *loads,
                  const uint8_t *fixed, double dt, double *out, double *partials, void *stream) {
    if (n_sites <= 0 || !mass || !v || !external || !loads || !fixed || !out || !partials) return DPF_ERR_ARGUMENT;
    rhs_scale_kernel<<<reduce_grid(6 * n_sites), kThreads, 0, (cudaStream_t)stream>>>(
        n_sites, mass, v, external, loads, fixed, dt, 0.5 * dt * dt, out, partials);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_masked_scale(int64_t n_sites, const double *a, const double *units, const uint8_t *fixed, double *out,
                     void *stream) {
    if (n_sites <= 0 || !a || !units || !fixed || !out) return DPF_ERR_ARGUMENT;
    masked_scale_kernel<<<reduce_grid(6 * n_sites), kThreads, 0, (cudaStream_t)stream>>>(n_sites, a, units, fixed,
                                                                                         out);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

}  // extern "C"
