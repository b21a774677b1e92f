// Shared device code for the bonded-DEM kernels: 3-vector math, the contact
// transport of the rate law, block reductions and a time-limited grid barrier.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "dpf_gb300.h"

namespace dpf {

constexpr int kThreads = 256;
// cos(0.25) rounded to double, the threshold of the reference transport guard.
constexpr double kCosQuarter = 0.9689124217106447;
// Grid barriers give up after this many nanoseconds and report
// DPF_ERR_BARRIER_TIMEOUT instead of waiting forever.
constexpr unsigned long long kBarrierTimeoutNs = 1000000000ull;

struct d3 {
    double x, y, z;
};

__device__ __forceinline__ d3 mk(double a, double b, double c) { return {a, b, c}; }
__device__ __forceinline__ d3 operator+(d3 a, d3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ d3 operator-(d3 a, d3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ d3 operator-(d3 a) { return {-a.x, -a.y, -a.z}; }
__device__ __forceinline__ d3 operator*(double s, d3 a) { return {s * a.x, s * a.y, s * a.z}; }
// One reciprocal and three products: a float64 division costs many times a
// multiply on GB300's float64 pipe.
__device__ __forceinline__ d3 operator/(d3 a, double s) {
    const double inv = 1.0 / s;
    return {a.x * inv, a.y * inv, a.z * inv};
}
__device__ __forceinline__ double dot(d3 a, d3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ d3 cross(d3 a, d3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ double norm(d3 a) { return sqrt(dot(a, a)); }
// acc + a x b and acc - a x b in six fused multiply-adds (the sum of a product
// and a vector written out costs nine operations).
__device__ __forceinline__ d3 cross_add(d3 acc, d3 a, d3 b) {
    return {fma(a.y, b.z, fma(-a.z, b.y, acc.x)), fma(a.z, b.x, fma(-a.x, b.z, acc.y)),
            fma(a.x, b.y, fma(-a.y, b.x, acc.z))};
}
__device__ __forceinline__ d3 cross_sub(d3 acc, d3 a, d3 b) { return cross_add(acc, b, a); }
__device__ __forceinline__ double dot_add(double acc, d3 a, d3 b) {
    return fma(a.x, b.x, fma(a.y, b.y, fma(a.z, b.z, acc)));
}
__device__ __forceinline__ d3 axpy(double s, d3 a, d3 b) {
    return {fma(s, a.x, b.x), fma(s, a.y, b.y), fma(s, a.z, b.z)};
}

__device__ __forceinline__ d3 ld3(const double *p) { return {p[0], p[1], p[2]}; }
__device__ __forceinline__ d3 ld3(const double *p, int64_t i) { return ld3(p + 3 * i); }
__device__ __forceinline__ void st3(double *p, d3 v) { p[0] = v.x; p[1] = v.y; p[2] = v.z; }
__device__ __forceinline__ void st3(double *p, int64_t i, d3 v) { st3(p + 3 * i, v); }

__device__ __forceinline__ void edge(const int64_t *edges, int64_t b, int64_t &i, int64_t &j) {
    const longlong2 e = reinterpret_cast<const longlong2 *>(edges)[b];
    i = e.x;
    j = e.y;
}

// Rotation that carries vectors from a bond frame with normal n0 to one with
// normal n1 (shortest arc) and then spins them about n1 by spin . bisector:
// the `transport` of experiments/bonded_dem_finite_gpu.py:22-32.
struct Transport {
    d3 k, n1;
    double inv1pc, c, s;
};

__device__ __forceinline__ Transport make_transport(d3 n0, d3 n1, d3 spin, int &flags) {
    Transport t;
    t.k = cross(n0, n1);
    const double cosine = fmin(fmax(dot(n0, n1), -1.0), 1.0);
    if (cosine < kCosQuarter) flags |= DPF_ERR_NORMAL_TURN;
    t.inv1pc = 1.0 / (1.0 + cosine);
    d3 b = n0 + n1;
    b = b / fmax(norm(b), 1e-12);
    sincos(dot(spin, b), &t.s, &t.c);
    t.n1 = n1;
    return t;
}

__device__ __forceinline__ d3 apply(const Transport &t, d3 v) {
    const d3 kv = cross(t.k, v);
    d3 out = v + kv;
    out = out + t.inv1pc * cross(t.k, kv);
    return t.c * out + t.s * cross(t.n1, out) + ((1.0 - t.c) * dot(t.n1, out)) * t.n1;
}

// ---- the same transport for unit normals, with few float64 operations --------
//
// The float64 bond passes are bound by the float64 pipe (two lanes per SM and
// clock: about 3.1 us per operation and bond at 2M bonds, against 2.3 us to
// read eight bytes per bond), so what they gain is operations left out.  With
// |n0| = |n1| = 1 the shortest-arc rotation is the unit quaternion
// r (1 + c, n0 x n1), r = 1/sqrt(2 + 2 c), c = n0 . n1; followed by the spin
// about n1 by the angle r spin.(n0 + n1) it is
//   w = r cos(h) (1 + c),  v = r (cos(h) n0 x n1 + sin(h) (n0 + n1)),
// h half that angle, because n1 x (n0 x n1) = n0 - c n1.  One reciprocal root
// and two short series instead of a root, two divisions and a sincos, and 15
// operations a rotated vector instead of 37.

struct Turn {
    double w;
    d3 v, v2;        // vector part and twice it
    d3 sum;          // n0 + n1
    double r, half, sh, ch;
};

// sin h and cos h: Maclaurin series for |h| < 0.25 (relative truncation below
// 1e-17 and 2e-17 there; the rotation guard keeps a step's |h| below 0.125).
__device__ __forceinline__ void sincos_small(double h, double &s, double &c) {
    if (fabs(h) < 0.25) {
        const double q = h * h;
        double a = -1.0 / 39916800.0;               // 1/11!
        a = fma(a, q, 1.0 / 362880.0);              // 1/9!
        a = fma(a, q, -1.0 / 5040.0);               // 1/7!
        a = fma(a, q, 1.0 / 120.0);                 // 1/5!
        a = fma(a, q, -1.0 / 6.0);                  // 1/3!
        s = fma(a * q, h, h);
        double b = 1.0 / 479001600.0;               // 1/12!
        b = fma(b, q, -1.0 / 3628800.0);            // 1/10!
        b = fma(b, q, 1.0 / 40320.0);               // 1/8!
        b = fma(b, q, -1.0 / 720.0);                // 1/6!
        b = fma(b, q, 1.0 / 24.0);                  // 1/4!
        b = fma(b, q, -0.5);
        c = fma(b, q, 1.0);
    } else {
        sincos(h, &s, &c);
    }
}

// A normal that geometry() formed has |n|^2 = 1 within a few 1e-16.
__device__ __forceinline__ bool is_unit(d3 n) { return fabs(dot(n, n) - 1.0) < 1e-12; }

// All three numbers are +0 or -0 (integer tests: the float64 pipe is the scarce one).
__device__ __forceinline__ bool is_zero(d3 a) {
    return ((__double_as_longlong(a.x) | __double_as_longlong(a.y) | __double_as_longlong(a.z)) << 1) == 0;
}

__device__ __forceinline__ Turn make_turn(d3 n0, d3 n1, d3 spin, int &flags) {
    Turn t;
    const double c = dot(n0, n1);
    if (!(c >= kCosQuarter)) flags |= DPF_ERR_NORMAL_TURN;
    t.sum = n0 + n1;
    t.r = rsqrt(2.0 + 2.0 * c);
    t.half = 0.5 * t.r * dot(spin, t.sum);
    sincos_small(t.half, t.sh, t.ch);
    const double rc = t.r * t.ch, rs = t.r * t.sh;
    t.w = rc + rc * c;
    t.v = axpy(rs, t.sum, rc * cross(n0, n1));
    t.v2 = t.v + t.v;
    return t;
}

__device__ __forceinline__ d3 apply(const Turn &t, d3 a) {
    const d3 x = cross(t.v2, a);
    return cross_add(axpy(t.w, x, a), t.v, x);
}

// Angular velocity of the transport when its normal moves by dn and its spin
// by dspin: d(R a) = omega x (R a) for every vector a.  The shortest-arc
// rotation is a half turn about the committed normal followed by one about
// the middle of the two normals, so it turns with (n0 + n) x dn / (1 + c);
// the spin by the angle th about n adds th' n + sin(th) dn +
// (1 - cos(th)) n x dn and rotates the former.
__device__ __forceinline__ d3 turn_rate(const Turn &t, d3 n, d3 dn, d3 spin, d3 dspin) {
    const double sine = 2.0 * t.sh * t.ch, versine = 2.0 * t.sh * t.sh;
    const d3 arc = (2.0 * t.r * t.r) * cross(t.sum, dn);
    const double dth = t.r * dot_add(dot_add(-(2.0 * t.half * t.r) * dot(t.sum, dn), spin, dn), dspin, t.sum);
    const d3 side = axpy(sine, arc, versine * cross_add(dn, n, arc));
    return cross_add(axpy(dth, n, axpy(sine, dn, arc)), n, side);
}

// Normal turns more than 0.25 rad (or is not a number) from unit n to the
// direction of d: n . d >= cos(0.25) |d| without forming |d|.
__device__ __forceinline__ bool turned(d3 n, d3 d, double d2) {
    const double c = dot(n, d);
    return !(c > 0.0 && c * c >= (kCosQuarter * kCosQuarter) * d2);
}

// Wrench [F_i, T_i, T_j] of the frozen tangent on one bond (F_j = -F_i):
// du = u_j - u_i + w_j x r_j - w_i x r_i, dw = w_j - w_i,
// f = ks du + (kn - ks)(du.n) n, m likewise of dw; F_i = -f,
// T_i = -(r_i x f) - m, T_j = r_j x f + m.  52 float64 operations.
struct Wrench {
    d3 f, ti, tj;
};

__device__ __forceinline__ Wrench stiffness_wrench(d3 n, d3 ri, d3 rj, double kn, double ks, double kb, double kt,
                                                   const double *qi, const double *qj) {
    const d3 wi = ld3(qi + 3), wj = ld3(qj + 3);
    const d3 du = cross_sub(cross_add(ld3(qj) - ld3(qi), wj, rj), wi, ri);
    const d3 dw = wj - wi;
    const d3 f = axpy((kn - ks) * dot(du, n), n, ks * du);
    const d3 m = axpy((kt - kb) * dot(dw, n), n, kb * dw);
    return {-f, cross_add(-m, f, ri), cross_add(m, rj, f)};
}

// A warp's 32 consecutive wrenches (bonds first, first + 1, ..; `count` of
// them exist) to memory through the warp's 288 doubles of shared memory, in
// consecutive addresses: stored by the lanes one number at a time, at a stride
// of 72 bytes, every store instruction touched 32 sectors of L2.
__device__ __forceinline__ void store_wrenches(double *wrench, int64_t first, int count, const Wrench &w,
                                               double *stage) {
    const int lane = threadIdx.x & 31;
    double *p = stage + 9 * lane;
    st3(p, w.f);
    st3(p + 3, w.ti);
    st3(p + 6, w.tj);
    __syncwarp();
    double *out = wrench + 9 * first;
#pragma unroll
    for (int k = 0; k < 9; ++k)
        if (32 * k + lane < 9 * count) out[32 * k + lane] = stage[32 * k + lane];
    __syncwarp();
}

// Sum over the incidences of site s of the bond wrenches [F, T_i, T_j]
// (nine doubles per bond; the j end receives (-F, T_j)), in incidence order.
__device__ __forceinline__ void gather_wrench(const int32_t *__restrict__ ptr, const int32_t *__restrict__ inc,
                                              const double *__restrict__ w, int64_t s, double acc[6]) {
#pragma unroll
    for (int c = 0; c < 6; ++c) acc[c] = 0.0;
    const int e1 = ptr[s + 1];
    for (int e = ptr[s]; e < e1; ++e) {
        const int v = inc[e];
        if (v >= 0) {
            const double *p = w + 9 * (int64_t)v;
#pragma unroll
            for (int c = 0; c < 6; ++c) acc[c] += p[c];
        } else {
            const double *p = w + 9 * (int64_t)(~v);
            acc[0] -= p[0];
            acc[1] -= p[1];
            acc[2] -= p[2];
            acc[3] += p[6];
            acc[4] += p[7];
            acc[5] += p[8];
        }
    }
}

// Half of gather_wrench: the force (part 0) or the torque (part 1) of site s,
// for site passes that give a site two neighbouring lanes.  The same sums in
// the same order; the sign and the place of the end's three numbers are
// chosen without a branch so that the loads of several incidences are in
// flight together, and the site's other work is split by rows of its 6x6
// block.  Reads `w` with plain loads when the caller's launch writes it too.
template <bool kConst = true>
__device__ __forceinline__ d3 gather_half(const int32_t *__restrict__ ptr, const int32_t *__restrict__ inc,
                                          const double *w, int64_t s, int part) {
    d3 acc = mk(0.0, 0.0, 0.0);
    const int e1 = ptr[s + 1];
#pragma unroll 4
    for (int e = ptr[s]; e < e1; ++e) {
        const int v = inc[e];
        const int j = v >> 31;               // 0: i end, -1: j end
        const double *p = w + 9 * (int64_t)(v ^ j) + (part ? 3 - 3 * j : 0);
        const unsigned long long flip = part ? 0ull : (unsigned long long)((unsigned)j & 0x80000000u) << 32;
        const double x = kConst ? __ldg(p) : p[0], y = kConst ? __ldg(p + 1) : p[1], z = kConst ? __ldg(p + 2) : p[2];
        acc.x += __longlong_as_double(__double_as_longlong(x) ^ (long long)flip);
        acc.y += __longlong_as_double(__double_as_longlong(y) ^ (long long)flip);
        acc.z += __longlong_as_double(__double_as_longlong(z) ^ (long long)flip);
    }
    return acc;
}

// The other lane's half of a site vector (lanes 2k and 2k + 1 share a site;
// both call it), and this lane's three rows of a 6x6 block times the vector
// whose halves are `own` and `other`.
__device__ __forceinline__ d3 other_half(d3 a) {
    return mk(__shfl_xor_sync(0xffffffffu, a.x, 1), __shfl_xor_sync(0xffffffffu, a.y, 1),
              __shfl_xor_sync(0xffffffffu, a.z, 1));
}

__device__ __forceinline__ d3 half_rows(const double *__restrict__ P, int part, d3 own, d3 other) {
    const d3 lo = part ? other : own, hi = part ? own : other;
    double r[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double *row = P + 18 * part + 6 * c;
        double v = row[0] * lo.x;
        v += row[1] * lo.y;
        v += row[2] * lo.z;
        v += row[3] * hi.x;
        v += row[4] * hi.y;
        v += row[5] * hi.z;
        r[c] = v;
    }
    return mk(r[0], r[1], r[2]);
}

// a / u for one half of a site's units: [r, r, r] or [1, 1, 1] in every solver
// of this library, so one division instead of three, or none.
__device__ __forceinline__ d3 over_units(d3 a, d3 u) {
    if (u.x == u.y && u.x == u.z) return u.x == 1.0 ? a : (1.0 / u.x) * a;
    return mk(a.x / u.x, a.y / u.y, a.z / u.z);
}

// Inverse of a symmetric positive definite 6x6 matrix via Cholesky
// (A = L L^T, A^-1 = L^-T L^-1), fully unrolled into registers: every loop
// has a constant trip count so all indices fold.  L's diagonal is kept as
// its reciprocal.
__device__ __forceinline__ void spd_inverse6(const double A[36], double P[36]) {
    double L[36];
#pragma unroll
    for (int c = 0; c < 36; ++c) L[c] = 0.0;
#pragma unroll
    for (int jj = 0; jj < 6; ++jj) {
        double s = A[6 * jj + jj];
#pragma unroll
        for (int kk = 0; kk < 6; ++kk)
            if (kk < jj) s -= L[6 * jj + kk] * L[6 * jj + kk];
        // only the reciprocal of the diagonal is used: one reciprocal root
        // instead of a root and two divisions
        const double inv = rsqrt(s);
        L[6 * jj + jj] = inv;
#pragma unroll
        for (int ii = 0; ii < 6; ++ii) {
            if (ii > jj) {
                double v = A[6 * ii + jj];
#pragma unroll
                for (int kk = 0; kk < 6; ++kk)
                    if (kk < jj) v -= L[6 * ii + kk] * L[6 * jj + kk];
                L[6 * ii + jj] = v * inv;
            }
        }
    }
    double W[36];  // W = L^-1 (lower triangular)
#pragma unroll
    for (int c = 0; c < 36; ++c) W[c] = 0.0;
#pragma unroll
    for (int ii = 0; ii < 6; ++ii) {
        W[6 * ii + ii] = L[6 * ii + ii];
#pragma unroll
        for (int jj = 0; jj < 6; ++jj) {
            if (jj < ii) {
                double v = 0.0;
#pragma unroll
                for (int kk = 0; kk < 6; ++kk)
                    if (kk >= jj && kk < ii) v += L[6 * ii + kk] * W[6 * kk + jj];
                W[6 * ii + jj] = -v * W[6 * ii + ii];
            }
        }
    }
#pragma unroll
    for (int ii = 0; ii < 6; ++ii)
#pragma unroll
        for (int jj = 0; jj < 6; ++jj) {
            if (jj <= ii) {
                double v = 0.0;
#pragma unroll
                for (int kk = 0; kk < 6; ++kk)
                    if (kk >= ii) v += W[6 * kk + ii] * W[6 * kk + jj];
                P[6 * ii + jj] = v;
                P[6 * jj + ii] = v;
            }
        }
}

// The midpoint step's end velocity 2 y / dt - v (bonded_dem_newton.py:150).  Every kernel
// that accepts a step takes it from here: a step committed again from its increment gives
// the bits of the first time.
__device__ __forceinline__ double end_velocity(double two_over_dt, double y, double v) {
    return fma(two_over_dt, y, -v);
}
__device__ __forceinline__ d3 end_velocity(double two_over_dt, d3 y, d3 v) {
    return {end_velocity(two_over_dt, y.x, v.x), end_velocity(two_over_dt, y.y, v.y),
            end_velocity(two_over_dt, y.z, v.z)};
}

// out = exp([w]x) R of one body (bonded_dem_finite_gpu.py:35-43); out may be R.
__device__ __forceinline__ void rotate_site(d3 w, const double *R, double *out) {
    // Rodrigues coefficients A = sin(a)/a and B = (1 - cos a)/a^2 of a = |w|.
    // Both are even in a: for a^2 < 1/4 (every step the rotation guard lets
    // through has a <= 0.25) their Maclaurin series in a^2, 8 terms each,
    // are exact to a few 1e-17 and need no float64 transcendental, which is
    // slow on this part.  Larger angles take the closed form.
    const double theta = w.x * w.x + w.y * w.y + w.z * w.z;
    double A, B;
    if (theta < 0.25) {
        // Horner in theta: A = sum (-theta)^k/(2k+1)!, B = sum (-theta)^k/(2k+2)!, k = 0..7
        A = 1.0 / 1307674368000.0;                 // 1/15!
        A = fma(-theta, A, 1.0 / 6227020800.0);    // 1/13!
        A = fma(-theta, A, 1.0 / 39916800.0);      // 1/11!
        A = fma(-theta, A, 1.0 / 362880.0);        // 1/9!
        A = fma(-theta, A, 1.0 / 5040.0);          // 1/7!
        A = fma(-theta, A, 1.0 / 120.0);           // 1/5!
        A = fma(-theta, A, 1.0 / 6.0);             // 1/3!
        A = fma(-theta, A, 1.0);
        B = 1.0 / 20922789888000.0;                // 1/16!
        B = fma(-theta, B, 1.0 / 87178291200.0);   // 1/14!
        B = fma(-theta, B, 1.0 / 479001600.0);     // 1/12!
        B = fma(-theta, B, 1.0 / 3628800.0);       // 1/10!
        B = fma(-theta, B, 1.0 / 40320.0);         // 1/8!
        B = fma(-theta, B, 1.0 / 720.0);           // 1/6!
        B = fma(-theta, B, 1.0 / 24.0);            // 1/4!
        B = fma(-theta, B, 0.5);
    } else {
        const double angle = sqrt(theta);
        double sh, ch;
        sincos(0.5 * angle, &sh, &ch);
        A = sin(angle) / angle;
        const double q = sh / (0.5 * angle);
        B = 0.5 * q * q;
    }
    const double S[9] = {0.0, -w.z, w.y, w.z, 0.0, -w.x, -w.y, w.x, 0.0};
    double E[9];
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const double ss = S[3 * p] * S[q] + S[3 * p + 1] * S[3 + q] + S[3 * p + 2] * S[6 + q];
            E[3 * p + q] = (p == q ? 1.0 : 0.0) + A * S[3 * p + q] + B * ss;
        }
    double Rn[9];
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int q = 0; q < 3; ++q) Rn[3 * p + q] = E[3 * p] * R[q] + E[3 * p + 1] * R[3 + q] + E[3 * p + 2] * R[6 + q];
#pragma unroll
    for (int c = 0; c < 9; ++c) out[c] = Rn[c];
}

// Threads a block for `work` independent items of a float64-bound kernel: the
// largest of 128, 64 and 32 that still gives every SM four blocks (the float64
// pipe belongs to the SM, so a few items packed into few blocks leave most
// pipes idle and an uneven last wave costs whole blocks), else 32.  Against blocks
// of 128 throughout: 3% of a float64 step at 512 sites / 3k bonds (40 us), 3% of the
// adjoint's passes at 8k sites.
constexpr int kSMs = 152;
inline int spread_threads(int64_t work) {
    for (int t = 128; t > 32; t /= 2)
        if (work >= (int64_t)t * 4 * kSMs) return t;
    return 32;
}

// The same for passes that end in a reduction over their blocks: more blocks
// than SMs cost more in the reduction than they gain (37k sites: residual pass
// 25 us with 286 blocks, 35 us with 571).
inline int reduce_threads(int64_t work) {
    return work >= (int64_t)kThreads * kSMs ? kThreads : spread_threads(work);
}

// Blocks of a grid-stride pass: no more than are resident at once, `resident` of
// kThreads threads an SM (the kernel's launch bounds).  With 1024 blocks a kernel of
// six blocks an SM ran a second wave of 112 blocks, nearly empty and as long as the
// first (residual pass of 262k sites 83 us, now 64).
inline int wave_grid(int64_t work, int resident, int threads = kThreads) {
    const int64_t g = (work + threads - 1) / threads, cap = (int64_t)kSMs * resident * kThreads / threads;
    return (int)(g < 1 ? 1 : g < cap ? g : cap);
}

// ---- reductions -----------------------------------------------------------

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Block-wide sum (all threads get the result).  Fixed order: deterministic.
// The threads' numbers go to shared memory and one warp adds them: 12 float64
// warp instructions a block of 256 where a shuffle tree in every warp takes 45
// (each of them 16 cycles of the SM's float64 pipe, and the PCGs sum twice an
// iteration).
__device__ __forceinline__ double block_sum(double v) {
    __shared__ double buf[kThreads + 1];
    __syncthreads();
    if (blockDim.x <= kThreads) {
        buf[threadIdx.x] = v;
    } else {                       // larger blocks: their warps' sums
        v = warp_sum(v);
        if ((threadIdx.x & 31) == 0) buf[threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int count = blockDim.x <= kThreads ? (int)blockDim.x : (int)(blockDim.x + 31) >> 5;
        double s = 0.0, t = 0.0;
        for (int k = threadIdx.x; k < count; k += 64) {
            s += buf[k];
            if (k + 32 < count) t += buf[k + 32];
        }
        s = warp_sum(s + t);
        if (threadIdx.x == 0) buf[kThreads] = s;
    }
    __syncthreads();
    return buf[kThreads];
}

__device__ __forceinline__ double block_max(double v) {
    __shared__ double buf[kThreads + 1];
    __syncthreads();
    if (blockDim.x <= kThreads) {
        buf[threadIdx.x] = v;
    } else {
        v = warp_max(v);
        if ((threadIdx.x & 31) == 0) buf[threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int count = blockDim.x <= kThreads ? (int)blockDim.x : (int)(blockDim.x + 31) >> 5;
        double m = -INFINITY;
        for (int k = threadIdx.x; k < count; k += 32) m = fmax(m, buf[k]);
        m = warp_max(m);
        if (threadIdx.x == 0) buf[kThreads] = m;
    }
    __syncthreads();
    return buf[kThreads];
}

// K reductions over the block's threads (at most kThreads), number k a maximum where
// bit k of kMaxMask is set; every thread gets the totals.  A warp takes an array, as
// block_sum does for one, so three cost little more than one (a float64 instruction
// holds its scheduler for 64 cycles: one after the other they took 1.1 us a block).
template <int K, unsigned kMaxMask>
__device__ __forceinline__ void block_reduce(double (&v)[K]) {
    __shared__ double buf[K][kThreads];
    __shared__ double total[K];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) buf[k][threadIdx.x] = v[k];
    __syncthreads();
    const int warps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if ((int)(threadIdx.x >> 5) != k % warps) continue;
        const bool most = ((kMaxMask >> k) & 1u) != 0;
        double s = most ? -INFINITY : 0.0, t = s;
        for (int e = threadIdx.x & 31; e < (int)blockDim.x; e += 64) {
            s = most ? fmax(s, buf[k][e]) : s + buf[k][e];
            if (e + 32 < (int)blockDim.x) t = most ? fmax(t, buf[k][e + 32]) : t + buf[k][e + 32];
        }
        s = most ? warp_max(fmax(s, t)) : warp_sum(s + t);
        if ((threadIdx.x & 31) == 0) total[k] = s;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = total[k];
}

// Sum or maximum of `count` partials by one warp, valid in every lane.  A lane has
// 16 loads in flight (one to four at a time, 1024 partials cost a last block 8 to 32
// round trips to L2: the norms of 262k sites 32.5 us, now 28.6); the sums go through
// four accumulators in a fixed order.
__device__ __forceinline__ double warp_array(const double *p, int count, int stride, bool most) {
    const int lane = threadIdx.x & 31;
    const double none = most ? -INFINITY : 0.0;
    double s[4] = {none, none, none, none};
    for (int base = 0; base < count; base += 512) {
        double v[16];
#pragma unroll
        for (int c = 0; c < 16; ++c) {
            const int k = base + 32 * c + lane;
            v[c] = k < count ? p[(int64_t)k * stride] : none;
        }
#pragma unroll
        for (int c = 0; c < 16; ++c)
            if (base + 32 * c < count) s[c & 3] = most ? fmax(s[c & 3], v[c]) : s[c & 3] + v[c];
    }
    return most ? warp_max(fmax(fmax(s[0], s[1]), fmax(s[2], s[3]))) : warp_sum((s[0] + s[1]) + (s[2] + s[3]));
}

// The K interleaved partial arrays p[k + K b] reduced over b, array k a maximum where
// bit k of kMaxMask is set; a warp an array.  Every thread gets the totals.
template <int K, unsigned kMaxMask>
__device__ __forceinline__ void block_arrays(const double *p, int count, double (&out)[K]) {
    __shared__ double total[K];
    __syncthreads();
    const int warps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k)
        if ((int)(threadIdx.x >> 5) == k % warps) {
            const double v = warp_array(p + k, count, K, ((kMaxMask >> k) & 1u) != 0);
            if ((threadIdx.x & 31) == 0) total[k] = v;
        }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) out[k] = total[k];
}

// Sum of `count` values spaced `stride` apart, in a fixed order (every block that
// calls this with the same data gets the bit-identical result); one warp adds, the
// others wait.  For the few hundred partials of a grid barrier.
__device__ __forceinline__ double block_sum_array(const double *p, int count, int stride = 1) {
    __shared__ double total;
    __syncthreads();
    if (threadIdx.x < 32) {
        double s[4] = {0.0, 0.0, 0.0, 0.0};
        for (int k = threadIdx.x; k < count; k += 128)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (k + 32 * c < count) s[c] += p[(int64_t)(k + 32 * c) * stride];
        const double v = warp_sum((s[0] + s[1]) + (s[2] + s[3]));
        if (threadIdx.x == 0) total = v;
    }
    __syncthreads();
    return total;
}

__device__ __forceinline__ double block_max_array(const double *p, int count, int stride = 1) {
    __shared__ double total;
    __syncthreads();
    if (threadIdx.x < 32) {
        const double m = warp_array(p, count, stride, true);
        if (threadIdx.x == 0) total = m;
    }
    __syncthreads();
    return total;
}

// ---- conversions between float32 and float64 in integer arithmetic ------------
// The conversion instructions run on the float64 pipe, which takes a warp's
// instruction in 16 cycles; re-biasing the exponent and moving the fraction are a
// handful of integer instructions.  Same results as the casts: what is neither zero
// nor normal in both formats takes the cast.

__device__ __forceinline__ double widen(float f) {
    const unsigned u = __float_as_uint(f), t = u & 0x7fffffffu;
    if (t != 0u && t - 0x00800000u >= 0x7f000000u) return (double)f;  // subnormal, infinite, not a number
    const unsigned hi = (u & 0x80000000u) | (t ? (t >> 3) + 0x38000000u : 0u);
    return __hiloint2double((int)hi, (int)(u << 29));
}

// round to nearest, ties to even
__device__ __forceinline__ float narrow(double d) {
    const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d), t = hi & 0x7fffffffu;
    if ((t | lo) != 0u && t - 0x38100000u >= 0x0fe00000u) return (float)d;  // outside float32's normal range
    const unsigned m = ((t - 0x38000000u) << 3) | (lo >> 29);
    const unsigned up = ((lo & 0x1fffffffu) + 0x0fffffffu + (m & 1u)) >> 29;
    return __uint_as_float((hi & 0x80000000u) | ((t | lo) ? m + up : 0u));
}

// ---- sums as float32 pairs ---------------------------------------------------
// A float32 pair (hi, lo) carries a sum to about 48 bits with float32
// arithmetic only (TwoSum); float64 arithmetic is scarce on this part, and a
// block reduction of doubles costs every thread a float64 add per shuffle
// level.  TwoSum's error term is exact whatever the order of its operands,
// so an xor-shuffle tree leaves the same pair in every lane.

__device__ __forceinline__ void pair_add(float &hi, float &lo, float h, float l) {
    const float t = hi + h;
    const float hp = t - hi;
    lo += ((hi - (t - hp)) + (h - hp)) + l;
    hi = t;
}

__device__ __forceinline__ void warp_pair_sum(float &hi, float &lo) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float h = __shfl_xor_sync(0xffffffffu, hi, o), l = __shfl_xor_sync(0xffffffffu, lo, o);
        pair_add(hi, lo, h, l);
    }
}

// Block sum of per-thread pairs; every thread gets the total pair.
__device__ __forceinline__ float2 block_pair_sum(float hi, float lo) {
    __shared__ float2 buf[32];
    __shared__ float2 total;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    warp_pair_sum(hi, lo);
    __syncthreads();
    if (lane == 0) buf[warp] = make_float2(hi, lo);
    __syncthreads();
    if (warp == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        float h = lane < nw ? buf[lane].x : 0.0f, l = lane < nw ? buf[lane].y : 0.0f;
        warp_pair_sum(h, l);
        if (lane == 0) total = make_float2(h, l);
    }
    __syncthreads();
    return total;
}

__device__ __forceinline__ float block_max_float(float v) {
    __shared__ float buf[32];
    __shared__ float total;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if (lane == 0) buf[warp] = v;
    __syncthreads();
    if (warp == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        float m = lane < nw ? buf[lane] : -INFINITY;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0) total = m;
    }
    __syncthreads();
    return total;
}

// The block's partial of a per-thread float32 value, as a pair, into part[blockIdx.x].
__device__ __forceinline__ void block_pair_partial(float v, float2 *part) {
    const float2 t = block_pair_sum(v, 0.0f);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
}

// Sum of `count` partial pairs in float64 by one warp, valid in its lane 0; 8 loads
// in flight a lane.
__device__ __forceinline__ double warp_pair_array(const float2 *part, int count) {
    float hi = 0.0f, lo = 0.0f;
    for (int k0 = threadIdx.x & 31; k0 < count; k0 += 256) {
        float2 p[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) p[c] = k0 + 32 * c < count ? part[k0 + 32 * c] : make_float2(0.0f, 0.0f);
#pragma unroll
        for (int c = 0; c < 8; ++c) pair_add(hi, lo, p[c].x, p[c].y);
    }
    warp_pair_sum(hi, lo);
    return (double)hi + (double)lo;
}

// Sum of `count` block partial pairs, in float64, the same in every block
// (one warp adds them in a fixed order; the others wait at the block barrier).
__device__ __forceinline__ double pair_total(const float2 *part, int count) {
    __shared__ double total;
    __syncthreads();  // the previous total has been read
    if (threadIdx.x < 32) {
        const double v = warp_pair_array(part, count);
        if (threadIdx.x == 0) total = v;
    }
    __syncthreads();
    return total;
}

// a / b formed by thread 0 and shared with the block: one float64 division
// per block instead of one per thread (float64 division is slow on this
// part).  Every thread of the block calls it, with the same a and b.
__device__ __forceinline__ double block_divide(double a, double b) {
    __shared__ double quotient;
    __syncthreads();  // the previous quotient has been read
    if (threadIdx.x == 0) quotient = a / b;
    __syncthreads();
    return quotient;
}

// "Last block finishes" protocol: every block has written its partial(s);
// returns true in exactly one block, after all partials are visible.  The
// counter lives in device memory, starts at zero and is reset by the last block.
__device__ __forceinline__ bool last_block(unsigned *counter) {
    __shared__ bool is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned ticket = atomicAdd(counter, 1u);
        is_last = (ticket == gridDim.x - 1);
        if (is_last) *counter = 0u;
    }
    __syncthreads();
    if (is_last) __threadfence();
    return is_last;
}

// ---- grid barrier for cooperative (co-resident) launches --------------------

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// One atomic per block and barrier: block 0 adds 2^31 - (parties - 1), every
// other block 1, so the top bit of barrier[0] flips exactly when all parties
// have arrived (and the low bits return to where they were); a block waits
// until the bit differs from the value its own add returned.  Release add and
// acquire loads order the blocks' writes before and after the barrier.
// barrier[0] starts at 0 (the launching entry point clears it).  Returns false when the wait ran past timeout_ns (the status word
// then carries the error).  parties: arrivals that release the barrier (0 =
// every block of the grid).
//
// grid_arrive and grid_wait are its halves: thread 0 may work between them while
// the other blocks arrive.
__device__ __forceinline__ unsigned grid_arrive(unsigned *barrier, unsigned parties = 0) {
    __syncthreads();
    unsigned old = 0;
    if (threadIdx.x == 0) {
        const unsigned n = parties ? parties : gridDim.x;
        const unsigned add = blockIdx.x == 0 ? 0x80000000u - (n - 1) : 1u;
        asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(barrier), "r"(add) : "memory");
    }
    return old;
}

__device__ __forceinline__ bool grid_wait(unsigned *barrier, unsigned old, int *status,
                                          unsigned long long timeout_ns = kBarrierTimeoutNs) {
    __shared__ int ok;
    if (threadIdx.x == 0) {
        ok = 1;
        unsigned polls = 0;
        const unsigned long long t0 = global_ns();
        while (((ld_acquire(barrier) ^ old) & 0x80000000u) == 0) {
            if ((++polls & 63u) == 0 && global_ns() - t0 > timeout_ns) {
                atomicOr(status, DPF_ERR_BARRIER_TIMEOUT);
                ok = 0;
                break;
            }
        }
    }
    __syncthreads();
    return ok != 0;
}

__device__ __forceinline__ bool grid_barrier(unsigned *barrier, int *status,
                                             unsigned long long timeout_ns = kBarrierTimeoutNs,
                                             unsigned parties = 0) {
    const unsigned old = grid_arrive(barrier, parties);
    return grid_wait(barrier, old, status, timeout_ns);
}

}  // namespace dpf

#define DPF_CHECK_LAUNCH()                                   \
    do {                                                     \
        if (cudaGetLastError() != cudaSuccess) return DPF_ERR_CUDA; \
    } while (0)
