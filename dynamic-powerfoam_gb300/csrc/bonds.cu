// Bond sweeps of the finite-motion rate law (float64).
//
// Every sweep is two passes with no atomics: a bond pass computes, once per
// bond, the wrench it applies to its two endpoints and stores it as nine
// doubles [F, T_i, T_j] (endpoint i receives (F, T_i), endpoint j (-F, T_j));
// a site pass walks the site's incidence list in the reference's index_add_
// order and sums them.  Results are deterministic run to run.

#include "common.cuh"
#include "internal.cuh"

namespace dpf {

constexpr int kMaxReduceBlocks = 1024;
constexpr int64_t kPartialsOffset = 8;  // doubles reserved for counters

__device__ __forceinline__ unsigned *counter_slot(double *partials, int slot) {
    return reinterpret_cast<unsigned *>(partials) + slot;
}

__device__ __forceinline__ void store_wrench(double *w, int64_t b, d3 f, d3 ti, d3 tj) {
    double *p = w + 9 * b;
    st3(p, f);
    st3(p + 3, ti);
    st3(p + 6, tj);
}

// ---------------------------------------------------------------------------
// Constitutive trial (experiments/bonded_dem_finite_gpu.py:87-116).

struct TrialBondArgs {
    int64_t m;
    const int64_t *edges;
    dpf_stiffness k;
    dpf_history h;
    const double *y, *mid, *end;
    int want_end;
    double *n, *ri, *rj;
    double *normal_end, *offset_end, *fs_end, *mb_end, *fn_end, *mt_end;
    double *wrench;
    int *status;
    double *linear, *general;   // residual_pass: the linearisation's planes and its flag
};

// The three carried vectors where the committed normal is not a unit vector
// (a state assigned from outside): the transport as the reference writes it.
__device__ __noinline__ void carry_general(d3 n0, d3 n1, d3 spin, d3 &a, d3 &b, d3 &c, int &flags) {
    const Transport t = make_transport(n0, n1, spin, flags);
    a = apply(t, a);
    b = apply(t, b);
    c = apply(t, c);
}

// One thread per bond; bound by the float64 pipe.  The midpoint direction
// comes from one reciprocal root, the transport is a quaternion (make_turn)
// whose application costs 15 operations, an offset of exactly zero (classical
// contacts, which every transport keeps at zero) is not rotated, and where the
// end state is not wanted its guards are tested without forming it: 230 to 250
// float64 instructions (ncu's count; 280 to 310 with the end state) against 480
// operations with root, divisions, sincos and rotations written out.  262k sites /
// 1.9M bonds: 1.50 -> 0.79 ms, with the end state 0.96 ms.
//
// kLinearise: what jvp_linear_bonds reads, in planes of one double a bond.
__device__ __forceinline__ void put(const TrialBondArgs &a, int plane, int64_t b, double v) {
    a.linear[plane * a.m + b] = v;
}
__device__ __forceinline__ void put(const TrialBondArgs &a, int plane, int64_t b, d3 v) {
    put(a, plane, b, v.x);
    put(a, plane + 1, b, v.y);
    put(a, plane + 2, b, v.z);
}

template <bool kLinearise>
__global__ void __launch_bounds__(128) trial_bonds(TrialBondArgs a) {
    const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (b >= a.m) return;
    int flags = 0;
    int64_t i, j;
    edge(a.edges, b, i, j);
    const double *yi = a.y + 6 * i, *yj = a.y + 6 * j;
    const d3 ui = ld3(yi), wi = ld3(yi + 3), uj = ld3(yj), wj = ld3(yj + 3);
    const d3 xi = ld3(a.h.x, i), xj = ld3(a.h.x, j);
    const d3 mi = a.mid ? ld3(a.mid, i) : xi + 0.5 * ui;
    const d3 mj = a.mid ? ld3(a.mid, j) : xj + 0.5 * uj;
    const d3 ei = a.end ? ld3(a.end, i) : xi + ui;
    const d3 ej = a.end ? ld3(a.end, j) : xj + uj;
    // geometry(mid)  (bonded_dem_finite_gpu.py:66-73)
    const d3 dm = mj - mi;
    const double lm2 = dot(dm, dm);
    if (lm2 <= 1e-24) flags |= DPF_ERR_COINCIDENT;
    const double inv = rsqrt(lm2);
    const d3 nm = inv * dm;
    const d3 half_spin = 0.25 * (wi + wj);
    const d3 n0 = ld3(a.h.normal, b);
    d3 offset = ld3(a.h.offset, b), fs0 = ld3(a.h.fs, b), mb0 = ld3(a.h.mb, b);
    if (is_unit(n0)) {
        const Turn to_mid = make_turn(n0, nm, half_spin, flags);
        if (!is_zero(offset)) offset = apply(to_mid, offset);
        fs0 = apply(to_mid, fs0);
        mb0 = apply(to_mid, mb0);
        if (kLinearise) {
            put(a, 4, b, to_mid.sum);
            put(a, 7, b, 2.0 * to_mid.r * to_mid.r);
            put(a, 8, b, 2.0 * to_mid.sh * to_mid.ch);
            put(a, 9, b, 2.0 * to_mid.sh * to_mid.sh);
            put(a, 10, b, to_mid.r);
            put(a, 11, b, 2.0 * to_mid.half * to_mid.r);
        }
    } else {
        carry_general(n0, nm, half_spin, offset, fs0, mb0, flags);
        if (kLinearise) *a.general = 1.0;
    }
    // levers of the contact (mi + mj)/2 + (radi - radj)/2 nm + offset
    const double rad = 0.5 * (a.h.radii[i] - a.h.radii[j]);
    const d3 lever = axpy(rad, nm, offset);
    const d3 ri = axpy(0.5, dm, lever), rj = axpy(-0.5, dm, lever);
    const d3 du = cross_sub(cross_add(uj - ui, wj, rj), wi, ri);
    const d3 dw = wj - wi;
    const double dn = dot(du, nm), twist = dot(dw, nm);
    const double kn = a.k.kn[b], ks = a.k.ks[b], kb = a.k.kb[b], kt = a.k.kt[b];
    const double fn_c = a.h.fn[b], mt_c = a.h.mt[b];
    const d3 slide = ks * axpy(-dn, nm, du), bend = kb * axpy(-twist, nm, dw);
    const double fn_mid = fma(0.5 * kn, dn, fn_c), mt_mid = fma(0.5 * kt, twist, mt_c);
    const d3 f = axpy(fn_mid, nm, axpy(0.5, slide, fs0));
    const d3 couple = axpy(mt_mid, nm, axpy(0.5, bend, mb0));
    if (kLinearise) {
        const double hks = 0.5 * ks, hkb = 0.5 * kb;
        put(a, 0, b, nm);
        put(a, 3, b, 0.5 * inv);
        put(a, 12, b, half_spin);
        put(a, 15, b, offset);
        put(a, 18, b, fs0);
        put(a, 21, b, mb0);
        put(a, 24, b, rad);
        put(a, 25, b, ri);
        put(a, 28, b, rj);
        put(a, 31, b, du);
        put(a, 34, b, dw);
        put(a, 37, b, f);
        put(a, 40, b, fma(-hks, dn, fn_mid));
        put(a, 41, b, fma(-hkb, twist, mt_mid));
        put(a, 42, b, hks);
        put(a, 43, b, hkb);
        put(a, 44, b, 0.5 * kn - hks);
        put(a, 45, b, 0.5 * kt - hkb);
    }
    if (a.wrench) store_wrench(a.wrench, b, f, cross_add(couple, ri, f), cross_sub(-couple, rj, f));
    if (a.n) st3(a.n, b, nm);
    if (a.ri) st3(a.ri, b, ri);
    if (a.rj) st3(a.rj, b, rj);
    // geometry(end) and the end-of-step transport; its guards hold even when unused
    const d3 de = ej - ei;
    const double le2 = dot(de, de);
    if (le2 <= 1e-24) flags |= DPF_ERR_COINCIDENT;
    if (a.want_end) {
        const d3 ne = rsqrt(le2) * de;
        const Turn to_end = make_turn(nm, ne, half_spin, flags);
        if (a.normal_end) st3(a.normal_end, b, ne);
        if (a.fn_end) a.fn_end[b] = fn_c + kn * dn;
        if (a.mt_end) a.mt_end[b] = mt_c + kt * twist;
        if (a.fs_end) st3(a.fs_end, b, apply(to_end, fs0 + slide));
        if (a.mb_end) st3(a.mb_end, b, apply(to_end, mb0 + bend));
        if (a.offset_end) st3(a.offset_end, b, is_zero(offset) ? offset : apply(to_end, offset));
    } else if (turned(nm, de, le2)) {
        flags |= DPF_ERR_NORMAL_TURN;
    }
    if (flags) atomicOr(a.status, flags);
}

// Site pass of trial/residual: force gather, rotation guard, end positions,
// midpoint residual (bonded_dem_newton.py:83-86), block scaling
// (bonded_dem_newton.py:104-105) and the three norms of NewtonBonds.step.
struct SiteResidualArgs {
    int64_t n;
    const int32_t *ptr, *inc;
    const double *wrench;
    const double *y, *x, *end;
    double *force, *x_end;
    // residual part (residual != nullptr)
    const double *v, *external, *mass;
    const uint8_t *fixed;
    double dt, half_dt2;
    double *residual;
    const double *P, *units;
    double *scaled, *norms, *partials;
    int *status;
};

// Two neighbouring lanes a site: the force with its three rows, and the torque
// with its.  A pass of one thread a site waited on its 15 incidences one after
// the other (two loads deep each) with 36 strided reads of P behind them.
// 262k sites: 146 -> 106 us (site_jvp 159 -> 105 us).
__global__ void __launch_bounds__(kThreads) site_residual(SiteResidualArgs a) {
    double sum_r = 0.0, max_s = 0.0, sum_s = 0.0;
    int flags = 0;
    const int side = threadIdx.x & 1;
    const int64_t stride = (int64_t)gridDim.x * (blockDim.x / 2);
    const int64_t rounds = (a.n + stride - 1) / stride;   // the same for every lane: the lanes of a site meet below
    int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / 2;
    for (int64_t k = 0; k < rounds; ++k, s += stride) {
        const bool live = s < a.n;
        d3 acc = mk(0.0, 0.0, 0.0), ys = acc, r = acc;
        if (live) {
            acc = gather_half(a.ptr, a.inc, a.wrench, s, side);
            ys = ld3(a.y + 6 * s + 3 * side);
            if (a.force) st3(a.force + 6 * s + 3 * side, acc);
            if (side) {
                if (dot(ys, ys) > 0.0625) flags |= DPF_ERR_ROTATION;
            } else if (a.x_end) {
                st3(a.x_end, s, a.end ? ld3(a.end, s) : ld3(a.x, s) + ys);
            }
        }
        if (!a.residual) continue;
        const int64_t at = 6 * s + 3 * side;
        if (live) {
            const d3 m = ld3(a.mass + at), v = ld3(a.v + at), ext = ld3(a.external + at);
            r = a.fixed[s] ? ys
                           : mk(m.x * (ys.x - a.dt * v.x) - a.half_dt2 * (acc.x + ext.x),
                                m.y * (ys.y - a.dt * v.y) - a.half_dt2 * (acc.y + ext.y),
                                m.z * (ys.z - a.dt * v.z) - a.half_dt2 * (acc.z + ext.z));
            st3(a.residual + at, r);
            sum_r += dot(r, r);
        }
        if (a.P) {
            const d3 other = other_half(r);
            if (live) {
                const d3 pr = half_rows(a.P + 36 * s, side, r, other), u = ld3(a.units + at);
                const d3 val = over_units(pr, u);
                if (a.scaled) st3(a.scaled + at, val);
                max_s = fmax(max_s, fmax(fabs(val.x), fmax(fabs(val.y), fabs(val.z))));
                sum_s += dot(val, val);
            }
        }
    }
    if (flags) atomicOr(a.status, flags);
    if (!a.norms) return;
    double v[3] = {sum_r, max_s, sum_s};
    block_reduce<3, 2u>(v);
    double *part = a.partials + kPartialsOffset;
    if (threadIdx.x == 0) {
        part[3 * blockIdx.x + 0] = v[0];
        part[3 * blockIdx.x + 1] = v[1];
        part[3 * blockIdx.x + 2] = v[2];
    }
    if (last_block(counter_slot(a.partials, 0))) {
        block_arrays<3, 2u>(part, gridDim.x, v);
        if (threadIdx.x == 0) {
            a.norms[0] = sqrt(v[0]);
            a.norms[1] = v[1];
            a.norms[2] = sqrt(v[2]);
            if (!isfinite(v[0]) || !isfinite(v[2])) atomicOr(a.status, DPF_ERR_NONFINITE);
        }
    }
}

// ---------------------------------------------------------------------------
// Analytic JVP of the midpoint force (experiments/bonded_dem_jvp_warp.py:17-97).

// Shared part of `transport` and its derivative for one bond: the same
// (n0, n, spin) rotate offset, fs and mb.
struct TransportJvp {
    d3 k, dk, n, dn, b;
    double inv, dc, c, s, da;
};

__device__ __forceinline__ TransportJvp make_transport_jvp(d3 n0, d3 n, d3 dn, d3 spin, d3 dspin) {
    TransportJvp t;
    const double raw = dot(n0, n);
    const double cosine = fmin(fmax(raw, -1.0), 1.0);
    t.dc = (raw < -1.0 || raw > 1.0) ? 0.0 : dot(n0, dn);
    t.k = cross(n0, n);
    t.dk = cross(n0, dn);
    t.inv = 1.0 / (1.0 + cosine);
    const d3 sum = n0 + n;
    const double length = norm(sum);
    t.b = sum / length;
    const d3 db = (dn - dot(t.b, dn) * t.b) / length;
    const double angle = dot(spin, t.b);
    t.da = dot(dspin, t.b) + dot(spin, db);
    sincos(angle, &t.s, &t.c);
    t.n = n;
    t.dn = dn;
    return t;
}

__device__ __forceinline__ void apply_jvp(const TransportJvp &t, d3 v, d3 &value, d3 &deriv) {
    const d3 kv = cross(t.k, v);
    const d3 kkv = cross(t.k, kv);
    const d3 tv = v + kv + t.inv * kkv;
    const d3 dkv = cross(t.dk, v);
    d3 dt = dkv + t.inv * (cross(t.dk, kv) + cross(t.k, dkv));
    dt = dt - (t.dc * t.inv * t.inv) * kkv;
    const double nt = dot(t.n, tv);
    const d3 nxt = cross(t.n, tv);
    value = t.c * tv + t.s * nxt + ((1.0 - t.c) * nt) * t.n;
    d3 d = t.c * dt - (t.s * t.da) * tv + (t.c * t.da) * nxt;
    d = d + t.s * (cross(t.dn, tv) + cross(t.n, dt)) + (t.s * t.da * nt) * t.n;
    deriv = d + (1.0 - t.c) * ((dot(t.dn, tv) + dot(t.n, dt)) * t.n + nt * t.dn);
}

struct JvpBondArgs {
    int64_t m;
    const int64_t *edges;
    dpf_stiffness k;
    dpf_history h;
    const double *y, *direction, *units;
    double *wrench;
};

__device__ __forceinline__ void load_direction(const double *d, const double *units, int64_t s, d3 &u, d3 &w) {
    const double *p = d + 6 * s;
    u = ld3(p);
    w = ld3(p + 3);
    if (units) {
        const double *q = units + 6 * s;
        u = mk(u.x * q[0], u.y * q[1], u.z * q[2]);
        w = mk(w.x * q[3], w.y * q[4], w.z * q[5]);
    }
}

// Carried vectors and their derivatives for a committed normal that is not a
// unit vector (a state assigned from outside): the general derivative.
__device__ __noinline__ void carry_jvp_general(d3 n0, d3 n, d3 dn, d3 spin, d3 dspin, d3 &a, d3 &da, d3 &b, d3 &db,
                                               d3 &c, d3 &dc) {
    const TransportJvp t = make_transport_jvp(n0, n, dn, spin, dspin);
    const d3 a0 = a, b0 = b, c0 = c;
    apply_jvp(t, a0, a, da);
    apply_jvp(t, b0, b, db);
    apply_jvp(t, c0, c, dc);
}

// One thread per bond; bound by the float64 pipe.  A transported vector's
// derivative is one cross product with the transport's angular velocity
// (turn_rate), so the three vectors share what the derivative costs: 380
// float64 instructions a bond (ncu, given contacts) against 770 with every vector's
// derivative written out.  262k sites / 1.9M bonds: 2.46 -> 1.20 ms; 101k sites with
// given contacts: 0.95 -> 0.49 ms.
__global__ void __launch_bounds__(128) jvp_bonds(JvpBondArgs a) {
    const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (b >= a.m) return;
    int64_t i, j;
    edge(a.edges, b, i, j);
    const d3 ui = ld3(a.y + 6 * i), wi = ld3(a.y + 6 * i + 3);
    const d3 uj = ld3(a.y + 6 * j), wj = ld3(a.y + 6 * j + 3);
    d3 dui, dwi, duj, dwj;
    load_direction(a.direction, a.units, i, dui, dwi);
    load_direction(a.direction, a.units, j, duj, dwj);
    const d3 disp = (ld3(a.h.x, j) + 0.5 * uj) - (ld3(a.h.x, i) + 0.5 * ui);
    const double inv = rsqrt(dot(disp, disp));
    const d3 n = inv * disp;
    const d3 e = duj - dui, dd = (0.5 * inv) * e;
    const d3 dn = dd - dot(n, dd) * n;
    const d3 spin = 0.25 * (wi + wj), dspin = 0.25 * (dwi + dwj);
    const d3 n0 = ld3(a.h.normal, b);
    d3 offset = ld3(a.h.offset, b), fs0 = ld3(a.h.fs, b), mb0 = ld3(a.h.mb, b);
    d3 doffset = mk(0.0, 0.0, 0.0), dfs0, dmb0;
    if (is_unit(n0)) {
        int flags = 0;
        const Turn t = make_turn(n0, n, spin, flags);
        const d3 rate = turn_rate(t, n, dn, spin, dspin);
        if (!is_zero(offset)) {
            offset = apply(t, offset);
            doffset = cross(rate, offset);
        }
        fs0 = apply(t, fs0);
        dfs0 = cross(rate, fs0);
        mb0 = apply(t, mb0);
        dmb0 = cross(rate, mb0);
    } else {
        carry_jvp_general(n0, n, dn, spin, dspin, offset, doffset, fs0, dfs0, mb0, dmb0);
    }
    // levers: the contact minus the two midpoints, and their derivatives
    const double rad = 0.5 * (a.h.radii[i] - a.h.radii[j]);
    const d3 lever = axpy(rad, n, offset), dlever = axpy(rad, dn, doffset);
    const d3 ri = axpy(0.5, disp, lever), rj = axpy(-0.5, disp, lever);
    const d3 dri = axpy(0.25, e, dlever), drj = axpy(-0.25, e, dlever);
    const d3 du = cross_sub(cross_add(uj - ui, wj, rj), wi, ri);
    const d3 ddu = cross_sub(cross_add(cross_sub(cross_add(e, dwj, rj), dwi, ri), wj, drj), wi, dri);
    const d3 dw = wj - wi, ddw = dwj - dwi;
    const double nd = dot(du, n), tw = dot(dw, n);
    const double dnd = dot_add(dot(du, dn), ddu, n);
    const double dtw = dot_add(dot(dw, dn), ddw, n);
    const double hkn = 0.5 * a.k.kn[b], hks = 0.5 * a.k.ks[b], hkb = 0.5 * a.k.kb[b], hkt = 0.5 * a.k.kt[b];
    const double fn_mid = a.h.fn[b] + hkn * nd, mt_mid = a.h.mt[b] + hkt * tw;
    const d3 f = axpy(fn_mid, n, axpy(hks, axpy(-nd, n, du), fs0));
    // df = d(fn n) + dfs0 + ks/2 (ddu - d(nd n)), gathered by direction: along ddu, n and dn
    const d3 df = axpy(fn_mid - hks * nd, dn, axpy((hkn - hks) * dnd, n, axpy(hks, ddu, dfs0)));
    const d3 dcouple = axpy(mt_mid - hkb * tw, dn, axpy((hkt - hkb) * dtw, n, axpy(hkb, ddw, dmb0)));
    store_wrench(a.wrench, b, df, cross_add(cross_add(dcouple, dri, f), ri, df),
                 cross_sub(cross_sub(-dcouple, drj, f), rj, df));
}

// The same product from the linearisation that the residual pass at y stored:
// everything that does not depend on the direction (geometry, transport, carried
// forces, levers, the force itself) is read instead of formed again, 170 float64
// instructions a bond (ncu) and 46 coalesced doubles, whose loads hide behind
// them.  With dri = e/4 + dl and drj = -e/4 + dl the spins' share of the relative
// motion is dw x dl - spin x e.  A step's FGMRES takes two or three of these an
// iterate for one linearisation (its stores: 5% of the trial pass).
// 262k sites: 1.20 -> 0.55 ms; a step there 27.0 -> 23.2 ms, at 37k sites 3.72 -> 3.33 ms.
__global__ void __launch_bounds__(128) jvp_linear_bonds(int64_t m, const int64_t *edges, const double *lin,
                                                        const double *direction, double *wrench) {
    const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (b >= m) return;
    const auto get = [&](int plane) { return __ldg(lin + plane * m + b); };
    const auto get3 = [&](int plane) { return mk(get(plane), get(plane + 1), get(plane + 2)); };
    int64_t i, j;
    edge(edges, b, i, j);
    const d3 dui = ld3(direction + 6 * i), dwi = ld3(direction + 6 * i + 3);
    const d3 duj = ld3(direction + 6 * j), dwj = ld3(direction + 6 * j + 3);
    const d3 n = get3(0), sum = get3(4), spin = get3(12);
    const d3 e = duj - dui, dd = get(3) * e;
    const d3 dn = axpy(-dot(n, dd), n, dd);
    // angular velocity of the transport (turn_rate)
    const double r = get(10);
    const d3 arc = get(7) * cross(sum, dn);
    const double dth = r * dot_add(fma(-get(11), dot(sum, dn), 0.25 * dot(sum, dwi + dwj)), spin, dn);
    const double sine = get(8);
    const d3 side = axpy(sine, arc, get(9) * cross_add(dn, n, arc));
    const d3 rate = cross_add(axpy(dth, n, axpy(sine, dn, arc)), n, side);
    d3 dlever = get(24) * dn;
    const d3 offset = get3(15);
    if (!is_zero(offset)) dlever = cross_add(dlever, rate, offset);
    const d3 ri = get3(25), rj = get3(28), dw = get3(34), ddw = dwj - dwi;
    const d3 ddu = cross_sub(cross_add(cross_sub(cross_add(e, dwj, rj), dwi, ri), dw, dlever), spin, e);
    const double dnd = dot_add(dot(get3(31), dn), ddu, n);
    const double dtw = dot_add(dot(dw, dn), ddw, n);
    const d3 f = get3(37);
    const d3 df = axpy(get(40), dn, axpy(get(44) * dnd, n, cross_add(get(42) * ddu, rate, get3(18))));
    const d3 dcouple = axpy(get(41), dn, axpy(get(45) * dtw, n, cross_add(get(43) * ddw, rate, get3(21))));
    const d3 dri = axpy(0.25, e, dlever), drj = axpy(-0.25, e, dlever);
    store_wrench(wrench, b, df, cross_add(cross_add(dcouple, dri, f), ri, df),
                 cross_sub(cross_sub(-dcouple, drj, f), rj, df));
}

// Site pass of the JVP: out = M d - dt^2/2 g, fixed rows d; optional P(.)/units.
// Two neighbouring lanes a site, as in site_residual.
struct SiteJvpArgs {
    int64_t n;
    const int32_t *ptr, *inc;
    const double *wrench, *direction, *units, *mass, *P;
    const uint8_t *fixed;
    double half_dt2;
    double *out;
    int scaled;     // the direction is in the scaled coordinates (d = units direction)
};

__global__ void __launch_bounds__(kThreads) site_jvp(SiteJvpArgs a) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, s = t / 2;
    const int part = (int)(t & 1);
    const bool live = s < a.n;
    const int64_t at = 6 * s + 3 * part;
    d3 r = mk(0.0, 0.0, 0.0), u = r;
    if (live) {
        const d3 acc = gather_half(a.ptr, a.inc, a.wrench, s, part);
        d3 d = ld3(a.direction + at);
        if (a.units) {
            u = ld3(a.units + at);
            if (a.scaled) d = mk(d.x * u.x, d.y * u.y, d.z * u.z);
        }
        const d3 m = ld3(a.mass + at);
        r = a.fixed[s] ? d
                       : mk(m.x * d.x - a.half_dt2 * acc.x, m.y * d.y - a.half_dt2 * acc.y,
                            m.z * d.z - a.half_dt2 * acc.z);
        if (!a.P) st3(a.out + at, r);
    }
    if (a.P) {
        const d3 other = other_half(r);
        if (live) {
            const d3 pr = half_rows(a.P + 36 * s, part, r, other);
            st3(a.out + at, over_units(pr, u));
        }
    }
}

// ---------------------------------------------------------------------------
// Frozen tangent K q (experiments/bonded_dem_linear_gpu.py:42-52).

struct StiffnessBondArgs {
    int64_t m;
    const int64_t *edges;
    dpf_stiffness k;
    dpf_tangent t;
    const double *q;
    double *wrench;
};

__global__ void __launch_bounds__(kThreads) stiffness_bonds(StiffnessBondArgs a) {
    __shared__ double stage[9 * kThreads];
    const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, first = b - (threadIdx.x & 31);
    if (first >= a.m) return;
    Wrench w{};
    if (b < a.m) {
        int64_t i, j;
        edge(a.edges, b, i, j);
        w = stiffness_wrench(ld3(a.t.n, b), ld3(a.t.ri, b), ld3(a.t.rj, b), a.k.kn[b], a.k.ks[b], a.k.kb[b],
                             a.k.kt[b], a.q + 6 * i, a.q + 6 * j);
    }
    store_wrenches(a.wrench, first, (int)(a.m - first < 32 ? a.m - first : 32), w, stage + 9 * (threadIdx.x & ~31));
}

// Two lanes a site: its force and its torque.
__global__ void __launch_bounds__(kThreads) site_gather(int64_t n, const int32_t *ptr, const int32_t *inc,
                                                         const double *wrench, double *out) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, s = t / 2;
    if (s >= n) return;
    st3(out, t, gather_half(ptr, inc, wrench, s, (int)(t & 1)));
}

// ---------------------------------------------------------------------------
// Diagonal blocks (bonded_dem_linear_gpu.py:54-72) and block scaling
// (bonded_dem_newton.py:94-102), one thread per site over its incidences.

// With S the matrix of the cross product with the lever r, a = n x r (so that
// S^T n = a up to sign), g = kn - ks and h = kt - kb, a bond end adds
//   ks I + g n n^T,   -(ks S + g n a^T) and its transpose,
//   ks (|r|^2 I - r r^T) + g a a^T + kb I + h n n^T
// to its site's blocks.  Only the 21 entries of a symmetric matrix are summed,
// the multiples of I and S as four numbers (sum ks, sum ks r): about 65
// float64 operations an end against 135 for the products of full 3x3 matrices.
// The scaling pass at 262k sites: 1.29 -> 0.70 ms, bound by the float64 pipe.
struct BlockSum {
    double uu[6], uw[9], ww[6];   // upper triangles xx xy xz yy yz zz; uw = g n a^T
    double k, w;                  // sums of ks, and of kb + ks |r|^2
    d3 kr;                        // sum of ks r
};

__device__ __forceinline__ void add_outer(double m[6], d3 a, d3 b) {
    m[0] += a.x * b.x;
    m[1] += a.x * b.y;
    m[2] += a.x * b.z;
    m[3] += a.y * b.y;
    m[4] += a.y * b.z;
    m[5] += a.z * b.z;
}

__device__ __forceinline__ void add_bond_block(BlockSum &B, d3 n, d3 r, double kn, double ks, double kb, double kt) {
    const d3 a = cross(n, r), gn = (kn - ks) * n, kr = ks * r;
    add_outer(B.uu, gn, n);
    B.uw[0] += gn.x * a.x;
    B.uw[1] += gn.x * a.y;
    B.uw[2] += gn.x * a.z;
    B.uw[3] += gn.y * a.x;
    B.uw[4] += gn.y * a.y;
    B.uw[5] += gn.y * a.z;
    B.uw[6] += gn.z * a.x;
    B.uw[7] += gn.z * a.y;
    B.uw[8] += gn.z * a.z;
    add_outer(B.ww, (kn - ks) * a, a);
    add_outer(B.ww, (kt - kb) * n, n);
    add_outer(B.ww, -kr, r);
    B.k += ks;
    B.w += kb + dot(kr, r);
    B.kr = B.kr + kr;
}

// kLanes neighbouring lanes share a site: each sums every kLanes-th of its ends,
// then all hold the site's block.
template <int kLanes>
__device__ __forceinline__ void site_diagonal(const int32_t *ptr, const int32_t *inc, const dpf_stiffness &k,
                                              const dpf_tangent &t, int64_t s, int lane, double D[36]) {
    BlockSum B;
#pragma unroll
    for (int c = 0; c < 6; ++c) B.uu[c] = B.ww[c] = 0.0;
#pragma unroll
    for (int c = 0; c < 9; ++c) B.uw[c] = 0.0;
    B.k = B.w = 0.0;
    B.kr = mk(0.0, 0.0, 0.0);
    const int e1 = s < 0 ? 0 : ptr[s + 1];
    for (int e = s < 0 ? 0 : ptr[s] + lane; e < e1; e += kLanes) {
        const int v = inc[e];
        const int64_t b = v >= 0 ? v : ~v;
        const d3 r = ld3(v >= 0 ? t.ri : t.rj, b);
        add_bond_block(B, ld3(t.n, b), r, k.kn[b], k.ks[b], k.kb[b], k.kt[b]);
    }
    if (kLanes > 1) {
        double *all = reinterpret_cast<double *>(&B);
#pragma unroll
        for (int o = 1; o < kLanes; o <<= 1)
#pragma unroll
            for (int c = 0; c < (int)(sizeof(B) / sizeof(double)); ++c)
                all[c] += __shfl_xor_sync(0xffffffffu, all[c], o);
    }
    const int at[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5};
    const double S[9] = {0.0, -B.kr.z, B.kr.y, B.kr.z, 0.0, -B.kr.x, -B.kr.y, B.kr.x, 0.0};
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const int c = at[3 * p + q];
            D[6 * p + q] = p == q ? B.uu[c] + B.k : B.uu[c];
            D[6 * (3 + p) + 3 + q] = p == q ? B.ww[c] + B.w : B.ww[c];
            // d S = ks S + g n (S^T n)^T with S^T n = (S applied from the left to n) = n x r
            D[6 * p + 3 + q] = -(S[3 * p + q] + B.uw[3 * p + q]);
            D[6 * (3 + q) + p] = -(S[3 * p + q] + B.uw[3 * p + q]);
        }
}

struct ScalingArgs {
    int64_t n;
    const int32_t *ptr, *inc;
    dpf_stiffness k;
    dpf_tangent t;
    const double *mass, *radii;
    const uint8_t *fixed;
    double alpha;  // dt^2 / 4
    double *diagonal, *block, *P, *units;
};

// Lane `lane` of a site's kLanes writes every kLanes-th entry.
template <int kLanes>
__device__ __forceinline__ void put_block(double *out, int64_t s, int lane, const double M[36]) {
#pragma unroll
    for (int c = 0; c < 36; ++c)
        if (kLanes == 1 || c % kLanes == lane) out[36 * s + c] = M[c];
}

// One lane a site where there are sites for every scheduler; four where there
// are not: a warp instruction of the float64 pipe takes 64 cycles of its
// scheduler's share however few warps there are, so a site's 1,300 operations
// one after the other took 57 us at 512 sites.  With four lanes (the ends dealt
// among them, the inverse formed by each): 29 us; 8k sites 64 -> 43 us, 10.6k sites 60 (one
// lane: 62).
template <int kLanes>
__global__ void __launch_bounds__(128) scaling_sites(ScalingArgs a) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, s = t / kLanes;
    const int lane = (int)(t % kLanes);
    const bool live = s < a.n;
    if (kLanes == 1 && !live) return;
    double D[36];
    site_diagonal<kLanes>(a.ptr, a.inc, a.k, a.t, live ? s : -1, lane, D);
    if (!live) return;
    if (a.diagonal) put_block<kLanes>(a.diagonal, s, lane, D);
    if (!a.P && !a.block) return;
    const bool fx = a.fixed[s] != 0;
    double B[36];
#pragma unroll
    for (int p = 0; p < 6; ++p)
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const double val = (p == q ? a.mass[6 * s + p] : 0.0) + a.alpha * D[6 * p + q];
            B[6 * p + q] = fx ? (p == q ? 1.0 : 0.0) : val;
        }
    if (a.block) put_block<kLanes>(a.block, s, lane, B);
    if (a.P) {
        double P[36];
        spd_inverse6(B, P);
        put_block<kLanes>(a.P, s, lane, P);
    }
    if (a.units && lane == 0) {
        const double r = fx ? 1.0 : a.radii[s];
#pragma unroll
        for (int c = 0; c < 6; ++c) a.units[6 * s + c] = c < 3 ? r : 1.0;
    }
}

template <int kLanes>
__global__ void __launch_bounds__(128) diagonal_sites(int64_t n, const int32_t *ptr, const int32_t *inc,
                                                      dpf_stiffness k, dpf_tangent t, double *out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, s = i / kLanes;
    const int lane = (int)(i % kLanes);
    double D[36];
    site_diagonal<kLanes>(ptr, inc, k, t, s < n ? s : -1, lane, D);
    if (s < n) put_block<kLanes>(out, s, lane, D);
}

// Sites from which one lane each fills the machine.
constexpr int64_t kFewSites = 12288;

// ---------------------------------------------------------------------------
// Loads of the committed state (experiments/bonded_dem_finite_gpu.py:82-85).

__global__ void __launch_bounds__(kThreads) loads_bonds(int64_t m, const int64_t *edges, dpf_history h,
                                                         double *wrench, int *status) {
    const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (b >= m) return;
    int64_t i, j;
    edge(edges, b, i, j);
    const d3 xi = ld3(h.x, i), xj = ld3(h.x, j);
    const d3 d = xj - xi;
    const double d2 = dot(d, d);
    if (d2 <= 1e-24 && status) atomicOr(status, DPF_ERR_COINCIDENT);
    const d3 n = rsqrt(d2) * d;
    const d3 lever = axpy(0.5 * (h.radii[i] - h.radii[j]), n, ld3(h.offset, b));
    const d3 ri = axpy(0.5, d, lever), rj = axpy(-0.5, d, lever);
    const d3 f = axpy(h.fn[b], n, ld3(h.fs, b));
    const d3 couple = axpy(h.mt[b], n, ld3(h.mb, b));
    store_wrench(wrench, b, f, cross_add(couple, ri, f), cross_sub(-couple, rj, f));
}

inline int blocks_for(int64_t n, int threads) { return (int)((n + threads - 1) / threads); }

// Bond setup of LinearBondsGPU / FiniteBondsGPU (experiments/bonded_dem_linear_gpu.py:15-40,
// experiments/bonded_dem_finite_gpu.py:49-63) on the device: normal, contact
// levers, stiffnesses and the contact offset from the classical contact.
struct BondSetupArgs {
    int64_t m;
    const int64_t *edges;
    const double *points, *radii, *areas, *contacts, *young_b, *shear_b;
    double young, shear;
    double *n, *ri, *rj, *kn, *ks, *kb, *kt, *offset;
};

// One-time setup arithmetic, written with correctly rounded divisions and no
// fused multiply-adds so that it gives the bits of the reference's host
// formulas (n = d / |d|, c = (p_i + p_j)/2 + (r_i - r_j)/2 n, k = E A / L, ..).
__global__ void __launch_bounds__(kThreads) bond_setup_kernel(BondSetupArgs a) {
    const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (b >= a.m) return;
    int64_t i, j;
    edge(a.edges, b, i, j);
    const d3 pi = ld3(a.points, i), pj = ld3(a.points, j);
    const d3 d = mk(__dsub_rn(pj.x, pi.x), __dsub_rn(pj.y, pi.y), __dsub_rn(pj.z, pi.z));
    const double length = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(d.x, d.x), __dmul_rn(d.y, d.y)), __dmul_rn(d.z, d.z)));
    const d3 n = mk(__ddiv_rn(d.x, length), __ddiv_rn(d.y, length), __ddiv_rn(d.z, length));
    const double half = __dmul_rn(0.5, __dsub_rn(a.radii[i], a.radii[j]));
    const d3 classical = mk(__dadd_rn(__dmul_rn(0.5, __dadd_rn(pi.x, pj.x)), __dmul_rn(half, n.x)),
                            __dadd_rn(__dmul_rn(0.5, __dadd_rn(pi.y, pj.y)), __dmul_rn(half, n.y)),
                            __dadd_rn(__dmul_rn(0.5, __dadd_rn(pi.z, pj.z)), __dmul_rn(half, n.z)));
    const d3 c = a.contacts ? ld3(a.contacts, b) : classical;
    st3(a.n, b, n);
    st3(a.ri, b, mk(__dsub_rn(c.x, pi.x), __dsub_rn(c.y, pi.y), __dsub_rn(c.z, pi.z)));
    st3(a.rj, b, mk(__dsub_rn(c.x, pj.x), __dsub_rn(c.y, pj.y), __dsub_rn(c.z, pj.z)));
    if (a.offset)
        st3(a.offset, b, mk(__dsub_rn(c.x, classical.x), __dsub_rn(c.y, classical.y), __dsub_rn(c.z, classical.z)));
    const double area = a.areas[b];
    const double second = __ddiv_rn(__dmul_rn(area, area), 4.0 * 3.14159265358979323846);
    const double E = a.young_b ? a.young_b[b] : a.young, G = a.shear_b ? a.shear_b[b] : a.shear;
    a.kn[b] = __ddiv_rn(__dmul_rn(E, area), length);
    a.ks[b] = __ddiv_rn(__dmul_rn(G, area), length);
    a.kb[b] = __ddiv_rn(__dmul_rn(E, second), length);
    a.kt[b] = __ddiv_rn(__dmul_rn(G, __dmul_rn(2.0, second)), length);
}

__global__ void __launch_bounds__(kThreads) site_mass_kernel(int64_t n, const double *masses, const double *radii,
                                                             double *mass6) {
    const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (s >= n) return;
    const double m = masses[s], r = radii[s];
    const double inertia = __dmul_rn(__dmul_rn(__dmul_rn(0.4, m), r), r);
#pragma unroll
    for (int c = 0; c < 6; ++c) mass6[6 * s + c] = c < 3 ? m : inertia;
}

}  // namespace dpf

using namespace dpf;

extern "C" {

int64_t dpf_wrench_scratch_doubles(int64_t n_bonds) { return 9 * n_bonds; }

int64_t dpf_partials_doubles(void) { return kPartialsOffset + 2 * 64 * (int64_t)kMaxReduceBlocks; }

static bool graph_ok(const dpf_graph *g) {
    return g && g->n_sites > 0 && g->n_bonds >= 0 && g->n_bonds < (int64_t(1) << 31) && g->inc_ptr &&
           (g->n_bonds == 0 || (g->edges && g->inc_bond));
}

int dpf_stiffness_apply(const dpf_graph *g, const dpf_stiffness *k, const dpf_tangent *t, const double *q,
                        double *out, double *wrench, void *stream) {
    if (!graph_ok(g) || !k || !t || !q || !out || (g->n_bonds && !wrench)) return DPF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    if (g->n_bonds) {
        StiffnessBondArgs a{g->n_bonds, g->edges, *k, *t, q, wrench};
        stiffness_bonds<<<blocks_for(g->n_bonds, kThreads), kThreads, 0, st>>>(a);
    }
    site_gather<<<blocks_for(2 * g->n_sites, kThreads), kThreads, 0, st>>>(g->n_sites, g->inc_ptr, g->inc_bond,
                                                                        wrench, out);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_diagonal_blocks(const dpf_graph *g, const dpf_stiffness *k, const dpf_tangent *t, double *diagonal,
                        void *stream) {
    if (!graph_ok(g) || !k || !t || !diagonal) return DPF_ERR_ARGUMENT;
    const int lanes = g->n_sites < kFewSites ? 4 : 1, threads = spread_threads(lanes * g->n_sites);
    (lanes == 4 ? diagonal_sites<4> : diagonal_sites<1>)<<<blocks_for(lanes * g->n_sites, threads), threads, 0,
                                                           (cudaStream_t)stream>>>(g->n_sites, g->inc_ptr, g->inc_bond,
                                                                                   *k, *t, diagonal);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_prepare_scaling(const dpf_graph *g, const dpf_stiffness *k, const dpf_tangent *t, const double *mass,
                        const uint8_t *fixed, const double *radii, double dt, double *diagonal, double *block,
                        double *preconditioner, double *units, void *stream) {
    if (!graph_ok(g) || !k || !t || !mass || !fixed || !radii || !preconditioner) return DPF_ERR_ARGUMENT;
    ScalingArgs a{g->n_sites, g->inc_ptr, g->inc_bond, *k, *t, mass, radii, fixed, 0.25 * dt * dt,
                  diagonal, block, preconditioner, units};
    const int lanes = g->n_sites < kFewSites ? 4 : 1, threads = spread_threads(lanes * g->n_sites);
    (lanes == 4 ? scaling_sites<4> : scaling_sites<1>)<<<blocks_for(lanes * g->n_sites, threads), threads, 0,
                                                         (cudaStream_t)stream>>>(a);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

static int launch_trial_bonds(const dpf_graph *g, const dpf_stiffness *k, const dpf_history *h, const double *y,
                              const double *mid, const double *end, int want_end, const dpf_trial_out *out,
                              double *wrench, int *status, cudaStream_t st, double *linear = nullptr,
                              double *general = nullptr) {
    if (!g->n_bonds) return DPF_OK;
    TrialBondArgs a{};
    a.m = g->n_bonds;
    a.edges = g->edges;
    a.k = *k;
    a.h = *h;
    a.y = y;
    a.mid = mid;
    a.end = end;
    a.want_end = want_end;
    if (out) {
        a.n = out->n;
        a.ri = out->ri;
        a.rj = out->rj;
        a.normal_end = out->normal_end;
        a.offset_end = out->offset_end;
        a.fs_end = out->fs_end;
        a.mb_end = out->mb_end;
        a.fn_end = out->fn_end;
        a.mt_end = out->mt_end;
    }
    a.wrench = wrench;
    a.status = status;
    a.linear = linear;
    a.general = general;
    const int threads = spread_threads(g->n_bonds);
    if (linear)
        trial_bonds<true><<<blocks_for(g->n_bonds, threads), threads, 0, st>>>(a);
    else
        trial_bonds<false><<<blocks_for(g->n_bonds, threads), threads, 0, st>>>(a);
    return DPF_OK;
}

// Per-bond history arrays may be null (empty) when the graph has no bonds.
static bool history_ok(const dpf_history *h, int64_t n_bonds = 1) {
    return h && h->x && h->radii &&
           (n_bonds == 0 || (h->normal && h->offset && h->fn && h->fs && h->mt && h->mb));
}

int dpf_trial(const dpf_graph *g, const dpf_stiffness *k, const dpf_history *h, const double *y,
              const double *mid_positions, const double *end_positions, int want_end, const dpf_trial_out *out,
              double *wrench, int *status, void *stream) {
    if (!graph_ok(g) || !k || !history_ok(h, g->n_bonds) || !y || !out || !out->force || !status ||
        (g->n_bonds && !wrench))
        return DPF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    launch_trial_bonds(g, k, h, y, mid_positions, end_positions, want_end, out, wrench, status, st);
    SiteResidualArgs a{};
    a.n = g->n_sites;
    a.ptr = g->inc_ptr;
    a.inc = g->inc_bond;
    a.wrench = wrench;
    a.y = y;
    a.x = h->x;
    a.end = end_positions;
    a.force = out->force;
    a.x_end = want_end ? out->x_end : nullptr;
    a.status = status;
    const int threads = spread_threads(2 * g->n_sites);
    site_residual<<<blocks_for(2 * g->n_sites, threads), threads, 0, st>>>(a);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_commit_state(const dpf_graph *g, const dpf_stiffness *k, const dpf_history *h, const double *y,
                     const dpf_trial_out *out, int *status, void *stream) {
    if (!graph_ok(g) || !k || !history_ok(h, g->n_bonds) || !y || !out || !status) return DPF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    launch_trial_bonds(g, k, h, y, nullptr, nullptr, 1, out, nullptr, status, st);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

static int residual_launch(const dpf_graph *g, const dpf_stiffness *k, const dpf_history *h, const double *y,
                           const double *v, const double *external, const double *mass, const uint8_t *fixed,
                           double dt, const dpf_trial_out *trial, const double *preconditioner, const double *units,
                           double *residual, double *scaled, double *norms, double *wrench, double *partials,
                           int *status, double *linear, double *general, cudaStream_t st) {
    if (!graph_ok(g) || !k || !history_ok(h, g->n_bonds) || !y || !v || !external || !mass || !fixed || !residual ||
        !status || (g->n_bonds && !wrench) || (norms && !partials) || (preconditioner && !units))
        return DPF_ERR_ARGUMENT;
    launch_trial_bonds(g, k, h, y, nullptr, nullptr, 0, trial, wrench, status, st, linear, general);
    SiteResidualArgs a{};
    a.n = g->n_sites;
    a.ptr = g->inc_ptr;
    a.inc = g->inc_bond;
    a.wrench = wrench;
    a.y = y;
    a.x = h->x;
    a.force = trial ? trial->force : nullptr;
    a.v = v;
    a.external = external;
    a.mass = mass;
    a.fixed = fixed;
    a.dt = dt;
    a.half_dt2 = 0.5 * dt * dt;
    a.residual = residual;
    a.P = preconditioner;
    a.units = units;
    a.scaled = scaled;
    a.norms = norms;
    a.partials = partials;
    a.status = status;
    const int threads = reduce_threads(2 * g->n_sites);
    int grid = blocks_for(2 * g->n_sites, threads);
    if (grid > kMaxReduceBlocks) grid = kMaxReduceBlocks;
    site_residual<<<grid, threads, 0, st>>>(a);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_residual(const dpf_graph *g, const dpf_stiffness *k, const dpf_history *h, const double *y,
                 const double *v, const double *external, const double *mass, const uint8_t *fixed, double dt,
                 const dpf_trial_out *trial, const double *preconditioner, const double *units, double *residual,
                 double *scaled, double *norms, double *wrench, double *partials, int *status, void *stream) {
    return residual_launch(g, k, h, y, v, external, mass, fixed, dt, trial, preconditioner, units, residual, scaled,
                           norms, wrench, partials, status, nullptr, nullptr, (cudaStream_t)stream);
}

int dpf_jacobian_vector(const dpf_graph *g, const dpf_stiffness *k, const dpf_history *h, const double *y,
                        const double *direction, const double *mass, const uint8_t *fixed, double dt,
                        const double *units, const double *preconditioner, double *out, double *wrench,
                        void *stream) {
    if (!graph_ok(g) || !k || !history_ok(h, g->n_bonds) || !y || !direction || !mass || !fixed || !out ||
        (g->n_bonds && !wrench) || (preconditioner && !units))
        return DPF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    if (g->n_bonds) {
        JvpBondArgs a{g->n_bonds, g->edges, *k, *h, y, direction, units, wrench};
        const int threads = spread_threads(g->n_bonds);
        jvp_bonds<<<blocks_for(g->n_bonds, threads), threads, 0, st>>>(a);
    }
    SiteJvpArgs s{g->n_sites, g->inc_ptr, g->inc_bond, wrench, direction, units, mass, preconditioner, fixed,
                  0.5 * dt * dt, out, 1};
    const int threads = spread_threads(2 * g->n_sites);
    site_jvp<<<blocks_for(2 * g->n_sites, threads), threads, 0, st>>>(s);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_bond_setup(int64_t n_sites, int64_t n_bonds, const int64_t *edges, const double *points, const double *radii,
                   const double *areas, const double *contacts, const double *masses, double young, double shear,
                   const double *young_b, const double *shear_b, double *n, double *ri, double *rj, double *kn,
                   double *ks, double *kb, double *kt, double *offset, double *mass6, void *stream) {
    if (n_sites <= 0 || n_bonds < 0 || (n_bonds && (!edges || !areas || !n || !ri || !rj || !kn || !ks || !kb || !kt)) ||
        !points || !radii || (mass6 && !masses))
        return DPF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    if (n_bonds) {
        BondSetupArgs a{n_bonds, edges, points, radii, areas, contacts, young_b, shear_b, young, shear,
                        n, ri, rj, kn, ks, kb, kt, offset};
        bond_setup_kernel<<<blocks_for(n_bonds, kThreads), kThreads, 0, st>>>(a);
    }
    if (mass6) site_mass_kernel<<<blocks_for(n_sites, kThreads), kThreads, 0, st>>>(n_sites, masses, radii, mass6);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_loads(const dpf_graph *g, const dpf_history *h, double *out, double *wrench, void *stream) {
    if (!graph_ok(g) || !history_ok(h, g->n_bonds) || !out || (g->n_bonds && !wrench)) return DPF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    const int rc = dpf::loads_bonds_pass(g, h, wrench, st);
    if (rc) return rc;
    site_gather<<<blocks_for(2 * g->n_sites, kThreads), kThreads, 0, st>>>(g->n_sites, g->inc_ptr, g->inc_bond,
                                                                        wrench, out);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

}  // extern "C"

namespace dpf {

int loads_bonds_pass(const dpf_graph *g, const dpf_history *h, double *wrench, cudaStream_t st) {
    if (!graph_ok(g) || !history_ok(h, g->n_bonds) || (g->n_bonds && !wrench)) return DPF_ERR_ARGUMENT;
    if (g->n_bonds)
        loads_bonds<<<blocks_for(g->n_bonds, 128), 128, 0, st>>>(g->n_bonds, g->edges, *h, wrench, nullptr);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int residual_pass(const dpf_graph *g, const dpf_stiffness *k, const dpf_history *h, const double *y, const double *v,
                  const double *external, const double *mass, const uint8_t *fixed, double dt,
                  const dpf_trial_out *trial, const double *preconditioner, const double *units, double *residual,
                  double *norms, double *wrench, double *partials, int *status, double *linear, double *general,
                  cudaStream_t stream) {
    return residual_launch(g, k, h, y, v, external, mass, fixed, dt, trial, preconditioner, units, residual, nullptr,
                           norms, wrench, partials, status, linear, general, stream);
}

int jacobian_pass(const dpf_graph *g, const double *linear, const double *direction, const double *mass,
                  const uint8_t *fixed, double dt, const double *units, const double *preconditioner, double *out,
                  double *wrench, cudaStream_t stream) {
    if (g->n_bonds) {
        const int threads = spread_threads(g->n_bonds);
        jvp_linear_bonds<<<blocks_for(g->n_bonds, threads), threads, 0, stream>>>(g->n_bonds, g->edges, linear,
                                                                                  direction, wrench);
    }
    SiteJvpArgs s{g->n_sites, g->inc_ptr, g->inc_bond, wrench, direction, units, mass, preconditioner, fixed,
                  0.5 * dt * dt, out, 0};
    const int threads = spread_threads(2 * g->n_sites);
    site_jvp<<<blocks_for(2 * g->n_sites, threads), threads, 0, stream>>>(s);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

}  // namespace dpf

// ---------------------------------------------------------------------------
// K q without any allocation by anyone: the bond-wrench scratch lives in a
// file-scope device array instead of a caller buffer.  For callers that
// cannot call cudaMalloc (see dpf_stiffness_apply_static in dpf_gb300.h).

namespace {

__device__ __align__(256) double g_static_wrench[9 * DPF_STATIC_MAX_BONDS];

// Device address of g_static_wrench on the current device.  The host-side
// name is only a stand-in for the device symbol, so the address is looked up
// with cudaGetSymbolAddress while the device is current.  It is looked up on
// every call (cheap once the module is loaded) rather than cached, so a
// device reset or a re-created primary context never leaves a stale address.
int static_wrench(double **out) {
    void *ptr = nullptr;
    if (cudaGetSymbolAddress(&ptr, g_static_wrench) != cudaSuccess || !ptr) {
        cudaGetLastError();
        return DPF_ERR_CUDA;
    }
    *out = static_cast<double *>(ptr);
    return DPF_OK;
}

}  // namespace

extern "C" {

int64_t dpf_static_max_bonds(void) { return DPF_STATIC_MAX_BONDS; }

int dpf_stiffness_apply_static(const dpf_graph *g, const dpf_stiffness *k, const dpf_tangent *t, const double *q,
                               double *out, void *stream) {
    if (!graph_ok(g) || !k || !t || !q || !out) return DPF_ERR_ARGUMENT;
    if (g->n_bonds > DPF_STATIC_MAX_BONDS) return DPF_ERR_TOO_LARGE;
    double *wrench = nullptr;
    const int rc = static_wrench(&wrench);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    // Every bond slot read by site_gather is written by stiffness_bonds first
    // in the same call, so the array needs no clearing between calls.
    if (g->n_bonds) {
        StiffnessBondArgs a{g->n_bonds, g->edges, *k, *t, q, wrench};
        stiffness_bonds<<<blocks_for(g->n_bonds, kThreads), kThreads, 0, st>>>(a);
    }
    site_gather<<<blocks_for(2 * g->n_sites, kThreads), kThreads, 0, st>>>(g->n_sites, g->inc_ptr, g->inc_bond,
                                                                        wrench, out);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

}  // extern "C"
