// Adjoint of the rate-law implicit step (implicit-function theorem).
//
// The per-bond constitutive trial (experiments/bonded_dem_finite_gpu.py:87-116:
// midpoint wrench and end-of-step history) is differentiated by hand, in
// reverse: bond_reverse contracts given adjoints of its outputs with its
// derivative in every input, at three to four times the trial's own operations.
//   * dpf_adjoint_bond_vjp returns input adjoints per bond (history,
//     stiffness) and per site (increment, position; a deterministic incidence
//     gather) for output adjoints (wrench adjoints from a site vector,
//     end-history adjoints per bond);
//   * dpf_adjoint_local_jacobian stores B_b = d[F, T_i, T_j]/d[y_i, y_j] (9 x 12)
//     per bond, so J^T lambda costs one sparse transposed product;
//   * dpf_adjoint_apply_jt applies J^T (free rows) for the adjoint Krylov solve.
#include "common.cuh"
#include "internal.cuh"

namespace dpf {
namespace adj {

// ---- the transport and its reverse ---------------------------------------------

// transport (bonded_dem_finite_gpu.py:22-32) as the reference writes it, for
// any n0 (its adjoint in n0 has a radial part that unit normals never see).
// Torch's conventions: the clamp of the cosine has derivative zero outside
// [-1, 1], the floor of |n0 + n1| derivative zero below it.
struct Rot {
    d3 n0, n1, k, b, spin;
    double inv1pc, inv_length, c, s;
    bool inside, floored;
};

__device__ __forceinline__ Rot make_rot(d3 n0, d3 n1, d3 spin) {
    Rot t;
    t.n0 = n0;
    t.n1 = n1;
    t.spin = spin;
    t.k = cross(n0, n1);
    const double raw = dot(n0, n1);
    t.inside = !(raw < -1.0 || raw > 1.0);
    t.inv1pc = 1.0 / (1.0 + fmin(fmax(raw, -1.0), 1.0));
    const d3 sum = n0 + n1;
    const double length = norm(sum);
    t.floored = !(length > 1e-12);
    t.inv_length = 1.0 / fmax(length, 1e-12);
    t.b = t.inv_length * sum;
    sincos_small(dot(spin, t.b), t.s, t.c);
    return t;
}

// v after the shortest arc, before the spin
__device__ __forceinline__ d3 arc(const Rot &t, d3 v, d3 &kv, d3 &kkv) {
    kv = cross(t.k, v);
    kkv = cross(t.k, kv);
    return axpy(t.inv1pc, kkv, v + kv);
}

__device__ __forceinline__ d3 rot_apply(const Rot &t, d3 v) {
    d3 kv, kkv;
    const d3 o = arc(t, v, kv, kkv);
    return axpy(t.c, o, axpy(t.s, cross(t.n1, o), ((1.0 - t.c) * dot(t.n1, o)) * t.n1));
}

// Adjoints of a transport's own quantities, summed over the vectors it carries.
struct RotBar {
    d3 k, n1;
    double c, s, inv;
};

// Adjoint of v for the adjoint g of rot_apply(t, v); adds to the transport's.
__device__ __forceinline__ d3 rot_reverse(const Rot &t, d3 v, d3 g, RotBar &bar) {
    d3 kv, kkv;
    const d3 o = arc(t, v, kv, kkv);
    const double p = dot(t.n1, o), gn = dot(g, t.n1), versine = 1.0 - t.c;
    const d3 go = cross(o, g);
    bar.c += dot(g, o) - p * gn;
    bar.s += dot(t.n1, go);
    bar.n1 = axpy(t.s, go, axpy(versine * p, g, axpy(versine * gn, o, bar.n1)));
    const d3 ob = axpy(t.c, g, axpy(t.s, cross(g, t.n1), (versine * gn) * t.n1));
    bar.inv = dot_add(bar.inv, ob, kkv);
    const d3 kvb = axpy(t.inv1pc, cross(ob, t.k), ob);
    bar.k = cross_add(axpy(t.inv1pc, cross(kv, ob), bar.k), v, kvb);
    return cross_add(ob, kvb, t.k);
}

__device__ __forceinline__ void rot_finish(const Rot &t, const RotBar &bar, d3 &n0b, d3 &n1b, d3 &spinb) {
    const double angle = bar.s * t.c - bar.c * t.s;
    spinb = axpy(angle, t.b, spinb);
    d3 sum = (angle * t.inv_length) * t.spin;
    if (!t.floored) sum = axpy(-dot(t.b, sum), t.b, sum);
    const double cosine = t.inside ? -bar.inv * t.inv1pc * t.inv1pc : 0.0;
    n0b = cross_add(axpy(cosine, t.n1, n0b + sum), t.n1, bar.k);
    n1b = cross_add(axpy(cosine, t.n0, n1b + sum + bar.n1), bar.k, t.n0);
}

// ---- the trial's reverse -----------------------------------------------------------

struct BondSide {
    d3 u, w, x;
};

struct Bond {
    BondSide i, j;
    double rad;        // (radius_i - radius_j)/2
    d3 normal, offset, fs, mb;
    double fn, mt, kn, ks, kb, kt;
};

// Adjoints of the outputs: the midpoint wrench [F, T_i, T_j] (site i gets
// (F, T_i), site j (-F, T_j)) and the end history.
struct OutBar {
    d3 f, ti, tj;
    d3 normal, offset, fs, mb;
    double fn, mt;
};

// Adjoints of the inputs.  Returned in place: i, j (u, w, x) and the history
// and stiffness of the bond.  kEnd: the end history has adjoints.
template <bool kEnd>
__device__ __forceinline__ void bond_reverse(const Bond &a, const OutBar &g, Bond &bar) {
    const d3 mi = axpy(0.5, a.i.u, a.i.x), mj = axpy(0.5, a.j.u, a.j.x);
    const d3 dm = mj - mi;
    const double inv_m = rsqrt(dot(dm, dm));
    const d3 n = inv_m * dm;
    const d3 spin = 0.25 * (a.i.w + a.j.w);
    const Rot r1 = make_rot(a.normal, n, spin);
    const bool flat = is_zero(a.offset);
    const d3 offset = flat ? a.offset : rot_apply(r1, a.offset);
    const d3 fs0 = rot_apply(r1, a.fs), mb0 = rot_apply(r1, a.mb);
    const d3 lever = axpy(a.rad, n, offset);
    const d3 ri = axpy(0.5, dm, lever), rj = axpy(-0.5, dm, lever);
    const d3 du = cross_sub(cross_add(a.j.u - a.i.u, a.j.w, rj), a.i.w, ri), dw = a.j.w - a.i.w;
    const double dn = dot(du, n), twist = dot(dw, n);
    const d3 slide = axpy(-dn, n, du), bend = axpy(-twist, n, dw);
    const double fm = fma(0.5 * a.kn, dn, a.fn), mm = fma(0.5 * a.kt, twist, a.mt);
    const d3 f = axpy(fm, n, axpy(0.5 * a.ks, slide, fs0));
    // wrench: T_i = r_i x f + c, T_j = -(r_j x f) - c, f = fm n + (fs0 + fs1)/2, c likewise
    const d3 cb = g.ti - g.tj;
    const d3 fb = cross_sub(cross_add(g.f, g.ti, ri), g.tj, rj);
    d3 rib = cross(f, g.ti), rjb = cross(g.tj, f);
    const double fmb = dot(fb, n), mmb = dot(cb, n);
    d3 nb = axpy(fm, fb, mm * cb);
    d3 fs0b = 0.5 * fb, fs1b = fs0b, mb0b = 0.5 * cb, mb1b = mb0b, offsetb = mk(0.0, 0.0, 0.0), spinb = offsetb;
    double fn1b = 0.5 * fmb, mt1b = 0.5 * mmb;
    bar.fn = fn1b;
    bar.mt = mt1b;
    bar.i.x = bar.j.x = mk(0.0, 0.0, 0.0);
    if (kEnd) {
        const d3 de = (a.j.x + a.j.u) - (a.i.x + a.i.u);
        const double inv_e = rsqrt(dot(de, de));
        const d3 ne = inv_e * de;
        const Rot r2 = make_rot(n, ne, spin);
        RotBar rb{};
        fs1b = fs1b + rot_reverse(r2, axpy(a.ks, slide, fs0), g.fs, rb);
        mb1b = mb1b + rot_reverse(r2, axpy(a.kb, bend, mb0), g.mb, rb);
        offsetb = rot_reverse(r2, offset, g.offset, rb);
        d3 neb = g.normal;
        rot_finish(r2, rb, nb, neb, spinb);
        const d3 eb = inv_e * axpy(-dot(ne, neb), ne, neb);
        bar.j.x = eb;
        bar.i.x = -eb;
        fn1b += g.fn;
        mt1b += g.mt;
        bar.fn += g.fn;
        bar.mt += g.mt;
    }
    bar.j.u = bar.j.x;
    bar.i.u = bar.i.x;
    // history update: fn1 = fn + kn dn, fs1 = fs0 + ks slide and the couple's
    bar.fn += 0.5 * fmb;
    bar.mt += 0.5 * mmb;
    bar.kn = dn * fn1b;
    bar.kt = twist * mt1b;
    fs0b = fs0b + fs1b;
    mb0b = mb0b + mb1b;
    bar.ks = dot(slide, fs1b);
    bar.kb = dot(bend, mb1b);
    const d3 sb = a.ks * fs1b, bb = a.kb * mb1b;
    const double dnb = a.kn * fn1b - dot(sb, n), twistb = a.kt * mt1b - dot(bb, n);
    nb = axpy(-dn, sb, axpy(dnb, du, axpy(-twist, bb, axpy(twistb, dw, nb))));
    const d3 dub = axpy(dnb, n, sb), dwb = axpy(twistb, n, bb);
    // du = u_j - u_i + w_j x r_j - w_i x r_i, dw = w_j - w_i
    bar.j.w = cross_add(dwb, rj, dub);
    bar.i.w = -cross_add(dwb, ri, dub);
    rjb = cross_add(rjb, dub, a.j.w);
    rib = cross_sub(rib, dub, a.i.w);
    // r_i = dm/2 + rad n + offset, r_j = -dm/2 + rad n + offset
    const d3 leverb = rib + rjb;
    nb = axpy(a.rad, leverb, nb);
    offsetb = offsetb + leverb;
    RotBar rb{};
    bar.fs = rot_reverse(r1, a.fs, fs0b, rb);
    bar.mb = rot_reverse(r1, a.mb, mb0b, rb);
    bar.offset = rot_reverse(r1, a.offset, offsetb, rb);
    bar.normal = mk(0.0, 0.0, 0.0);
    rot_finish(r1, rb, bar.normal, nb, spinb);
    const d3 dmb = axpy(0.5, rib - rjb, inv_m * axpy(-dot(n, nb), n, nb));
    bar.j.x = bar.j.x + dmb;
    bar.i.x = bar.i.x - dmb;
    bar.j.u = axpy(0.5, dmb, bar.j.u + dub);
    bar.i.u = axpy(-0.5, dmb, bar.i.u - dub);
    bar.j.w = axpy(0.25, spinb, bar.j.w);
    bar.i.w = axpy(0.25, spinb, bar.i.w);
}

struct BondSources {
    const int64_t *edges;
    const double *y, *x, *radii, *normal, *offset, *fn, *fs, *mt, *mb, *kn, *ks, *kb, *kt;
};

__device__ __forceinline__ Bond load_bond(const BondSources &s, int64_t b, int64_t &i, int64_t &j) {
    edge(s.edges, b, i, j);
    Bond a;
    a.i = {ld3(s.y + 6 * i), ld3(s.y + 6 * i + 3), ld3(s.x, i)};
    a.j = {ld3(s.y + 6 * j), ld3(s.y + 6 * j + 3), ld3(s.x, j)};
    a.rad = 0.5 * (s.radii[i] - s.radii[j]);
    a.normal = ld3(s.normal, b);
    a.offset = ld3(s.offset, b);
    a.fs = ld3(s.fs, b);
    a.mb = ld3(s.mb, b);
    a.fn = s.fn[b];
    a.mt = s.mt[b];
    a.kn = s.kn[b];
    a.ks = s.ks[b];
    a.kb = s.kb[b];
    a.kt = s.kt[b];
    return a;
}

// Column `dir` (entries 0 .. 8) of a bond's B (9 x 12, row-major by output).
__device__ __forceinline__ void put_column(double *B, int dir, double sign, d3 f, d3 ti, d3 tj) {
    B[dir] = sign * f.x;
    B[12 + dir] = sign * f.y;
    B[24 + dir] = sign * f.z;
    B[36 + dir] = sign * ti.x;
    B[48 + dir] = sign * ti.y;
    B[60 + dir] = sign * ti.z;
    B[72 + dir] = sign * tj.x;
    B[84 + dir] = sign * tj.y;
    B[96 + dir] = sign * tj.z;
}

// The same block by rows, one reverse pass an output: for committed normals
// that are not unit vectors.
__device__ __noinline__ void jacobian_rows(const Bond &a, double *B) {
    for (int o = 0; o < 9; ++o) {
        OutBar g{};
        const d3 e = mk(o % 3 == 0 ? 1.0 : 0.0, o % 3 == 1 ? 1.0 : 0.0, o % 3 == 2 ? 1.0 : 0.0);
        (o < 3 ? g.f : o < 6 ? g.ti : g.tj) = e;
        Bond bar;
        bond_reverse<false>(a, g, bar);
        st3(B + 12 * o, bar.i.u);
        st3(B + 12 * o + 3, bar.i.w);
        st3(B + 12 * o + 6, bar.j.u);
        st3(B + 12 * o + 9, bar.j.w);
    }
}

// B_b (9 x 12, row-major by output) for every bond, bound by the float64 pipe.
// The wrench depends on u_i and u_j through u_j - u_i alone (three columns,
// the others their negatives), and on a rotation through its lever and one
// scalar, the spin angle: 990 float64 instructions a bond (ncu) against twelve
// forward-mode passes of the whole trial at 1,200 each.
// 8k sites / 55k bonds: 978 -> 106 us.
__global__ void __launch_bounds__(128) local_jacobian_kernel(int64_t m, BondSources s, double *B) {
    const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (b >= m) return;
    int64_t i, j;
    const Bond a = load_bond(s, b, i, j);
    double *out = B + 108 * b;
    if (!is_unit(a.normal)) {
        jacobian_rows(a, out);
        return;
    }
    const d3 dm = axpy(0.5, a.j.u - a.i.u, a.j.x - a.i.x);
    const double inv = rsqrt(dot(dm, dm));
    const d3 n = inv * dm, spin = 0.25 * (a.i.w + a.j.w);
    int flags = 0;
    const Turn t = make_turn(a.normal, n, spin, flags);
    const d3 offset = apply(t, a.offset), fs0 = apply(t, a.fs), mb0 = apply(t, a.mb);
    const d3 lever = axpy(a.rad, n, offset);
    const d3 ri = axpy(0.5, dm, lever), rj = axpy(-0.5, dm, lever);
    const d3 du = cross_sub(cross_add(a.j.u - a.i.u, a.j.w, rj), a.i.w, ri), dw = a.j.w - a.i.w;
    const double hkn = 0.5 * a.kn, hks = 0.5 * a.ks, hkb = 0.5 * a.kb, hkt = 0.5 * a.kt;
    const double nd = dot(du, n), tw = dot(dw, n);
    const double fn_mid = fma(hkn, nd, a.fn), mt_mid = fma(hkt, tw, a.mt);
    const d3 f = axpy(fn_mid, n, axpy(hks, axpy(-nd, n, du), fs0));
    const d3 zero = mk(0.0, 0.0, 0.0);
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
        const d3 e = mk(c == 0 ? 1.0 : 0.0, c == 1 ? 1.0 : 0.0, c == 2 ? 1.0 : 0.0);
        const double nc = c == 0 ? n.x : c == 1 ? n.y : n.z, sc = c == 0 ? t.sum.x : c == 1 ? t.sum.y : t.sum.z;
        // u_j - u_i along e
        const d3 dn = (0.5 * inv) * axpy(-nc, n, e);
        const d3 rate = turn_rate(t, n, dn, spin, zero);
        const d3 dlever = cross_add(a.rad * dn, rate, offset);
        const d3 dri = axpy(0.25, e, dlever), drj = axpy(-0.25, e, dlever);
        const d3 ddu = cross_sub(cross_add(e, a.j.w, drj), a.i.w, dri);
        const double dnd = dot_add(dot(du, dn), ddu, n), dtw = dot(dw, dn);
        const d3 df = axpy(fn_mid - hks * nd, dn, axpy((hkn - hks) * dnd, n, cross_add(hks * ddu, rate, fs0)));
        const d3 dc = axpy(mt_mid - hkb * tw, dn, axpy((hkt - hkb) * dtw, n, cross(rate, mb0)));
        const d3 ti = cross_add(cross_add(dc, dri, f), ri, df), tj = cross_sub(cross_sub(-dc, drj, f), rj, df);
        put_column(out, c, -1.0, df, ti, tj);
        put_column(out, 6 + c, 1.0, df, ti, tj);
        // w_i and w_j along e: the spin angle turns by r sum.e/4 about n, the lever sweeps
        const double turn = 0.25 * t.r * sc;
        const d3 about = turn * n, doffset = cross(about, offset), swept = cross(dw, doffset);
        const d3 dfs = cross(about, fs0), dmb = cross(about, mb0), arm = cross(doffset, f);
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const double sign = side ? 1.0 : -1.0;
            const d3 wdu = side ? cross_add(swept, e, rj) : cross_sub(swept, e, ri);
            const d3 wdf = axpy((hkn - hks) * dot(wdu, n), n, axpy(hks, wdu, dfs));
            const d3 wdc = axpy(sign * hkb, e, axpy(sign * (hkt - hkb) * nc, n, dmb));
            put_column(out, 3 + 6 * side + c, 1.0, wdf, cross_add(wdc + arm, ri, wdf),
                       cross_sub(-(wdc + arm), rj, wdf));
        }
    }
}

// Per-bond adjoints of the 9 wrench outputs from a site vector lam (N, 6):
// F -> lam_i[0:3] - lam_j[0:3], T_i -> lam_i[3:6], T_j -> lam_j[3:6].
__device__ __forceinline__ void wrench_adjoint(const double *lam, int64_t i, int64_t j, double w[9]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        w[c] = lam[6 * i + c] - lam[6 * j + c];
        w[3 + c] = lam[6 * i + 3 + c];
        w[6 + c] = lam[6 * j + 3 + c];
    }
}

// J^T product, bond pass: slots[b] = [ (B_b^T w)_i (6), (B_b^T w)_j (6) ].
__global__ void __launch_bounds__(kThreads) jt_bonds_kernel(int64_t m, const int64_t *edges, const double *B,
                                                            const double *lam, double *slots) {
    const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (b >= m) return;
    int64_t i, j;
    edge(edges, b, i, j);
    double w[9];
    wrench_adjoint(lam, i, j, w);
    const double *Bb = B + 108 * b;
#pragma unroll
    for (int k = 0; k < 12; ++k) {
        double acc = 0.0;
#pragma unroll
        for (int o = 0; o < 9; ++o) acc += w[o] * Bb[12 * o + k];
        slots[12 * b + k] = acc;
    }
}

// Three of the numbers of site s summed over its per-bond slots of width 2K
// ([i-side K, j-side K]): those from `first` on.  A site's lanes take three
// each, so that the loads of an incidence are contiguous over them.
template <int K>
__device__ __forceinline__ d3 gather_slots(const int32_t *ptr, const int32_t *inc, const double *slots, int64_t s,
                                           int first) {
    d3 acc = mk(0.0, 0.0, 0.0);
    const int e1 = ptr[s + 1];
#pragma unroll 4
    for (int e = ptr[s]; e < e1; ++e) {
        const int v = inc[e], j = v >> 31;
        acc = acc + ld3(slots + 2 * K * (int64_t)(v ^ j) - (int64_t)K * j + first);
    }
    return acc;
}

// out = M lam - h sum B^T w on free rows, lam on fixed rows (lam's fixed rows are
// zero); times units when given.  Two lanes a site.
__global__ void __launch_bounds__(128) jt_sites_kernel(int64_t n, const int32_t *ptr, const int32_t *inc,
                                                       const double *slots, const double *mass, const uint8_t *fixed,
                                                       double half_dt2, const double *lam, const double *units,
                                                       double *out) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, s = t / 2;
    if (s >= n) return;
    const d3 acc = gather_slots<6>(ptr, inc, slots, s, 3 * (int)(t & 1)), l = ld3(lam, t), m = ld3(mass, t);
    d3 o = fixed[s] ? l : mk(m.x * l.x - half_dt2 * acc.x, m.y * l.y - half_dt2 * acc.y, m.z * l.z - half_dt2 * acc.z);
    if (units) {
        const d3 u = ld3(units, t);
        o = mk(u.x * o.x, u.y * o.y, u.z * o.z);
    }
    st3(out, t, o);
}

// lam = P (mu / units): from the scaled adjoint system's unknown to the
// multiplier.  Two lanes a site.  The scaled system's operator is three launches
// (this, the bonds' transposed products, the sites' sums with the units folded in)
// and its preconditioner one (the elastic PCG reads vector / units and writes
// units (block x)); with the divisions, products and 6x6 products as separate
// passes over the sites an 8k-site, 8-step rollout with its gradient took 13.4 ms,
// with them folded in 11.1 ms.
__global__ void __launch_bounds__(128) multiplier_kernel(int64_t n, const double *P, const double *units,
                                                         const double *mu, double *lam) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, s = t / 2;
    const bool live = s < n;
    const d3 v = live ? over_units(ld3(mu, t), ld3(units, t)) : mk(0.0, 0.0, 0.0), other = other_half(v);
    if (live) st3(lam, t, half_rows(P + 36 * s, (int)(t & 1), v, other));
}

// The site passes around the adjoint's bond passes and its Krylov solve, two lanes a
// site, each in place of five or six passes over the sites' vectors (an 8k-site,
// 3-step gradient: 10.9 -> 9.9 ms with what fgmres in newton.py leaves out).
//
// The commit map: y_bar = [x_bar, 0] + (2/dt) v_bar, x_next = x_bar + g, v_next = -v_bar.
__global__ void __launch_bounds__(128) commit_map_kernel(int64_t n, double two_over_dt, const double *x_bar,
                                                         const double *v_bar, const double *g, double *y_bar,
                                                         double *x_next, double *v_next) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, s = t / 2;
    if (s >= n) return;
    const d3 v = ld3(v_bar, t);
    d3 y = two_over_dt * v;
    if (!(t & 1)) {
        const d3 x = ld3(x_bar, s);
        y = y + x;
        st3(x_next, s, x + ld3(g, s));
    }
    st3(y_bar, t, y);
    st3(v_next, t, -v);
}

// rhs = units y_bar, zero rows on fixed sites
__global__ void __launch_bounds__(128) adjoint_rhs_kernel(int64_t n, const double *y_bar, const double *units,
                                                          const uint8_t *fixed, double *rhs) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, s = t / 2;
    if (s >= n) return;
    const d3 y = ld3(y_bar, t), u = ld3(units, t);
    st3(rhs, t, fixed[s] ? mk(0.0, 0.0, 0.0) : mk(u.x * y.x, u.y * y.y, u.z * y.z));
}

// load_bar = dt^2/2 lam, v_next += dt mass lam
__global__ void __launch_bounds__(128) adjoint_loads_kernel(int64_t n, double dt, double half_dt2, const double *mass,
                                                            const double *lam, double *load_bar, double *v_next) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= 2 * n) return;
    const d3 l = ld3(lam, t), m = ld3(mass, t), v = ld3(v_next, t);
    st3(load_bar, t, half_dt2 * l);
    st3(v_next, t, mk(fma(dt * m.x, l.x, v.x), fma(dt * m.y, l.y, v.y), fma(dt * m.z, l.z, v.z)));
}

// Input adjoints of one bond for output adjoints: wrench part = coef * (wrench
// adjoint of lam), end part = end-history adjoints of the bond (optional).
// Per-bond inputs: history adjoints (14: normal 3, offset 3, fn, fs 3, mt, mb 3,
// the end-history layout) ADDED to hist_adj, stiffness adjoints (kn ks kb kt)
// ADDED to stiff_adj; per-site inputs (y_i, y_j, x_i, x_j) written to slots
// [i: y 6, x 3 | j: y 6, x 3] (18 per bond) for the site gather.
struct VjpArgs {
    int64_t m;
    BondSources s;
    const double *lam;        // (N, 6) or null
    double coef;
    const double *end_adj;    // (M, 14) or null
    int with_increment;       // 0: the increment's slots are zero
    double *hist_adj;         // (M, 14) accumulated
    double *stiff_adj;        // (M, 4) accumulated
    double *slots;            // (M, 18) written
};

// One reverse pass of the trial a bond (by ncu 1,210 float64 instructions with
// end-history adjoints, 740 without, at 85-87% of the float64 pipe) where one
// forward-mode pass for each of 36 inputs was taken before.  8k sites / 55k bonds:
// 4.35 ms -> 0.13 ms.
template <bool kEnd>
__global__ void __launch_bounds__(128) vjp_kernel(VjpArgs a) {
    const int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (b >= a.m) return;
    int64_t i, j;
    const Bond in = load_bond(a.s, b, i, j);
    OutBar g{};
    if (a.lam) {
        const double *li = a.lam + 6 * i, *lj = a.lam + 6 * j;
        g.f = a.coef * (ld3(li) - ld3(lj));
        g.ti = a.coef * ld3(li + 3);
        g.tj = a.coef * ld3(lj + 3);
    }
    if (kEnd) {
        const double *e = a.end_adj + 14 * b;
        g.normal = ld3(e);
        g.offset = ld3(e + 3);
        g.fn = e[6];
        g.fs = ld3(e + 7);
        g.mt = e[10];
        g.mb = ld3(e + 11);
    }
    Bond bar;
    bond_reverse<kEnd>(in, g, bar);
    const d3 zero = mk(0.0, 0.0, 0.0);
    double *sl = a.slots + 18 * b;
    st3(sl, a.with_increment ? bar.i.u : zero);
    st3(sl + 3, a.with_increment ? bar.i.w : zero);
    st3(sl + 6, bar.i.x);
    st3(sl + 9, a.with_increment ? bar.j.u : zero);
    st3(sl + 12, a.with_increment ? bar.j.w : zero);
    st3(sl + 15, bar.j.x);
    double *ha = a.hist_adj + 14 * b;
    st3(ha, ld3(ha) + bar.normal);
    st3(ha + 3, ld3(ha + 3) + bar.offset);
    ha[6] += bar.fn;
    st3(ha + 7, ld3(ha + 7) + bar.fs);
    ha[10] += bar.mt;
    st3(ha + 11, ld3(ha + 11) + bar.mb);
    double *ka = a.stiff_adj + 4 * b;
    ka[0] += bar.kn;
    ka[1] += bar.ks;
    ka[2] += bar.kb;
    ka[3] += bar.kt;
}

// Site adjoints from the VJP slots: y_adj (N, 6) and x_adj (N, 3), ADDED.  Three
// lanes a site.
__global__ void __launch_bounds__(96) vjp_sites_kernel(int64_t n, const int32_t *ptr, const int32_t *inc,
                                                       const double *slots, double *y_adj, double *x_adj) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, s = t / 3;
    const int part = (int)(t - 3 * s);
    if (s >= n || !(part < 2 ? y_adj : x_adj)) return;
    double *out = part < 2 ? y_adj + 6 * s + 3 * part : x_adj + 3 * s;
    st3(out, ld3(out) + gather_slots<9>(ptr, inc, slots, s, 3 * part));
}

inline int blocks_for(int64_t n, int threads) { return (int)((n + threads - 1) / threads); }

}  // namespace adj
}  // namespace dpf

using namespace dpf;
using namespace dpf::adj;

extern "C" {

static bool adj_ok(const dpf_graph *g, const dpf_stiffness *k, const dpf_history *h, const double *y) {
    return g && g->n_sites > 0 && g->inc_ptr && (g->n_bonds == 0 || (g->edges && g->inc_bond)) && k && h && h->x &&
           h->radii && h->normal && h->offset && h->fn && h->fs && h->mt && h->mb && y;
}

static BondSources sources(const dpf_graph *g, const dpf_stiffness *k, const dpf_history *h, const double *y) {
    return BondSources{g->edges, y, h->x, h->radii, h->normal, h->offset, h->fn, h->fs, h->mt, h->mb,
                       k->kn, k->ks, k->kb, k->kt};
}

int64_t dpf_adjoint_jacobian_doubles(int64_t n_bonds) { return 108 * n_bonds; }

int64_t dpf_adjoint_slot_doubles(int64_t n_bonds) { return 18 * n_bonds; }

int dpf_adjoint_local_jacobian(const dpf_graph *g, const dpf_stiffness *k, const dpf_history *h, const double *y,
                               double *jacobian, void *stream) {
    if (!adj_ok(g, k, h, y) || (g->n_bonds && !jacobian)) return DPF_ERR_ARGUMENT;
    if (g->n_bonds)
        local_jacobian_kernel<<<blocks_for(g->n_bonds, spread_threads(g->n_bonds)), spread_threads(g->n_bonds), 0,
                                (cudaStream_t)stream>>>(g->n_bonds, sources(g, k, h, y), jacobian);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

static int apply_jt(const dpf_graph *g, const double *jacobian, const double *mass, const uint8_t *fixed, double dt,
                    const double *lam, const double *units, double *out, double *slots, void *stream) {
    if (!g || g->n_sites <= 0 || !mass || !fixed || !lam || !out || (g->n_bonds && (!jacobian || !slots)))
        return DPF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    if (g->n_bonds)
        jt_bonds_kernel<<<blocks_for(g->n_bonds, kThreads), kThreads, 0, st>>>(g->n_bonds, g->edges, jacobian, lam,
                                                                               slots);
    const int threads = spread_threads(2 * g->n_sites);
    jt_sites_kernel<<<blocks_for(2 * g->n_sites, threads), threads, 0, st>>>(
        g->n_sites, g->inc_ptr, g->inc_bond, slots, mass, fixed, 0.5 * dt * dt, lam, units, out);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_adjoint_apply_jt(const dpf_graph *g, const double *jacobian, const double *mass, const uint8_t *fixed,
                         double dt, const double *lam, double *out, double *slots, void *stream) {
    return apply_jt(g, jacobian, mass, fixed, dt, lam, nullptr, out, slots, stream);
}

int dpf_adjoint_multiplier(int64_t n_sites, const double *preconditioner, const double *units, const double *mu,
                           double *lam, void *stream) {
    if (n_sites <= 0 || !preconditioner || !units || !mu || !lam) return DPF_ERR_ARGUMENT;
    const int threads = spread_threads(2 * n_sites);
    multiplier_kernel<<<blocks_for(2 * n_sites, threads), threads, 0, (cudaStream_t)stream>>>(
        n_sites, preconditioner, units, mu, lam);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_adjoint_commit_map(int64_t n_sites, double dt, const double *x_bar, const double *v_bar, const double *g,
                           double *y_bar, double *x_next, double *v_next, void *stream) {
    if (n_sites <= 0 || !(dt > 0.0) || !x_bar || !v_bar || !g || !y_bar || !x_next || !v_next)
        return DPF_ERR_ARGUMENT;
    const int threads = spread_threads(2 * n_sites);
    commit_map_kernel<<<blocks_for(2 * n_sites, threads), threads, 0, (cudaStream_t)stream>>>(
        n_sites, 2.0 / dt, x_bar, v_bar, g, y_bar, x_next, v_next);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_adjoint_rhs(int64_t n_sites, const double *y_bar, const double *units, const uint8_t *fixed, double *rhs,
                    void *stream) {
    if (n_sites <= 0 || !y_bar || !units || !fixed || !rhs) return DPF_ERR_ARGUMENT;
    const int threads = spread_threads(2 * n_sites);
    adjoint_rhs_kernel<<<blocks_for(2 * n_sites, threads), threads, 0, (cudaStream_t)stream>>>(n_sites, y_bar, units,
                                                                                            fixed, rhs);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_adjoint_loads(int64_t n_sites, double dt, const double *mass, const double *lam, double *load_bar,
                      double *v_next, void *stream) {
    if (n_sites <= 0 || !mass || !lam || !load_bar || !v_next) return DPF_ERR_ARGUMENT;
    const int threads = spread_threads(2 * n_sites);
    adjoint_loads_kernel<<<blocks_for(2 * n_sites, threads), threads, 0, (cudaStream_t)stream>>>(
        n_sites, dt, 0.5 * dt * dt, mass, lam, load_bar, v_next);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

int dpf_adjoint_operator(const dpf_graph *g, const double *jacobian, const double *mass, const uint8_t *fixed,
                         const double *preconditioner, const double *units, double dt, const double *mu, double *out,
                         double *lam, double *slots, void *stream) {
    if (!g || !units) return DPF_ERR_ARGUMENT;
    const int rc = dpf_adjoint_multiplier(g->n_sites, preconditioner, units, mu, lam, stream);
    return rc ? rc : apply_jt(g, jacobian, mass, fixed, dt, lam, units, out, slots, stream);
}

int dpf_adjoint_precondition(const dpf_graph *g, const dpf_stiffness *k, const dpf_tangent *t, const double *mass,
                             const uint8_t *fixed, const double *block, const double *preconditioner,
                             const double *units, const double *vector, double dt, double tolerance,
                             int max_iterations, double *out, int *iterations, double *wrench, double *workspace,
                             unsigned *barrier, int *status, void *stream) {
    return elastic_pass(g, k, t, mass, fixed, block, preconditioner, units, vector, dt, tolerance, max_iterations, out,
                        iterations, wrench, workspace, barrier, nullptr, status, kElasticT, (cudaStream_t)stream);
}

int dpf_adjoint_bond_vjp(const dpf_graph *g, const dpf_stiffness *k, const dpf_history *h, const double *y,
                         const double *lam, double coef, const double *end_adjoint, int with_increment,
                         double *history_adjoint, double *stiffness_adjoint, double *y_adjoint, double *x_adjoint,
                         double *slots, void *stream) {
    if (!adj_ok(g, k, h, y) || (g->n_bonds && (!slots || !history_adjoint || !stiffness_adjoint)))
        return DPF_ERR_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    if (g->n_bonds) {
        VjpArgs a{g->n_bonds, sources(g, k, h, y), lam, coef, end_adjoint, with_increment ? 1 : 0,
                  history_adjoint, stiffness_adjoint, slots};
        const int threads = spread_threads(g->n_bonds);
        (end_adjoint ? vjp_kernel<true> : vjp_kernel<false>)<<<blocks_for(g->n_bonds, threads), threads, 0, st>>>(a);
    }
    if ((y_adjoint || x_adjoint) && g->n_bonds)
        vjp_sites_kernel<<<blocks_for(3 * g->n_sites, 96), 96, 0, st>>>(
            g->n_sites, g->inc_ptr, g->inc_bond, slots, with_increment ? y_adjoint : nullptr, x_adjoint);
    DPF_CHECK_LAUNCH();
    return DPF_OK;
}

}  // extern "C"
