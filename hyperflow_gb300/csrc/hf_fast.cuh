// The MUSCL-Hancock predictor, the HLLC face and the update of ordinary states, with every product,
// quotient and root on the integer pipes and without a branch per operation.
//
// What bounds the stencils is the FP64 pipe: a warp's FP64 addition or product holds it for 19 cycles of the SM
// (measured; a fused multiply-add 16), the time of 76 instructions on the other pipes.  With
// divisions and roots on the integer pipes the step was at that bound, two fifths of its FP64
// instructions products; an exact product costs 29 integer instructions (prod).  A range check and a
// branch per product cost half as much again and cut the code into pieces too short to overlap, so the
// functions here compute straight through as if every value were in a comfortable range, note on the
// way whether one was not (Window, two instructions a value), and the caller repeats such an item with
// the general code.  Halvings are folded into FP64 fused multiply-adds (0.5 x is exact, so the fused
// result is the rounded sum itself), which takes them off the integer pipes.
//
// Measured on GB300 (2048^2 MUSCL-Hancock MinBee, waves everywhere): 1521 Mcell-updates/s with FP64
// products, 1600 - 1700 with one checked integer product at a time or in groups, 1973 like this (2107 with
// a CTA per tile, hf_cart.cu); Van Leer 1469 -> 1964 (2097), the developed forward-facing step 1639 -> 2038
// (2171).  FP64 instructions a cell update 305 -> 194, all instructions 7,300 -> 11,000; issue slots 58 % busy,
// FP64 pipe 76 % of what it can take, the integer (ALU) pipe 62 %.  It is no longer the FP64 pipe alone: with 8 %
// of the FP64 instructions moved too (the limiter's 1 + r and slope product, 17 and 31 integer ones each) it
// ran between 1.5 % slower and 1 % faster, and stays as it is.
#pragma once

#include "hf_device.cuh"

namespace hf {

// The window: |x| in [2^-255, 2^257), told by two bits of the exponent plus a constant.  Values are
// collected in one word that is looked at once.  A product or quotient of two values inside lies in
// [2^-513, 2^514), of three in [2^-769, 2^771): normal, so those need no look of their own.
struct Window {
    uint32_t any = 0, pos = 0;
};
HF_HD uint32_t off_window(double x) { return (hi32(f64_bits(x)) + 0x10000000u) ^ 0x40000000u; }
HF_HD void see(Window& w, double x) { w.any |= off_window(x); }
HF_HD void see_pos(Window& w, double x) { w.pos |= off_window(x); }          // and positive
HF_HD void see0(Window& w, double x, bool zero) { if (!zero) w.any |= off_window(x); }   // or zero
HF_HD bool outside(const Window& w) { return ((w.any & 0x60000000u) | (w.pos & 0xE0000000u)) != 0; }
HF_HD bool zero(double x) { return (f64_bits(x) << 1) == 0; }

HF_HD double fma_rn(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}

// The correctly rounded product of normal operands with a normal product: the 53-bit mantissas as
// 21 + 32 bits, four 32 x 32 -> 64 products whose sums need no carries, the top 53 bits of the 105
// or 106 taken by one funnel shift and rounded by the rest, ties to even.  z: a factor is zero.
template <bool Z>
HF_HD double prod(double a, double b, bool z) {
    const uint64_t A = f64_bits(a), B = f64_bits(b);
    const uint32_t ha = hi32(A), hb = hi32(B);
    const uint32_t a1 = (ha & kMantHi) | kOneHi, b1 = (hb & kMantHi) | kOneHi;
    const uint64_t p0 = wide(lo32(A), lo32(B));
    const uint64_t p1 = wide(lo32(A), b1) + (wide(a1, lo32(B)) + hi32(p0));
    const uint64_t p2 = wide(a1, b1) + hi32(p1);                  // the product / 2^64, 41 or 42 bits
    const uint32_t s = 12u - (hi32(p2) >> 9);
    const uint32_t w1 = fshl32(hi32(p2), lo32(p2), s), w0 = fshl32(lo32(p2), lo32(p1), s);
    const uint32_t l = lo32(p1) << s;                             // the bits below, and lo32(p0) under them
    uint64_t r = u64_of(w1, w0) + (l >> 31);
    if (((l ^ 0x80000000u) | lo32(p0)) == 0u) r &= ~1ull;         // a tie: to even
    const uint32_t e = (ha & kExpHi) + (hb & kExpHi) - (1012u << 20) - (s << 20), sg = (ha ^ hb) & 0x80000000u;
    if (Z && z) return f64_from(u64_of(sg, 0u));
    return f64_from(u64_of(hi32(r) + e + sg, lo32(r)));
}
HF_HD double mulw(double a, double b) { return prod<false>(a, b, false); }
HF_HD double mulz(double a, double b, bool z) { return prod<true>(a, b, z); }
HF_HD double quot(double a, double b, uint32_t X) { return quot32(f64_bits(a), f64_bits(b), X); }
HF_HD double quotz(double a, double b, uint32_t X, bool z) {
    const double q = quot(a, b, X);
    return z ? f64_from((f64_bits(a) ^ f64_bits(b)) & 0x8000000000000000ull) : q;
}
HF_HD uint32_t rcp32(double b) { return recip32(f64_bits(b)); }

// the primitives of a state (n, t: the velocity normal and tangential to the faces)
struct PrimN {
    double r, n, t, p, q;
    bool zn, zt;
    uint32_t X;   // the reciprocal of r
};
HF_HD PrimN prim_n(Window& w, double g1, const double* c) {
    PrimN a;
    a.r = c[0];
    a.X = rcp32(a.r);
    a.zn = zero(c[1]);
    a.zt = zero(c[2]);
    see_pos(w, a.r);
    see0(w, c[1], a.zn);
    see0(w, c[2], a.zt);
    a.n = quotz(c[1], a.r, a.X, a.zn);
    a.t = quotz(c[2], a.r, a.X, a.zt);
    see0(w, a.n, a.zn);
    see0(w, a.t, a.zt);
    a.q = mulz(a.n, a.n, a.zn) + mulz(a.t, a.t, a.zt);
    const bool zq = a.zn && a.zt;
    see0(w, a.q, zq);
    see_pos(w, c[3]);
    // E - (r / 2) q: halving is exact, and what it loses below the window does not reach E's last bit
    const double E = fma_rn(-0.5, mulz(a.r, a.q, zq), c[3]);
    see_pos(w, E);
    a.p = mulw(g1, E);
    see_pos(w, a.p);
    return a;
}
// the total energy from the primitives
HF_HD double energy_n(Window& w, double g1, const PrimN& a) {
    const double rg = mulw(a.r, g1);
    const double h = fma_rn(0.5, a.q, quot(a.p, rg, rcp32(rg)));
    see_pos(w, h);
    return mulw(a.r, h);
}
// the flux along n; y: the products of the tangential momentum as cons_flux_y orders them
HF_HD void flux_n(Window& w, bool y, const PrimN& a, double Et, double* f) {
    f[0] = mulz(a.r, a.n, a.zn);
    f[1] = mulz(f[0], a.n, a.zn) + a.p;
    const double rt = mulz(a.r, y ? a.t : a.n, y ? a.zt : a.zn);
    f[2] = mulz(rt, y ? a.n : a.t, a.zn || a.zt);
    const double s = Et + a.p;
    see(w, s);
    f[3] = mulz(a.n, s, a.zn);
}

// One cell of the half-step predictor along a direction (variables in n, t order) from ordinary
// states: the limited slopes, the extrapolated face states, their fluxes, the evolved states lo and
// hi.  False: some value is outside the window, and lo, hi are not valid.
template <int LIM>
HF_HD bool predict_fast(bool y, const double* um, const double* u0, const double* up, double g1, double h,
                        double* lo, double* hi) {
    Window w;
    double e0[4], e1[4];
    see(w, h);
    see(w, g1);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const double dl = u0[v] - um[v], dr = up[v] - u0[v];
        const double cl = clamp_tol(dl), cr = clamp_tol(dr);
        see(w, cl);
        see(w, cr);
        const double r = quot(cl, cr, rcp32(cr));
        const uint64_t rb = f64_bits(r);
        const bool in = rb <= 0x3FF0000000000000ull, neg = (rb >> 63) != 0;
        const double den = 1.0 + r;
        // the limiters' second quotient; a negative ratio's divisor is replaced (its limiter is zero).  The
        // clamped differences lie within [1e-6, 2^257), so 1 + r and the quotients are normal.
        const double dd = neg ? 2.0 : den, num = LIM == 1 && in ? f64_from(rb + (1ull << 52)) : 2.0;
        double xi = quot(num, dd, rcp32(dd));
        if (LIM == 0) xi = in ? r : xi;
        xi = neg ? 0.0 : xi;
        // s / 2 = xi (dl / 2 + dr / 2) / 2 = t / 4: beside a cell value inside the window, or beside zero
        // when t itself is inside, no scaling by 2 or 4 loses a bit of the result
        const double t = xi * (dl + dr);
        e0[v] = fma_rn(-0.25, t, u0[v]);
        e1[v] = fma_rn(0.25, t, u0[v]);
        const bool z = zero(u0[v]);
        see0(w, z ? t : u0[v], z && zero(t));
    }
    const PrimN a = prim_n(w, g1, e0), b = prim_n(w, g1, e1);
    const double Ea = energy_n(w, g1, a), Eb = energy_n(w, g1, b);
    double f0[4], f1[4];
    flux_n(w, y, a, Ea, f0);
    flux_n(w, y, b, Eb, f1);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const double df = f0[v] - f1[v];
        const bool z = zero(df);
        see0(w, df, z);
        const double d = mulz(h, df, z);
        lo[v] = e0[v] + d;
        hi[v] = e1[v] + d;
    }
    return !outside(w);
}

// a < b for values that are not NaN
HF_HD bool less(double a, double b) { return order_key(a) < order_key(b); }

HF_HD double sound_n(double g, const PrimN& a) { return root32(f64_bits(quot(mulw(g, a.p), a.r, a.X))); }

// The HLLC flux (n, t order) from the two sides' primitives and sound speeds (E: and total energies, in
// place of the reciprocals); only the side the branches select forms its energy, flux and star state.
template <bool E>
HF_HD bool hllc_sides(Window& w, bool y, double g1, const PrimN& L, const PrimN& R, double aL, double aR, double EL,
                      double ER, const double* UL, const double* UR, double* F) {
    const double l0 = L.n - aL, r0 = R.n - aR, l1 = L.n + aL, r1 = R.n + aR;
    const double SL = less(r0, l0) ? r0 : l0, SR = less(l1, r1) ? r1 : l1;
    if (outside(w)) return false;
    bool left = true, star = false;
    double Ss = 0.0;
    if (!ge0(SL)) {
        const double dl = SL - L.n, dr = SR - R.n;
        see(w, dl);
        see(w, dr);
        const double num = R.p - L.p + mulz(mulz(L.r, L.n, L.zn), dl, L.zn) -
                           mulz(mulz(R.r, R.n, R.zn), dr, R.zn);
        const double den = mulw(L.r, dl) - mulw(R.r, dr);
        const bool z = zero(num);
        see0(w, num, z);
        see(w, den);
        if (outside(w)) return false;
        Ss = quotz(num, den, rcp32(den), z);
        // the branches of riemann_hllc.cpp:179-211 with SL < 0 and no NaN: star left, star right, right
        left = ge0(Ss);
        star = left || ge0(SR);
    }
    PrimN a;
    a.r = left ? L.r : R.r;
    a.n = left ? L.n : R.n;
    a.t = left ? L.t : R.t;
    a.p = left ? L.p : R.p;
    a.q = left ? L.q : R.q;
    a.zn = left ? L.zn : R.zn;
    a.zt = left ? L.zt : R.zt;
    if (!E) a.X = left ? L.X : R.X;
    const double Et = E ? (left ? EL : ER) : energy_n(w, g1, a);
    double f[4];
    flux_n(w, y, a, Et, f);
    if (star) {
        const double S = left ? SL : SR, dk = S - a.n, ds = S - Ss, rd = mulw(a.r, dk), sn = Ss - a.n;
        const bool zs = zero(Ss), zsn = zero(sn);
        see(w, S);
        see(w, dk);
        see(w, ds);
        see0(w, Ss, zs);
        see0(w, sn, zsn);
        const double c = mulw(a.r, quot(dk, ds, rcp32(ds)));
        see(w, c);
        const double k = Ss + quot(a.p, rd, rcp32(rd));
        see(w, k);
        const double m = quot(Et, a.r, E ? rcp32(a.r) : a.X) + mulz(sn, k, zsn);
        see(w, m);
        const double us[4] = {c, mulz(c, Ss, zs), mulz(c, a.t, a.zt), mulw(c, m)};
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const double d = us[v] - (left ? UL[v] : UR[v]);
            const bool z = zero(d);
            see0(w, d, z);
            f[v] = f[v] + mulz(S, d, z);
        }
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) F[v] = f[v];
    return !outside(w);
}

// The HLLC flux (n, t order) between ordinary states; false: some value is outside the window
HF_HD bool hllc_fast(bool y, double g, double g1, const double* UL, const double* UR, double* F) {
    Window w;
    see(w, g);
    see(w, g1);
    const PrimN L = prim_n(w, g1, UL), R = prim_n(w, g1, UR);
    return hllc_sides<false>(w, y, g1, L, R, sound_n(g, L), sound_n(g, R), 0.0, 0.0, UL, UR, F);
}

// TimeStep's terms |u| + c and |v| + c of an ordinary state (wave_terms); its density and pressure are positive
HF_HD bool speeds_fast(double g, double g1, const double* U, double& sx, double& sy) {
    Window w;
    see(w, g);
    see(w, g1);
    const PrimN a = prim_n(w, g1, U);
    const double c = sound_n(g, a);
    sx = f64_from(f64_bits(a.n) & kAbs) + c;
    sy = f64_from(f64_bits(a.t) & kAbs) + c;
    return !outside(w);
}
static __host__ __device__ __noinline__ bool speeds_any(double g, double g1, double r, double ru, double rv, double E,
                                                        double* s) {
    return wave_terms(g, g1, r, ru, rv, E, s[0], s[1]);
}
// false: density or pressure not positive
HF_HD bool speeds(double g, double g1, const double* U, double& sx, double& sy) {
    if (speeds_fast(g, g1, U, sx, sy)) return true;
    double s[2];
    const bool ok = speeds_any(g, g1, U[0], U[1], U[2], U[3], s);
    sx = s[0];
    sy = s[1];
    return ok;
}

// A Godunov cell: q = u, v, p, Et, a (its primitives, total energy and sound speed), formed once for its
// four faces
HF_HD bool cell_fast(double g, double g1, const double* U, double* q) {
    Window w;
    see(w, g);
    see(w, g1);
    const PrimN a = prim_n(w, g1, U);
    q[0] = a.n;
    q[1] = a.t;
    q[2] = a.p;
    q[3] = energy_n(w, g1, a);
    q[4] = sound_n(g, a);
    return !outside(w);
}
static __host__ __device__ __noinline__ void cell_any(double g, double g1, double r, double ru, double rv, double E,
                                                      double* q) {
    const Prim w = to_prim(g1, r, ru, rv, E);
    q[0] = w.u;
    q[1] = w.v;
    q[2] = w.p;
    q[3] = w.Et;
    q[4] = sound(g, w.r, w.p);
}
// the sides of a Godunov face from their cells' values (n, t order)
HF_HD PrimN prim_of(Window& w, const double* U, const double* q) {
    PrimN a;
    a.r = U[0];
    a.n = q[0];
    a.t = q[1];
    a.p = q[2];
    a.q = 0.0;
    a.X = 0u;
    a.zn = zero(a.n);
    a.zt = zero(a.t);
    see_pos(w, a.r);
    see0(w, a.n, a.zn);
    see0(w, a.t, a.zt);
    see_pos(w, a.p);
    see_pos(w, q[3]);
    see_pos(w, q[4]);
    return a;
}
HF_HD bool face_fast(bool y, const double* UL, const double* qL, const double* UR, const double* qR, double* F) {
    Window w;
    const PrimN L = prim_of(w, UL, qL), R = prim_of(w, UR, qR);
    return hllc_sides<true>(w, y, 0.0, L, R, qL[4], qR[4], qL[3], qR[3], UL, UR, F);
}
static __host__ __device__ __noinline__ int face_any(bool y, const double* UL, const double* qL, const double* UR,
                                                     const double* qR, double* F) {
    const double* const U[2] = {UL, UR};
    const double* const q[2] = {qL, qR};
    const int n = y ? 2 : 1, t = 3 - n;
    Prim w[2];
    double V[2][4], f[2][4], G[4];
    for (int k = 0; k < 2; ++k) {
        V[k][0] = U[k][0];
        V[k][n] = U[k][1];
        V[k][t] = U[k][2];
        V[k][3] = U[k][3];
        w[k].r = U[k][0];
        w[k].u = y ? q[k][1] : q[k][0];
        w[k].v = y ? q[k][0] : q[k][1];
        w[k].p = q[k][2];
        w[k].Et = q[k][3];
        w[k].q = 0.0;
        if (y) flux<1>(w[k], f[k]);
        else flux<0>(w[k], f[k]);
    }
    const int bad = y ? hllc<1>(V[0], w[0], qL[4], f[0], V[1], w[1], qR[4], f[1], G)
                      : hllc<0>(V[0], w[0], qL[4], f[0], V[1], w[1], qR[4], f[1], G);
    F[0] = G[0];
    F[1] = G[n];
    F[2] = G[t];
    F[3] = G[3];
    return bad;
}

// dt (one_dx (F_l - F_r) + one_dy (G_b - G_t)) + U of four variables; false: outside the window
HF_HD bool update_fast(const double* a, const double* b, const double* u, double dt, double one_dx, double one_dy,
                       double* un) {
    Window w;
    see(w, dt);
    see(w, one_dx);
    see(w, one_dy);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const bool za = zero(a[v]), zb = zero(b[v]);
        see0(w, a[v], za);
        see0(w, b[v], zb);
        const double l = mulz(one_dx, a[v], za) + mulz(one_dy, b[v], zb);
        const bool zl = zero(l);
        see0(w, l, zl);
        un[v] = mulz(dt, l, zl) + u[v];
    }
    return !outside(w);
}
// the general form, for values outside the window
static __host__ __device__ __noinline__ double update_any(double a, double b, double u, double dt, double one_dx,
                                                          double one_dy) {
    return dt * (one_dx * a + one_dy * b) + u;
}

// The general predictor and face, for items with a value outside the window (n, t order).
template <int LIM>
static __host__ __device__ __noinline__ void predict_any(bool y, const double* um, const double* u0, const double* up, double g1,
                                         double h, double* lo, double* hi) {
    double e0[4], e1[4], f0[4], f1[4];
    for (int v = 0; v < 4; ++v) {
        const double s = slope<LIM>(um[v], u0[v], up[v]);
        const double hs = half(s);
        e0[v] = u0[v] - hs;
        e1[v] = u0[v] + hs;
    }
    const int n = y ? 2 : 1, t = 3 - n;
    Prim w0 = to_prim(g1, e0[0], e0[n], e0[t], e0[3]);
    Prim w1 = to_prim(g1, e1[0], e1[n], e1[t], e1[3]);
    if (y) {
        flux<1>(w0, f0);
        flux<1>(w1, f1);
    } else {
        flux<0>(w0, f0);
        flux<0>(w1, f1);
    }
    for (int v = 0; v < 4; ++v) {
        const int k = v == 0 || v == 3 ? v : (v == 1 ? n : t);
        const double d = h * (f0[k] - f1[k]);
        lo[v] = e0[v] + d;
        hi[v] = e1[v] + d;
    }
}
static __host__ __device__ __noinline__ int hllc_any(bool y, double g, double g1, const double* UL, const double* UR, double* F) {
    if (!y) return hllc_cons<0>(g, g1, UL, UR, F);
    const double L[4] = {UL[0], UL[2], UL[1], UL[3]}, R[4] = {UR[0], UR[2], UR[1], UR[3]};
    double G[4];
    const int bad = hllc_cons<1>(g, g1, L, R, G);
    F[0] = G[0]; F[1] = G[2]; F[2] = G[1]; F[3] = G[3];
    return bad;
}

// A state's momentum turned by an angle (euler_ideal_gas.cpp:152-165): (c m1 + s m2, c m2 - s m1)
HF_HD void turn_fast(Window& w, double c, double s, const double* f, double* o) {
    const bool zc = zero(c), zs = zero(s), z1 = zero(f[1]), z2 = zero(f[2]);
    see0(w, c, zc);
    see0(w, s, zs);
    see0(w, f[1], z1);
    see0(w, f[2], z2);
    o[0] = f[0];
    o[1] = mulz(c, f[1], zc || z1) + mulz(s, f[2], zs || z2);
    o[2] = mulz(c, f[2], zc || z2) - mulz(s, f[1], zs || z1);
    o[3] = f[3];
}
// The flux through an unstructured edge of length len between the states U and V: turned into the edge's
// frame (c, s), the HLLC flux there, turned back (cn, sn) and scaled
HF_HD bool edge_fast(double c, double s, double cn, double sn, double len, double g, double g1, const double* U,
                     const double* V, double* f) {
    Window w;
    double a[4], b[4], F[4], t[4];
    turn_fast(w, c, s, U, a);
    turn_fast(w, c, s, V, b);
    if (outside(w) || !hllc_fast(false, g, g1, a, b, F)) return false;
    turn_fast(w, cn, sn, F, t);
    see(w, len);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const bool z = zero(t[v]);
        see0(w, t[v], z);
        f[v] = mulz(len, t[v], z);
    }
    return !outside(w);
}
// The unstructured update dt (-(inv acc)) + U of a cell, and its TimeStep term r_in / (|V| + c)
HF_HD bool uns_update_fast(double g, double g1, double dt, double inv, double rin, const double* acc, const double* U,
                           double* un, double& term) {
    Window w;
    see(w, g);
    see(w, g1);
    see(w, dt);
    see(w, inv);
    see_pos(w, rin);
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        const bool z = zero(acc[v]);
        see0(w, acc[v], z);
        un[v] = U[v] - mulz(dt, mulz(inv, acc[v], z), z);
    }
    const PrimN a = prim_n(w, g1, un);
    const double c = sound_n(g, a), sp = (a.zn && a.zt ? 0.0 : root32(f64_bits(a.q))) + c;
    see_pos(w, sp);
    term = quot(rin, sp, rcp32(sp));
    return !outside(w);
}

}  // namespace hf
