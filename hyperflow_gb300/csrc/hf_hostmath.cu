// Host build of the kernels' arithmetic (hf_device.cuh, hf_intdiv.cuh) for the CPU test
// suite: the same source the GPU kernels compile, exposed as plain C functions so the
// tests can compare it with the oracle and with IEEE division / sqrt without a GPU; and the rules
// of the host side that can be told apart there (ranges of pinned memory, the graphs of a batched run).
// Built as a separate library (libhf_hostmath.so); the product library does not use it.
#include <cstdint>

#include "hf_cart.h"
#include "hf_device.cuh"
#include "hf_fast.cuh"
#include "hf_pinned.h"

extern "C" {

int64_t hm_batch_graph_steps(int64_t left, int graphs) { return hf::batch_graph_steps(left, graphs); }

// host_covered over n ranges [begin[k], begin[k] + size[k])
int hm_host_covered(const uint64_t* begin, const uint64_t* size, int n, uint64_t p, uint64_t bytes) {
    return hf::host_covered((uintptr_t)p, (size_t)bytes, [&](uintptr_t q) {
        for (int k = 0; k < n; ++k)
            if (q >= begin[k] && q < begin[k] + size[k])
                return hf::HostRange{(uintptr_t)begin[k], (uintptr_t)(begin[k] + size[k])};
        return hf::HostRange{0, 0};
    });
}

void hm_div(const double* a, const double* b, double* out, int64_t n) {
    for (int64_t i = 0; i < n; ++i) out[i] = hf::div_rn(a[i], b[i]);
}

void hm_half(const double* x, double* out, int64_t n) {
    for (int64_t i = 0; i < n; ++i) out[i] = hf::half(x[i]);
}

void hm_sqrt(const double* x, double* out, int64_t n) {
    for (int64_t i = 0; i < n; ++i) out[i] = hf::sqrt_rn(x[i]);
}

int hm_hllc(double gamma, const double* ul, const double* ur, int dir, double* f) {
    return dir == 0 ? hf::hllc_cons<0>(gamma, gamma - 1.0, ul, ur, f)
                    : hf::hllc_cons<1>(gamma, gamma - 1.0, ul, ur, f);
}

double hm_limiter(int kind, double r) { return kind == 0 ? hf::limiter<0>(r) : hf::limiter<1>(r); }

double hm_slope(int kind, double um, double u0, double up) {
    return kind == 0 ? hf::slope<0>(um, u0, up) : hf::slope<1>(um, u0, up);
}

// bit 0 lt(a,b), 1 le0(a), 2 ge0(a), 3 abs_le(a, 1e-6); out[0] smin, out[1] smax, out[2] nmax(|b|, a)
int hm_compare(double a, double b, double* out) {
    out[0] = hf::smin(a, b);
    out[1] = hf::smax(a, b);
    out[2] = hf::nmax(std::fabs(b), a);
    return (hf::lt(a, b) ? 1 : 0) | (hf::le0(a) ? 2 : 0) | (hf::ge0(a) ? 4 : 0) |
           (hf::abs_le(a, 1e-6) ? 8 : 0);
}

void hm_wave_terms(double gamma, const double* u, double* s2) {
    hf::wave_terms(gamma, gamma - 1.0, u[0], u[1], u[2], u[3], s2[0], s2[1]);
}

// The straight-through functions of hf_fast.cuh and the general ones on the same n items: c [n][3][4] the
// states around a cell (normal, tangential order), each item along x (y = 0) or y.  ok[k] is 1 where the
// item stayed in the window; fast and any get [n][8] evolved states.
void hm_predict(int lim, int y, const double* c, double g1, double h, int64_t n, int* ok, double* fast, double* any) {
    for (int64_t k = 0; k < n; ++k) {
        const double* a = c + 12 * k;
        double *f = fast + 8 * k, *s = any + 8 * k;
        if (lim == 0) {
            ok[k] = hf::predict_fast<0>(y != 0, a, a + 4, a + 8, g1, h, f, f + 4);
            hf::predict_any<0>(y != 0, a, a + 4, a + 8, g1, h, s, s + 4);
        } else {
            ok[k] = hf::predict_fast<1>(y != 0, a, a + 4, a + 8, g1, h, f, f + 4);
            hf::predict_any<1>(y != 0, a, a + 4, a + 8, g1, h, s, s + 4);
        }
    }
}

// the face between c[k][0] and c[k][2]; [n][4] fluxes (normal, tangential order), bad: zero-flux fallbacks
void hm_face(int y, const double* c, double g, double g1, int64_t n, int* ok, int* bad, double* fast, double* any) {
    for (int64_t k = 0; k < n; ++k) {
        ok[k] = hf::hllc_fast(y != 0, g, g1, c + 12 * k, c + 12 * k + 8, fast + 4 * k);
        bad[k] = hf::hllc_any(y != 0, g, g1, c + 12 * k, c + 12 * k + 8, any + 4 * k);
    }
}

// the update of c[k][1] with c[k][0] and c[k][2] as the flux differences
void hm_update(const double* c, double dt, double one_dx, double one_dy, int64_t n, int* ok, double* fast, double* any) {
    for (int64_t k = 0; k < n; ++k) {
        const double* a = c + 12 * k;
        ok[k] = hf::update_fast(a, a + 8, a + 4, dt, one_dx, one_dy, fast + 4 * k);
        for (int v = 0; v < 4; ++v) any[4 * k + v] = hf::update_any(a[v], a[8 + v], a[4 + v], dt, one_dx, one_dy);
    }
}

// Godunov: the cells c[k][0] and c[k][2] (n, t order; q [n][2][5]) and the face between them; and TimeStep's
// terms of c[k][0] (s [n][2]).  Bits of ok: 1 both cells, 2 the face (from the general cells), 4 the terms.
void hm_godunov(int y, const double* c, double g, double g1, int64_t n, int* ok, int* bad, double* fq, double* aq,
                double* ff, double* af, double* fs, double* as) {
    for (int64_t k = 0; k < n; ++k) {
        const double *l = c + 12 * k, *r = l + 8;
        double *f = fq + 10 * k, *a = aq + 10 * k;
        ok[k] = hf::cell_fast(g, g1, l, f) & hf::cell_fast(g, g1, r, f + 5) ? 1 : 0;
        hf::cell_any(g, g1, l[0], l[1], l[2], l[3], a);
        hf::cell_any(g, g1, r[0], r[1], r[2], r[3], a + 5);
        ok[k] |= hf::face_fast(y != 0, l, a, r, a + 5, ff + 4 * k) ? 2 : 0;
        bad[k] = hf::face_any(y != 0, l, a, r, a + 5, af + 4 * k);
        ok[k] |= hf::speeds_fast(g, g1, l, fs[2 * k], fs[2 * k + 1]) ? 4 : 0;
        hf::speeds_any(g, g1, l[0], l[1], l[2], l[3], as + 2 * k);
    }
}

// The flux through an unstructured edge between c[k][0] and c[k][2], geo [n][5] = cos, sin, cos and sin of the
// opposite angle, length; and the update of c[k][1] with c[k][0] as the flux sum: [n][5] with the TimeStep
// term.  Bits of ok: 1 the edge, 2 the update.
void hm_uns(const double* c, const double* geo, double g, double g1, double dt, double rin, int64_t n, int* ok,
            int* bad, double* ff, double* af, double* fu, double* au) {
    auto rot = [](double a, double b, const double* f, double* o) {
        o[0] = f[0];
        o[1] = a * f[1] + b * f[2];
        o[2] = (-b) * f[1] + a * f[2];
        o[3] = f[3];
    };
    for (int64_t k = 0; k < n; ++k) {
        const double *l = c + 12 * k, *m = l + 4, *r = l + 8, *q = geo + 5 * k;
        ok[k] = hf::edge_fast(q[0], q[1], q[2], q[3], q[4], g, g1, l, r, ff + 4 * k) ? 1 : 0;
        double a[4], b[4], F[4];
        rot(q[0], q[1], l, a);
        rot(q[0], q[1], r, b);
        bad[k] = hf::hllc_cons<0>(g, g1, a, b, F);
        rot(q[2], q[3], F, a);
        for (int v = 0; v < 4; ++v) af[4 * k + v] = q[4] * a[v];
        double* u = au + 5 * k;
        ok[k] |= hf::uns_update_fast(g, g1, dt, q[4], rin, l, m, fu + 5 * k, fu[5 * k + 4]) ? 2 : 0;
        for (int v = 0; v < 4; ++v) u[v] = dt * (-(q[4] * l[v])) + m[v];
        double uu, vv, p;
        hf::to_prim_short(g1, u[0], u[1], u[2], u[3], uu, vv, p);
        u[4] = hf::div_rn(rin, std::fabs(hf::sqrt_rn(uu * uu + vv * vv)) + hf::sound(g, u[0], p));
    }
}

}  // extern "C"
