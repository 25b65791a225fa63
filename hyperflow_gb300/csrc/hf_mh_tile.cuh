// The MUSCL-Hancock tile computation shared by the Cartesian stencils (hf_cart.cu) and the
// batched step kernel (hf_batch.cu).
//
// Input: sU, the tile's conservative state plus a 2-cell halo in shared memory,
// [4][ty+4][tx+4].  Output, in sA: the HLLC fluxes of the tile's x and y faces, each in the place of
// the evolved state on the face's low side (which that face alone reads).
// The reference steps restated here: calculate_slope_limiters_{x,y} + calculate_slopes_{x,y}
// (muscl_hancock.cpp:67-206), calculate_boundary_extrapolations (209-240),
// evolve_boundary_reconstruction (243-281), calculate_fluxes_{x,y} (284-345).
//
// Both directions run the same code, a warp's items at a time (y is uniform over a warp; the momentum
// components are taken as normal and tangential to the faces): a copy of the code per direction
// missed the instruction cache (1546 against 1651 Mcell-updates/s at 2048^2 when it was measured).  All
// predictor cells, then all faces: two phases of two directions leave the CTA's warps unevenly
// loaded half as often as four phases of one, and need no room for fluxes beside the states.
#pragma once

#include "hf_cart.h"
#include "hf_device.cuh"
#include "hf_fast.cuh"

namespace hf {

// A tile of tx x ty cells: the row of item `it` of a list whose rows are tx, tx + 1 or tx + 2 long.
struct RowShape {
    TileShape t;
    __device__ int tx() const { return t.tx; }
    __device__ int ty() const { return t.ty; }
    __device__ int row0(int it) const { return (int)(((uint32_t)it * t.m[0]) >> 21); }
    __device__ int row1(int it) const { return (int)(((uint32_t)it * t.m[1]) >> 21); }
    __device__ int row2(int it) const { return (int)(((uint32_t)it * t.m[2]) >> 21); }
};
// doubles of shared memory a tile takes: the state with its halo, the evolved states
inline int mh_tile_doubles(int tx, int ty) {
    return 4 * (tx + 4) * (ty + 4) + 8 * ((tx + 2) * ty + tx * (ty + 2));
}

// A face on a tile edge is formed by both tiles that share it, and partial tiles form
// faces past the block.  Only the owner counts an HLLC zero-flux fallback, so the count
// equals the reference's: face index gf (0..n along the normal) of row gr, local index lf.
__device__ __forceinline__ bool owned_face(int gf, int lf, int T, int n, int gr, int nr) {
    return gr < nr && gf <= n && (lf < T || gf == n);
}

// One cell of the half-step predictor (u points at its variable 0; plane and stride step to the next
// variable and the next cell along the direction): the evolved states to lo[v * ls] (minus side) and
// lo[(4 + v) * ls], in n, t order, as the faces of this direction read them back.
template <int LIM>
__device__ __forceinline__ void mh_predict(bool y, const double* u, int plane, int stride, double g1, double h,
                                           double* lo, int ls) {
    double um[4], u0[4], up[4], e[4], f[4];
    const int pn = (y ? 2 : 1) * plane, pt = (y ? 1 : 2) * plane;
    const double* const q[4] = {u, u + pn, u + pt, u + 3 * plane};
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        um[v] = q[v][-stride];
        u0[v] = q[v][0];
        up[v] = q[v][stride];
    }
    if (!predict_fast<LIM>(y, um, u0, up, g1, h, e, f)) {
        double xm[4], x0[4], xp[4], r0[4], r1[4];   // copies, so that the fast path's stay in registers
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            xm[v] = q[v][-stride];
            x0[v] = q[v][0];
            xp[v] = q[v][stride];
        }
        predict_any<LIM>(y, xm, x0, xp, g1, h, r0, r1);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            e[v] = r0[v];
            f[v] = r1[v];
        }
    }
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        lo[v * ls] = e[v];
        lo[(4 + v) * ls] = f[v];
    }
}

// One face: HLLC between the evolved states l[v * ls] (minus side) and r[v * ls]; the flux, in the
// variables' order, replaces l.  Returns 1 for the zero-flux fallback.
__device__ __forceinline__ int mh_face(bool y, double* l, const double* r, int ls, double g, double g1) {
    double UL[4], UR[4], F[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        UL[v] = l[v * ls];
        UR[v] = r[v * ls];
    }
    int bad = 0;
    if (!hllc_fast(y, g, g1, UL, UR, F)) {
        double xl[4], xr[4], xf[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            xl[v] = l[v * ls];
            xr[v] = r[v * ls];
        }
        bad = hllc_any(y, g, g1, xl, xr, xf);
#pragma unroll
        for (int v = 0; v < 4; ++v) F[v] = xf[v];
    }
    l[0] = F[0];
    l[(y ? 2 : 1) * ls] = F[1];
    l[(y ? 1 : 2) * ls] = F[2];
    l[3 * ls] = F[3];
    return bad;
}

// Computes the face fluxes in sA from sU.  Ends with __syncthreads().  Returns the number of owned
// faces whose HLLC took the zero-flux branch (tile origin x0, y0 in interior cells); with
// first_bad, each such face's face_key (key_base: its step and block bits) is min-reduced there.
// Items past the block (cells beyond the first ghost layer, faces beyond the last face) are skipped:
// no in-block cell reads them, and their zero-filled states would only take the general path.
template <int NT, int LIM, class S>
__device__ __forceinline__ int mh_tile_fluxes(const S& s, const double* sU, double* sA, double g, double g1, double hdx,
                                              double hdy, int x0, int y0, int nx, int ny,
                                              unsigned long long* first_bad = nullptr,
                                              unsigned long long key_base = 0) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll 1
    for (int w = warp;; w += NT / 32) {
        const int tx = s.tx(), ty = s.ty(), ux = tx + 4, plane = ux * (ty + 4);
        const int nax = (tx + 2) * ty, nay = tx * (ty + 2), px = (nax + 31) >> 5;
        if (w >= px + ((nay + 31) >> 5)) break;
        double* const sY = sA + 8 * nax;
        const bool y = w >= px;
        const int it = (y ? w - px : w) * 32 + lane, n = y ? nay : nax;
        const int row = y ? s.row0(it) : s.row2(it);
        const int cx = it - row * (y ? tx : tx + 2) - (y ? 0 : 1), cy = row - (y ? 1 : 0);   // the cell in the tile
        if (it >= n || x0 + cx >= nx + (y ? 0 : 1) || y0 + cy >= ny + (y ? 1 : 0)) continue;
        mh_predict<LIM>(y, sU + (cy + 2) * ux + cx + 2, plane, y ? ux : 1, g1, y ? hdy : hdx, (y ? sY : sA) + it, n);
    }
    __syncthreads();
    int herr = 0;
#pragma unroll 1
    for (int w = warp;; w += NT / 32) {
        const int tx = s.tx(), ty = s.ty(), nfx = (tx + 1) * ty, nfy = tx * (ty + 1);
        const int nax = (tx + 2) * ty, nay = tx * (ty + 2), fx = (nfx + 31) >> 5;
        if (w >= fx + ((nfy + 31) >> 5)) break;
        double* const sY = sA + 8 * nax;
        const bool y = w >= fx;
        const int it = (y ? w - fx : w) * 32 + lane, n = y ? nay : nax;
        const int row = y ? s.row0(it) : s.row1(it), col = it - row * (y ? tx : tx + 1);
        if (it >= (y ? nfy : nfx) || x0 + col >= nx + (y ? 0 : 1) || y0 + row >= ny + (y ? 1 : 0)) continue;
        double* const lo = (y ? sY : sA) + row * (y ? tx : tx + 2) + col;   // the cell on the low side
        const int bad = mh_face(y, lo + 4 * n, lo + (y ? tx : 1), n, g, g1);
        if (bad && (y ? owned_face(y0 + row, row, ty, ny, x0 + col, nx) : owned_face(x0 + col, col, tx, nx, y0 + row, ny))) {
            ++herr;
            if (first_bad) atomicMin(first_bad, key_base | face_key(0, 0, y ? 1 : 0, y0 + row, x0 + col));
        }
    }
    __syncthreads();
    return herr;
}

// Conservative update + forward Euler of output cell (ox, oy) of the tile
// (calculate_spatial_update, muscl_hancock.cpp:348-376; forward_euler.cpp:19-29)
template <class S>
__device__ __forceinline__ void mh_update(const S& s, const double* sU, const double* sA, int ox, int oy, double dt,
                                          double one_dx, double one_dy, double* un) {
    const int tx = s.tx(), ty = s.ty(), nax = (tx + 2) * ty, nay = tx * (ty + 2);
    const double* F = sA + 4 * nax + oy * (tx + 2) + ox;
    const double* G = sA + 8 * nax + 4 * nay + oy * tx + ox;
    const double* U = sU + (oy + 2) * (tx + 4) + ox + 2;
    double a[4], b[4], u[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        a[v] = F[v * nax] - F[v * nax + 1];
        b[v] = G[v * nay] - G[v * nay + tx];
        u[v] = U[v * (tx + 4) * (ty + 4)];
    }
    if (!update_fast(a, b, u, dt, one_dx, one_dy, un))
#pragma unroll
        for (int v = 0; v < 4; ++v) un[v] = update_any(a[v], b[v], u[v], dt, one_dx, one_dy);
}

}  // namespace hf
