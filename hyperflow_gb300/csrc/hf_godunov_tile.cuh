// The first-order Godunov tile computation shared by the Cartesian stencils (hf_cart.cu) and the
// batched step kernel (hf_batch.cu): GodunovScheme::calculate_fluxes_{x,y} +
// calculate_spatial_update (src/fvm_2d_cart/scheme/godunov/godunov.cpp:27-118) with the
// forward-Euler update (forward_euler.cpp:19-29).
//
// Input: sU, the tile's conservative state plus a 1-cell halo in shared memory, [4][ty+2][tx+2].  Each
// cell's primitives, total energy and sound speed are formed once (sQ [5][cells]) for the faces that use
// them.  Output: sF / sG, the HLLC fluxes of the tile's x faces [4][ty][tx+1] and y faces [4][ty+1][tx].
//
// As the MUSCL-Hancock tile: FP64 issue bounds it, the products go to the integer pipes (hf_fast.cuh) and
// both directions run one copy of the code.  A face forms the flux of the one side it uses: with both
// fluxes of every cell in sQ (12 values) a CTA's tile was 32 x 10 cells and a quarter of its cells halo.
#pragma once

#include "hf_cart.h"
#include "hf_device.cuh"
#include "hf_fast.cuh"
#include "hf_mh_tile.cuh"   // tile shapes, owned_face

namespace hf {

// doubles of shared memory a tile takes: the state with its halo, the cells' values, the fluxes
inline int go_tile_doubles(int tx, int ty) {
    return 9 * (tx + 2) * (ty + 2) + 4 * ty * (tx + 1) + 4 * (ty + 1) * tx;
}

// One face between the tile cells l and r = l + step (nc cells a plane); its flux, in the variables'
// order, to f[v * fs].  Returns 1 for the zero-flux fallback.
__device__ __forceinline__ int go_face(bool y, const double* sU, const double* sQ, int l, int step, int nc, double* f,
                                       int fs) {
    const int pn = y ? 2 * nc : nc, pt = 3 * nc - pn, qn = y ? nc : 0, qt = nc - qn;
    double U[2][4], q[2][5], F[4];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const double* u = sU + l + k * step;
        const double* w = sQ + l + k * step;
        U[k][0] = u[0]; U[k][1] = u[pn]; U[k][2] = u[pt]; U[k][3] = u[3 * nc];
        q[k][0] = w[qn]; q[k][1] = w[qt]; q[k][2] = w[2 * nc]; q[k][3] = w[3 * nc]; q[k][4] = w[4 * nc];
    }
    int bad = 0;
    if (!face_fast(y, U[0], q[0], U[1], q[1], F)) {
        double V[2][4], r[2][5], G[4];   // copies, so that the fast path's stay in registers
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const double* u = sU + l + k * step;
            const double* w = sQ + l + k * step;
            V[k][0] = u[0]; V[k][1] = u[pn]; V[k][2] = u[pt]; V[k][3] = u[3 * nc];
            r[k][0] = w[qn]; r[k][1] = w[qt]; r[k][2] = w[2 * nc]; r[k][3] = w[3 * nc]; r[k][4] = w[4 * nc];
        }
        bad = face_any(y, V[0], r[0], V[1], r[1], G);
#pragma unroll
        for (int v = 0; v < 4; ++v) F[v] = G[v];
    }
    f[0] = F[0];
    f[(y ? 2 : 1) * fs] = F[1];
    f[(y ? 1 : 2) * fs] = F[2];
    f[3 * fs] = F[3];
    return bad;
}

// Computes the fluxes in sW (after the cells' values there) from sU (tile origin x0, y0 in interior cells
// of an nx x ny block).  Ends with __syncthreads().  Returns the number of owned faces whose HLLC took
// the zero-flux branch; with first_bad, each such face's face_key (key_base: its step and block bits) is
// min-reduced there.  Cells beyond the first ghost layer and faces beyond the last face are skipped: no
// in-block cell reads them, and zero-filled states would only take the general path.
template <int NT, class S>
__device__ __forceinline__ int go_tile_fluxes(const S& s, const double* sU, double* sW, double g, double g1, int x0, int y0,
                                              int nx, int ny, unsigned long long* first_bad = nullptr,
                                              unsigned long long key_base = 0) {
    const int tx = s.tx(), ty = s.ty(), ux = tx + 2, nc = ux * (ty + 2);
    const int nfx = (tx + 1) * ty, nfy = tx * (ty + 1);
    double* const sQ = sW;
    double* const sF = sW + 5 * nc;
    double* const sG = sF + 4 * nfx;
#pragma unroll 1
    for (int cell = threadIdx.x; cell < nc; cell += NT) {
        const int row = s.row2(cell);
        if (x0 - 1 + cell - row * ux > nx || y0 - 1 + row > ny) continue;
        const double U[4] = {sU[cell], sU[nc + cell], sU[2 * nc + cell], sU[3 * nc + cell]};
        double q[5];
        if (!cell_fast(g, g1, U, q)) {
            double r[5];
            cell_any(g, g1, U[0], U[1], U[2], U[3], r);
#pragma unroll
            for (int k = 0; k < 5; ++k) q[k] = r[k];
        }
#pragma unroll
        for (int k = 0; k < 5; ++k) sQ[k * nc + cell] = q[k];
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int fx = (nfx + 31) >> 5, fxy = fx + ((nfy + 31) >> 5);
    int herr = 0;
#pragma unroll 1
    for (int w = warp; w < fxy; w += NT / 32) {
        const bool y = w >= fx;
        const int it = (y ? w - fx : w) * 32 + lane, row = y ? s.row0(it) : s.row1(it), col = it - row * (y ? tx : tx + 1);
        if (it >= (y ? nfy : nfx) || x0 + col >= nx + (y ? 0 : 1) || y0 + row >= ny + (y ? 1 : 0)) continue;
        // face f of row r sits between tile cells (f-1, r) and (f, r), or (r, f-1) and (r, f)
        const int l = (row + (y ? 0 : 1)) * ux + col + (y ? 1 : 0);
        const int bad = go_face(y, sU, sQ, l, y ? ux : 1, nc, (y ? sG : sF) + it, y ? nfy : nfx);
        if (bad && (y ? owned_face(y0 + row, row, ty, ny, x0 + col, nx) : owned_face(x0 + col, col, tx, nx, y0 + row, ny))) {
            ++herr;
            if (first_bad) atomicMin(first_bad, key_base | face_key(0, 0, y ? 1 : 0, y0 + row, x0 + col));
        }
    }
    __syncthreads();
    return herr;
}

// Conservative update + forward Euler of output cell (ox, oy) of the tile
// (godunov.cpp:97-113; forward_euler.cpp:19-29)
template <class S>
__device__ __forceinline__ void go_update(const S& s, const double* sU, const double* sW, int ox, int oy, double dt,
                                          double one_dx, double one_dy, double* un) {
    const int tx = s.tx(), ty = s.ty(), nc = (tx + 2) * (ty + 2), nfx = (tx + 1) * ty, nfy = tx * (ty + 1);
    const double* F = sW + 5 * nc + oy * (tx + 1) + ox;
    const double* G = sW + 5 * nc + 4 * nfx + oy * tx + ox;
    const double* U = sU + (oy + 1) * (tx + 2) + ox + 1;
    double a[4], b[4], u[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
        a[v] = F[v * nfx] - F[v * nfx + 1];
        b[v] = G[v * nfy] - G[v * nfy + tx];
        u[v] = U[v * nc];
    }
    if (!update_fast(a, b, u, dt, one_dx, one_dy, un))
#pragma unroll
        for (int v = 0; v < 4; ++v) un[v] = update_any(a[v], b[v], u[v], dt, one_dx, one_dy);
}

}  // namespace hf
