// Cartesian time-step kernels for sm_103a.
//
//   fill_cfl      ghost/halo fill, Mesh::apply_bcs (src/fvm_2d_cart/mesh/mesh/mesh.cpp:31-39), TimeStep over
//                 the ghost cells and the step dt (timestep.cpp:29-68)
//   upload,       a block's state from and into host memory the GPU maps, the upload with the TimeStep
//   download      terms of its interior; interior_cfl: those terms after another upload
//   godunov       fused x/y HLLC + update, GodunovScheme (godunov.cpp:27-118) + ForwardEuler
//   mh            fused slopes/limiter/predictor/HLLC/update, MUSCLHancockScheme
//                 (muscl_hancock.cpp:41-376) + ForwardEuler, with the next step's TimeStep
//                 terms reduced in the epilogue
//   *_step        the same for every block of a step, a CTA per tile, the last of which ends the step
//   solo          a whole step of a small single block, its ghosts included
//
// Layout: per block, SoA FP64 [var][total_y][pitch] (x contiguous), ghosts included, two
// buffers alternating by step parity.  The stencil CTAs stage one tile plus its halo with a
// single 3-D TMA load (box = tile + 2*ghost in x and y, all four variables) into shared
// memory; halos come from the neighbouring tiles' cells in HBM, never from another CTA.
#include <algorithm>
#include <cstdio>

#include "hf_cart.h"
#include "hf_device.cuh"
#include "hf_godunov_tile.cuh"
#include "hf_mh_tile.cuh"

namespace hf {

constexpr unsigned kWaitLimit = 1u << 22;   // bounded mbarrier polls before giving up

// stop the device loop before this step?  At t_end; in strict mode once a failure is recorded; while the
// frame ring lacks room for the two frames a step takes at most.
__device__ __forceinline__ bool loop_done(const Ctrl* c) {
    if (c->clamp && c->t == c->t_end) return true;
    if (c->strict && (c->first_bad != ~0ull || c->first_nonpos != ~0ull)) return true;
    return c->clamp && c->frames && c->captured - c->drained > c->ring_slots - 2;
}

// the accumulators of a step whose starting state has parity p, cleared
__device__ void clear_step(Ctrl* __restrict__ c, int p, int nblocks) {
    for (int b = 0; b < nblocks; ++b) {
        c->ghost_s[b][0] = c->ghost_s[b][1] = 0ull;
        c->int_s[p ^ 1][b][0] = c->int_s[p ^ 1][b][1] = 0ull;
        c->step_hllc[b] = 0;
        c->step_bad[b] = c->step_nonpos[b] = ~0ull;
    }
    c->ticket = 0u;
}

// Start of a step that no finished step prepared (after an upload, a restore, a ghost fill on its own): its
// stop flag, and its accumulators cleared, also where the loop has ended: the step that comes next counts on
// it.  A finished step clears the next one's itself (finish_step) and the fill takes the stop flag, so a
// loop's steps need no launch for this.
__global__ void step_begin_kernel(Ctrl* __restrict__ c) {
    c->done = loop_done(c);
    c->snap_pre = c->snap_post = 0;
    clear_step(c, (int)(c->step & 1), c->nblocks);
}

// ------------------------------------------------------------------------------------
// TimeStep over the ghost cells; the last CTA forms the step dt
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void ghost_cell_ij(const BlockDev& B, int g, long long k, int& i, int& j) {
    const long long row_cells = (long long)g * B.tx;
    if (k < row_cells) {                      // bottom ghost rows
        j = (int)(k / B.tx); i = (int)(k % B.tx);
    } else if (k < 2 * row_cells) {           // top ghost rows
        k -= row_cells;
        j = B.ty - g + (int)(k / B.tx); i = (int)(k % B.tx);
    } else {                                  // left/right ghost columns of interior rows
        k -= 2 * row_cells;
        j = g + (int)(k / (2 * g));
        int c = (int)(k % (2 * g));
        i = c < g ? c : B.tx - 2 * g + c;
    }
}

constexpr int kRedThreads = 256;

__device__ void form_step_dt(Ctrl* __restrict__ c, int p, StepState* __restrict__ ss);

// block b's dx / max(|u| + c) and dy / max(|v| + c), ghost cells and the interior of parity p, read past L1
__device__ __forceinline__ void block_dt(const Ctrl* c, int b, int p, double& dtx, double& dty) {
    const volatile Ctrl* vc = c;
    dtx = div_rn(c->dx[b], smax(bitsd(vc->ghost_s[b][0]), bitsd(vc->int_s[p][b][0])));
    dty = div_rn(c->dy[b], smax(bitsd(vc->ghost_s[b][1]), bitsd(vc->int_s[p][b][1])));
}

// the predictor scalars of block b from its predictor dt (muscl_hancock.cpp:248-249, 352-353)
__device__ __forceinline__ void step_scalars(const Ctrl* c, StepState* ss, int b, double dtp) {
    ss->sc[b][0] = div_rn(0.5 * dtp, c->dx[b]);
    ss->sc[b][1] = div_rn(0.5 * dtp, c->dy[b]);
    ss->sc[b][2] = div_rn(1.0, c->dx[b]);
    ss->sc[b][3] = div_rn(1.0, c->dy[b]);
    ss->sc[b][4] = dtp;
}

// form_dt = 0: the ghost maxima only (for a predictor TimeStep in a step whose dt the caller gave)
__global__ void __launch_bounds__(kRedThreads) ghost_cfl_kernel(Ctrl* __restrict__ c,
                                                                const MeshDev* __restrict__ m, int form_dt) {
    if (c->done) return;
    const int p = (int)(c->step & 1);
    const double g = c->gamma, g1 = c->g1;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (int b = 0; b < m->nblocks; ++b) {
        const BlockDev& B = m->b[b];
        const size_t plane = (size_t)B.ty * B.pitch;
        const double* __restrict__ U = B.buf[p];
        double mx = 0.0, my = 0.0;
        for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < B.ghost_count;
             k += stride) {
            int i, j;
            ghost_cell_ij(B, m->ghost, k, i, j);
            size_t o = (size_t)j * B.pitch + i;
            if (!hf_in((long long)o, (long long)plane, &c->err)) continue;
            double sx, sy;
            wave_terms(g, g1, U[o], U[plane + o], U[2 * plane + o], U[3 * plane + o], sx, sy);
            mx = nmax(mx, sx);
            my = nmax(my, sy);
        }
        block_max2_atomic<kRedThreads>(mx, my, &c->ghost_s[b][0], &c->ghost_s[b][1]);
        __syncthreads();
    }
    if (form_dt) form_step_dt(c, p, nullptr);
}

// The last CTA of a ghost-maxima launch to finish forms the step's dt: TimeStep call number
// `calls` over every block (timestep.cpp:29-68), then Simulation::solve's clamps and frame points.
// With ss, also the all-blocks launch's scalars: each block's predictor dt from the same maxima (the
// predictor's TimeStep call, muscl_hancock.cpp:246-249, over the step's starting state).  A block per
// thread: the quotients take about 300 cycles each, one after the other on one thread more than the fill.
__device__ void form_step_dt(Ctrl* __restrict__ c, int p, StepState* __restrict__ ss) {
    __shared__ bool last;
    __shared__ double s_dt[HF_MAXB][2], s_min;
    __threadfence();
    if (threadIdx.x == 0) last = (atomicAdd(&c->ticket, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int nb = c->nblocks;
    const long long call = c->calls;
    const double cfl = c->cfl;
    if ((int)threadIdx.x < nb) block_dt(c, threadIdx.x, p, s_dt[threadIdx.x][0], s_dt[threadIdx.x][1]);
    __syncthreads();
    if (threadIdx.x == 0) {
        double dtx = 1e16, dty = 1e16;
        for (int b = 0; b < nb; ++b) {
            dtx = smin(dtx, s_dt[b][0]);
            dty = smin(dty, s_dt[b][1]);
        }
        s_min = smin(dtx, dty);
        double dt = ((call + 1 <= 10) ? 0.2 * cfl : cfl) * s_min;
        c->dt_cfl = dt;
        const double t = c->t;
        c->snap_pre = c->snap_post = 0;
        if (c->clamp && t + dt > c->t_end) dt = c->t_end - t;        // simulation.cpp:88-90
        if (c->clamp && c->frames) {
            const double cur = c->frame_next;
            c->snap_pre = (cur == 0.0);                              // simulation.cpp:93-96
            if ((t + dt > cur) && (cur > 0.0)) dt = cur - t;         // simulation.cpp:98-102
            if (fabs(t - cur) < 1e-12) {                             // simulation.cpp:106-113
                c->snap_post = 1;
                c->frame_next = cur + c->frame_interval;
            }
            c->snap_t = t;
        }
        c->dt = dt;
        c->done = 0;
        c->calls = call + 1;
        c->ticket = 0u;
    }
    if (!ss) return;
    __syncthreads();
    if ((int)threadIdx.x < nb) {
        const int b = threadIdx.x;
        const double dtp = ((call + 1 + b + 1 <= 10) ? 0.2 * cfl : cfl) * s_min;
        step_scalars(c, ss, b, dtp);
    }
}

// the block of ghost cell k of the all-blocks enumeration
__device__ __forceinline__ int ghost_block(const MeshDev* __restrict__ m, long long k) {
    int b = 0;
    while (b + 1 < m->nblocks && k >= m->b[b + 1].ghost_off) ++b;
    return b;
}

// Mesh::apply_bcs (mesh.cpp:31-39) for every block in one launch: ghost cell k takes its final
// value from the fill program (a copy of one cell's pre-fill value or of a Dirichlet side's state,
// with the reflective sides' negations: transmissive_boundary.cpp, reflective_boundary.cpp,
// dirichlet_boundary.cpp, internal_boundary.cpp replayed in the reference's order on the host),
// then its TimeStep terms feed the block's ghost maxima.  With ss (a step of the loop) the stop flag is
// taken here: nothing it depends on changes before the last CTA forms the dt.
__global__ void __launch_bounds__(kRedThreads) fill_cfl_kernel(Ctrl* __restrict__ c, const MeshDev* __restrict__ m,
                                                               int form_dt, StepState* __restrict__ ss) {
    // (a chain of loads: those that need no other's result first)
    const long long total = m->total_ghost;
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    FillOp op{};
    if (k < total) op = m->fill[k];
    const int p = (int)(c->step & 1);
    const double g = c->gamma, g1 = c->g1;
    const int gh = m->ghost;
    if (ss ? loop_done(c) : c->done != 0) {
        if (ss && blockIdx.x == 0 && threadIdx.x == 0) {
            c->done = 1;
            c->snap_pre = c->snap_post = 0;
        }
        return;
    }
    const long long k0 = (long long)blockIdx.x * blockDim.x;
    const long long k1 = (k0 + blockDim.x < total ? k0 + blockDim.x : total) - 1;
    int b = -1;
    double sx = 0.0, sy = 0.0;
    if (k < total) {
        b = ghost_block(m, k);
        const BlockDev& B = m->b[b];
        int i, j;
        ghost_cell_ij(B, gh, k - B.ghost_off, i, j);
        double u[4];
        if (op.kind == 2) {
            const BlockDev& S = m->b[op.block];
#pragma unroll
            for (int v = 0; v < 4; ++v) u[v] = S.bc_state[op.side][v];
        } else {
            const BlockDev& S = m->b[op.block];
            const size_t splane = (size_t)S.ty * S.pitch;
            const double* __restrict__ src = S.buf[op.kind == 0 ? p : p ^ 1];
            if (hf_in(op.src, (long long)splane, &c->err)) {
#pragma unroll
                for (int v = 0; v < 4; ++v) u[v] = src[v * splane + op.src];
            } else {
#pragma unroll
                for (int v = 0; v < 4; ++v) u[v] = 0.0;
            }
        }
        if (op.neg & 1) u[1] = -1.0 * u[1];
        if (op.neg & 2) u[2] = -1.0 * u[2];
        const size_t plane = (size_t)B.ty * B.pitch, o = (size_t)j * B.pitch + i;
        if (hf_in((long long)o, (long long)plane, &c->err)) {
            double* __restrict__ dst = B.buf[p];
#pragma unroll
            for (int v = 0; v < 4; ++v) dst[v * plane + o] = u[v];
        }
        double tx_, ty_;
        wave_terms(g, g1, u[0], u[1], u[2], u[3], tx_, ty_);
        sx = nmax(0.0, tx_);   // NaN terms are skipped, as TimeStep's std::min skips them
        sy = nmax(0.0, ty_);
    }
    // one atomic pair per block this CTA touched (its cells are consecutive in block order)
    const int b0 = ghost_block(m, k0), b1 = ghost_block(m, k1);
    for (int bb = b0; bb <= b1; ++bb)
        block_max2_atomic<kRedThreads>(b == bb ? sx : 0.0, b == bb ? sy : 0.0, &c->ghost_s[bb][0],
                                       &c->ghost_s[bb][1]);
    if (form_dt) form_step_dt(c, p, ss);
}

// the current buffer's ghost cells into the other buffer (after a fill no stencil follows)
__global__ void __launch_bounds__(256) ghost_mirror_kernel(const Ctrl* __restrict__ c, const MeshDev* __restrict__ m) {
    const int p = (int)(c->step & 1);
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= m->total_ghost) return;
    const int b = ghost_block(m, k);
    const BlockDev& B = m->b[b];
    int i, j;
    ghost_cell_ij(B, m->ghost, k - B.ghost_off, i, j);
    const size_t plane = (size_t)B.ty * B.pitch, o = (size_t)j * B.pitch + i;
#pragma unroll
    for (int v = 0; v < 4; ++v) B.buf[p ^ 1][v * plane + o] = B.buf[p][v * plane + o];
}

// TimeStep terms over one block's interior (after an upload of new state)
__global__ void __launch_bounds__(kRedThreads) interior_cfl_kernel(Ctrl* __restrict__ c,
                                                                   const MeshDev* __restrict__ m,
                                                                   int b, int parity) {
    const BlockDev& B = m->b[b];
    const int g = m->ghost;
    const size_t plane = (size_t)B.ty * B.pitch;
    const double* __restrict__ U = B.buf[parity];
    const double gm = c->gamma, g1 = c->g1;
    double mx = 0.0, my = 0.0;
    const long long n = (long long)B.nx * B.ny;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
         k += (long long)gridDim.x * blockDim.x) {
        int i = (int)(k % B.nx) + g, j = (int)(k / B.nx) + g;
        size_t o = (size_t)j * B.pitch + i;
        double sx, sy;
        wave_terms(gm, g1, U[o], U[plane + o], U[2 * plane + o], U[3 * plane + o], sx, sy);
        mx = nmax(mx, sx);
        my = nmax(my, sy);
    }
    block_max2_atomic<kRedThreads>(mx, my, &c->int_s[parity][b][0], &c->int_s[parity][b][1]);
}

// A block's whole state ([4][total_y][total_x], ghosts included) read from host memory the GPU
// maps (pinned), written into both buffers, with the TimeStep terms of the interior cells -- the
// upload, buffer copy and interior_cfl of a host-buffer step or a state upload in one pass over the
// link.  A warp takes a row's cells 32 at a time, and the next row when it has them all.
// Bound by the link: 4096^2 cells (538 MB) in 2.86 ms, 188 GB/s; 3.43 with the copy engine, a device copy to the
// other buffer and interior_cfl behind it; 1000 x 1000 in 0.20 ms, before 0.35; 300 x 8000 in 0.43, before 1.68.
// (a row of CTAs per block from b0 on: a launch per block left the link idle between them)
__global__ void __launch_bounds__(kRedThreads) upload_kernel(Ctrl* __restrict__ c, const MeshDev* __restrict__ m,
                                                             int b0, int parity, const HostBlocks h) {
    const int b = b0 + blockIdx.y;
    const double* __restrict__ hin = h.p[blockIdx.y];
    const BlockDev& B = m->b[b];
    const int g = m->ghost;
    const size_t plane = (size_t)B.ty * B.pitch, hplane = (size_t)B.ty * B.tx;
    double* __restrict__ U0 = B.buf[parity];
    double* __restrict__ U1 = B.buf[parity ^ 1];
    const double gm = c->gamma, g1 = c->g1;
    double mx = 0.0, my = 0.0;
    const int segs = (B.tx + 31) >> 5, lane = threadIdx.x & 31;
    const long long n = (long long)segs * B.ty;
    for (long long w = (blockIdx.x * (long long)kRedThreads + threadIdx.x) >> 5; w < n;
         w += (long long)gridDim.x * (kRedThreads / 32)) {
        const int j = (int)(w / segs), i = (int)(w - (long long)j * segs) * 32 + lane;
        if (i >= B.tx) continue;
        const size_t o = (size_t)j * B.pitch + i, h = (size_t)j * B.tx + i;
        if (!hf_in((long long)o, (long long)plane, &c->err)) continue;
        double u[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) u[v] = __ldcs(&hin[v * hplane + h]);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            U0[v * plane + o] = u[v];
            U1[v * plane + o] = u[v];
        }
        if (i >= g && i < B.tx - g && j >= g && j < B.ty - g) {
            double sx, sy;
            wave_terms(gm, g1, u[0], u[1], u[2], u[3], sx, sy);
            mx = nmax(mx, sx);
            my = nmax(my, sy);
        }
    }
    block_max2_atomic<kRedThreads>(mx, my, &c->int_s[parity][b][0], &c->int_s[parity][b][1]);
}

// A block's whole state into host memory the GPU maps.  Bound by the link, which a store of a whole line uses
// best: the array is taken in pieces that start on its 256-byte lines, whatever its rows' length, a warp four
// lines at a time.  us for 1000 rows of 65, 191, 1003, 2049 cells: 37, 58, 193, 366; from each row's start 38, 64,
// 236, 456; the copy engine 47, 61, 193, 455, with the same 191 GB/s at 4096^2 (2.82 ms) but for 4 to 10 ms in one
// copy of ten there, and up to 20 the first time it writes an array.
constexpr int kDownLines = 4;
__global__ void __launch_bounds__(kRedThreads) download_kernel(Ctrl* __restrict__ c, const MeshDev* __restrict__ m, int b,
                                                               int parity, double* __restrict__ hout) {
    const BlockDev& B = m->b[b];
    const unsigned tx = (unsigned)B.tx;
    const long long n = 4LL * B.ty * B.tx, all = 4LL * B.ty * B.pitch;
    const double* __restrict__ U = B.buf[parity];
    const int lead = (int)(reinterpret_cast<uintptr_t>(hout) >> 3) & 31, lane = threadIdx.x & 31;
    for (long long w = (blockIdx.x * (long long)kRedThreads + threadIdx.x) >> 5; w * 32 * kDownLines - lead < n;
         w += (long long)gridDim.x * (kRedThreads / 32)) {
        const long long f0 = w * 32 * kDownLines - lead, from = f0 < 0 ? 0 : f0;
        const long long row = from / tx;                 // of the array's 4 total_y rows
        const int col = (int)(from - row * tx);
        double u[kDownLines];
        bool in[kDownLines];
#pragma unroll
        for (int k = 0; k < kDownLines; ++k) {
            const long long f = f0 + 32 * k + lane;
            const unsigned at = (unsigned)(col + (int)(f - from)), down = at / tx;
            const long long o = (row + down) * B.pitch + (at - down * tx);
            in[k] = f >= 0 && f < n && hf_in(o, all, &c->err);
            if (in[k]) u[k] = U[o];
        }
#pragma unroll
        for (int k = 0; k < kDownLines; ++k)
            if (in[k]) __stcs(&hout[f0 + 32 * k + lane], u[k]);
    }
}

// The ghost cells filled this step into host memory the GPU maps: with the stencil's own host
// stores of the updated cells, the whole block downloaded.
__global__ void __launch_bounds__(256) ghost_store_kernel(Ctrl* __restrict__ c, const MeshDev* __restrict__ m,
                                                          int parity, const HostBlocks h) {
    const BlockDev& B = m->b[blockIdx.y];
    double* __restrict__ hout = h.p[blockIdx.y];
    const int g = m->ghost;
    const size_t plane = (size_t)B.ty * B.pitch, hplane = (size_t)B.ty * B.tx;
    const double* __restrict__ U = B.buf[parity];    // filled this step; the stencil copies them later
    const long long rows = (long long)g * B.tx;          // cells in the g bottom (or top) rows
    const long long n = 2 * rows + 2LL * g * B.ny;       // + g columns each side of the interior rows
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n;
         k += (long long)gridDim.x * blockDim.x) {
        int i, j;
        if (k < 2 * rows) {
            const long long r = k < rows ? k : k - rows;
            i = (int)(r % B.tx);
            j = (int)(r / B.tx) + (k < rows ? 0 : B.ty - g);
        } else {
            const long long r = k - 2 * rows;
            const int col = (int)(r % (2 * g));
            j = g + (int)(r / (2 * g));
            i = col < g ? col : B.tx - 2 * g + col;
        }
        const size_t o = (size_t)j * B.pitch + i, h = (size_t)j * B.tx + i;
        if (!hf_in((long long)o, (long long)plane, &c->err) || !hf_in((long long)h, (long long)hplane, &c->err))
            continue;
#pragma unroll
        for (int v = 0; v < 4; ++v) __stcs(&hout[v * hplane + h], U[v * plane + o]);
    }
}

__global__ void set_dt_kernel(Ctrl* c, double dt) { c->dt = dt; }

// Frames of this step into the device ring: the interior of every block, SoA per block,
// packed ([b][var][y][x]); the state before the update is still in buffer `step & 1` and the
// updated one in the other buffer until finalize flips the parity.
__global__ void __launch_bounds__(256) frame_copy_kernel(const Ctrl* __restrict__ c,
                                                         const MeshDev* __restrict__ m,
                                                         FrameRing ring) {
    if (c->done) return;
    const int pre = c->snap_pre, post = c->snap_post;
    if (!pre && !post) return;
    const int p = (int)(c->step & 1);
    const long long R = c->ring_slots;
    const long long slot_pre = c->captured % R, slot_post = (c->captured + pre) % R;
    const int g = m->ghost;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (int which = 0; which < 2; ++which) {
        if (which == 0 ? !pre : !post) continue;
        double* __restrict__ dst = ring.base + (which == 0 ? slot_pre : slot_post) * ring.slot_len;
        for (int b = 0; b < m->nblocks; ++b) {
            const BlockDev& B = m->b[b];
            const double* __restrict__ src = B.buf[which == 0 ? p : p ^ 1];
            const long long plane = (long long)B.nx * B.ny, n = 4 * plane;
            double* __restrict__ d = dst + ring.off[b];
            for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
                const long long v = k / plane, r = k - v * plane;
                const int j = (int)(r / B.nx), i = (int)(r - (long long)j * B.nx);
                d[k] = src[(size_t)v * B.ty * B.pitch + (size_t)(j + g) * B.pitch + (i + g)];
            }
        }
    }
}

// end of step: t += dt; the MUSCL-Hancock predictor calls advance the counter; record this
// step's frames; flip parity; clear the next step's accumulators
// (One thread's work at the end of every step: all it reads, first, so that the loads are one latency.)
__device__ void finish_step(Ctrl* __restrict__ c, StepOut* out = nullptr) {
    const int nb = c->nblocks, scheme = c->scheme;
    const bool snap = c->clamp && c->frames;
    const double t = c->t, dt = c->dt;
    const long long calls = c->calls, step = c->step + 1;
    if (snap) {
        for (int which = 0; which < 2; ++which) {
            if (which == 0 ? !c->snap_pre : !c->snap_post) continue;
            const long long slot = c->captured % c->ring_slots;
            c->ring_t[slot] = c->snap_t;
            c->ring_idx[slot] = c->frame_idx;
            c->frame_idx = c->frame_idx + 1;
            c->captured = c->captured + 1;
        }
    }
    c->t = t + dt;
    if (scheme == 1) c->calls = calls + nb;
    c->step = step;
    clear_step(c, (int)(step & 1), nb);
    if (out) {   // (visible to the host once it has waited for the launch)
        out->dt = dt;
        out->step = step;
    }
}

__global__ void finalize_kernel(Ctrl* c) {
    if (!c->done) finish_step(c);
}

// ------------------------------------------------------------------------------------
// shared helpers for the stencils
// ------------------------------------------------------------------------------------
// wait (bounded) for the tile's first TMA load, which thread 0 issued; false if the wait gave up
__device__ __forceinline__ bool wait_tile(uint64_t* bar, Ctrl* c) {
    __syncthreads();
    const bool ok = mbar_wait_bounded(bar, 0, kWaitLimit);
    if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) {
            raise_error(c, HF_DEV_TIMEOUT);
            mbar_wait_bounded(bar, 0, kWaitLimit);   // let an in-flight copy land before exit
        }
        __syncthreads();
        return false;
    }
    return true;
}

// The ghost cells in a tile's halo (loaded after this step's fill), from shared memory into the
// step's output buffer, so the updated state carries the ghost values the reference's mesh holds
// after the step (its update leaves ghost cells as filled) and the next fill finds this fill's
// values in its other buffer.  Each ghost cell is stored by the one tile holding its nearest
// interior cell; only tiles on the block's edge hold any.  sU is [4][ty + 2G][tx + 2G].
template <int G, int NT>
__device__ __forceinline__ void store_ghosts(const double* __restrict__ sU, const BlockDev& B, int tx, int ty, int x0,
                                             int y0, double* __restrict__ out, int* err) {
    if (x0 > 0 && y0 > 0 && x0 + tx < B.nx && y0 + ty < B.ny) return;
    const int ux = tx + 2 * G, uy = ty + 2 * G;
    const size_t plane = (size_t)B.ty * B.pitch;
    for (int it = threadIdx.x; it < ux * uy; it += NT) {
        const int lx = it % ux, ly = it / ux;
        const int x = x0 - G + lx, y = y0 - G + ly;   // interior coordinates
        if (x < -G || y < -G || x >= B.nx + G || y >= B.ny + G) continue;
        if (x >= 0 && y >= 0 && x < B.nx && y < B.ny) continue;
        const int cx = x < 0 ? 0 : (x >= B.nx ? B.nx - 1 : x);
        const int cy = y < 0 ? 0 : (y >= B.ny ? B.ny - 1 : y);
        if (cx < x0 || cx >= x0 + tx || cy < y0 || cy >= y0 + ty) continue;
        const size_t o = (size_t)(y + G) * B.pitch + (x + G);
        if (!hf_in((long long)o, (long long)plane, err)) continue;
#pragma unroll
        for (int v = 0; v < 4; ++v) out[v * plane + o] = sU[(v * uy + ly) * ux + lx];
    }
}

// The tile's update (G ghost layers: 1 Godunov, 2 MUSCL-Hancock) of its cells into out (and hout), the next
// step's TimeStep terms into mx and my, the earliest non-positive cell into *nonpos.
template <int NT, int G>
__device__ __forceinline__ void store_tile(const RowShape& S, const double* sU, const double* sA, const BlockDev& B, int x0,
                                         int y0, double* __restrict__ out, double* __restrict__ hout, double dt,
                                         double one_dx, double one_dy, double g, double g1, unsigned long long* nonpos,
                                         unsigned long long key, double& mx, double& my, int* err) {
    const int tx = S.tx(), n = tx * S.ty();
    const size_t plane = (size_t)B.ty * B.pitch;
    for (int it = threadIdx.x; it < n; it += NT) {
        const int oy = S.row0(it), ox = it - oy * tx;
        const int gxx = x0 + ox, gyy = y0 + oy;
        if (gxx < B.nx && gyy < B.ny) {
            double un[4];
            const size_t o = (size_t)(gyy + G) * B.pitch + (gxx + G);
            const size_t h = (size_t)(gyy + G) * B.tx + gxx + G;
            if (!hf_in((long long)o, (long long)plane, err) || !hf_in((long long)h, (long long)B.ty * B.tx, err)) continue;
            if (G == 1) go_update(S, sU, sA, ox, oy, dt, one_dx, one_dy, un);
            else mh_update(S, sU, sA, ox, oy, dt, one_dx, one_dy, un);
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                out[v * plane + o] = un[v];
                if (hout) __stcs(&hout[(size_t)v * B.ty * B.tx + h], un[v]);
            }
            double sx, sy;
            if (!speeds(g, g1, un, sx, sy)) atomicMin(nonpos, key | face_key(0, 0, 0, gyy, gxx));
            mx = nmax(mx, sx);
            my = nmax(my, sy);
        }
    }
}

// ------------------------------------------------------------------------------------
// MUSCL-Hancock, fused
// ------------------------------------------------------------------------------------
// Two 448-thread CTAs per SM (72 registers; 110.9 KB of shared memory each, which a 32 x 19 tile fills):
// the tile's 42 warp-items of predictor cells are three rounds of the 14 warps, its 40 of faces too.
// Measured at 2048^2 (Mcell-updates/s, in a persistent kernel): 1973; 512 threads and 64 registers 1962, 320 threads and 32 x 18
// tiles 1933, 256 threads and 32 x 14 1880, three CTAs of 256 threads and 32 x 12 tiles 1751.
constexpr int kNT = kTileThreads;

template <int LIM>
__global__ void __launch_bounds__(kNT, 2) mh_kernel(Ctrl* __restrict__ c, const MeshDev* __restrict__ m, int b,
                                                      const TileShape tile, const __grid_constant__ CUtensorMap tm0,
                                                      const __grid_constant__ CUtensorMap tm1,
                                                      double* __restrict__ hout) {
    extern __shared__ __align__(1024) double smem[];
    __shared__ uint64_t bar;
    const RowShape S{tile};
    const int tx = tile.tx, ty = tile.ty, usize = 4 * (tx + 4) * (ty + 4);
    double* sU = smem;
    double* sA = smem + usize;
    if (c->done) return;

    const BlockDev& B = m->b[b];
    const int p = (int)(c->step & 1);
    const int tiles_x = (B.nx + tx - 1) / tx;
    const int x0 = (blockIdx.x % tiles_x) * tx, y0 = (blockIdx.x / tiles_x) * ty;

    // scalars of this step, formed once per CTA by thread 0 while the tile is in flight and
    // published by the barrier in load_tile
    __shared__ double sc[5];
    const double g = c->gamma, g1 = c->g1;
    const double dt = c->dt;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_expect_tx(&bar, usize * 8);
        tma_load_3d(sU, p ? &tm1 : &tm0, &bar, x0, y0, 0);
        // the predictor's own TimeStep call (muscl_hancock.cpp:246): blocks < b already advanced
        const double dtp = cfl_dt(c, c->calls + b, b, p, p ^ 1);
        const double dx = c->dx[b], dy = c->dy[b];
        sc[0] = div_rn(0.5 * dtp, dx);   // 248-249
        sc[1] = div_rn(0.5 * dtp, dy);
        sc[2] = div_rn(1.0, dx);         // 352-353
        sc[3] = div_rn(1.0, dy);
        if (blockIdx.x == 0) c->dt_pred[b] = dtp;
    }
    if (!wait_tile(&bar, c)) return;
    const double hdx = sc[0], hdy = sc[1], one_dx = sc[2], one_dy = sc[3];

    const int herr = mh_tile_fluxes<kNT, LIM>(S, sU, sA, g, g1, hdx, hdy, x0, y0, B.nx, B.ny, &c->first_bad,
                                                face_key(c->step, b, 0, 0, 0));
    double mx = 0.0, my = 0.0;
    store_tile<kNT, 2>(S, sU, sA, B, x0, y0, B.buf[p ^ 1], hout, dt, one_dx, one_dy, g, g1, &c->first_nonpos,
                    face_key(c->step, b, 0, 0, 0), mx, my, &c->err);
    store_ghosts<2, kNT>(sU, B, tx, ty, x0, y0, B.buf[p ^ 1], &c->err);
    block_max2_atomic<kNT>(mx, my, &c->int_s[p ^ 1][b][0], &c->int_s[p ^ 1][b][1]);
    if (herr) atomicAdd(reinterpret_cast<unsigned long long*>(&c->hllc_errors), (unsigned long long)herr);
}

// ------------------------------------------------------------------------------------
// MUSCL-Hancock, every block of a step in one launch
// ------------------------------------------------------------------------------------
// The reference updates the blocks one after the other, and block b's half-step predictor takes
// its dt from a TimeStep call over a mesh whose blocks < b are already updated
// (muscl_hancock.cpp:246, called from simulation.cpp:106-110).  One launch per block leaves a
// partly filled last wave of CTAs at the end of every block, and its launches.  Here one launch
// holds the tiles of all blocks, in block order, so one block's tail overlaps the next block's
// start, and runs every block with the predictor dt of a TimeStep call over the step's starting
// state.  For block 0 that is the reference's value.  For block b > 0 it is the reference's value
// whenever updating blocks 0..b-1 leaves the largest wave speed TimeStep sees unchanged, the usual
// case.  The last CTA to finish forms the true predictor dt block by block (the reference's call:
// blocks < b from their updated state); at the first whose bits differ from the value used it
// leaves that block to the re-run launch that follows (one for every block but the first; with
// nothing to do it leaves at once), whose last CTA goes on from there.  A step never writes a
// block's input buffer, so the second run gives exactly the sequential result; a block's
// wave-speed maxima and numerical-failure records are kept per block and folded into the totals
// only when every block is final, so a discarded run leaves nothing behind.  The CTA that finds
// every block final also ends the step, so a step is this launch, the fill and the re-runs.
//
// (It was a persistent cooperative launch with a grid barrier per block, tiles from a counter:
// 1958 Mcell-updates/s at 2048^2 where a CTA per tile gives 2062, and two launches more a step.)

// the last CTA's thread 0: the next block from b on whose predictor dt was not the reference's, its
// scalars and records made ready; the step's end when there is none.
__device__ void settle_step(Ctrl* __restrict__ c, StepState* __restrict__ ss, int b, int finish, StepOut* out) {
    const int p = (int)(c->step & 1), nb = c->nblocks;
    for (; b < nb; ++b) {
        const double dtp = cfl_dt_fresh(c, c->calls + b, b, p, p ^ 1);
        if (f64_bits(dtp) == f64_bits(ss->sc[b][4])) continue;
        step_scalars(c, ss, b, dtp);
        c->int_s[p ^ 1][b][0] = c->int_s[p ^ 1][b][1] = 0ull;   // forget the first run's records
        c->step_hllc[b] = 0;
        c->step_bad[b] = c->step_nonpos[b] = ~0ull;
        c->blocks_rerun = c->blocks_rerun + 1;
        ss->rerun = b;
        return;
    }
    ss->rerun = 0;
    const volatile Ctrl* vc = c;
    long long herr = 0;
    for (b = 0; b < nb; ++b) {   // every block final: fold this step's records
        herr += vc->step_hllc[b];
        const unsigned long long fb = vc->step_bad[b], fn = vc->step_nonpos[b];
        if (fb < c->first_bad) c->first_bad = fb;
        if (fn < c->first_nonpos) c->first_nonpos = fn;
        c->dt_pred[b] = ss->sc[b][4];
    }
    c->hllc_errors = c->hllc_errors + herr;
    if (finish) finish_step(c, out);
}

// this CTA's work is done; true in thread 0 of the last of the launch's CTAs
__device__ __forceinline__ bool last_cta(unsigned int* ctr) {
    __syncthreads();
    if (threadIdx.x != 0) return false;
    __threadfence();
    const bool last = atomicAdd(ctr, 1u) == gridDim.x - 1;
    if (last) {
        *ctr = 0u;
        __threadfence();
    }
    return last;
}

// One tile of block b (local tile index `local`): its TMA load (mbarrier phase `phase`), the
// fused fluxes with the block's predictor scalars, the update and the block's records.
template <int LIM>
__device__ __forceinline__ void mh_plan_tile(Ctrl* __restrict__ c, const MeshDev* __restrict__ m, const StepState* ss,
                                             const StepPlan& plan, int b, int local, uint64_t* bar, uint32_t phase) {
    extern __shared__ __align__(1024) double smem[];
    const int p = (int)(c->step & 1);
    const RowShape S{plan.tile};
    const int tx = plan.tile.tx, ty = plan.tile.ty, usize = 4 * (tx + 4) * (ty + 4);
    double* sU = smem;
    double* sA = smem + usize;
    const BlockDev& B = m->b[b];
    const int x0 = (local % plan.tiles_x[b]) * tx, y0 = (local / plan.tiles_x[b]) * ty;
    if (threadIdx.x == 0) {
        // the previous tile's reads of sU (generic proxy) are ordered before this copy's writes
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(bar, usize * 8);
        tma_load_3d(sU, &plan.tm[b][p], bar, x0, y0, 0);
    }
    const double hdx = ss->sc[b][0], hdy = ss->sc[b][1];
    const bool ok = mbar_wait_bounded(bar, phase, kWaitLimit);
    if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) {
            raise_error(c, HF_DEV_TIMEOUT);
            mbar_wait_bounded(bar, phase, kWaitLimit);   // let an in-flight copy land before exit
        }
        __syncthreads();
        return;
    }
    const double g = c->gamma, g1 = c->g1;
    const unsigned long long key = face_key(c->step, b, 0, 0, 0);
    const int herr = mh_tile_fluxes<kNT, LIM>(S, sU, sA, g, g1, hdx, hdy, x0, y0, B.nx, B.ny, &c->step_bad[b], key);
    double mx = 0.0, my = 0.0;
    store_tile<kNT, 2>(S, sU, sA, B, x0, y0, B.buf[p ^ 1], plan.hout[b], c->dt, ss->sc[b][2], ss->sc[b][3], g, g1,
                    &c->step_nonpos[b], key, mx, my, &c->err);
    store_ghosts<2, kNT>(sU, B, tx, ty, x0, y0, B.buf[p ^ 1], &c->err);
    block_max2_atomic<kNT>(mx, my, &c->int_s[p ^ 1][b][0], &c->int_s[p ^ 1][b][1]);
    if (herr) atomicAdd(reinterpret_cast<unsigned long long*>(&c->step_hllc[b]), (unsigned long long)herr);
}

template <int LIM>
__global__ void __launch_bounds__(kNT, 2) mh_step_kernel(Ctrl* __restrict__ c, const MeshDev* __restrict__ m,
                                                           StepState* __restrict__ ss,
                                                           const __grid_constant__ StepPlan plan) {
    if (c->done) return;   // set before this launch: every CTA leaves
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    int b = 0;
    while (b + 1 < plan.nb && (int)blockIdx.x >= plan.tile_start[b + 1]) ++b;
    mh_plan_tile<LIM>(c, m, ss, plan, b, blockIdx.x - plan.tile_start[b], &bar, 0u);
    if (last_cta(&ss->tiles)) settle_step(c, ss, 1, plan.finish, plan.out);
}

// the block a launch before this one left to be run again, if any, on the resident CTAs
template <int LIM>
__global__ void __launch_bounds__(kNT, 2) mh_rerun_kernel(Ctrl* __restrict__ c, const MeshDev* __restrict__ m,
                                                            StepState* __restrict__ ss,
                                                            const __grid_constant__ StepPlan plan) {
    const int b = c->done ? 0 : ss->rerun;
    if (b == 0) return;
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    uint32_t phase = 0u;
    for (int t = plan.tile_start[b] + blockIdx.x; t < plan.tile_start[b + 1]; t += gridDim.x) {
        mh_plan_tile<LIM>(c, m, ss, plan, b, t - plan.tile_start[b], &bar, phase);
        phase ^= 1u;
        __syncthreads();   // the tile's last reads of shared memory come before the next one's load
    }
    if (last_cta(&ss->tiles)) settle_step(c, ss, b + 1, plan.finish, plan.out);
}

// ------------------------------------------------------------------------------------
// Godunov, fused: per-cell primitives once, then x/y HLLC, then update
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void godunov_tile(Ctrl* __restrict__ c, const MeshDev* __restrict__ m, int b, int local,
                                             const TileShape& tile, const CUtensorMap* tm, double* __restrict__ hout) {
    extern __shared__ __align__(1024) double smem[];
    __shared__ uint64_t bar;
    const RowShape S{tile};
    const int tx = tile.tx, ty = tile.ty, usize = 4 * (tx + 2) * (ty + 2);
    double* sU = smem;
    double* sW = smem + usize;

    const BlockDev& B = m->b[b];
    const int p = (int)(c->step & 1);
    const int tiles_x = (B.nx + tx - 1) / tx;
    const int x0 = (local % tiles_x) * tx, y0 = (local / tiles_x) * ty;
    const double g = c->gamma, g1 = c->g1;
    const double dt = c->dt;
    __shared__ double sc[2];
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_expect_tx(&bar, usize * 8);
        tma_load_3d(sU, tm, &bar, x0, y0, 0);
        sc[0] = div_rn(1.0, c->dx[b]);   // godunov.cpp:97-98
        sc[1] = div_rn(1.0, c->dy[b]);
    }
    if (!wait_tile(&bar, c)) return;

    const int herr = go_tile_fluxes<kNT>(S, sU, sW, g, g1, x0, y0, B.nx, B.ny, &c->first_bad,
                                         face_key(c->step, b, 0, 0, 0));
    double mx = 0.0, my = 0.0;
    store_tile<kNT, 1>(S, sU, sW, B, x0, y0, B.buf[p ^ 1], hout, dt, sc[0], sc[1], g, g1, &c->first_nonpos,
                       face_key(c->step, b, 0, 0, 0), mx, my, &c->err);
    store_ghosts<1, kNT>(sU, B, tx, ty, x0, y0, B.buf[p ^ 1], &c->err);
    block_max2_atomic<kNT>(mx, my, &c->int_s[p ^ 1][b][0], &c->int_s[p ^ 1][b][1]);
    if (herr) atomicAdd(reinterpret_cast<unsigned long long*>(&c->hllc_errors), (unsigned long long)herr);
}

// one block (hf_advance_block, meshes of many blocks)
__global__ void __launch_bounds__(kNT, 2) godunov_kernel(Ctrl* __restrict__ c, const MeshDev* __restrict__ m, int b,
                                                         const TileShape tile, const __grid_constant__ CUtensorMap tm0,
                                                         const __grid_constant__ CUtensorMap tm1,
                                                         double* __restrict__ hout) {
    if (c->done) return;
    godunov_tile(c, m, b, blockIdx.x, tile, (c->step & 1) ? &tm1 : &tm0, hout);
}

// every block of a step in one launch, whose last CTA ends the step
__global__ void __launch_bounds__(kNT, 2) godunov_step_kernel(Ctrl* __restrict__ c, const MeshDev* __restrict__ m,
                                                              StepState* __restrict__ ss,
                                                              const __grid_constant__ StepPlan plan) {
    if (c->done) return;
    int b = 0;
    while (b + 1 < plan.nb && (int)blockIdx.x >= plan.tile_start[b + 1]) ++b;
    godunov_tile(c, m, b, blockIdx.x - plan.tile_start[b], plan.tile, &plan.tm[b][c->step & 1], plan.hout[b]);
    if (last_cta(&ss->tiles) && plan.finish) finish_step(c, plan.out);
}

// ------------------------------------------------------------------------------------
// a step of one block in one launch
// ------------------------------------------------------------------------------------
// Where every ghost cell takes an interior cell's value (transmissive and reflective sides, up to the sign of
// a momentum) or a Dirichlet state, TimeStep's largest wave speed over the ghost cells is one of the
// interior's or of those states, so dt is known before any ghost is filled: every CTA forms it from the
// maxima the last step left, writes the ghosts of its own tile's halo in shared memory, and stores them with
// its update.  The fill, a chain of dependent loads, quotients and a reduction over few cells, took 9 to
// 11 us a step beside 20 to 25 us for the stencil of a small mesh (100 x 5, 256^2).  A step in the loop, before
// and now: MUSCL-Hancock 100 x 5 72 and 17.2 us, Godunov 256^2 68 and 23.7.  Steps with frames, strict mode
// (whose records change during a step) or one launch per block keep the fill.
__global__ void prepare_solo_kernel(Ctrl* c, const MeshDev* m, StepState* ss) {
    double mx = 0.0, my = 0.0;
    for (int side = 0; side < 4; ++side) {
        if (m->b[0].bc_type[side] != BC_DIRICHLET) continue;
        const double* u = m->b[0].bc_state[side];
        double sx, sy;
        wave_terms(c->gamma, c->g1, u[0], u[1], u[2], u[3], sx, sy);
        mx = nmax(mx, sx);
        my = nmax(my, sy);
    }
    ss->solo[0] = mx;
    ss->solo[1] = my;
    ss->solo[2] = div_rn(1.0, c->dx[0]);
    ss->solo[3] = div_rn(1.0, c->dy[0]);
}

// The ghost cell at position it = lx + ly * ux of the tile's halo by the fill program, from the interior
// cells of U, into u; false where there is none
template <int G>
__device__ __forceinline__ bool tile_ghost(const MeshDev* __restrict__ m, const BlockDev& B, const double* __restrict__ U,
                                           int nx, int ny, int ux, int it, int x0, int y0, double* u, int* err) {
    const int ly = it / ux, lx = it - ly * ux, i = x0 + lx, j = y0 + ly;   // in the block, ghosts included
    const int bx = nx + 2 * G, by = ny + 2 * G;
    if (i >= bx || j >= by || (i >= G && i < bx - G && j >= G && j < by - G)) return false;
    const long long k = j < G ? (long long)j * bx + i
                      : j >= by - G ? (long long)(G + j - (by - G)) * bx + i
                      : 2LL * G * bx + (long long)(j - G) * (2 * G) + (i < G ? i : i - (bx - 2 * G));
    const FillOp op = m->fill[k];
    const size_t plane = (size_t)by * B.pitch;
    if (op.kind == 2) {
#pragma unroll
        for (int v = 0; v < 4; ++v) u[v] = B.bc_state[op.side][v];
    } else {
        if (!hf_in(op.src, (long long)plane, err)) return false;
#pragma unroll
        for (int v = 0; v < 4; ++v) u[v] = U[v * plane + op.src];
    }
    if (op.neg & 1) u[1] = -1.0 * u[1];
    if (op.neg & 2) u[2] = -1.0 * u[2];
    return true;
}

// SCHEME 0 Godunov, 1 MUSCL-Hancock with limiter LIM
template <int SCHEME, int LIM>
__global__ void __launch_bounds__(kNT, 2) solo_kernel(Ctrl* __restrict__ c, const MeshDev* __restrict__ m,
                                                      StepState* __restrict__ ss, const TileShape tile,
                                                      const __grid_constant__ CUtensorMap tm0,
                                                      const __grid_constant__ CUtensorMap tm1, int nx, int ny,
                                                      int tiles_x, StepOut* out) {
    constexpr int G = SCHEME == 0 ? 1 : 2;
    extern __shared__ __align__(1024) double smem[];
    __shared__ uint64_t bar;
    // the step's scalars live here, not in registers across the stencil: dx and dy quotients, 0.5 dtp / dx, 0.5 dtp / dy, dt, dt before its clamp, dtp
    __shared__ double s_v[7];
    const int clamp = c->clamp, p = (int)(c->step & 1);
    const double t = c->t, t_end = c->t_end;
    if (clamp && t == t_end) {   // the loop stops here
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            c->done = 1;
            c->snap_pre = c->snap_post = 0;
        }
        return;
    }
    const RowShape S{tile};
    const int tx = tile.tx, ty = tile.ty, ux = tx + 2 * G, uxy = ux * (ty + 2 * G);
    double* sU = smem;
    double* sW = smem + 4 * uxy;
    const BlockDev& B = m->b[0];
    const int x0 = (blockIdx.x % tiles_x) * tx, y0 = (blockIdx.x / tiles_x) * ty;
    // TimeStep (timestep.cpp:29-68), its clamp (simulation.cpp:88-90) and the predictor's call
    // (muscl_hancock.cpp:246-249) while the tile is in flight; a direction's quotients per thread
    const bool forms = threadIdx.x == 0 || threadIdx.x == 32;
    const int d = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_expect_tx(&bar, 4 * uxy * 8);
        tma_load_3d(sU, p ? &tm1 : &tm0, &bar, x0, y0, 0);
    }
    // a ghost cell per thread of a tile on the block's edge, read while the tile is in flight
    const bool edge = x0 < G || y0 < G || x0 + tx + G > nx || y0 + ty + G > ny;
    double u[4];
    const bool ghost = edge && (int)threadIdx.x < uxy &&
                       tile_ghost<G>(m, B, B.buf[p], nx, ny, ux, threadIdx.x, x0, y0, u, &c->err);
    if (forms) s_v[d] = div_rn(d ? c->dy[0] : c->dx[0], smax(ss->solo[d], bitsd(c->int_s[p][0][d])));
    __syncthreads();
    if (forms) {
        const double least = smin(smin(1e16, s_v[0]), smin(1e16, s_v[1])), cfl = c->cfl;
        const long long call = c->calls;
        if (SCHEME == 1) {
            const double dtp = ((call + 2 <= 10) ? 0.2 * cfl : cfl) * least;
            s_v[2 + d] = div_rn(0.5 * dtp, d ? c->dy[0] : c->dx[0]);
            if (d == 0) s_v[6] = dtp;
        }
        if (d == 0) {
            const double dt = ((call + 1 <= 10) ? 0.2 * cfl : cfl) * least;
            s_v[4] = clamp && t + dt > t_end ? t_end - t : dt;
            s_v[5] = dt;
        }
    }
    if (wait_tile(&bar, c)) {
        if (edge) {
            if (ghost)
#pragma unroll
                for (int v = 0; v < 4; ++v) sU[v * uxy + threadIdx.x] = u[v];
            for (int it = threadIdx.x + kNT; it < uxy; it += kNT)
                if (tile_ghost<G>(m, B, B.buf[p], nx, ny, ux, it, x0, y0, u, &c->err))
#pragma unroll
                    for (int v = 0; v < 4; ++v) sU[v * uxy + it] = u[v];
            __syncthreads();
        }
        const double g = c->gamma, g1 = c->g1;
        const int herr = SCHEME == 0
            ? go_tile_fluxes<kNT>(S, sU, sW, g, g1, x0, y0, nx, ny, &c->first_bad, face_key(c->step, 0, 0, 0, 0))
            : mh_tile_fluxes<kNT, LIM>(S, sU, sW, g, g1, s_v[2], s_v[3], x0, y0, nx, ny, &c->first_bad,
                                       face_key(c->step, 0, 0, 0, 0));
        double mx = 0.0, my = 0.0;
        store_tile<kNT, G>(S, sU, sW, B, x0, y0, B.buf[p ^ 1], nullptr, s_v[4], ss->solo[2], ss->solo[3], g, g1,
                           &c->first_nonpos, face_key(c->step, 0, 0, 0, 0), mx, my, &c->err);
        store_ghosts<G, kNT>(sU, B, tx, ty, x0, y0, B.buf[p ^ 1], &c->err);
        block_max2_atomic<kNT>(mx, my, &c->int_s[p ^ 1][0][0], &c->int_s[p ^ 1][0][1]);
        if (herr) atomicAdd(reinterpret_cast<unsigned long long*>(&c->hllc_errors), (unsigned long long)herr);
    }
    if (!last_cta(&ss->tiles)) return;
    c->done = 0;
    c->snap_pre = c->snap_post = 0;
    c->dt_cfl = s_v[5];
    c->dt = s_v[4];
    if (SCHEME == 1) c->dt_pred[0] = s_v[6];
    c->calls = c->calls + 1;
    finish_step(c, out);
}

// ------------------------------------------------------------------------------------
// launchers
// ------------------------------------------------------------------------------------
TileShape tile_shape(int tx, int ty) {
    TileShape t;
    t.tx = tx;
    t.ty = ty;
    for (int k = 0; k < 3; ++k) t.m[k] = ((1u << 21) + (unsigned)(tx + k) - 1) / (unsigned)(tx + k);
    return t;
}

bool tile_fits(int scheme, int tx, int ty) {
    return (scheme == 0 ? go_tile_doubles(tx, ty) : mh_tile_doubles(tx, ty)) <= kTileDoubles;
}

// What a tile costs: microseconds of an SM that has enough of them (`work`), and from start to end of a
// CTA alone on its SM (`alone`): the warp-items of its phases at their instruction counts, a time per tile,
// and (model 0) what the rounds of the CTA's 14 warps leave idle.  Fitted to steps of many tiles and of one
// per SM: MUSCL-Hancock tiles of 32 x 19, 16 x 16 and 32 x 4 cells take 44.5, 22.2 and 13.4 us of an SM (both
// models within 7 %); with 32 x 14, alone, 55.5, 30.8, 18.0 and 47.5 us.
TileCost tile_cost(int scheme, int model, int tx, int ty) {
    constexpr int W = kNT / 32;
    auto warps = [](int items) { return (items + 31) / 32; };
    const int faces = warps((tx + 1) * ty) + warps(tx * (ty + 1)), cells = warps(tx * ty);
    const int first = scheme == 0 ? warps((tx + 2) * (ty + 2)) : warps((tx + 2) * ty) + warps(tx * (ty + 2));
    const double items = scheme == 0 ? 0.55 * first + 0.95 * faces + 0.75 * cells : 2.0 * first + 2.2 * faces + 0.8 * cells;
    const double rounds = (scheme == 0 ? 0.35 : 1.0) * ((std::max(first, faces) + W - 1) / W);
    return {model == 0 ? 1.9 + 0.196 * items + 2.34 * rounds : 2.5 + 0.23 * items, 3.0 + 0.165 * items + 7.2 * rounds};
}

// The tile: of the even widths (a TMA copy starts on 16 bytes) and heights that fit a CTA's shared memory,
// the one whose tiles are done first on the 2 x sms resident CTAs.  A mesh of many tiles gets the shape with
// the fewest wasted lanes and halo items, by the rounds of a CTA's 14 warps over the tile's cells and faces at
// their instruction counts; a small one, of fewer cells than one round of the largest tiles holds, a shape that
// fills the GPU once, by tile_cost's model of the work (256^2 in 32 x 19 tiles would leave 44 of 152 SMs
// without any).  Measured, us a step by the first and by the second: Godunov 256^2 29.1, 26.8, 512^2 69.2, 77.9;
// MUSCL-Hancock 256^2 55.4, 49.3, 400^2 98.4, 94.6, 777 x 1000 384, 402.
TileShape choose_tile(int scheme, const int* nx, const int* ny, int nb, int sms) {
    constexpr int W = kNT / 32;
    auto warps = [](int items) { return (items + 31) / 32; };
    auto rounds = [](int w) { return (w + W - 1) / W; };
    long long cells = 0;
    for (int b = 0; b < nb; ++b) cells += (long long)nx[b] * ny[b];
    const bool small = cells < 2LL * sms * 32 * 19;
    double best = 0.0;
    int bx = 8, by = 2;
    for (int tx = 8; tx <= 64; tx += 2)
        for (int ty = 2; ty <= 32; ++ty) {
            if (!tile_fits(scheme, tx, ty)) continue;
            long long n = 0;
            for (int b = 0; b < nb; ++b) n += (long long)((nx[b] + tx - 1) / tx) * ((ny[b] + ty - 1) / ty);
            double shared, alone;   // a tile's time beside another one on its SM, and alone there
            if (small) {
                const TileCost t = tile_cost(scheme, 1, tx, ty);
                shared = std::max(2.0 * t.work, t.alone);
                alone = t.alone;
            } else {
                const int faces = rounds(warps((tx + 1) * ty) + warps(tx * (ty + 1))), own = rounds(warps(tx * ty));
                shared = scheme == 0
                    ? 550.0 * rounds(warps((tx + 2) * (ty + 2))) + 950.0 * faces + 750.0 * own + 400.0
                    : 2000.0 * rounds(warps((tx + 2) * ty) + warps(tx * (ty + 2))) + 2200.0 * faces + 800.0 * own + 600.0;
                alone = 0.6 * shared;
            }
            const long long rest = n % (2 * sms);
            const double time = (double)(n / (2 * sms)) * shared + (rest == 0 ? 0.0 : rest <= sms ? alone : shared);
            if (best == 0.0 || time < best) {
                best = time;
                bx = tx;
                by = ty;
            }
        }
    return tile_shape(bx, by);
}

void step_plan_tiles(StepPlan& plan, int b, int nx, int ny) {
    plan.tiles_x[b] = (nx + plan.tile.tx - 1) / plan.tile.tx;
    plan.tile_start[b + 1] = plan.tile_start[b] + plan.tiles_x[b] * ((ny + plan.tile.ty - 1) / plan.tile.ty);
}

cudaError_t launch_step(Ctrl* c, const MeshDev* m, StepState* ss, const StepPlan& plan, int scheme, int limiter,
                        cudaStream_t s) {
    if (plan.nb < 1 || plan.nb > kStepMaxBlocks) return cudaErrorInvalidValue;
    const int tiles = plan.tile_start[plan.nb];
    if (scheme == 0) {
        godunov_step_kernel<<<tiles, kNT, kTileBytes, s>>>(c, m, ss, plan);
        return cudaGetLastError();
    }
    if (limiter == 0) mh_step_kernel<0><<<tiles, kNT, kTileBytes, s>>>(c, m, ss, plan);
    else mh_step_kernel<1><<<tiles, kNT, kTileBytes, s>>>(c, m, ss, plan);
    // a block run again on a fixed grid: with nothing to do (nearly always) few CTAs come and go
    const int again = tiles < 2 * 152 ? tiles : 2 * 152;
    for (int b = 1; b < plan.nb; ++b) {
        if (limiter == 0) mh_rerun_kernel<0><<<again, kNT, kTileBytes, s>>>(c, m, ss, plan);
        else mh_rerun_kernel<1><<<again, kNT, kTileBytes, s>>>(c, m, ss, plan);
    }
    return cudaGetLastError();
}

cudaError_t prepare_solo(Ctrl* c, const MeshDev* m, StepState* ss, cudaStream_t s) {
    prepare_solo_kernel<<<1, 1, 0, s>>>(c, m, ss);
    return cudaGetLastError();
}

cudaError_t launch_solo(Ctrl* c, const MeshDev* m, StepState* ss, int nx, int ny, int scheme, int limiter,
                        const TileShape& tile, const CUtensorMap* tm0, const CUtensorMap* tm1, cudaStream_t s,
                        StepOut* out) {
    const int across = (nx + tile.tx - 1) / tile.tx, tiles = across * ((ny + tile.ty - 1) / tile.ty);
    if (scheme == 0) solo_kernel<0, 0><<<tiles, kNT, kTileBytes, s>>>(c, m, ss, tile, *tm0, *tm1, nx, ny, across, out);
    else if (limiter == 0) solo_kernel<1, 0><<<tiles, kNT, kTileBytes, s>>>(c, m, ss, tile, *tm0, *tm1, nx, ny, across, out);
    else solo_kernel<1, 1><<<tiles, kNT, kTileBytes, s>>>(c, m, ss, tile, *tm0, *tm1, nx, ny, across, out);
    return cudaGetLastError();
}

// (of the scheme's kernels alone: an opt-in costs a creation about a microsecond)
cudaError_t stencil_prepare(int scheme, int limiter) {
    const void* const kernels[3][4] = {
        {(const void*)godunov_step_kernel, (const void*)godunov_kernel, (const void*)solo_kernel<0, 0>, nullptr},
        {(const void*)mh_step_kernel<0>, (const void*)mh_rerun_kernel<0>, (const void*)mh_kernel<0>, (const void*)solo_kernel<1, 0>},
        {(const void*)mh_step_kernel<1>, (const void*)mh_rerun_kernel<1>, (const void*)mh_kernel<1>, (const void*)solo_kernel<1, 1>}};
    for (const void* k : kernels[scheme == 0 ? 0 : limiter == 0 ? 1 : 2]) {
        const cudaError_t e = k ? cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileBytes)
                                : cudaSuccess;
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_step_begin(Ctrl* c, cudaStream_t s) {
    step_begin_kernel<<<1, 1, 0, s>>>(c);
    return cudaGetLastError();
}

cudaError_t launch_fill_cfl(Ctrl* c, const MeshDev* m, long long total_ghost, cudaStream_t s, int form_dt,
                            StepState* ss) {
    long long grid = (total_ghost + kRedThreads - 1) / kRedThreads;
    fill_cfl_kernel<<<(unsigned)(grid < 1 ? 1 : grid), kRedThreads, 0, s>>>(c, m, form_dt, ss);
    return cudaGetLastError();
}

cudaError_t launch_ghost_mirror(Ctrl* c, const MeshDev* m, long long total_ghost, cudaStream_t s) {
    long long grid = (total_ghost + 255) / 256;
    ghost_mirror_kernel<<<(unsigned)(grid < 1 ? 1 : grid), 256, 0, s>>>(c, m);
    return cudaGetLastError();
}

cudaError_t launch_ghost_cfl(Ctrl* c, const MeshDev* m, long long total_ghost, cudaStream_t s, int form_dt) {
    long long want = (total_ghost + kRedThreads - 1) / kRedThreads;
    int grid = (int)(want < 1 ? 1 : (want > 4 * 152 ? 4 * 152 : want));
    ghost_cfl_kernel<<<grid, kRedThreads, 0, s>>>(c, m, form_dt);
    return cudaGetLastError();
}

cudaError_t launch_interior_cfl(Ctrl* c, const MeshDev* m, int b, int nx, int ny, int parity,
                                cudaStream_t s) {
    long long want = ((long long)nx * ny + kRedThreads - 1) / kRedThreads;
    int grid = (int)(want < 1 ? 1 : (want > 8 * 152 ? 8 * 152 : want));
    interior_cfl_kernel<<<grid, kRedThreads, 0, s>>>(c, m, b, parity);
    return cudaGetLastError();
}

cudaError_t launch_set_dt(Ctrl* c, double dt, cudaStream_t s) {
    set_dt_kernel<<<1, 1, 0, s>>>(c, dt);
    return cudaGetLastError();
}

// k x k box average of one block's interior in FP64, stored as FP32 [4][ny/k][nx/k]
__global__ void __launch_bounds__(256) coarsen_kernel(const Ctrl* __restrict__ c,
                                                      const MeshDev* __restrict__ m, int b, int k,
                                                      float* __restrict__ out) {
    const BlockDev& B = m->b[b];
    const double* __restrict__ U = B.buf[(int)(c->step & 1)];
    const int g = m->ghost, cx = B.nx / k, cy = B.ny / k;
    const long long n = 4LL * cx * cy;
    const double inv = 1.0 / ((double)k * (double)k);
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x) {
        const int v = (int)(q / ((long long)cx * cy));
        const long long r = q - (long long)v * cx * cy;
        const int j = (int)(r / cx), i = (int)(r - (long long)j * cx);
        const double* base = U + (size_t)v * B.ty * B.pitch + (size_t)(j * k + g) * B.pitch + (i * k + g);
        double acc = 0.0;
        for (int jj = 0; jj < k; ++jj)
            for (int ii = 0; ii < k; ++ii) acc += base[(size_t)jj * B.pitch + ii];
        out[q] = (float)(acc * inv);
    }
}

cudaError_t launch_coarsen(const Ctrl* c, const MeshDev* m, int b, int k, long long n, float* out,
                           cudaStream_t s) {
    long long want = (n + 255) / 256;
    int grid = (int)(want < 1 ? 1 : (want > 8 * 152 ? 8 * 152 : want));
    coarsen_kernel<<<grid, 256, 0, s>>>(c, m, b, k, out);
    return cudaGetLastError();
}

cudaError_t launch_frame_copy(Ctrl* c, const MeshDev* m, const FrameRing& ring, cudaStream_t s) {
    frame_copy_kernel<<<4 * 152, 256, 0, s>>>(c, m, ring);
    return cudaGetLastError();
}

cudaError_t launch_finalize(Ctrl* c, cudaStream_t s) {
    finalize_kernel<<<1, 1, 0, s>>>(c);
    return cudaGetLastError();
}

cudaError_t launch_stencil(Ctrl* c, const MeshDev* m, int b, int nx, int ny, int scheme, int limiter,
                           const TileShape& tile, const CUtensorMap* tm0, const CUtensorMap* tm1, cudaStream_t s,
                           double* hout) {
    const int tiles = ((nx + tile.tx - 1) / tile.tx) * ((ny + tile.ty - 1) / tile.ty);
    if (scheme == 0)
        godunov_kernel<<<tiles, kNT, kTileBytes, s>>>(c, m, b, tile, *tm0, *tm1, hout);
    else if (limiter == 0)
        mh_kernel<0><<<tiles, kNT, kTileBytes, s>>>(c, m, b, tile, *tm0, *tm1, hout);
    else
        mh_kernel<1><<<tiles, kNT, kTileBytes, s>>>(c, m, b, tile, *tm0, *tm1, hout);
    return cudaGetLastError();
}

// CTAs of the copies over the host link: a warp per 32 cells, at most as many as keep the link busy
static int link_grid(int tx, int ty) {
    const long long want = ((long long)((tx + 31) / 32) * ty + kRedThreads / 32 - 1) / (kRedThreads / 32);
    return (int)(want < 1 ? 1 : (want > 8 * 152 ? 8 * 152 : want));
}

cudaError_t launch_upload(Ctrl* c, const MeshDev* m, int b0, int nb, const int* tx, const int* ty, int parity,
                          const HostBlocks& h, cudaStream_t s) {
    int grid = 1;
    for (int k = 0; k < nb; ++k) grid = std::max(grid, link_grid(tx[k], ty[k]));
    upload_kernel<<<dim3((unsigned)grid, (unsigned)nb), kRedThreads, 0, s>>>(c, m, b0, parity, h);
    return cudaGetLastError();
}

cudaError_t launch_download(Ctrl* c, const MeshDev* m, int b, int tx, int ty, int parity, double* hout, cudaStream_t s) {
    const long long want = (4LL * tx * ty + 31) / (4 * kRedThreads) + 1;   // (the array may start inside a line)
    static_assert(kDownLines == 4, "a CTA takes 4 doubles a thread");
    download_kernel<<<(unsigned)(want > 8 * 152 ? 8 * 152 : want), kRedThreads, 0, s>>>(c, m, b, parity, hout);
    return cudaGetLastError();
}

cudaError_t launch_ghost_store(Ctrl* c, const MeshDev* m, int nb, const int* tx, const int* ty, int ghost, int parity,
                               const HostBlocks& h, cudaStream_t s) {
    long long n = 1;
    for (int k = 0; k < nb; ++k) n = std::max(n, 2LL * ghost * (tx[k] + ty[k]));
    ghost_store_kernel<<<dim3((unsigned)((n + 255) / 256), (unsigned)nb), 256, 0, s>>>(c, m, parity, h);
    return cudaGetLastError();
}

}  // namespace hf
