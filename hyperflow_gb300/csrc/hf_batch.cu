// Batched single-block cases: hundreds of independent, all-transmissive cases of different
// sizes advanced together, one launch per step, a run of steps captured in a
// CUDA graph, each case with its own CFL dt.  C ABI in include/hyperflow_gb300_batch.h.
//
// Each case is the reference's single-block MUSCL-Hancock step
// (src/fvm_2d_cart/scheme/muscl_hancock/muscl_hancock.cpp:41-376 + TimeStep +
// ForwardEuler) or Godunov step (src/fvm_2d_cart/scheme/godunov/godunov.cpp:27-118 + TimeStep +
// ForwardEuler); all cases of a batch use the same scheme.  With transmissive boundaries on all
// four sides every ghost value is a mirror copy of an interior value
// (transmissive_boundary.cpp:25-104; the fill order makes corner ghosts mirror in x and in y).
// So the tile loader reads the mirrored interior cell directly and the state is stored without
// ghosts, and the CFL maximum over ghost cells equals the maximum over the interior.
//
// Work decomposition: every case is cut into tiles; the tiles of all cases form one list, the
// dearest first, a CTA each.  The CFL maxima rotate through three slots: read (this step's
// dt), write (the next step's, by the update epilogue), and one that the step before cleared; the
// last CTA of a step clears the slot just read and counts the step.
//
// (A step was a round of a persistent cooperative kernel: one launch per run, a grid barrier per
// step.  The loop's state cost the tile computation registers, and a CTA's next tile waited for its
// descriptor: with the same tiles 54.3 against 52.6 ms for 100 steps of 24 cases of 64^2 .. 385^2,
// Godunov 22.7 against 21.0, and 2.39 against 2.23 for two cases of 16^2 and 81^2.  Letting the next
// step's CTAs take their places during a step's tail gave nothing on large batches and put two on
// one SM where there are fewer tiles than SMs: 9.7 against 6.0 ms for one case of 256^2.)
//
// Autotuning: two configurations give each case a tile shape of its own (case_tiles), the others one
// shape for all; the autotuner times each on the real batch and keeps the fastest.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <string>
#include <vector>

#include "../../include/hyperflow_gb300_batch.h"
#include "hf_cart.h"
#include "hf_device.cuh"
#include "hf_trace.h"
#include "hf_godunov_tile.cuh"
#include "hf_mh_tile.cuh"

namespace hf {

struct BatchInst {
    int n;                 // cells per side
    int pitch;             // doubles per row: n rounded up to even (a TMA row stride is a multiple of 16 bytes)
    long long off;         // offset (doubles) of the case's [4][n][pitch] state
    double dx, dy, one_dx, one_dy;   // and 1 / dx, 1 / dy
};

// One tile of the batch
struct __align__(16) BatchTile {
    int inst, x0, y0;        // interior cells
    int n, pitch;            // the case's
    int tx, ty;
    unsigned int m[3];       // TileShape's
    long long off;           // the case's
};
static_assert(sizeof(BatchTile) == 48, "a tile is copied in 16-byte pieces");

struct BatchCtrl {
    double gamma, g1, cfl;
    long long calls;        // TimeStep calls made by every case so far
    long long step;         // steps completed
    int ninst;
    int err;
    unsigned int tiles_done;           // of the running step
    long long hllc_errors;
    unsigned long long first_nonpos;   // least batch_key of a cell a step left with density or
                                       // pressure not positive, ~0 when none
};

// Key of a cell for the earliest non-positive record: the step (24 bits, saturating), then the
// cell's offset in the batch state (40 bits: the case's offset + j * n + i), which orders by case,
// row, column.
__device__ __forceinline__ unsigned long long batch_key(long long step, long long off) {
    const unsigned long long s = step > 0xFFFFFFll ? 0xFFFFFFull : (unsigned long long)step;
    return (s << 40) | ((unsigned long long)off & 0xFFFFFFFFFFull);
}

struct BatchDev {
    BatchCtrl* ctrl;
    const BatchInst* inst;
    const CUtensorMap* maps;       // MUSCL-Hancock: per state parity, per case, [2][ninst]
    int ninst;
    const BatchTile* tiles;        // [ntiles]
    long long ntiles;
    double* U[2];
    unsigned long long* acc;       // [3][ninst][2]
    double* t;                     // [ninst]
    double* last_dt;               // [ninst]
};

__device__ __forceinline__ int mirror(int x, int n) {
    x = x < 0 ? -1 - x : (x >= n ? 2 * n - 1 - x : x);
    return x < 0 ? 0 : (x >= n ? n - 1 : x);   // positions past the 2-cell halo are never used
}

constexpr unsigned kBatchWaitLimit = 1u << 22;   // bounded mbarrier polls before giving up

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// The halo positions outside the case (within 2 cells of it) take the mirrored interior values,
// the transmissive ghosts (transmissive_boundary.cpp:25-104; corners mirrored in x and in y).
// Every source is an interior cell inside the same box.  Positions further out are never read.
// A warp's row at a time; ends with __syncthreads() where there was something to write.
template <int NT>
__device__ __forceinline__ void mirror_halo(double* sU, int tx, int ty, int x0, int y0, int n) {
    constexpr int H = 2;
    if (x0 >= H && y0 >= H && x0 + tx + H <= n && y0 + ty + H <= n) return;   // the box lies inside the case
    const int ux = tx + 2 * H, uy = ty + 2 * H;
    for (int r = threadIdx.x >> 5; r < 4 * uy; r += NT / 32) {
        const int ly = r % uy, gy = y0 + ly - H;
        if (gy < -H || gy >= n + H) continue;
        double* const row = sU + r * ux;
        const double* const from = row + (mirror(gy, n) - gy) * ux;
        for (int lx = threadIdx.x & 31; lx < ux; lx += 32) {
            const int gx = x0 + lx - H;
            if (gx < -H || gx >= n + H || (gx >= 0 && gx < n && gy >= 0 && gy < n)) continue;
            row[lx] = from[lx + mirror(gx, n) - gx];
        }
    }
    __syncthreads();
}

// One step of every case, a CTA per tile.
// What bounds it: the FP64 and integer pipes of the tile computation, as in the Cartesian step kernel,
// whose CTA it shares (two per SM, any tile that fits 110.9 KB); beyond that the lanes a
// tile wastes on the part of it outside its case, and the tail of a step.  So a case has a tile that
// divides it well, and the dearest tiles are dispatched first.  Measured (Mcell-updates/s, 100 steps;
// before: the best of the fixed shapes, in a persistent kernel): 24 cases of 64^2 .. 385^2 1902 (1738),
// Godunov 4753 (4036); 64 of 48^2 .. 97^2 1729 (1148); 8 of 128^2 1526 (1327); 40 of 83^2 .. 501^2 1963.
// One block of 2048^2 on the Cartesian path, without a tail or partial tiles to speak of, has 2108.
//
// MUSCL-Hancock tiles come by TMA: one 3-D box (the tile and its 2-cell halo, all four variables) of
// the case's state, issued by thread 0; positions outside the case arrive as zeros and mirror_halo
// then writes the transmissive ghosts there.  (The box's x start, x0 - 2, is even, as a TMA copy of
// FP64 needs; Godunov's 1-cell halo would start at an odd x, so Godunov batches load by element.)
template <int NT, int SCHEME, int LIM>
__global__ void __launch_bounds__(NT, 2) batch_kernel(const __grid_constant__ BatchDev d) {
    constexpr int H = SCHEME == 1 ? 2 : 1;
    constexpr int CALLS = SCHEME == 1 ? 2 : 1;   // TimeStep calls per step (+ the predictor's)
    extern __shared__ __align__(1024) double smem[];
    double* const sU = smem;
    __shared__ double sc[3];
    __shared__ uint64_t bar;
    BatchCtrl* const c = d.ctrl;
    const BatchTile T = d.tiles[blockIdx.x];
    const RowShape S{{T.tx, T.ty, {T.m[0], T.m[1], T.m[2]}}};
    const int usize = 4 * (T.tx + 2 * H) * (T.ty + 2 * H);
    double* const sW = smem + usize;
    const int p = (int)(c->step & 1), ar = (int)(c->step % 3);
    if (threadIdx.x == 0) {
        if (SCHEME == 1) {
            mbar_init(&bar, 1);
            mbar_expect_tx(&bar, usize * 8);
            tma_load_3d(sU, &d.maps[(size_t)p * d.ninst + T.inst], &bar, T.x0 - H, T.y0 - H, 0);
        }
        // TimeStep::operator() for this case (timestep.cpp:29-68) from last step's maxima
        const unsigned long long* a = d.acc + ((size_t)ar * d.ninst + T.inst) * 2;
        const double dx = d.inst[T.inst].dx, dy = d.inst[T.inst].dy, cfl = c->cfl;
        const double dtx = smin(1e16, div_rn(dx, bitsd(a[0])));
        const double dty = smin(1e16, div_rn(dy, bitsd(a[1])));
        const double dt = ((c->calls + 1 <= 10) ? 0.2 * cfl : cfl) * smin(dtx, dty);    // the step's call
        sc[0] = dt;
        if (SCHEME == 1) {
            const double dtp = ((c->calls + 2 <= 10) ? 0.2 * cfl : cfl) * smin(dtx, dty);   // the predictor's
            sc[1] = div_rn(0.5 * dtp, dx);   // muscl_hancock.cpp:248-249
            sc[2] = div_rn(0.5 * dtp, dy);
        }
        if (T.x0 == 0 && T.y0 == 0) {
            d.t[T.inst] = d.t[T.inst] + dt;
            d.last_dt[T.inst] = dt;
        }
    }
    if (SCHEME == 1) {
        __syncthreads();   // the mbarrier is initialised
        const bool ok = mbar_wait_bounded(&bar, 0u, kBatchWaitLimit);
        if (__syncthreads_or(!ok || (threadIdx.x == 0 && c->err != 0))) {
            if (!ok && threadIdx.x == 0) {
                atomicCAS(&c->err, 0, (int)HF_DEV_TIMEOUT);
                mbar_wait_bounded(&bar, 0u, kBatchWaitLimit);   // let the copy in flight land before exit
            }
            __syncthreads();
            return;        // this step and those after it are not counted
        }
        mirror_halo<NT>(sU, T.tx, T.ty, T.x0, T.y0, T.n);
    } else {
        const double* __restrict__ base = d.U[p] + T.off;
        const int uxy = (T.tx + 2) * (T.ty + 2);
        for (int k = threadIdx.x; k < uxy; k += NT) {
            const int ly = S.row2(k), lx = k - ly * (T.tx + 2);
            const double* q = base + (size_t)mirror(T.y0 + ly - H, T.n) * T.pitch + mirror(T.x0 + lx - H, T.n);
#pragma unroll
            for (int v = 0; v < 4; ++v) cp_async8(sU + v * uxy + k, q + (size_t)v * T.pitch * T.n);
        }
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
        __syncthreads();
    }
    const double g = c->gamma, g1 = c->g1;
    const int herr = SCHEME == 0 ? go_tile_fluxes<NT>(S, sU, sW, g, g1, T.x0, T.y0, T.n, T.n)
                                 : mh_tile_fluxes<NT, LIM>(S, sU, sW, g, g1, sc[1], sc[2], T.x0, T.y0, T.n, T.n);
    double mx = 0.0, my = 0.0;
    const double dt = sc[0], one_dx = d.inst[T.inst].one_dx, one_dy = d.inst[T.inst].one_dy;
    const size_t plane = (size_t)T.pitch * T.n;
#pragma unroll 1
    for (int it = threadIdx.x; it < T.tx * T.ty; it += NT) {
        const int oy = S.row0(it), ox = it - oy * T.tx;
        const int gx = T.x0 + ox, gy = T.y0 + oy;
        if (gx >= T.n || gy >= T.n) continue;
        double un[4];
        if (SCHEME == 0) go_update(S, sU, sW, ox, oy, dt, one_dx, one_dy, un);
        else mh_update(S, sU, sW, ox, oy, dt, one_dx, one_dy, un);
        const long long at = T.off + (long long)gy * T.pitch + gx;
        double* const out = d.U[p ^ 1] + at;
#pragma unroll
        for (int v = 0; v < 4; ++v) out[v * plane] = un[v];
        double sx, sy;
        if (!speeds(g, g1, un, sx, sy)) atomicMin(&c->first_nonpos, batch_key(c->step, at));
        mx = nmax(mx, sx);
        my = nmax(my, sy);
    }
    unsigned long long* const aw = d.acc + ((size_t)(ar == 2 ? 0 : ar + 1) * d.ninst + T.inst) * 2;
    block_max2_atomic<NT>(mx, my, aw, aw + 1);
    if (herr) atomicAdd(reinterpret_cast<unsigned long long*>(&c->hllc_errors), (unsigned long long)herr);
    // the last CTA ends the step: the maxima just read are cleared (the next step but one writes them)
    __shared__ int last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(&c->tiles_done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    for (int i = threadIdx.x; i < 2 * d.ninst; i += NT) d.acc[(size_t)ar * 2 * d.ninst + i] = 0ull;
    if (threadIdx.x == 0) {
        c->tiles_done = 0u;
        c->step = c->step + 1;
        c->calls = c->calls + CALLS;
    }
}

// CFL maxima of the current state, into slot step % 3 (after an upload): a row of CTAs per case from
// `first`
constexpr int kCflThreads = 256;
__global__ void __launch_bounds__(kCflThreads) batch_cfl_kernel(BatchDev d, int first, int count) {
    BatchCtrl* c = d.ctrl;
    const long long step = c->step;
    const int p = (int)(step & 1), ar = (int)(step % 3);
    const double g = c->gamma, g1 = c->g1;
    for (int i = blockIdx.y; i < count; i += gridDim.y) {
        const BatchInst I = d.inst[first + i];
        const double* U = d.U[p] + I.off;
        const size_t plane = (size_t)I.pitch * I.n;
        double mx = 0.0, my = 0.0;
        for (int gy = blockIdx.x; gy < I.n; gy += gridDim.x)
            for (int gx = threadIdx.x; gx < I.n; gx += kCflThreads) {
                const size_t o = (size_t)gy * I.pitch + gx;
                const double u[4] = {U[o], U[plane + o], U[2 * plane + o], U[3 * plane + o]};
                double sx, sy;
                speeds(g, g1, u, sx, sy);
                mx = nmax(mx, sx);
                my = nmax(my, sy);
            }
        unsigned long long* a = d.acc + ((size_t)ar * c->ninst + first + i) * 2;
        block_max2_atomic<kCflThreads>(mx, my, a, a + 1);
        __syncthreads();   // block_max2_atomic's shared memory is used again
    }
}

// A configuration's tile shape and CTA.  tx = 0: each case has its own (case_tiles), by a model that
// counts what the rounds of a CTA's warps leave idle beside the work, or (model 1) the work alone: the first
// was better for batches of several rounds of tiles (24 cases of 64^2 .. 385^2: 52.5 against 56.3 ms for 100
// steps), the second for smaller ones (8 of 128^2: 9.61, 8.66; one of 256^2: 5.28, 4.68).  Of the fixed
// shapes, timed on 72 batches of 1 to 200 cases, the fifth beat both by up to 9 % on five (8 of 128^2, Godunov: 36.8
// against 40.6 us a step, MUSCL-Hancock 84.6, 88.7) and the sixth by up to 15 % on three (8 of 64^2,
// MUSCL-Hancock: 36.6, 43.1); the third and fourth by no more than 0.1 % on any: they stay for callers that
// select a configuration by its number.
struct BatchConfig {
    int tx, ty, threads, model;
};
constexpr BatchConfig kConfigs[] = {{0, 0, 448, 0},   {0, 0, 448, 1},   {32, 19, 448, 0},
                                    {24, 25, 448, 0}, {32, 14, 256, 0}, {32, 4, 448, 0}};
constexpr int kNumConfigs = 6;

template <int NT>
cudaError_t launch_threads(int scheme, int limiter, const BatchDev& d, long long nsteps, cudaStream_t s) {
    auto k = scheme == 0 ? batch_kernel<NT, 0, 0> : limiter == 0 ? batch_kernel<NT, 1, 0> : batch_kernel<NT, 1, 1>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileBytes);
    if (e != cudaSuccess) return e;
    for (long long i = 0; i < nsteps && e == cudaSuccess; ++i) {
        k<<<(unsigned)d.ntiles, NT, kTileBytes, s>>>(d);
        e = cudaGetLastError();
    }
    return e;
}

cudaError_t launch_batch(int k, int scheme, int limiter, const BatchDev& d, long long nsteps, cudaStream_t s) {
    return kConfigs[k].threads == 256 ? launch_threads<256>(scheme, limiter, d, nsteps, s)
                                      : launch_threads<448>(scheme, limiter, d, nsteps, s);
}

// The tile shape of each case (sides n) by a model.  A case takes, of the shapes whose whole
// tile is within a limit, the one whose tiles are the least work (the last row of tiles has as many rows
// as the case has left); the limit is the one with which the tiles, dealt dearest first to the
// 2 x sms resident CTAs, are done first.  No limit wastes the fewest lanes and halo items and suits a batch
// of many rounds of tiles; a small batch needs more, smaller tiles.
std::vector<TileShape> case_tiles(int scheme, int model, const std::vector<int>& n, int sms) {
    struct Shape {
        int tx, ty;
        double time;   // of a whole tile beside another on its SM
        int order;
    };
    auto shared_time = [](const TileCost& c) { return std::max(2.0 * c.work, c.alone); };
    // the model's costs, once: a case looks up a whole tile and its last row for every shape
    std::vector<TileCost> costs(29 * 32);
    auto cost = [&](int tx, int ty) -> TileCost& { return costs[(tx - 8) / 2 * 32 + ty - 1]; };
    std::vector<Shape> shapes;
    double lo = 0.0, hi = 0.0;
    for (int tx = 8; tx <= 64; tx += 2)
        for (int ty = 1; ty <= 32; ++ty) {
            cost(tx, ty) = tile_cost(scheme, model, tx, ty);
            if (ty < 2 || !tile_fits(scheme, tx, ty)) continue;
            const double t = shared_time(cost(tx, ty));
            shapes.push_back({tx, ty, t, (int)shapes.size()});
            lo = lo == 0.0 ? t : std::min(lo, t);
            hi = std::max(hi, t);
        }
    std::sort(shapes.begin(), shapes.end(),
              [](const Shape& a, const Shape& b) { return a.time < b.time || (a.time == b.time && a.order < b.order); });
    std::vector<double> limits;
    for (double l = hi; l > lo; l *= 0.85) limits.push_back(l);
    limits.push_back(lo);
    // per distinct side and limit: the shape of the least work, the narrower and lower of two alike (the shapes
    // by their time, so one pass serves every limit)
    std::map<int, std::vector<int>> best;
    for (int side : n) {
        if (best.count(side)) continue;
        std::vector<int> at(limits.size(), -1);
        int pick = -1, across[29], whole[33], rest[33];   // by tx, and by ty
        for (int i = 0; i < 29; ++i) across[i] = (side + 7 + 2 * i) / (8 + 2 * i);
        for (int ty = 1; ty <= 32; ++ty) {
            whole[ty] = side / ty;
            rest[ty] = side % ty;
        }
        double least = 0.0;
        size_t k = 0;
        for (size_t l = limits.size(); l-- > 0;) {
            for (; k < shapes.size() && shapes[k].time <= limits[l]; ++k) {
                const Shape& s = shapes[k];
                const double column = (double)whole[s.ty] * cost(s.tx, s.ty).work +
                                      (rest[s.ty] ? cost(s.tx, rest[s.ty]).work : 0.0);
                const double work = column * across[(s.tx - 8) / 2];
                if (pick < 0 || work < least || (work == least && s.order < shapes[pick].order)) {
                    least = work;
                    pick = (int)k;
                }
            }
            at[l] = pick;
        }
        best.emplace(side, std::move(at));
    }
    size_t pick = 0;
    double done = 0.0;
    for (size_t l = 0; l < limits.size(); ++l) {
        std::map<double, std::pair<long long, double>> kinds;   // shared time -> tiles, their time alone
        double work = 0.0;
        long long tiles = 0;
        auto add = [&](int tx, int ty, long long k) {
            const TileCost c = cost(tx, ty);
            auto& e = kinds[shared_time(c)];
            e.first += k;
            e.second = c.alone;
            work += c.work * (double)k;
            tiles += k;
        };
        for (int side : n) {
            const Shape& s = shapes[best[side][l]];
            const long long across = (side + s.tx - 1) / s.tx;
            if (side >= s.ty) add(s.tx, s.ty, across * (side / s.ty));
            if (side % s.ty) add(s.tx, side % s.ty, across);
        }
        double end = 0.0;
        if (tiles <= sms) {
            for (auto& e : kinds) end = std::max(end, e.second.second);
        } else if (tiles <= 24LL * sms) {
            // each tile to the CTA that is done first, alike ones together: end -> CTAs
            std::map<double, long long> cta{{0.0, 2LL * sms}};
            for (auto e = kinds.rbegin(); e != kinds.rend(); ++e)
                for (long long k = e->second.first; k > 0;) {
                    auto first = cta.begin();
                    const long long m = std::min(k, first->second);
                    cta[first->first + e->first] += m;
                    k -= m;
                    if ((first->second -= m) == 0) cta.erase(first);
                }
            // an SM's two CTAs: while one is done the other runs faster, but not twice as fast
            std::vector<double> f;
            for (auto& c : cta) f.insert(f.end(), (size_t)c.second, c.first);
            for (int k = 0; k < sms; ++k) end = std::max(end, f[k] + 0.65 * (f[2 * sms - 1 - k] - f[k]));
        } else {
            end = work / sms + 0.3 * kinds.rbegin()->first;   // of many rounds: their mean and a tail
        }
        if (l == 0 || end < done) {
            done = end;
            pick = l;
        }
    }
    std::vector<TileShape> out;
    for (int side : n) {
        const Shape& s = shapes[best[side][pick]];
        out.push_back(tile_shape(s.tx, s.ty));
    }
    return out;
}

}  // namespace hf

// =====================================================================================
// host side
// =====================================================================================
struct hf_batch {
    cudaStream_t stream = nullptr;
    int sms = 0;
    double gamma = 1.4, cfl = 0.8;
    int limiter = 0;
    int scheme = 1;             // 0 Godunov, 1 MUSCL-Hancock
    std::vector<hf::BatchInst> inst;
    long long total_cells = 0;
    long long total_doubles = 0;   // the state buffer: every case's [4][n][pitch]
    std::vector<void*> allocs;
    hf::BatchCtrl* dctrl = nullptr;
    hf::BatchInst* dinst = nullptr;
    double* U[2] = {nullptr, nullptr};
    unsigned long long* acc = nullptr;
    double* t = nullptr;
    double* last_dt = nullptr;
    // per configuration: device tile lists
    std::vector<hf::TileShape> shapes[hf::kNumConfigs];
    hf::BatchTile* tiles[hf::kNumConfigs] = {};
    long long ntiles[hf::kNumConfigs] = {};
    CUtensorMap* maps[hf::kNumConfigs] = {};   // MUSCL-Hancock: the TMA maps of the cases' tile boxes
    int config = 0;
    // graphs: key = (config, nsteps), a bounded number per configuration (batch_graph_steps)
    struct G { int config; long long nsteps; cudaGraphExec_t exec; };
    std::vector<G> graphs;
    std::string err;
};

namespace {

int bfail(hf_batch* b, int code, const std::string& m) {
    if (b) b->err = m;
    return code;
}

#define BCK(call)                                                                              \
    do {                                                                                       \
        cudaError_t e_ = (call);                                                               \
        if (e_ != cudaSuccess)                                                                 \
            return bfail(b, HF_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));  \
    } while (0)

int ensure_tiles(hf_batch* b, int k) {
    if (b->tiles[k]) return HF_OK;
    const hf::BatchConfig C = hf::kConfigs[k];
    const size_t n = b->inst.size();
    std::vector<int> sides(n);
    for (size_t i = 0; i < n; ++i) sides[i] = b->inst[i].n;
    b->shapes[k] = C.tx ? std::vector<hf::TileShape>(n, hf::tile_shape(C.tx, C.ty))
                        : hf::case_tiles(b->scheme, C.model, sides, b->sms);
    // rows of tiles, the dearest first
    struct Row {
        double time;
        int inst, y0;
    };
    std::vector<Row> rows;
    size_t ntiles = 0;
    for (size_t i = 0; i < n; ++i) {
        const hf::TileShape& s = b->shapes[k][i];
        for (int y0 = 0; y0 < sides[i]; y0 += s.ty)
            rows.push_back({hf::tile_cost(b->scheme, C.model, s.tx, std::min(s.ty, sides[i] - y0)).work, (int)i, y0});
        ntiles += (size_t)((sides[i] + s.tx - 1) / s.tx) * ((sides[i] + s.ty - 1) / s.ty);
    }
    std::stable_sort(rows.begin(), rows.end(), [](const Row& a, const Row& c) { return a.time > c.time; });
    std::vector<hf::BatchTile> tiles;
    tiles.reserve(ntiles);
    for (const Row& r : rows) {
        const hf::TileShape& s = b->shapes[k][r.inst];
        const hf::BatchInst& I = b->inst[r.inst];
        for (int x0 = 0; x0 < I.n; x0 += s.tx)
            tiles.push_back({r.inst, x0, r.y0, I.n, I.pitch, s.tx, s.ty, {s.m[0], s.m[1], s.m[2]}, I.off});
    }
    hf::BatchTile* dt = nullptr;
    BCK(cudaMalloc(&dt, tiles.size() * sizeof(hf::BatchTile)));
    b->allocs.push_back(dt);
    BCK(cudaMemcpy(dt, tiles.data(), tiles.size() * sizeof(hf::BatchTile), cudaMemcpyHostToDevice));
    b->ntiles[k] = (long long)tiles.size();
    b->tiles[k] = dt;
    return HF_OK;
}

// The TMA maps of configuration k (MUSCL-Hancock batches): per state parity and case, the case's
// [4][n][pitch] state as a 3-D tensor {n, n, 4} with the box of its tile and the 2-cell halo.
int ensure_maps(hf_batch* b, int k) {
    if (b->scheme != 1 || b->maps[k]) return HF_OK;
    hf::EncodeTiledFn enc = hf::tensor_map_encoder();
    if (!enc) return bfail(b, HF_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
    const size_t n = b->inst.size();
    std::vector<CUtensorMap> maps(2 * n);
    for (int par = 0; par < 2; ++par)
        for (size_t i = 0; i < n; ++i) {
            const hf::BatchInst& I = b->inst[i];
            cuuint64_t dims[3] = {(cuuint64_t)I.n, (cuuint64_t)I.n, 4};
            cuuint64_t strides[2] = {(cuuint64_t)I.pitch * 8, (cuuint64_t)I.pitch * I.n * 8};
            cuuint32_t box[3] = {(cuuint32_t)(b->shapes[k][i].tx + 4), (cuuint32_t)(b->shapes[k][i].ty + 4), 4};
            cuuint32_t es[3] = {1, 1, 1};
            CUresult r = enc(&maps[par * n + i], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, b->U[par] + I.off, dims, strides,
                             box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (r != CUDA_SUCCESS)
                return bfail(b, HF_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
        }
    BCK(cudaMalloc(&b->maps[k], maps.size() * sizeof(CUtensorMap)));
    b->allocs.push_back(b->maps[k]);
    BCK(cudaMemcpy(b->maps[k], maps.data(), maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice));
    return HF_OK;
}

// the tile list and maps of configuration k, from its selection on: a run allocates and copies nothing, so the
// first one too may be captured, or made in a thread that has no context yet
int prepare_config(hf_batch* b, int k) {
    const int r = ensure_tiles(b, k);
    return r ? r : ensure_maps(b, k);
}

hf::BatchDev devview(hf_batch* b, int k) {
    hf::BatchDev d{};
    d.ctrl = b->dctrl;
    d.inst = b->dinst;
    d.maps = b->maps[k];
    d.ninst = (int)b->inst.size();
    d.tiles = b->tiles[k];
    d.ntiles = b->ntiles[k];
    d.U[0] = b->U[0];
    d.U[1] = b->U[1];
    d.acc = b->acc;
    d.t = b->t;
    d.last_dt = b->last_dt;
    return d;
}

cudaGraphExec_t find_graph(const hf_batch* b, long long nsteps) {
    for (const auto& g : b->graphs)
        if (g.config == b->config && g.nsteps == nsteps) return g.exec;
    return nullptr;
}

long long read_step(hf_batch* b) {
    long long s = 0;
    cudaStreamSynchronize(b->stream);
    cudaMemcpy(&s, &b->dctrl->step, sizeof s, cudaMemcpyDeviceToHost);
    return s;
}

// refresh the read slot's CFL maxima of `count` cases from `first` on (after their upload)
int refresh_cfl(hf_batch* b, long long step, int first, int count) {
    const int ar = (int)(step % 3);
    const size_t n = b->inst.size();
    BCK(cudaMemsetAsync(b->acc + ((size_t)ar * n + first) * 2, 0, 2 * (size_t)count * sizeof(unsigned long long),
                        b->stream));
    int rows = 1;
    for (int i = first; i < first + count; ++i) rows = std::max(rows, b->inst[i].n);
    hf::batch_cfl_kernel<<<dim3((unsigned)std::min(rows, 2 * b->sms), (unsigned)std::min(count, 65535)),
                           hf::kCflThreads, 0, b->stream>>>(devview(b, 0), first, count);
    BCK(cudaGetLastError());
    BCK(cudaStreamSynchronize(b->stream));
    return HF_OK;
}

int check_device_error(hf_batch* b) {
    int e = 0;
    BCK(cudaStreamSynchronize(b->stream));
    BCK(cudaMemcpy(&e, &b->dctrl->err, sizeof e, cudaMemcpyDeviceToHost));
    if (e) return bfail(b, HF_ERR_DEVICE, "device error word " + std::to_string(e));
    return HF_OK;
}

}  // namespace

extern "C" {

int hf_batch_create(const char* manifest, size_t len, hf_batch** out) {
    using hf::Json;
    if (!manifest || !out) return HF_ERR_ARG;
    hf_batch* b = new hf_batch();
    *out = b;
    std::vector<std::vector<double>> init;
    try {
        Json m = Json::parse(manifest, len);
        const Json& cs = m["cases"];
        if (cs.size() == 0) return bfail(b, HF_ERR_ARG, "manifest has no cases");
        for (size_t i = 0; i < cs.size(); ++i) {
            const Json& c = cs[i];
            if (c["model"]["model"].string() != "EulerIdealGas")
                return bfail(b, HF_ERR_UNSUPPORTED, "model must be EulerIdealGas");
            const Json& sch = c["scheme"];
            const std::string type = sch["type"].string();
            const int S = type == "Godunov" ? 0 : (type == "MUSCLHancock" ? 1 : -1);
            if (S < 0 || sch["riemann"].string() != "HLLCEuler" || sch["ode"].string() != "ForwardEuler")
                return bfail(b, HF_ERR_UNSUPPORTED,
                             "batched cases are Godunov or MUSCL-Hancock + HLLC + forward Euler");
            int L = 0;
            if (S == 1) {
                const std::string lim = sch["limiter"].string();
                L = lim == "MinBee" ? 0 : (lim == "VanLeer" ? 1 : -1);
                if (L < 0) return bfail(b, HF_ERR_UNSUPPORTED, "limiter '" + lim + "' not supported");
            }
            double gamma = c["model"]["gamma"].number(), cfl = c["simulation"]["cfl"].number();
            if (i == 0) { b->gamma = gamma; b->cfl = cfl; b->limiter = L; b->scheme = S; }
            else if (gamma != b->gamma || cfl != b->cfl || L != b->limiter || S != b->scheme)
                return bfail(b, HF_ERR_UNSUPPORTED, "all batched cases share scheme, gamma, cfl and limiter");
            const Json& blocks = c["mesh"]["blocks"];
            if (blocks.size() != 1) return bfail(b, HF_ERR_UNSUPPORTED, "batched cases have one block");
            const Json& blk = blocks[0];
            for (const char* side : {"bottom", "right", "top", "left"})
                if (blk["boundaries"][side]["type"].string() != "Transmissive")
                    return bfail(b, HF_ERR_UNSUPPORTED, "batched cases are transmissive on every side");
            const double cx = blk["x_cells"].number(), cy = blk["y_cells"].number();
            if (!(cx >= 4.0 && cx <= 65535.0) || cx != cy || cx != (double)(int)cx)
                return bfail(b, HF_ERR_UNSUPPORTED, "batched cases are square, 4..65535 cells per side");
            const int nx = (int)cx, ny = (int)cy;
            const Json& ex = blk["extents"];
            double xl = ex["x_left"].number(), xr = ex["x_right"].number();
            double yb = ex["y_bottom"].number(), yt = ex["y_top"].number();
            hf::BatchInst I{};
            I.n = nx;
            I.pitch = nx + (nx & 1);
            I.off = b->total_doubles;
            b->total_doubles += 4LL * I.pitch * nx;
            I.dx = (xr - xl) / nx;   // mesh_block.cpp:227-236
            I.dy = (yt - yb) / ny;
            I.one_dx = 1.0 / I.dx;   // muscl_hancock.cpp:352-353, godunov.cpp:97-98
            I.one_dy = 1.0 / I.dy;
            b->inst.push_back(I);
            b->total_cells += (long long)nx * ny;
            // the centroids depend on the ghost width in floating point (mesh_block.cpp:239-257),
            // so the initial condition is sampled on the scheme's own ghost layout
            const int gh = S == 0 ? 1 : 2;
            std::vector<double> soa;
            hf::BlockGeom G{nx + 2 * gh, ny + 2 * gh, xl, yb, I.dx, I.dy};
            hf::build_initial_state(c["initial_condition"], gamma, G, gh, soa);
            std::vector<double> inner((size_t)4 * nx * ny);
            for (int v = 0; v < 4; ++v)
                for (int j = 0; j < ny; ++j)
                    std::memcpy(&inner[((size_t)v * ny + j) * nx],
                                &soa[((size_t)v * (ny + 2 * gh) + j + gh) * (nx + 2 * gh) + gh], nx * sizeof(double));
            init.push_back(std::move(inner));
        }
    } catch (const std::exception& e) {
        return bfail(b, HF_ERR_PARSE, e.what());
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return bfail(b, HF_ERR_NO_DEVICE, "no CUDA device visible");
    int dev = 0;
    BCK(cudaGetDevice(&dev));
    BCK(cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, dev));
    BCK(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
    const size_t n = b->inst.size();
    for (int k = 0; k < 2; ++k) {
        BCK(cudaMalloc(&b->U[k], (size_t)b->total_doubles * sizeof(double)));
        BCK(cudaMemset(b->U[k], 0, (size_t)b->total_doubles * sizeof(double)));
        b->allocs.push_back(b->U[k]);
    }
    BCK(cudaMalloc(&b->acc, 3 * 2 * n * sizeof(unsigned long long)));
    BCK(cudaMalloc(&b->t, n * sizeof(double)));
    BCK(cudaMalloc(&b->last_dt, n * sizeof(double)));
    BCK(cudaMalloc(&b->dinst, n * sizeof(hf::BatchInst)));
    BCK(cudaMalloc(&b->dctrl, sizeof(hf::BatchCtrl)));
    for (void* p : {(void*)b->acc, (void*)b->t, (void*)b->last_dt, (void*)b->dinst, (void*)b->dctrl}) b->allocs.push_back(p);
    BCK(cudaMemset(b->acc, 0, 3 * 2 * n * sizeof(unsigned long long)));
    BCK(cudaMemset(b->t, 0, n * sizeof(double)));
    BCK(cudaMemset(b->last_dt, 0, n * sizeof(double)));
    BCK(cudaMemcpy(b->dinst, b->inst.data(), n * sizeof(hf::BatchInst), cudaMemcpyHostToDevice));
    hf::BatchCtrl C{};
    C.gamma = b->gamma;
    C.g1 = b->gamma - 1.0;
    C.cfl = b->cfl;
    C.ninst = (int)n;
    C.first_nonpos = ~0ull;
    BCK(cudaMemcpy(b->dctrl, &C, sizeof C, cudaMemcpyHostToDevice));
    for (size_t i = 0; i < n; ++i) {
        const hf::BatchInst& I = b->inst[i];
        BCK(cudaMemcpy2D(b->U[0] + I.off, (size_t)I.pitch * 8, init[i].data(), (size_t)I.n * 8, (size_t)I.n * 8,
                         (size_t)4 * I.n, cudaMemcpyHostToDevice));
    }
    const int r = prepare_config(b, 0);
    return r ? r : refresh_cfl(b, 0, 0, (int)n);
}

void hf_batch_destroy(hf_batch* b) {
    if (!b) return;
    if (b->stream) cudaStreamSynchronize(b->stream);
    for (auto& g : b->graphs) cudaGraphExecDestroy(g.exec);
    for (void* p : b->allocs) cudaFree(p);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
}

const char* hf_batch_last_error_message(const hf_batch* b) { return b ? b->err.c_str() : ""; }

int hf_batch_sizes(const hf_batch* b, int* ninst, int64_t* total_cells) {
    if (!b) return HF_ERR_ARG;
    if (ninst) *ninst = (int)b->inst.size();
    if (total_cells) *total_cells = b->total_cells;
    return HF_OK;
}

int hf_batch_instance_side(const hf_batch* b, int i, int* n) {
    if (!b || !n || i < 0 || i >= (int)b->inst.size()) return HF_ERR_ARG;
    *n = b->inst[i].n;
    return HF_OK;
}

int hf_batch_num_configs(int* n) {
    if (!n) return HF_ERR_ARG;
    *n = hf::kNumConfigs;
    return HF_OK;
}

int hf_batch_config_info(int k, int* tile_x, int* tile_y, int* threads, int* stages) {
    if (k < 0 || k >= hf::kNumConfigs) return HF_ERR_ARG;
    const hf::BatchConfig C = hf::kConfigs[k];
    if (tile_x) *tile_x = C.tx;
    if (tile_y) *tile_y = C.ty;
    if (threads) *threads = C.threads;
    if (stages) *stages = 1;
    return HF_OK;
}

int hf_batch_set_config(hf_batch* b, int k) {
    if (!b || k < 0 || k >= hf::kNumConfigs) return HF_ERR_ARG;
    const int r = prepare_config(b, k);
    if (r == HF_OK) b->config = k;
    return r;
}

int hf_batch_run(hf_batch* b, int64_t nsteps, int use_graph) {
    hf::TraceRange trace_("hf_batch_run");
    if (!b || nsteps < 0 || nsteps > (1 << 30)) return HF_ERR_ARG;
    if (nsteps == 0) return HF_OK;
    const int r = prepare_config(b, b->config);   // (there already, unless a call before failed)
    if (r) return r;
    hf::BatchDev d = devview(b, b->config);
    while (use_graph && nsteps > 0) {
        long long n = std::min<long long>(nsteps, hf::kBatchGraphSteps);
        cudaGraphExec_t exec = find_graph(b, n);
        if (!exec) {
            n = hf::batch_graph_steps(nsteps, (int)std::count_if(b->graphs.begin(), b->graphs.end(), [&](const hf_batch::G& g) {
                return g.config == b->config;
            }));
            exec = find_graph(b, n);
        }
        if (!exec) {
            cudaGraph_t graph;
            BCK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
            cudaError_t e = hf::launch_batch(b->config, b->scheme, b->limiter, d, n, b->stream);
            cudaError_t e2 = cudaStreamEndCapture(b->stream, &graph);
            if (e != cudaSuccess) return bfail(b, HF_ERR_CUDA, std::string("capture: ") + cudaGetErrorString(e));
            if (e2 != cudaSuccess) return bfail(b, HF_ERR_CUDA, std::string("end capture: ") + cudaGetErrorString(e2));
            BCK(cudaGraphInstantiate(&exec, graph, 0));
            cudaGraphDestroy(graph);
            b->graphs.push_back({b->config, n, exec});
        }
        BCK(cudaGraphLaunch(exec, b->stream));
        nsteps -= n;
    }
    BCK(hf::launch_batch(b->config, b->scheme, b->limiter, d, nsteps, b->stream));
    return HF_OK;
}

int hf_batch_sync(hf_batch* b) {
    if (!b) return HF_ERR_ARG;
    return check_device_error(b);
}

int hf_batch_autotune(hf_batch* b, int steps_per_trial, int* best, double* ms_per_step) {
    if (!b || steps_per_trial < 1) return HF_ERR_ARG;
    // trials advance a copy: save the live state, time each configuration, restore
    const size_t bytes = (size_t)b->total_doubles * sizeof(double);
    long long step = read_step(b);
    int p = (int)(step & 1);
    double* save = nullptr;
    BCK(cudaMalloc(&save, bytes));
    std::vector<unsigned long long> acc(3 * 2 * b->inst.size());
    std::vector<double> tt(b->inst.size()), ld(b->inst.size());
    hf::BatchCtrl C;
    BCK(cudaMemcpy(save, b->U[p], bytes, cudaMemcpyDeviceToDevice));
    BCK(cudaMemcpy(acc.data(), b->acc, acc.size() * 8, cudaMemcpyDeviceToHost));
    BCK(cudaMemcpy(tt.data(), b->t, tt.size() * 8, cudaMemcpyDeviceToHost));
    BCK(cudaMemcpy(ld.data(), b->last_dt, ld.size() * 8, cudaMemcpyDeviceToHost));
    BCK(cudaMemcpy(&C, b->dctrl, sizeof C, cudaMemcpyDeviceToHost));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int bestk = -1;
    double bestms = 1e300;
    for (int k = 0; k < hf::kNumConfigs; ++k) {
        int r = prepare_config(b, k);
        if (r) return r;
        hf::BatchDev d = devview(b, k);
        // warm (first launch pays the shared-memory opt-in), then time
        BCK(hf::launch_batch(k, b->scheme, b->limiter, d, 1, b->stream));
        cudaEventRecord(e0, b->stream);
        BCK(hf::launch_batch(k, b->scheme, b->limiter, d, steps_per_trial, b->stream));
        cudaEventRecord(e1, b->stream);
        int er = check_device_error(b);
        if (er) return er;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        double per = ms / steps_per_trial;
        if (ms_per_step) ms_per_step[k] = per;
        if (per < bestms) { bestms = per; bestk = k; }
        // restore
        BCK(cudaMemcpy(b->U[p], save, bytes, cudaMemcpyDeviceToDevice));
        BCK(cudaMemcpy(b->acc, acc.data(), acc.size() * 8, cudaMemcpyHostToDevice));
        BCK(cudaMemcpy(b->t, tt.data(), tt.size() * 8, cudaMemcpyHostToDevice));
        BCK(cudaMemcpy(b->last_dt, ld.data(), ld.size() * 8, cudaMemcpyHostToDevice));
        BCK(cudaMemcpy(b->dctrl, &C, sizeof C, cudaMemcpyHostToDevice));
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(save);
    b->config = bestk;
    if (best) *best = bestk;
    return HF_OK;
}

int hf_batch_get_state(hf_batch* b, int i, double* out) {
    if (!b || !out || i < 0 || i >= (int)b->inst.size()) return HF_ERR_ARG;
    long long step = read_step(b);
    const hf::BatchInst& I = b->inst[i];
    BCK(cudaMemcpy2D(out, (size_t)I.n * 8, b->U[step & 1] + I.off, (size_t)I.pitch * 8, (size_t)I.n * 8,
                     (size_t)4 * I.n, cudaMemcpyDeviceToHost));
    return HF_OK;
}

int hf_batch_set_state(hf_batch* b, int i, const double* in) {
    if (!b || !in || i < 0 || i >= (int)b->inst.size()) return HF_ERR_ARG;
    long long step = read_step(b);
    const hf::BatchInst& I = b->inst[i];
    BCK(cudaMemcpy2D(b->U[step & 1] + I.off, (size_t)I.pitch * 8, in, (size_t)I.n * 8, (size_t)I.n * 8,
                     (size_t)4 * I.n, cudaMemcpyHostToDevice));
    return refresh_cfl(b, step, i, 1);
}

int hf_batch_instance_time(hf_batch* b, int i, double* t, double* last_dt) {
    if (!b || i < 0 || i >= (int)b->inst.size()) return HF_ERR_ARG;
    BCK(cudaStreamSynchronize(b->stream));
    if (t) BCK(cudaMemcpy(t, b->t + i, sizeof(double), cudaMemcpyDeviceToHost));
    if (last_dt) BCK(cudaMemcpy(last_dt, b->last_dt + i, sizeof(double), cudaMemcpyDeviceToHost));
    return HF_OK;
}

int hf_batch_counters(hf_batch* b, int64_t* steps, int64_t* calls, int64_t* hllc_errors) {
    if (!b) return HF_ERR_ARG;
    hf::BatchCtrl C;
    BCK(cudaStreamSynchronize(b->stream));
    BCK(cudaMemcpy(&C, b->dctrl, sizeof C, cudaMemcpyDeviceToHost));
    if (steps) *steps = C.step;
    if (calls) *calls = C.calls;
    if (hllc_errors) *hllc_errors = C.hllc_errors;
    return HF_OK;
}

int hf_batch_last_nonpositive_cell(hf_batch* b, int* instance, int* i, int* j, int64_t* step) {
    if (!b) return HF_ERR_ARG;
    unsigned long long k = ~0ull;
    BCK(cudaStreamSynchronize(b->stream));
    BCK(cudaMemcpy(&k, &b->dctrl->first_nonpos, sizeof k, cudaMemcpyDeviceToHost));
    int ci = -1, cj = -1, cx = -1;
    long long st = -1;
    if (k != ~0ull) {
        const long long off = (long long)(k & 0xFFFFFFFFFFull);
        // the case whose state holds that offset (offsets ascend with the case index)
        size_t lo = 0, hi = b->inst.size();
        while (hi - lo > 1) {
            const size_t mid = (lo + hi) / 2;
            (b->inst[mid].off <= off ? lo : hi) = mid;
        }
        const long long rem = off - b->inst[lo].off;
        cx = (int)lo;
        cj = (int)(rem / b->inst[lo].pitch);
        ci = (int)(rem % b->inst[lo].pitch);
        st = (long long)(k >> 40);
    }
    if (instance) *instance = cx;
    if (i) *i = ci;
    if (j) *j = cj;
    if (step) *step = st;
    return HF_OK;
}

int hf_batch_clear_error_cell(hf_batch* b) {
    if (!b) return HF_ERR_ARG;
    const unsigned long long none = ~0ull;
    BCK(cudaMemcpyAsync(&b->dctrl->first_nonpos, &none, sizeof none, cudaMemcpyHostToDevice, b->stream));
    BCK(cudaStreamSynchronize(b->stream));
    return HF_OK;
}

int hf_batch_stream(hf_batch* b, void** stream) {
    if (!b || !stream) return HF_ERR_ARG;
    *stream = (void*)b->stream;
    return HF_OK;
}

}  // extern "C"
