// k_membrane.cu — immersed-boundary and geometry kernels.  Compiled with
// --fmad=false: every FP64 result is bit-identical to the reference.
//
//   force_eval       ForceSolver::calculateForce (ForceSolver.cpp:42-85) over a
//                    per-node CSR of force records in insertion order
//                    (ForceStructs.hpp:49-588).
//   spread           SimulationRunner::distributeForce + GeometryNode::distributeForce
//                    (SimulationRunner.cpp:425-453, GeometryNode.cpp:228-235) as a
//                    deterministic sum: each 16x16 lattice tile collects the
//                    membrane nodes whose 4x4 stencil overlaps it, sorts them by
//                    id and adds their contributions in id order (the
//                    reference's serial map order).  No floating-point atomics.
//   interp_move      GeometryNode::collectVelocity (GeometryNode.cpp:216-226, slot
//                    order (4x+y) mod 16 from GeometryHandler.cpp:641), the speed
//                    check (LagrangianPoint.cpp:92-103) and GeometryNode::move
//                    (GeometryNode.cpp:245-254); positions that need the
//                    reference's random perturbation (GeometryNode.cpp:153-214)
//                    are flagged for the host, which owns the generator.
//   crossings        Connection::generateBoundaryNodes / insertBoundaryNode
//                    (Connection.cpp:181-324): every crossing of a connection with
//                    a lattice line is a candidate for one (node, slot); the
//                    closest wins, ties keep the earlier connection.
//   reinit           PhysicalNode::updateDomainIdentifier + CDESolverD2Q5::reinitialise
//                    (PhysicalNode.cpp:109-124, CDESolverD2Q5.cpp:156-228) in
//                    row-major order semantics, processed in dependency rounds.
//   domain_fill      GeometryHandler::updateAllDomainIdentifiers (GeometryHandler.cpp:68-85).
#include <algorithm>

#include <cub/cub.cuh>

#include "kernels.cuh"
#include "lattice_math.cuh"
#include "remesh.cuh"

namespace lbib {

// ---------------------------------------------------------------------------
// fastCos and the Dirac weight: GeometryNode.cpp:55-94.
__device__ __forceinline__ double fast_cos(const double x) {
    const double halfPi = M_PI / 2.0;
    const double doublePi = 2.0 * M_PI;
    double cs;
    double tempx = x + halfPi;
    if (tempx > M_PI) tempx -= doublePi;
    if (tempx < .00) {
        cs = 1.27323954 * tempx + 0.405284735 * tempx * tempx;
    } else {
        cs = 1.27323954 * tempx - 0.405284735 * tempx * tempx;
    }
    if (cs < 0.0) {
        cs = 0.225 * (cs * -cs - cs) + cs;
    } else {
        cs = 0.225 * (cs * cs - cs) + cs;
    }
    return cs;
}

__device__ __forceinline__ double dirac(const double dx, const double dy) {
    const double halfPi = M_PI / 2.0;
    return ((1.0 + fast_cos(halfPi * dx)) * (1.0 + fast_cos(halfPi * dy))) / 16.0;
}

// ---------------------------------------------------------------------------
// Force evaluation

// The force of one record on the node at (x1, y1) (ForceStructs.hpp:49-588),
// added to (Fx, Fy); p0 is the record's first parameter, p its four, (x2, y2)
// the partner's position (types 0, 5, 6, 7).
__device__ __forceinline__ void add_force(int type, double p0, const double* p, double x1, double y1, double x2,
                                          double y2, double& Fx, double& Fy) {
    switch (type) {
        case 0: case 7: {  // spring between two nodes: f = k(|d| - l0), along d
            const double dist = sqrt((x2 - x1) * (x2 - x1) + (y2 - y1) * (y2 - y1));
            const double f = p0 * (dist - p[1]);
            Fx += ((x2 - x1) * f) / dist;
            Fy += ((y2 - y1) * f) / dist;
            break;
        }
        case 1: {  // anchor spring to (x, y)
            const double tx = p0, ty = p[1];
            const double dist = sqrt((tx - x1) * (tx - x1) + (ty - y1) * (ty - y1));
            const double f = p[2] * (dist - p[3]);
            if (dist != 0.0) {
                Fx += ((tx - x1) * f) / dist;
                Fy += ((ty - y1) * f) / dist;
            }
            break;
        }
        case 2:  // constant force
            Fx += p0;
            Fy += p[1];
            break;
        case 3: {  // horizontal slider at y
            const double dist = sqrt((x1 - x1) * (x1 - x1) + (p0 - y1) * (p0 - y1));
            const double f = p[1] * (dist - p[2]);
            Fx += 0.0;
            Fy += (y1 < p0) ? f : -f;
            break;
        }
        case 4: {  // vertical slider at x
            const double dist = sqrt((p0 - x1) * (p0 - x1) + (y1 - y1) * (y1 - y1));
            const double f = p[1] * (dist - p[2]);
            Fx += (x1 < p0) ? f : -f;
            Fy += 0.0;
            break;
        }
        default: {  // 5, 6: constant-magnitude pull toward the partner
            const double dist = sqrt((x2 - x1) * (x2 - x1) + (y2 - y1) * (y2 - y1));
            Fx += ((x2 - x1) * p0) / dist;
            Fy += ((y2 - y1) * p0) / dist;
            break;
        }
    }
}

// A node's entries in the slot lists of the (up to 2 x 2) tiles its stencil
// covers.  The lanes of a warp that enter the same tile share one atomic;
// tile_slots_take issues the four rounds' atomics, tile_slots_put, which
// waits for them, stores the entries: what stands between the two hides the
// round trips.  All lanes of the warp take part in both.
struct TileSlots {
    int tile[4];
    int base[4];
    unsigned group[4];
};
__device__ __forceinline__ TileSlots tile_slots_take(double bx, double by, const TileDev& t, int i, bool ok, int nx,
                                                     int ny, Status* st);
__device__ __forceinline__ void tile_slots_put(const TileDev& t, const TileSlots& s, int i, Status* st);

// `slots`: also enter the node in the per-tile lists of the spread (which left
// the tile counts at zero).
// Two records are read ahead (a membrane node has two tension records), and the
// slot lists' atomics are under way meanwhile: 5.5 -> 4.0 us for one cell, 8.3 ->
// 6.3 us for 150k nodes.
__global__ void __launch_bounds__(128) force_eval_kernel(MembraneDev m, Status* st, TileDev t, int nx,
                                                         int ny, int slots) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x, ic = min(i, m.Mcap - 1);
    int halt = st->halt, M = m.topo->M;
    double x1 = m.x[ic], y1 = m.y[ic], bx = m.bx[ic], by = m.by[ic];
    int r0 = m.foff[ic], r1 = m.foff[ic + 1];
    read_ahead(halt, M, x1, y1, bx, by, r0, r1);
    if (halt) return;
    if (i - (int)(threadIdx.x & 31) >= M) return;  // the whole warp
    bool live = i < M;
    if (!live) r0 = r1 = 0;
    TileSlots ts;
    if (slots) ts = tile_slots_take(bx, by, t, i, live, nx, ny, st);
    double Fx = 0.0, Fy = 0.0;
    for (int r = r0; r < r1; r += 2) {
        int type[2], j[2];
        double p0[2], x2[2] = {0.0, 0.0}, y2[2] = {0.0, 0.0};
        bool pair[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int rq = r + q < r1 ? r + q : r;
            type[q] = m.ftype[rq];
            j[q] = m.fpartner[rq];
            p0[q] = m.fpar[4 * (size_t)rq];
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            pair[q] = type[q] == 0 || type[q] == 7 || type[q] == 5 || type[q] == 6;
            if (pair[q] && j[q] >= 0 && j[q] < M) {
                x2[q] = m.x[j[q]];
                y2[q] = m.y[j[q]];
            }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (!live || r + q >= r1) break;
            if (pair[q] && (j[q] < 0 || j[q] >= M)) {
                raise_error(st, ERR_FORCE_NODE, i, ST_FORCE);
                live = false;
                break;
            }
            add_force(type[q], p0[q], m.fpar + 4 * (size_t)(r + q), x1, y1, x2[q], y2[q], Fx, Fy);
        }
        if (!live) break;
    }
    if (live) {
        m.fx[i] = Fx;
        m.fy[i] = Fy;
    }
    if (slots) tile_slots_put(t, ts, i, st);
}

// dL/d of every force record's parameters from dL/dF of the node forces
// (the membrane-force gradient of a differentiated run), through the
// record's force as force_eval_kernel forms it (ForceStructs.hpp:49-588):
// each record of node i adds to F_i only, so
// dL/dp = (dL/dF_i) . dF_i/dp, with the positions fixed.  Parameters a type
// does not read get 0.  gpar: 4 per record, in record order.
__global__ void force_param_grad_kernel(MembraneDev m, const double* gfx, const double* gfy, double* gpar) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.topo->M) return;
    const double x1 = m.x[i], y1 = m.y[i], gx = gfx[i], gy = gfy[i];
    for (int r = m.foff[i]; r < m.foff[i + 1]; ++r) {
        const int type = m.ftype[r];
        const double* p = m.fpar + 4 * (size_t)r;
        const int j = m.fpartner[r];
        double g[4] = {0.0, 0.0, 0.0, 0.0};
        switch (type) {
            case 0: case 7: case 5: case 6: {
                if (j < 0 || j >= m.topo->M) break;
                const double dx = m.x[j] - x1, dy = m.y[j] - y1;
                const double dist = sqrt(dx * dx + dy * dy);
                const double gd = (gx * dx + gy * dy) / dist;  // (dL/dF) . d / |d|
                if (type == 5 || type == 6) {
                    g[0] = gd;                      // F = f d/|d|
                } else {
                    g[0] = (dist - p[1]) * gd;      // F = k (|d| - l0) d/|d|
                    g[1] = -p[0] * gd;
                }
                break;
            }
            case 1: {  // F = k (|d| - l0) d/|d|, d = (tx, ty) - x; none at |d| = 0
                const double dx = p[0] - x1, dy = p[1] - y1;
                const double dist = sqrt(dx * dx + dy * dy);
                if (dist == 0.0) break;
                const double gdd = gx * dx + gy * dy;
                const double a = 1.0 - p[3] / dist, b = p[3] * gdd / (dist * dist * dist);
                g[0] = p[2] * (a * gx + b * dx);  // dF/dtx: k [(1 - l0/|d|) I + l0 d d^T / |d|^3]
                g[1] = p[2] * (a * gy + b * dy);
                g[2] = (dist - p[3]) * gdd / dist;
                g[3] = -p[2] * gdd / dist;
                break;
            }
            case 2:  // F = (fx, fy)
                g[0] = gx;
                g[1] = gy;
                break;
            case 3: case 4: {  // sliders: F_y (3) or F_x (4) = +-k (|c - y| - l0), + below c
                const double pos = type == 3 ? y1 : x1, gc = type == 3 ? gy : gx;
                const double dist = fabs(p[0] - pos);
                const double sgn = pos < p[0] ? 1.0 : -1.0;
                const double dd = p[0] > pos ? 1.0 : (p[0] < pos ? -1.0 : 0.0);  // d|c - pos| / dc
                g[0] = gc * sgn * p[1] * dd;
                g[1] = gc * sgn * (dist - p[2]);
                g[2] = -gc * sgn * p[1];
                break;
            }
            default:
                break;
        }
        for (int q = 0; q < 4; ++q) gpar[4 * (size_t)r + q] = g[q];
    }
}

void launch_force_param_grad(const MembraneDev& m, const double* gfx, const double* gfy, double* gpar,
                             cudaStream_t s) {
    if (m.Mcap == 0) return;
    force_param_grad_kernel<<<(m.Mcap + 127) / 128, 128, 0, s>>>(m, gfx, gfy, gpar);
}

void launch_force_eval(const MembraneDev& m, Status* st, cudaStream_t s, TileDev* tiles, int nx, int ny) {
    if (m.Mcap == 0) return;
    launch_pdl(force_eval_kernel, (m.Mcap + 127) / 128, 128, 0, s, m, st, tiles ? *tiles : TileDev{}, nx, ny,
               tiles ? 1 : 0);
}

// ---------------------------------------------------------------------------
// Spreading

// Stencil of a membrane node (GeometryHandler.cpp:613-643): the loop
//   for x in [ceil(X-2), floor(X+2)], for y in [ceil(Y-2), floor(Y+2)]:
//       slot[(4x + y) % 16] = node(x, y)
// binds 16 slots.  The ranges are 4 wide, except when rounding of X+2 or X-2
// makes them 5 wide (e.g. X = 32 - 1 ulp); then later writes replace earlier
// ones with the same slot, and the bound set is what the last writers leave.
struct Stencil {
    int x0, x1, y0, y1;
};

__device__ __forceinline__ bool stencil_on_lattice(const Stencil& s, int nx, int ny) {
    const int wx = s.x1 - s.x0, wy = s.y1 - s.y0;
    return wx >= 3 && wx <= 4 && wy >= 3 && wy <= 4 && s.x0 >= 0 && s.y0 >= 0 && s.x1 < nx && s.y1 < ny;
}

__device__ __forceinline__ bool stencil_range(double X, double Y, int nx, int ny, Stencil& s) {
    s.x0 = (int)ceil(X - 2.0);
    s.y0 = (int)ceil(Y - 2.0);
    s.x1 = (int)floor(X + 2.0);
    s.y1 = (int)floor(Y + 2.0);
    return stencil_on_lattice(s, nx, ny);
}

// Is lattice node (x, y) bound by the stencil (the last writer of its slot)?
__device__ __forceinline__ bool in_stencil(const Stencil& s, int x, int y) {
    if (x < s.x0 || x > s.x1 || y < s.y0 || y > s.y1) return false;
    if (s.x1 - s.x0 == 3 && s.y1 - s.y0 == 3) return true;
    const int slot = (4 * x + y) & 15;
    for (int xp = x; xp <= s.x1; ++xp)
        for (int yp = (xp == x ? y + 1 : s.y0); yp <= s.y1; ++yp)
            if (((4 * xp + yp) & 15) == slot) return false;
    return true;
}

// The lattice node bound to slot k (k = 0..15).
__device__ __forceinline__ void stencil_slot(const Stencil& s, int k, int& xk, int& yk) {
    if (s.x1 - s.x0 == 3 && s.y1 - s.y0 == 3) {
        const int base = ((4 * s.x0 + s.y0) % 16 + 16) % 16;
        const int r = (k - base + 16) & 15;
        xk = s.x0 + (r >> 2);
        yk = s.y0 + (r & 3);
        return;
    }
    xk = -1; yk = -1;
    for (int x = s.x0; x <= s.x1; ++x)
        for (int y = s.y0; y <= s.y1; ++y)
            if (((4 * x + y) & 15) == k) { xk = x; yk = y; }
}

__device__ __forceinline__ TileSlots tile_slots_take(double bx, double by, const TileDev& t, int i, bool ok, int nx,
                                                     int ny, Status* st) {
    Stencil sc{0, 0, 0, 0};
    if (ok && !stencil_range(bx, by, nx, ny, sc)) {
        raise_error(st, ERR_STENCIL, i, ST_SPREAD);
        ok = false;
    }
    const int tx0 = sc.x0 / kTile, tx1 = sc.x1 / kTile, ty0 = sc.y0 / kTile, ty1 = sc.y1 / kTile;
    const int lane = threadIdx.x & 31;
    TileSlots s;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int tx = tx0 + (j & 1), ty = ty0 + (j >> 1);
        s.tile[j] = ok && tx <= tx1 && ty <= ty1 ? ty * t.tilesX + tx : -1;
        s.group[j] = __match_any_sync(0xffffffffu, s.tile[j]);
        s.base[j] = 0;
        if (s.tile[j] >= 0 && lane == __ffs(s.group[j]) - 1)
            s.base[j] = atomicAdd(&t.count[s.tile[j]], __popc(s.group[j]));
    }
    return s;
}

__device__ __forceinline__ void tile_slots_put(const TileDev& t, const TileSlots& s, int i, Status* st) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int slot = __shfl_sync(0xffffffffu, s.base[j], __ffs(s.group[j]) - 1) +
                         __popc(s.group[j] & ((1u << lane) - 1u));
        if (s.tile[j] < 0) continue;
        if (slot < kTileSlots) t.slots[(size_t)s.tile[j] * kTileSlots + slot] = i;
        else raise_error(st, ERR_CAPACITY, s.tile[j], ST_SPREAD);
    }
}

__global__ void tile_slot_kernel(MembraneDev m, TileDev t, int nx, int ny, Status* st) {
    pdl_wait();
    if (st->halt) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = i < m.topo->M;
    tile_slots_put(t, tile_slots_take(live ? m.bx[i] : 0.0, live ? m.by[i] : 0.0, t, i, live, nx, ny, st), i, st);
}

// Per-tile entry: the stencil origin relative to the tile (+4) and the stencil
// widths, packed in one word: ox | oy << 8 | (x1-x0) << 16 | (y1-y0) << 20.
__device__ __forceinline__ int pack_stencil(const Stencil& s, int tileX0, int tileY0) {
    return (s.x0 - tileX0 + 4) | ((s.y0 - tileY0 + 4) << 8) | ((s.x1 - s.x0) << 16) | ((s.y1 - s.y0) << 20);
}

// The tile's list as the spread takes it: its length, noted for the readers of
// the force field, and the counter left at zero for the next step's lists (a
// memset node between two kernels of the step cost 3.5 us).
// -1 on a halted step.  `first`: the list's entry of that place, if it has one.
__device__ __forceinline__ int take_tile_count(const TileDev& t, int tile, const Status* st, int place, int& first) {
    int halt = st->halt, count = t.count[tile];
    first = t.slots[(size_t)tile * kTileSlots + place];
    read_ahead(halt, count, first);
    if (__syncthreads_or(halt)) return -1;  // (the block as one: the spread raises errors itself)
    if (threadIdx.x == 0) {
        t.active[tile] = count;
        if (count != 0) t.count[tile] = 0;
    }
    return count;
}

// FP64 runs, whose sums must be formed in the reference's order: each 16x16
// tile sorts its membrane nodes by index (= id order; the rank of an entry is
// the number of smaller ones) and forms per node the Dirac factors
// A_i = 1 + fastCos(pi/2 (x0 + i - X)) and B_j = 1 + fastCos(pi/2 (y0 + j - Y)),
// so that the weight of lattice node (x0+i, y0+j) is (A_i * B_j) / 16, the same
// expression as calculateDiscreteDeltaDirac (GeometryNode.cpp:89-94; A is kept
// as A / 16, an exact scaling).  Each warp owns two rows of the tile and takes,
// in id order, the entries whose stencil rows meet them; the lane of a lattice
// node adds an entry's products to it in registers, without a branch, so that
// the entries' loads and products overlap and only the additions form a chain.  Longer lists go through in chunks, in order.
// With lists built by count, scan and fill, a radix sort per tile and a lane per
// node testing every entry, the spread took 96 us for 150k nodes on 1024^2 and
// 21 us for one cell.  Adding each entry's 16 products to shared memory, a
// lane each, took 48 and 17 us (a chain of shared-memory round trips); this
// form takes 40 (issue in 55 % of the cycles; the barriers of unevenly filled tiles
// stall it first) and 6.5 us.  Four rows per warp of a 128-thread block: 40 and
// 8.2 us.
constexpr int kSpreadMax = 768;    // entries of a tile
constexpr int kSpreadChunk = 128;  // entries whose factors are held at once
template <typename Real>
__global__ void __launch_bounds__(256) spread_kernel(MembraneDev m, TileDev t, Real* force, int nx, int ny, size_t L,
                                                     Status* st) {
    pdl_wait();
    const int tile = blockIdx.x;
    int first;
    const int cnt = take_tile_count(t, tile, st, threadIdx.x, first);
    if (cnt <= 0) return;
    if (cnt > kSpreadMax) {
        if (threadIdx.x == 0) raise_error(st, ERR_CAPACITY, tile, ST_SPREAD);
        return;
    }
    __shared__ __align__(16) double fac[kSpreadChunk][10];  // A[5] / 16, B[5]
    __shared__ double2 sF[kSpreadChunk];
    __shared__ int code[kSpreadChunk];
    __shared__ int order[kSpreadMax];               // sorted membrane indices
    __shared__ unsigned wlist[8][kSpreadChunk];     // per warp: pack_stencil and the entry's place << 24
    {
        int* raw = (int*)fac;  // free until the factors are formed
        static_assert(sizeof(fac) >= (kSpreadMax + 3) * sizeof(int), "the unsorted list fits the factors' place");
        const int* list = t.slots + (size_t)tile * kTileSlots;
        const int cnt4 = (cnt + 3) & ~3;
        for (int k = threadIdx.x; k < cnt4; k += blockDim.x)
            raw[k] = k < cnt ? (k < (int)blockDim.x ? first : list[k]) : 0x7fffffff;
        __syncthreads();
        for (int k = threadIdx.x; k < cnt; k += blockDim.x) {
            const int v = raw[k];
            int r = 0;
            for (int j = 0; j < cnt4; j += 4) {
                const int4 w = *(const int4*)(raw + j);
                r += (w.x < v) + (w.y < v) + (w.z < v) + (w.w < v);
            }
            order[r] = v;
        }
        __syncthreads();
    }
    const int tx = tile % t.tilesX, ty = tile / t.tilesX;
    const int tileX0 = tx * kTile, tileY0 = ty * kTile;
    const double halfPi = M_PI / 2.0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wy0 = 2 * warp;  // the warp's first row in the tile
    const int lx = lane & 15, ly = wy0 + (lane >> 4);
    double ax = 0.0, ay = 0.0;
    for (int c0 = 0; c0 < cnt; c0 += kSpreadChunk) {
        const int nc = min(kSpreadChunk, cnt - c0);
        // two threads per entry: the column factors and the row factors
        for (int k2 = threadIdx.x; k2 < 2 * nc; k2 += blockDim.x) {
            const int k = k2 >> 1, half = k2 & 1;
            const int i = order[c0 + k];
            Stencil sc;
            stencil_range(m.bx[i], m.by[i], nx, ny, sc);
            const double X = half ? m.y[i] : m.x[i];
            const int o = half ? sc.y0 : sc.x0;
            const double scale = half ? 1.0 : 1.0 / 16.0;
            double* f = &fac[k][5 * half];
#pragma unroll
            for (int q = 0; q < 5; ++q) f[q] = (1.0 + fast_cos(halfPi * ((double)(o + q) - X))) * scale;
            reinterpret_cast<double*>(sF + k)[half] = half ? m.fy[i] : m.fx[i];
            if (half == 0) code[k] = pack_stencil(sc, tileX0, tileY0);
        }
        __syncthreads();
        // the entries whose stencil rows meet the warp's rows, in order
        int wn = 0;
        bool wide = false;
        for (int k0 = 0; k0 < nc; k0 += 32) {
            const int k = k0 + lane;
            bool rel = false;
            int c = 0;
            if (k < nc) {
                c = code[k];
                const int oy = ((c >> 8) & 0xff) - 4, hy = (c >> 20) & 0xf;
                rel = oy + hy >= wy0 && oy <= wy0 + 1;
                wide |= rel && (c >> 16) != 0x33;
            }
            const unsigned bal = __ballot_sync(0xffffffffu, rel);
            if (rel) wlist[warp][wn + __popc(bal & ((1u << lane) - 1u))] = (unsigned)c | ((unsigned)k << 24);
            wn += __popc(bal);
        }
        wide = __any_sync(0xffffffffu, wide);
        __syncwarp();
        if (!wide) {
#pragma unroll 4
            for (int e = 0; e < wn; ++e) {
                const unsigned c = wlist[warp][e];
                const unsigned k = c >> 24;
                const int dx = lx + 4 - (int)(c & 0xffu), dy = ly + 4 - (int)((c >> 8) & 0xffu);
                const bool hit = (unsigned)dx < 4u && (unsigned)dy < 4u;
                const double dl = fac[k][dx & 3] * fac[k][5 + (dy & 3)];
                const double2 F = sF[k];
                const double sx = ax + F.x * dl, sy = ay + F.y * dl;
                if (hit) {
                    ax = sx;
                    ay = sy;
                }
            }
        } else {
            // stencils of five columns or rows among them: the nodes bound by
            // the slots' last writers
            for (int e = 0; e < wn; ++e) {
                const unsigned c = wlist[warp][e];
                const int k = c >> 24;
                const int ox = (int)(c & 0xffu) - 4, oy = (int)((c >> 8) & 0xffu) - 4;
                const Stencil sc{ox + tileX0, ox + tileX0 + (int)((c >> 16) & 0xfu), oy + tileY0,
                                 oy + tileY0 + (int)((c >> 20) & 0xfu)};
                const int x = tileX0 + lx, y = tileY0 + ly;
                if (!in_stencil(sc, x, y)) continue;
                const double dl = fac[k][x - sc.x0] * fac[k][5 + y - sc.y0];
                ax += sF[k].x * dl;
                ay += sF[k].y * dl;
            }
        }
        __syncthreads();
    }
    const int x = tileX0 + lx, y = tileY0 + ly;
    if (x >= nx || y >= ny) return;
    const size_t n = (size_t)y * nx + x;
    force[n] = (Real)ax;
    force[L + n] = (Real)ay;
}

// FP32-shifted runs: each 16x16 tile scatters the contributions of the
// membrane nodes listed for it into 64-bit fixed-point accumulators (2^-44) in
// shared memory.  Each contribution dirac * F_i is formed in FP64 exactly as in
// the ordered gather and rounded once; the integer sums are exact, so the
// field does not depend on the order of the list (it is deterministic) and no
// sort is needed.  The rounding is far below FP32 resolution.
// Where tiles hold many nodes, the barriers between the staging of a chunk's
// factors and its scatter are the first stall and the scheduler issues in 44 % of
// the cycles (tiles are filled unevenly); where there is one cell, the chain of
// reads bounds it.  Two lanes form a node's factors, one per axis, the
// force is staged with the products' power of two (an exact scaling), and the
// usual 4 x 4 stencil has its own loop: 150k nodes on 1024^2 21.6 -> 19.0 us, one
// cell on 200^2 4.5 -> 3.9 us against a lane per node and one loop.  Blocks of 64
// to 192 threads, or a warp's entries spread along the list: no gain.
constexpr double kForceFix = 17592186044416.0;  // 2^44
constexpr int kScatterChunk = 256;
__global__ void __launch_bounds__(256) spread_fixed_kernel(MembraneDev m, TileDev t, float* force, int nx, int ny,
                                                           size_t L, Status* st) {
    pdl_wait();
    const int tile = blockIdx.x;
    int first;
    const int cnt = min(take_tile_count(t, tile, st, threadIdx.x >> 1, first), kTileSlots);
    if (cnt <= 0) return;
    // each 64-bit fixed-point sum is kept as a signed high part (bits 22..63)
    // and an unsigned low part (bits 0..21), each summed with 32-bit integer
    // atomics: the low parts of up to 1024 contributions cannot overflow
    __shared__ int accHi[2][kTile * kTile];
    __shared__ unsigned accLo[2][kTile * kTile];
    // per axis and node: the Dirac factors, the force (scaled), the stencil's origin + 4 and its width << 8
    __shared__ double fab[2][kScatterChunk][5], sF[2][kScatterChunk];
    __shared__ int org[2][kScatterChunk];
    for (int j = threadIdx.x; j < kTile * kTile; j += blockDim.x) {
        accHi[0][j] = accHi[1][j] = 0;
        accLo[0][j] = accLo[1][j] = 0u;
    }

    const int tx = tile % t.tilesX, ty = tile / t.tilesX;
    const int tileX0 = tx * kTile, tileY0 = ty * kTile;
    const int* list = t.slots + (size_t)tile * kTileSlots;
    const double halfPi = M_PI / 2.0;
    for (int c0 = 0; c0 < cnt; c0 += kScatterChunk) {
        const int nc = min(kScatterChunk, cnt - c0);
        __syncthreads();
        for (int j = threadIdx.x; j < 2 * nc; j += blockDim.x) {
            const int e = j >> 1, axis = j & 1;
            const int i = c0 == 0 && j == threadIdx.x ? first : list[c0 + e];
            const double X = axis ? m.y[i] : m.x[i], B = axis ? m.by[i] : m.bx[i];
            const double F = axis ? m.fy[i] : m.fx[i];
            const int lo = (int)ceil(B - 2.0), hi = (int)floor(B + 2.0);  // (stencil_range)
            org[axis][e] = (lo - (axis ? tileY0 : tileX0) + 4) | ((hi - lo) << 8);
#pragma unroll
            for (int q = 0; q < 5; ++q) fab[axis][e][q] = 1.0 + fast_cos(halfPi * ((double)(lo + q) - X));
            sF[axis][e] = F * (kForceFix / 16.0);
        }
        __syncthreads();
        // one item per (node, slot row r): slots k = 4 r .. 4 r + 3 of the
        // node's 16 (in a 4 x 4 stencil, column dx = r, rows dy = 0..3)
        for (int j = threadIdx.x; j < 4 * nc; j += blockDim.x) {
            const int e = j >> 2, r = j & 3;
            const int cx = org[0][e], cy = org[1][e];
            const int ox = (cx & 0xff) - 4, oy = (cy & 0xff) - 4, hx = cx >> 8, hy = cy >> 8;
            const double Fx = sF[0][e], Fy = sF[1][e];
            auto add = [&](int node, double w) {  // w: 16 x the Dirac weight
                const long long vx = __double2ll_rn(Fx * w);
                const long long vy = __double2ll_rn(Fy * w);
                atomicAdd(&accHi[0][node], (int)(vx >> 22));
                atomicAdd(&accLo[0][node], (unsigned)(vx & 0x3fffff));
                atomicAdd(&accHi[1][node], (int)(vy >> 22));
                atomicAdd(&accLo[1][node], (unsigned)(vy & 0x3fffff));
            };
            if (hx == 3 && hy == 3) {
                if ((unsigned)(ox + r) >= (unsigned)kTile) continue;  // the column lies outside the tile
                const double a = fab[0][e][r];
                const int node = oy * kTile + ox + r;
#pragma unroll
                for (int t4 = 0; t4 < 4; ++t4)
                    if ((unsigned)(oy + t4) < (unsigned)kTile) add(node + t4 * kTile, a * fab[1][e][t4]);
            } else {
                // wider stencil: the node bound to slot k (last writer of the slot)
                const Stencil sc{ox + tileX0, ox + tileX0 + hx, oy + tileY0, oy + tileY0 + hy};
                for (int t4 = 0; t4 < 4; ++t4) {
                    int xk, yk;
                    stencil_slot(sc, 4 * r + t4, xk, yk);
                    if (xk < 0) continue;
                    const int lx = xk - tileX0, ly = yk - tileY0;
                    if ((unsigned)lx >= (unsigned)kTile || (unsigned)ly >= (unsigned)kTile) continue;
                    add(ly * kTile + lx, fab[0][e][xk - sc.x0] * fab[1][e][yk - sc.y0]);
                }
            }
        }
    }
    __syncthreads();
    const int lx = threadIdx.x & 15, ly = threadIdx.x >> 4;
    const int x = tileX0 + lx, y = tileY0 + ly;
    if (x >= nx || y >= ny) return;
    const size_t n = (size_t)y * nx + x;
    const long long sx = (long long)accHi[0][threadIdx.x] * (1ll << 22) + (long long)accLo[0][threadIdx.x];
    const long long sy = (long long)accHi[1][threadIdx.x] * (1ll << 22) + (long long)accLo[1][threadIdx.x];
    force[n] = (float)((double)sx * (1.0 / kForceFix));
    force[L + n] = (float)((double)sy * (1.0 / kForceFix));
}

template <typename Real>
void launch_spread(const MembraneDev& m, TileDev& t, Real* force, int nx, int ny, size_t L, Status* st,
                   cudaStream_t s, bool slotsFilled) {
    if (m.Mcap == 0) {
        cudaMemsetAsync(t.active, 0, sizeof(int) * t.nTiles, s);
        return;
    }
    // fixed per-tile slot lists (filled by the force kernel when slotsFilled),
    // then the sums: FP64 in id order, FP32-shifted in exact fixed point
    if (!slotsFilled) launch_pdl(tile_slot_kernel, (m.Mcap + 127) / 128, 128, 0, s, m, t, nx, ny, st);
    if constexpr (sizeof(Real) == 4)
        launch_pdl(spread_fixed_kernel, t.nTiles, 256, 0, s, m, t, (float*)force, nx, ny, L, st);
    else
        launch_pdl(spread_kernel<Real>, t.nTiles, 256, 0, s, m, t, force, nx, ny, L, st);
}
template void launch_spread<double>(const MembraneDev&, TileDev&, double*, int, int, size_t, Status*,
                                    cudaStream_t, bool);
template void launch_spread<float>(const MembraneDev&, TileDev&, float*, int, int, size_t, Status*,
                                   cudaStream_t, bool);

// ---------------------------------------------------------------------------
// Interpolation and motion

__device__ __forceinline__ bool needs_perturbation(double X, double Y) {
    // The four tests of GeometryNode::perturbatePosition (GeometryNode.cpp:160, 174, 189, 202).
    if (fabs((double)(int)X - X) <= kEPSILON) return true;
    if (fabs((double)(int)Y - Y) <= kEPSILON) return true;
    if (fabs(Y - floor(Y) - (X - floor(X))) <= kEPSILON) return true;
    if (fabs(ceil(Y) - Y - (X - floor(X))) <= kEPSILON) return true;
    return false;
}

// Four lanes per membrane node, one per column of its stencil (eight nodes per
// warp).  A lane forms its column's and its row's Dirac factor (the rows'
// factors are shared by shuffles), loads the column's four rows of both
// velocity components at once and leaves the 16 products per component in
// shared memory by slot; then one lane per component adds them in slot order
// (the order of collectVelocity's sum is part of the result).
// With one thread per node the 16 loads, weights and additions formed one
// serial chain: 9.3 us for a single cell's 500 nodes and 14.3 us (FP64 18.1)
// for 150k nodes.  This form takes 2.8 us, and 11.2 us (FP64 13.7), where the
// L1 pipe (gathers, products) bounds it.
constexpr int kInterpBlock = 128;
constexpr int kInterpNodes = kInterpBlock / 4;  // nodes per block
// Place of (slot, node e) in a warp's products: eight nodes per slot, swapped
// about by the slot's column so that the four columns of two nodes, which a
// quarter warp stores at once, lie in different banks.
__device__ __forceinline__ int interp_place(int slot, int e) { return slot * 8 + (e ^ ((slot >> 2) << 1)); }

template <typename Real>
__global__ void __launch_bounds__(kInterpBlock) interp_move_kernel(MembraneDev m, const Real* u, int nx, int ny,
                                                                   size_t L, CrossDev c, Status* st) {
    pdl_wait();
    __shared__ double2 prod[kInterpBlock / 32][16 * 8];
    const int lane = threadIdx.x & 31, col = lane & 3, e = lane >> 2;
    double2* p = prod[threadIdx.x >> 5];
    const int i = blockIdx.x * kInterpNodes + (int)(threadIdx.x >> 2), ic = min(i, m.Mcap - 1);
    int halt = st->halt, M = m.topo->M;
    unsigned long long beside = st->beside;
    double X = m.x[ic], Y = m.y[ic], bind = (col < 2 ? m.bx : m.by)[ic];
    read_ahead(halt, beside, M, X, Y, bind);
    if (beside != 0) {  // the streams have joined: an error beside the step before stops the main sequence here
        if (blockIdx.x == 0 && threadIdx.x == 0) raise_halt(st, ST_INTERP_MOVE);
        return;
    }
    if (halt || i - e >= M) return;  // the whole warp
    const bool live = i < M;
    if (!live) X = Y = bind = 32.0;
    // stencil_range, one of its four bounds per lane
    const int bound = (col & 1) ? (int)floor(bind + 2.0) : (int)ceil(bind - 2.0);
    Stencil sc;
    sc.x0 = __shfl_sync(0xffffffffu, bound, lane & ~3);
    sc.x1 = __shfl_sync(0xffffffffu, bound, (lane & ~3) + 1);
    sc.y0 = __shfl_sync(0xffffffffu, bound, (lane & ~3) + 2);
    sc.y1 = __shfl_sync(0xffffffffu, bound, (lane & ~3) + 3);
    const bool ok = live && stencil_on_lattice(sc, nx, ny);
    if (live && !ok && col == 0) raise_error(st, ERR_STENCIL, i, ST_INTERP_MOVE);
    // the Dirac factors of the stencil's columns and rows, each formed once:
    // (fa * fb) / 16 is calculateDiscreteDeltaDirac's expression
    const double halfPi = M_PI / 2.0;
    const double fa = 1.0 + fast_cos(halfPi * ((double)(sc.x0 + col) - X));
    const double fbOwn = 1.0 + fast_cos(halfPi * ((double)(sc.y0 + col) - Y));
    double fb[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) fb[q] = __shfl_sync(0xffffffffu, fbOwn, (lane & ~3) + q);
    if (ok) {
        if (sc.x1 - sc.x0 == 3 && sc.y1 - sc.y0 == 3) {
            const size_t n0 = (size_t)sc.y0 * nx + (sc.x0 + col);
            Real ux[4], uy[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                ux[q] = u[n0 + (size_t)q * nx];
                uy[q] = u[L + n0 + (size_t)q * nx];
            }
            const int slot0 = 4 * (sc.x0 + col) + sc.y0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double dl = (fa * fb[q]) / 16.0;
                p[interp_place((slot0 + q) & 15, e)] = make_double2((double)ux[q] * dl, (double)uy[q] * dl);
            }
        } else {
            // wider stencil: the node bound to each slot (the slot's last writer)
            for (int k = 4 * col; k < 4 * col + 4; ++k) {
                int xk, yk;
                stencil_slot(sc, k, xk, yk);
                const size_t n = (size_t)yk * nx + xk;
                const double dl = dirac((double)xk - X, (double)yk - Y);
                p[interp_place(k, e)] = make_double2((double)u[n] * dl, (double)u[L + n] * dl);
            }
        }
    }
    __syncwarp();
    double v = 0.0;  // lane 0 of the node: x component, lane 1: y component
    if (ok && col < 2) {
#pragma unroll
        for (int k = 0; k < 16; ++k) v += reinterpret_cast<const double*>(p + interp_place(k, e))[col];
    }
    const double vOther = __shfl_xor_sync(0xffffffffu, v, 1);
    if (!ok || col > 1) return;
    const double vx = col == 0 ? v : vOther, vy = col == 0 ? vOther : v;
    const double CS = 1 / sqrt(3.0);
    const bool fast = ((vx * vx) + (vy * vy)) > CS;
    const double Xn = X + vx, Yn = Y + vy;
    if (col == 1) {
        m.vy[i] = vy;
        if (fast) return;
        m.oy[i] = Y;
        m.y[i] = Yn;
        return;
    }
    m.vx[i] = vx;
    if (fast) {
        raise_error(st, ERR_SPEED, i, ST_INTERP_MOVE);
        return;
    }
    m.ox[i] = X;
    m.x[i] = Xn;
    // listed for the host; the next kernel raises the halt, so that every
    // block here sees the same halt word and moves its nodes
    if (needs_perturbation(Xn, Yn)) {
        const int k = atomicAdd(&st->nPerturbNode, 1);
        if (k < c.perturbCap) c.perturbList[k] = i;
    }
}

template <typename Real>
void launch_interp_move(const MembraneDev& m, const Real* u, int nx, int ny, size_t L, CrossDev& c, Status* st,
                        cudaStream_t s) {
    if (m.Mcap == 0) return;
    launch_pdl(interp_move_kernel<Real>, (m.Mcap + kInterpNodes - 1) / kInterpNodes, kInterpBlock, 0, s, m, u, nx, ny, L,
               c, st);
}
template void launch_interp_move<double>(const MembraneDev&, const double*, int, int, size_t, CrossDev&, Status*,
                                         cudaStream_t);
template void launch_interp_move<float>(const MembraneDev&, const float*, int, int, size_t, CrossDev&, Status*,
                                        cudaStream_t);

// Adjoint of the spread for a differentiated run with frozen positions.  The
// spread adds dirac(x - X_i) * F_i to every lattice node x of node i's stencil
// (GeometryNode::distributeForce, GeometryNode.cpp:228-235), so
// dL/dF_i = sum over the same 16 slots of dirac * dL/dF(x): the interpolation
// of collectVelocity (GeometryNode.cpp:216-226) applied to G = dL/dF.
__global__ void force_adjoint_kernel(MembraneDev m, const double* G, int nx, int ny, size_t L, double* gfx,
                                     double* gfy) {
    pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.topo->M) return;
    const double X = m.x[i], Y = m.y[i];
    Stencil sc;
    double gx = 0.0, gy = 0.0;
    if (stencil_range(m.bx[i], m.by[i], nx, ny, sc)) {
        for (int k = 0; k < 16; ++k) {
            int xk, yk;
            stencil_slot(sc, k, xk, yk);
            const size_t n = (size_t)yk * nx + xk;
            const double dl = dirac((double)xk - X, (double)yk - Y);
            gx += G[n] * dl;
            gy += G[L + n] * dl;
        }
    }
    gfx[i] = gx;
    gfy[i] = gy;
}

void launch_force_adjoint(const MembraneDev& m, const double* G, int nx, int ny, size_t L, double* gfx,
                          double* gfy, cudaStream_t s) {
    if (m.Mcap == 0) return;
    launch_pdl(force_adjoint_kernel, (m.Mcap + 127) / 128, 128, 0, s, m, G, nx, ny, L, gfx, gfy);
}

// ---------------------------------------------------------------------------
// Crossings: three passes over the connections.
//   pass 0: closest distance per (node, slot) by atomicMin on the distance bits
//           (non-negative doubles order like their bit patterns);
//   pass 1: among records at that distance, the earliest connection;
//   pass 2: the winner writes its domain; the winner of a node's last present
//           slot (order E,N,W,S = the reference's boundaryNodes_ scan order)
//           decides the node's tentative domain (PhysicalNode.cpp:111-115).
constexpr unsigned long long kEmpty = ~0ull;

__device__ __forceinline__ int slot_code(int d) {  // E,N,W,S -> 0..3
    return d - 1;
}

// Pass 0: every crossing of a connection with a lattice line is a candidate
// boundary node for one (node, slot) key.  The closest distance per key is
// found by atomicMin on the distance's bits; each candidate is recorded for
// passes 1 and 2 and for the reset of its key at the end of the step.
//
// Almost every connection meets at most one vertical and one horizontal line:
// its (up to four) records are formed once, in registers.  A connection may be
// long (the cut across a cell that a division adds, until remeshing splits
// it): the general form enumerates the lattice lines between its end points,
// which the bounds test below keeps on the lattice, once to count and once to
// emit.  A block reserves its records with one atomic (a warp did: 4,700 of
// them on one address for 150k connections).  12.5 -> 7.8 us at 150k
// connections, 3.8 -> 3.6 us for one cell, with the perturbation test, a kernel
// of its own before (3.3 and 2.1 us), inside.

struct CrossRec {
    uint32_t key;
    uint32_t dom;
    unsigned long long bits;
};

__device__ __forceinline__ bool make_record(int nx, int ny, int px, int py, int dirSlot, double bx, double by,
                                            uint32_t bdom, CrossRec& r) {
    if (px < 0 || py < 0 || px >= nx || py >= ny) return false;
    const size_t node = (size_t)py * nx + px;
    const double d2 = ((double)px - bx) * ((double)px - bx) + ((double)py - by) * ((double)py - by);
    r.bits = (unsigned long long)__double_as_longlong(d2);
    r.key = (uint32_t)(node * 4 + slot_code(dirSlot));
    r.dom = bdom;
    return true;
}

// Calls fn(k, record) for the candidate records of connection cn in a fixed
// order (k = 0, 1, ...); returns the number of records, or -1 after raising
// the error of a connection that cannot be processed.  The kernel enumerates
// twice (count, emit) so that no per-thread record array is needed.
template <class Fn>
__device__ __forceinline__ int for_each_record(const MembraneDev& m, int cn, int nx, int ny, Status* st, bool report,
                                               Fn fn) {
    const int a = m.ca[cn], b = m.cb[cn];
    const double x1 = m.x[a], y1 = m.y[a], x2 = m.x[b], y2 = m.y[b];
    const uint32_t D = m.cdom[cn];
    const double maxX = x1 < x2 ? x2 : x1, maxY = y1 < y2 ? y2 : y1;
    const double minX = x2 < x1 ? x2 : x1, minY = y2 < y1 ? y2 : y1;
    const double mm = (y2 - y1) / (x2 - x1);
    const double nn = y1 - (y2 - y1) / (x2 - x1) * x1;
    if (!isfinite(mm)) {
        if (report) raise_error(st, ERR_VERTICAL, cn, ST_CROSSINGS);
        return -1;
    }
    if (!(minX >= -1.0 && maxX <= nx + 1.0 && minY >= -1.0 && maxY <= ny + 1.0)) {
        // keeps the line loops bounded for positions off the lattice
        if (report) raise_error(st, ERR_EDGE_W, cn, ST_CROSSINGS);
        return -1;
    }
    const bool eastward = x1 < x2, southward = y1 > y2;
    int k = 0;
    CrossRec r;
    for (int i = (int)ceil(minX); i <= (int)floor(maxX); i++) {
        const double yc = mm * i + nn;
        // fluidS gets its N slot, fluidN its S slot (Connection.cpp:273-279)
        if (!make_record(nx, ny, i, (int)floor(yc), N, (double)i, yc, eastward ? 0u : D, r)) break;
        fn(k++, r);
        if (!make_record(nx, ny, i, (int)ceil(yc), S, (double)i, yc, eastward ? D : 0u, r)) break;
        fn(k++, r);
    }
    for (int i = (int)ceil(minY); i <= (int)floor(maxY); i++) {
        const double xc = (i - nn) / mm;
        // fluidW gets its E slot, fluidE its W slot (Connection.cpp:307-313)
        if (!make_record(nx, ny, (int)floor(xc), i, E, xc, (double)i, southward ? 0u : D, r)) break;
        fn(k++, r);
        if (!make_record(nx, ny, (int)ceil(xc), i, W, xc, (double)i, southward ? D : 0u, r)) break;
        fn(k++, r);
    }
    const int want = 2 * (max(0, (int)floor(maxX) - (int)ceil(minX) + 1) + max(0, (int)floor(maxY) - (int)ceil(minY) + 1));
    if (k != want) {
        if (report) raise_error(st, ERR_EDGE_W, cn, ST_CROSSINGS);
        return -1;
    }
    return k;
}

// `check`: the first kernel after the move.  It raises the halt for the nodes
// that the move listed for the host's perturbation, and lists the connections
// whose end points share an x or a y to within EPSILON
// (Connection::perturbConnection's tests, Connection.cpp:339-340, 363-364) in
// `perturb` (up to perturbCap) instead of crossing them; the next kernel raises
// the halt for those, so that every block here sees the same halt word and the
// list is complete.  The halted step's records are reset like any other's
// (domain_fill_kernel), and the crossings run again once the host is done.
constexpr int kCrossBlock = 128;
__global__ void __launch_bounds__(kCrossBlock) crossings_kernel(MembraneDev m, CrossDev c, int nx, int ny, Status* st,
                                                                int check, int* perturb, int perturbCap) {
    pdl_wait();
    const int cn = blockIdx.x * kCrossBlock + threadIdx.x, cc = min(cn, max(m.Ccap, 1) - 1);
    const bool any = m.Ccap > 0;  // there are buffers to read from
    int halt = st->halt, nodes = st->nPerturbNode, C = m.topo->C, a = any ? m.ca[cc] : 0, b = any ? m.cb[cc] : 0;
    uint32_t D = any ? m.cdom[cc] : 0u;
    read_ahead(halt, nodes, C, a, b, D);
    // Other blocks may raise an error meanwhile, between the reads of two warps
    // of this block: a warp that sees it has no records, and takes part in the
    // block's count of them all the same.
    const bool wait = check && nodes > 0;
    if (wait && !halt && blockIdx.x == 0 && threadIdx.x == 0) raise_halt(st, ST_INTERP_MOVE);
    int nrec = 0;
    bool simple = false;
    CrossRec r[4];
    bool have[4] = {false, false, false, false};
    if (cn < C && !halt && !wait) {
        const double x1 = m.x[a], y1 = m.y[a], x2 = m.x[b], y2 = m.y[b];
        if (check && (fabs(x1 - x2) < kEPSILON || fabs(y1 - y2) < kEPSILON)) {
            const int k = atomicAdd(&st->nPerturbConn, 1);
            if (k < perturbCap) perturb[k] = cn;
        } else {
            const double maxX = x1 < x2 ? x2 : x1, maxY = y1 < y2 ? y2 : y1;
            const double minX = x2 < x1 ? x2 : x1, minY = y2 < y1 ? y2 : y1;
            const double mm = (y2 - y1) / (x2 - x1);
            const int iv = (int)ceil(minX), ih = (int)ceil(minY);
            const int nv = (int)floor(maxX) - iv + 1, nh = (int)floor(maxY) - ih + 1;
            // one line each way at most, inside the lattice with room to spare
            simple = isfinite(mm) && minX >= 1.0 && maxX <= nx - 2.0 && minY >= 1.0 && maxY <= ny - 2.0 && nv <= 1 &&
                     nh <= 1;
            if (simple) {
                const double nn = y1 - mm * x1;
                if (nv == 1) {
                    // fluidS gets its N slot, fluidN its S slot (Connection.cpp:273-279)
                    const double yc = mm * iv + nn;
                    const bool eastward = x1 < x2;
                    have[0] = make_record(nx, ny, iv, (int)floor(yc), N, (double)iv, yc, eastward ? 0u : D, r[0]);
                    have[1] = make_record(nx, ny, iv, (int)ceil(yc), S, (double)iv, yc, eastward ? D : 0u, r[1]);
                }
                if (nh == 1) {
                    // fluidW gets its E slot, fluidE its W slot (Connection.cpp:307-313)
                    const double xc = (ih - nn) / mm;
                    const bool southward = y1 > y2;
                    have[2] = make_record(nx, ny, (int)floor(xc), ih, E, xc, (double)ih, southward ? 0u : D, r[2]);
                    have[3] = make_record(nx, ny, (int)ceil(xc), ih, W, xc, (double)ih, southward ? D : 0u, r[3]);
                }
                nrec = have[0] + have[1] + have[2] + have[3];
                // a crossing off the lattice: the general form reports it
                simple = nrec == 2 * (max(nv, 0) + max(nh, 0));
            }
            if (!simple) {
                nrec = for_each_record(m, cn, nx, ny, st, true, [](int, const CrossRec&) {});
                if (nrec < 0) nrec = 0;
            }
        }
    }
    // the block's records, in any order (they also list the keys to reset at
    // the end of the step), and the closest distance per key
    __shared__ int warpSum[kCrossBlock / 32], blockBase;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = nrec;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += v;
    }
    if (lane == 31) warpSum[warp] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
        int total = 0;
#pragma unroll
        for (int w = 0; w < kCrossBlock / 32; ++w) {
            const int v = warpSum[w];
            warpSum[w] = total;
            total += v;
        }
        blockBase = total > 0 ? atomicAdd(&st->nCrossRec, total) : 0;
    }
    __syncthreads();
    if (nrec == 0) return;
    const int rb = blockBase + warpSum[warp] + incl - nrec;
    auto emit = [&](int k, const CrossRec& q) {
        const int idx = rb + k;
        if (idx < c.recCap) {
            c.recKey[idx] = q.key; c.recConn[idx] = (uint32_t)cn; c.recDom[idx] = q.dom; c.recDist[idx] = q.bits;
        } else {
            raise_error(st, ERR_CAPACITY, cn, ST_CROSSINGS);
        }
        atomicMin(&c.bnDist[q.key], q.bits);
    };
    if (simple) {
        int k = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (have[j]) emit(k++, r[j]);
    } else {
        for_each_record(m, cn, nx, ny, st, false, emit);
    }
}

// GeometryHandler::connectGeometryNodesToPhysicalNodes for one node
// (GeometryHandler.cpp:608-644): a node that left its previous unit cell
// (GeometryNode::isUpdateNeeded, GeometryNode.cpp:256-261, Rectangle.cpp
// pointWithinBounds) is bound again from its current position, after the
// edge test; the others keep their binding.  True if the test raised an error.
__device__ __forceinline__ bool edge_check_node(const MembraneDev& m, int i, int nx, int ny, Status* st, int stage) {
    const double X = m.x[i], Y = m.y[i], ox = m.ox[i], oy = m.oy[i];
    const bool within = (X >= floor(ox)) && (X < ceil(ox)) && (Y <= ceil(oy)) && (Y > floor(oy));
    if (within) return false;
    m.bx[i] = X;
    m.by[i] = Y;
    if (X - 2.0 < 0) raise_error(st, ERR_EDGE_W, i, stage);
    else if (Y - 2.0 < 0) raise_error(st, ERR_EDGE_S, i, stage);
    else if (X + 2.0 > nx) raise_error(st, ERR_EDGE_E, i, stage);
    else if (Y + 2.0 > ny) raise_error(st, ERR_EDGE_N, i, stage);
    else return false;
    return true;
}

// Pass 1: among records at the closest distance, the earliest connection.
// And, over the same grid, GeometryHandler::connectGeometryNodesToPhysicalNodes'
// edge test of the moved nodes, and the count of the connections that the
// remeshing pass will split (remesh.cuh; a kernel of its own, with the pass's
// decision in its last block, took 6.3 us at 150k connections).  The kernel
// first raises the halt for the connections that pass 0 listed for the host's
// perturbation.  It is the last kernel that decides whether the domain stages run:
// in a graph of several steps they run beside the main sequence, whose later
// stages may halt.
__global__ void __launch_bounds__(kRemeshBlock) cross_tie_kernel(CrossDev c, MembraneDev m, TopoDev t, int nx, int ny,
                                                                 Status* st) {
    pdl_wait();
    const int tid = blockIdx.x * kRemeshBlock + threadIdx.x, all = gridDim.x * kRemeshBlock;
    const int rc = min(tid, c.recCap - 1);
    int halt = st->halt, conns = st->nPerturbConn, n = st->nCrossRec, M = m.topo->M;
    uint32_t key = c.recKey[rc], conn = c.recConn[rc];
    unsigned long long dist = c.recDist[rc];
    read_ahead(halt, conns, n, M, key, conn, dist);
    if (tid == 0) st->domainGo = !halt && conns == 0;
    if (halt) return;
    if (conns > 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) raise_halt(st, ST_PERTURB_CONN);
        return;
    }
    n = min(n, c.recCap);
    for (int r = tid; r < n; r += all) {
        if (r != tid) {
            key = c.recKey[r];
            conn = c.recConn[r];
            dist = c.recDist[r];
        }
        if (c.bnDist[key] == dist) atomicMin(&c.bnConn[key], conn);
    }
    for (int i = tid; i < M; i += all)
        if (edge_check_node(m, i, nx, ny, st, ST_CROSSINGS)) st->domainStop = 1;
    if (t.flag != nullptr) remesh_count_block(m, t);  // (not at set-up)
}

// Pass 2: the winner writes its domain; the winner of a node's last present
// slot (order E,N,W,S = the reference's boundaryNodes_ scan order) decides the
// node's tentative domain (PhysicalNode.cpp:111-115).
// The boundary node of a winning record whose connection carries boundary
// solvers: its position on the lattice line (BoundaryNode(i, getYPos(m, i, n))
// or BoundaryNode(getXPos(m, i, n), i), Connection.cpp:243-312) and its
// velocity, interpolated along the connection (Connection::calculateVelocity,
// Connection.cpp:146-168), kept for the next step's no-flux solvers.
__device__ __forceinline__ void record_noflux(const MembraneDev& m, CrossDev& c, int conn, uint32_t key, int nx) {
    const int desc = m.cdesc[conn];
    if (desc < 0 || c.nfTab[desc].nSolvers == 0) return;
    const int a = m.ca[conn], b = m.cb[conn];
    const double x1 = m.x[a], y1 = m.y[a], x2 = m.x[b], y2 = m.y[b];
    const double mm = (y2 - y1) / (x2 - x1);
    const double nn = y1 - (y2 - y1) / (x2 - x1) * x1;
    const size_t node = key >> 2;
    const int s = (int)(key & 3u);  // E, N, W, S
    const int px = (int)(node % (size_t)nx), py = (int)(node / (size_t)nx);
    double bx, by;
    if (s == 1 || s == 3) {  // N / S slot: a crossing with the vertical line x = px
        bx = (double)px;
        by = mm * px + nn;
    } else {                 // E / W slot: a crossing with the horizontal line y = py
        bx = (py - nn) / mm;
        by = (double)py;
    }
    const double l = sqrt((x1 - bx) * (x1 - bx) + (y1 - by) * (y1 - by));
    const double Lc = sqrt((x2 - x1) * (x2 - x1) + (y2 - y1) * (y2 - y1));
    const double vx1 = m.vx[a], vy1 = m.vy[a], vx2 = m.vx[b], vy2 = m.vy[b];
    c.nfU[2 * (size_t)key] = (vx2 - vx1) * l / Lc + vx1;
    c.nfU[2 * (size_t)key + 1] = (vy2 - vy1) * l / Lc + vy1;
    c.nfSpec[key] = (uint8_t)(desc + 1);
    const int k = atomicAdd(c.nfN, 1);
    if (k < c.nfCap) c.nfKeys[k] = key;
}

__global__ void cross_win_kernel(CrossDev c, MembraneDev m, const uint32_t* dom, int nx, int ny, Status* st) {
    pdl_wait();
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, all = gridDim.x * blockDim.x, rc = min(tid, c.recCap - 1);
    int go = st->domainGo, stop = st->domainStop, n = st->nCrossRec;
    uint32_t key = c.recKey[rc], conn = c.recConn[rc], bdom = c.recDom[rc];
    unsigned long long dist = c.recDist[rc];
    read_ahead(go, stop, n, key, conn, bdom, dist);
    if (!go || stop) return;
    n = min(n, c.recCap);
    for (int r = tid; r < n; r += all) {
        if (r != tid) {
            key = c.recKey[r];
            conn = c.recConn[r];
            bdom = c.recDom[r];
            dist = c.recDist[r];
        }
        const size_t node = key >> 2;
        const int s = (int)(key & 3u);
        // the node's four slots and domain, whether or not the record wins
        const ulonglong2 d01 = *(const ulonglong2*)(c.bnDist + node * 4), d23 = *(const ulonglong2*)(c.bnDist + node * 4 + 2);
        const uint32_t winner = c.bnConn[key], old = dom[node];
        const unsigned long long at[4] = {d01.x, d01.y, d23.x, d23.y};
        if ((s == 0 ? at[0] : s == 1 ? at[1] : s == 2 ? at[2] : at[3]) != dist || winner != conn) continue;
        c.bnDom[key] = bdom;
        if (c.nfTab != nullptr) record_noflux(m, c, (int)conn, key, nx);
        if (c.bounceW != nullptr && s >= 2) {
            // DiracD2Q5's advect skips the swap with the W / S neighbour when
            // this node has a boundary node there (DiracD2Q5.cpp:166-180)
            (s == 2 ? c.bounceW : c.bounceS)[node] = 1;
            const int k = atomicAdd(c.bounceN, 1);
            if (k < c.bounceCap) c.bounceKeys[k] = key;
            else raise_error_beside(st, ERR_CAPACITY, (int)node, ST_CROSSINGS);
        }
        if (s == 2) {
            c.wDom[node] = bdom + 1;
            c.rowNow[(uint32_t)node / (uint32_t)nx] = 1;
        }
        const bool last = (s >= 1 || at[1] == kEmpty) && (s >= 2 || at[2] == kEmpty) && (s >= 3 || at[3] == kEmpty);
        if (last && bdom != old) {
            const int k = atomicAdd(&st->nChanged, 1);
            if (k < c.changedCap) {
                c.changedNode[k] = (uint32_t)node;
                c.changedDom[k] = bdom;
                c.rowNow[(uint32_t)node / (uint32_t)nx] = 1;
                c.mark[node] = k + 1;  // the node's position in the list, for the re-initialisation
            } else {
                raise_error_beside(st, ERR_CAPACITY, (int)node, ST_CROSSINGS);
            }
        }
    }
}

// Clears the previous step's no-flux boundary nodes (after the stream-collide
// that used them, before this step's crossings set the new ones).  A halted
// step, which ran no stream-collide, leaves them to the step that will.
__global__ void noflux_reset_kernel(CrossDev c, const Status* st) {
    pdl_wait();
    if (st->halt) return;
    const int n = min(*c.nfN, c.nfCap);
    for (int k = threadIdx.x; k < n; k += blockDim.x) c.nfSpec[c.nfKeys[k]] = 0;
    __syncthreads();
    if (threadIdx.x == 0) *c.nfN = 0;
}

// Clears the previous step's W / S boundary-node marks (after the
// stream-collide that used them, before this step's crossings set new ones);
// not on a halted step (noflux_reset_kernel).
__global__ void bounce_reset_kernel(CrossDev c, const Status* st) {
    pdl_wait();
    if (st->halt) return;
    const int n = min(*c.bounceN, c.bounceCap);
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        const uint32_t key = c.bounceKeys[k];
        ((key & 3u) == 2u ? c.bounceW : c.bounceS)[key >> 2] = 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) *c.bounceN = 0;
}

// GeometryHandler::connectGeometryNodesToPhysicalNodes' edge test for nodes
// that left their previous unit cell (GeometryHandler.cpp:610-636,
// GeometryNode.cpp:256-261, Rectangle.cpp pointWithinBounds).
__global__ void edge_check_kernel(MembraneDev m, int nx, int ny, Status* st, int stage) {
    pdl_wait();
    if (st->halt) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.topo->M) return;
    edge_check_node(m, i, nx, ny, st, stage);
}

void launch_crossings(const MembraneDev& m, CrossDev& c, int nx, int ny, Status* st, const TopoDev* remesh,
                       cudaStream_t s, bool check, int* perturb, int perturbCap) {
    const int blocks = (m.Ccap + kCrossBlock - 1) / kCrossBlock;
    if (m.Ccap == 0) {  // nodes without connections: the halt of the listed nodes alone
        if (check && m.Mcap > 0)
            launch_pdl(crossings_kernel, 1, kCrossBlock, 0, s, m, c, nx, ny, st, 1, perturb, perturbCap);
        return;
    }
    if (c.nfTab != nullptr) launch_pdl(noflux_reset_kernel, 1, 1024, 0, s, c, st);
    if (c.bounceW != nullptr) launch_pdl(bounce_reset_kernel, 1, 1024, 0, s, c, st);
    // the record count (st->nCrossRec) is zero here: cleared with the status
    // word before a run and at the end of each step's domain fill (end_step)
    launch_pdl(crossings_kernel, blocks, kCrossBlock, 0, s, m, c, nx, ny, st, check ? 1 : 0, perturb, perturbCap);
    // grid-stride over the step's records (their count is known on the device
    // only): up to 8 blocks per SM, so that each thread's chain of dependent
    // loads overlaps many others, and no more than 4 records per connection
    // fill
    const int recBlocks = std::min(148 * 8, (4 * m.Ccap + 255) / 256);
    launch_pdl(cross_tie_kernel, std::max(recBlocks, (m.Ccap + kRemeshBlock - 1) / kRemeshBlock), kRemeshBlock, 0, s, c, m,
               remesh ? *remesh : TopoDev{}, nx, ny, st);
}

void launch_cross_winners(const MembraneDev& m, CrossDev& c, const uint32_t* dom, int nx, int ny, Status* st,
                          cudaStream_t s, bool programmatic) {
    if (m.Ccap == 0) return;
    launch_ex(programmatic, cross_win_kernel, std::min(148 * 8, (4 * m.Ccap + 255) / 256), 256, 0, s, c, m, dom, nx, ny,
              st);
}

void launch_edge_check(const MembraneDev& m, int nx, int ny, Status* st, cudaStream_t s) {
    if (m.Mcap == 0) return;
    launch_pdl(edge_check_kernel, (m.Mcap + 127) / 128, 128, 0, s, m, nx, ny, st, ST_REMESH);
}

// ---------------------------------------------------------------------------
// Reinitialisation of the species at nodes whose domain changed.
//
// The reference visits all lattice nodes in row-major order; a changed node
// takes its new domain and re-initialises from its E,N,W,S neighbours of the
// same domain that have no boundary node on the link, reading neighbours that
// come earlier in the order with their new state and later ones with their old
// state.  So a changed node waits for the earlier changed nodes among its
// E,N,W,S,NE (read after write) and SW (write after read) neighbours; the
// nodes that wait for none (almost all of them) are re-initialised at once by
// the whole grid, the others by the grid's last block, in rounds.
//
// One warp per changed node: its lanes read what the update may need (the
// species' 25 neighbour values, the neighbours' domains and marks, the boundary
// slots, the velocity) in one go, and the arithmetic, which is the reference's
// in its order, runs alike in every lane.  With a thread per node (75 loads
// and 106 registers each) and the waiting nodes in a second one-block launch
// the stage took 16.6 us for 150 changed nodes of 1024^2 and 4.2 us for none;
// this form takes 11.1 (latency: five dependent reads, then those of the waiting
// nodes) and 1.6 us.
constexpr int kReinitMax = 4096;  // changed nodes per step
struct SpeciesSet {
    SpeciesConst s[kMaxSpecies];
};

// What a warp's lanes read for the re-initialisation of a node: lane 5 s + q
// slot q of neighbour s (E, N, W, S, NE) of each species; the domains, boundary
// slots and the velocity ride on lanes of their own.
template <typename Real>
struct ReinitLoads {
    Real gv[kMaxSpecies];
    uint32_t dom;
    bool bn;
    double u;
};

// Neighbour s of (x, y): E, N, W, S, NE, then the other diagonals NW, SW, SE.
__device__ __forceinline__ size_t reinit_neighbour(int x, int y, int nx, int ny, int s) {
    const int xm = x == 0 ? nx - 1 : x - 1, xp = x == nx - 1 ? 0 : x + 1;
    const int ym = y == 0 ? ny - 1 : y - 1, yp = y == ny - 1 ? 0 : y + 1;
    const int X = (s == 0 || s == 4 || s == 7) ? xp : ((s == 2 || s == 5 || s == 6) ? xm : x);
    const int Y = (s == 1 || s == 4 || s == 5) ? yp : ((s == 3 || s == 6 || s == 7) ? ym : y);
    return (size_t)Y * nx + X;
}

// The values other blocks may have written in this launch are read past the L1
// cache.
template <typename Real>
__device__ __forceinline__ ReinitLoads<Real> reinit_load(size_t n, const uint32_t* dom, const Real* g, const Real* u,
                                                         int nS, const CrossDev& c, int nx, int ny, size_t L) {
    const int lane = threadIdx.x & 31;
    const int x = (int)((uint32_t)n % (uint32_t)nx), y = (int)((uint32_t)n / (uint32_t)nx);
    const int s5 = lane / 5, q5 = lane - 5 * s5;
    const size_t nbv = reinit_neighbour(x, y, nx, ny, s5 < 5 ? s5 : 4);
    ReinitLoads<Real> r;
#pragma unroll
    for (int k = 0; k < kMaxSpecies; ++k)
        r.gv[k] = k < nS && lane < 25 ? __ldcg(g + ((size_t)k * 5 + q5) * L + nbv) : (Real)0;
    r.dom = lane < 8 ? __ldcg(dom + reinit_neighbour(x, y, nx, ny, lane)) : (lane == 8 ? __ldcg(dom + n) : 0u);
    r.bn = lane < 4 && __ldcg(c.bnDist + n * 4 + lane) != kEmpty;
    r.u = lane < 2 ? (double)u[(size_t)lane * L + n] : 0.0;
    return r;
}

// The warp re-initialises node n (all lanes take part).
template <typename Real>
__device__ __forceinline__ void reinit_node(const ReinitLoads<Real>& in, size_t n, uint32_t newDom, uint32_t* dom,
                                            Real* g, int nS, const SpeciesConst* sp, const double* srcTab,
                                            int nDomains, const uint32_t* ctypeTab, int cellTypesCopied, int nx,
                                            int ny, size_t L, Status* st, unsigned iteration) {
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned hasBN = __ballot_sync(all, in.bn);
    const unsigned same = __ballot_sync(all, lane < 8 && in.dom == newDom);  // bit s: neighbour s is of the new domain
    const uint32_t oldDom = __shfl_sync(all, in.dom, 8);
    const double ux = __shfl_sync(all, in.u, 0), uy = __shfl_sync(all, in.u, 1);
    if (lane == 0) dom[n] = newDom;
    // boundaryNodes_[NE] aliases (domainIdentifier_, cellType_): null only if both are 0.
    const uint32_t ctype = cellTypesCopied ? (oldDom < (uint32_t)nDomains ? ctypeTab[oldDom] : 1u) : 0u;
    const bool neNull = newDom == 0 && ctype == 0;
    double Cnew[2] = {0.0, 0.0};  // getC() of the first two species once re-initialised here
    bool coupled = false;
    for (int k = 0; k < nS; ++k) coupled |= sp[k].partner >= 0;
#pragma unroll 1
    for (int k = 0; k < nS; ++k) {
        const Real* gk = g + (size_t)k * 5 * L;
        // getC() of neighbour s in slot order after localSwap (T, W, S, E, N),
        // formed by lane s
        const double v = (double)(k == 0 ? in.gv[0] : k == 1 ? in.gv[1] : in.gv[2]);
        const int b = 5 * (lane < 5 ? lane : 0);
        double Cs = 0.0;
        Cs += __shfl_sync(all, v, b);
        Cs += __shfl_sync(all, v, b + 3);
        Cs += __shfl_sync(all, v, b + 4);
        Cs += __shfl_sync(all, v, b + 1);
        Cs += __shfl_sync(all, v, b + 2);
        const int style = sp[k].reinit;
        double sumC = 0.0;
        int counter = 0;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const double Cn = __shfl_sync(all, Cs, s);
            if (!((hasBN >> s) & 1u) && ((same >> s) & 1u)) {
                sumC += Cn;
                counter++;
            }
        }
        if (counter == 0 && style != RI_DIAG && neNull && ((same >> 4) & 1u)) {
            sumC += __shfl_sync(all, Cs, 4);
            counter++;
            if (lane == 0) atomicAdd(&st->nDiagReinit, 1);
        }
        if (counter == 0 && style == RI_DIAG) {
            // NE, NW, SW, SE of the same domain, no boundary-node test
            for (int s = 4; s < 8; ++s) {
                if (!((same >> s) & 1u)) continue;
                const size_t nd = reinit_neighbour((int)(n % nx), (int)(n / nx), nx, ny, s);
                double C = 0.0;
                C += (double)__ldcg(gk + nd);
                C += (double)__ldcg(gk + 3 * L + nd);
                C += (double)__ldcg(gk + 4 * L + nd);
                C += (double)__ldcg(gk + 1 * L + nd);
                C += (double)__ldcg(gk + 2 * L + nd);
                sumC += C;
                counter++;
            }
            if (counter != 0 && lane == 0) atomicAdd(&st->nDiagReinit, 1);
        }
        if (counter == 0 && style == RI_ALL4) {
            // all of E, N, W, S whatever their domain
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                sumC += __shfl_sync(all, Cs, s);
                counter++;
            }
        }
        if (counter == 0 && lane == 0) atomicAdd(&st->nFailedReinit, 1);
        sumC /= static_cast<double>(counter);
        double gi[5];
        for (int q = 0; q < 5; ++q) gi[q] = style == RI_DIAG ? sumC / 4.0 : sumC / 5.0;
        const double src = (srcTab != nullptr && newDom < (uint32_t)nDomains) ? srcTab[(size_t)k * nDomains + newDom]
                                                                            : 0.0;
        // a coupled reaction reads the partner's getC(): re-initialised
        // already (an earlier species), else its state from this step's collide
        double Cp = 0.0;
        const int pj = sp[k].partner;
        if (pj >= 0 && pj < nS) {
            if (pj < k) {
                Cp = pj == 0 ? Cnew[0] : Cnew[1];
            } else {
                const Real* gp = g + (size_t)pj * 5 * L + n;
                Cp += (double)__ldcg(gp);
                Cp += (double)__ldcg(gp + 3 * L);
                Cp += (double)__ldcg(gp + 4 * L);
                Cp += (double)__ldcg(gp + 1 * L);
                Cp += (double)__ldcg(gp + 2 * L);
            }
        }
        collide_cde64(gi, ux, uy, sp[k], src, Cp, newDom, ctype, iteration);
        if (coupled) {
            const double C = sum5_swapped(gi);
            if (k == 0) Cnew[0] = C;
            else Cnew[1] = C;
        }
        const double out = lane == 0 ? gi[0] : lane == 1 ? gi[1] : lane == 2 ? gi[2] : lane == 3 ? gi[3] : gi[4];
        if (lane < 5) g[((size_t)k * 5 + lane) * L + n] = (Real)out;
    }
}

// Place + 1 in the changed list of the earlier changed node that lane d < 8
// finds in direction d (0: none, or it is not waited for): E, N, W, S, NE, SW;
// with a species that falls back on all four diagonals (RI_DIAG) also NW, SE.
__device__ __forceinline__ int reinit_dep(const CrossDev& c, size_t n, int nx, int ny, int d) {
    if (d >= 8 || (d >= 6 && !c.diag8)) return 0;
    const int s = d == 5 ? 6 : d == 6 ? 5 : d;  // SW before NW
    const size_t nb = reinit_neighbour((int)((uint32_t)n % (uint32_t)nx), (int)((uint32_t)n / (uint32_t)nx), nx, ny, s);
    return nb < n ? c.mark[nb] : 0;
}

// (Each changed node's place in the list is marked where the crossings append
// it, in cross_win_kernel; the last block clears the marks.)  No two nodes that
// wait for none read each other (a changed neighbour in any of the directions
// makes one of the two wait for the other), so the order among them does not
// matter.
constexpr int kReinitBlock = 128;
template <typename Real>
__global__ void __launch_bounds__(kReinitBlock) reinit_kernel(CrossDev c, uint32_t* dom, Real* g, const Real* u, int nS,
                                                              const __grid_constant__ SpeciesSet species,
                                                              const double* srcTab, int nDomains,
                                                              const uint32_t* ctypeTab, int nx, int ny, size_t L,
                                                              Status* st) {
    pdl_wait();
    const int lane = threadIdx.x & 31, warps = kReinitBlock / 32, warp = threadIdx.x >> 5;
    const int k0 = blockIdx.x * warps + warp;
    int go = st->domainGo, stop = st->domainStop, cnt = st->nChanged, typesCopied = st->cellTypesCopied;
    uint32_t iteration = st->iteration, node0 = c.changedNode[min(k0, c.changedCap - 1)];
    read_ahead(go, stop, cnt, typesCopied, iteration, node0);
    if (!go || stop || cnt == 0) return;
    if (cnt > kReinitMax || cnt > c.changedCap) {
        if (blockIdx.x == 0 && threadIdx.x == 0) raise_error_beside(st, ERR_CAPACITY, cnt, ST_REINIT);
        return;
    }
    const SpeciesConst* sp = species.s;
    for (int k = k0; k < cnt; k += gridDim.x * warps) {
        const size_t n = k == k0 ? node0 : c.changedNode[k];
        const uint32_t newDom = c.changedDom[k];
        // read with the marks, before it is known that the node may go ahead
        const ReinitLoads<Real> in = reinit_load<Real>(n, dom, g, u, nS, c, nx, ny, L);
        const bool free = !__any_sync(0xffffffffu, reinit_dep(c, n, nx, ny, lane) > 0);
        if (lane == 0) {
            int done = 1;
            if (!free) {
                // listed for the last block; the place says where
                const int w = atomicAdd(&c.nWait[0], 1);
                c.waitList[w] = k;
                done = 2 + w;
            }
            c.reinitDone[k] = done;
        }
        if (free)
            reinit_node<Real>(in, n, newDom, dom, g, nS, sp, srcTab, nDomains, ctypeTab, typesCopied, nx, ny, L, st,
                              iteration);
    }
    // the last block to finish: the waiting nodes, usually few or none.  A node
    // waited for is done when the whole grid's pass did it (reinitDone 1) or
    // when this one has (done[w] of its place w in the wait list).
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd((unsigned*)&c.nWait[1], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int nw = __ldcg(&c.nWait[0]);
    __shared__ unsigned char done[kReinitMax];
    __shared__ int remaining;
    for (int w = threadIdx.x; w < nw; w += kReinitBlock) done[w] = 0;
    if (threadIdx.x == 0) remaining = nw;
    __syncthreads();
    // a round does every node whose earlier ones are done: at most nw rounds
    for (int round = 0; round < nw && remaining > 0; ++round) {
        __syncthreads();
        for (int w = warp; w < nw; w += warps) {
            if (done[w]) continue;
            const size_t n = c.changedNode[__ldcg(&c.waitList[w])];
            const int p = reinit_dep(c, n, nx, ny, lane);
            bool waits = false;
            if (p > 0) {
                const int v = __ldcg(&c.reinitDone[p - 1]);
                waits = v != 1 && done[v - 2] != 1;
            }
            // marked only after the round's tests: no node of the round sees it done
            if (!__any_sync(0xffffffffu, waits) && lane == 0) done[w] = 2;
        }
        __syncthreads();
        for (int w = warp; w < nw; w += warps) {
            if (done[w] != 2) continue;
            const int k = __ldcg(&c.waitList[w]);
            const size_t n = c.changedNode[k];
            reinit_node<Real>(reinit_load<Real>(n, dom, g, u, nS, c, nx, ny, L), n, c.changedDom[k], dom, g, nS, sp,
                              srcTab, nDomains, ctypeTab, typesCopied, nx, ny, L, st, iteration);
            if (lane == 0) atomicSub(&remaining, 1);
        }
        __syncthreads();
        for (int w = threadIdx.x; w < nw; w += kReinitBlock)
            if (done[w] == 2) done[w] = 1;
        __syncthreads();
    }
    for (int k = threadIdx.x; k < cnt; k += kReinitBlock) c.mark[(size_t)c.changedNode[k]] = 0;
    if (threadIdx.x < 2) c.nWait[threadIdx.x] = 0;
}

template <typename Real>
void launch_reinit(CrossDev& c, uint32_t* dom, Real* g, const Real* u, int nS, const SpeciesConst* sp,
                   const double* srcTab, int nDomains, const uint32_t* ctypeTab, int nx, int ny, size_t L, Status* st,
                   cudaStream_t s) {
    if (c.changedCap <= 0) return;
    const SpeciesSet species{{sp[0], sp[1], sp[2]}};
    launch_pdl(reinit_kernel<Real>, 148, kReinitBlock, 0, s, c, dom, g, u, nS, species, srcTab, nDomains, ctypeTab, nx,
               ny, L, st);
}
template void launch_reinit<double>(CrossDev&, uint32_t*, double*, const double*, int, const SpeciesConst*,
                                    const double*, int, const uint32_t*, int, int, size_t, Status*, cudaStream_t);
template void launch_reinit<float>(CrossDev&, uint32_t*, float*, const float*, int, const SpeciesConst*,
                                   const double*, int, const uint32_t*, int, int, size_t, Status*, cudaStream_t);

// ---------------------------------------------------------------------------
// Domain fill: one block per row; the row's domain id at x >= 1 is the domain
// of the last W-slot boundary node at x' in [1, x], else dom(0, y), which must
// be 0 (GeometryHandler.cpp:68-85).  Reads and clears the W-slot plane.
// The kernel also resets the (node, slot) entries the step's crossings wrote
// (every written key has a record), after the re-initialisation that read
// them; that part runs on a halted step too.
//
// Each warp takes eight segments of 32 nodes, all loaded before the first is
// used; the last mark at or before a node is a ballot and a shuffle, and the
// warps' last marks meet in shared memory.  Rows without a mark now and after
// the last fill, and without a changed node, hold the exterior throughout and
// are left as they are.  With a run of consecutive nodes per thread (strided
// access) and a block scan the kernel took 6.5 us for 1024^2 and 25 us for a
// 2048^2 lattice with cells in its middle; this form takes 6.1 and 9.1 us.
constexpr int kFillBlock = 128, kFillSeg = 8;
__device__ __forceinline__ void fill_row(const CrossDev& c, uint32_t* dom, int nx, int y, Status* st);

// The last block ends the step (end_step).  `gated`: the crossings' ties ran and
// decided whether the domain stages do (else, without connections, the halt word).
__global__ void __launch_bounds__(kFillBlock) domain_fill_kernel(CrossDev c, uint32_t* dom, int nx, int gated,
                                                                 Status* st) {
    pdl_wait();
    const int y = blockIdx.x;
    const size_t row = (size_t)y * nx;
    // everything the block's course depends on, read at once
    int nrec = st->nCrossRec, go = gated ? st->domainGo : !st->halt, stop = st->domainStop;
    int marked = c.rowNow[y] | c.rowHad[y];
    uint32_t left = dom[row];
    read_ahead(nrec, go, stop, marked, left);
    nrec = min(nrec, c.recCap);
    go = go && !stop;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nrec; k += gridDim.x * blockDim.x) {
        const uint32_t key = c.recKey[k];
        c.bnDist[key] = kEmpty;
        c.bnConn[key] = ~0u;
    }
    if (go && marked) {
        if (left == 0) fill_row(c, dom, nx, y, st);
        else if (threadIdx.x == 0) raise_error_beside(st, ERR_LEFT_DOMAIN, y, ST_DOMAIN);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd((unsigned*)&c.nWait[2], 1u) == gridDim.x - 1) {
            c.nWait[2] = 0;
            __threadfence();
            end_step(st, go);
        }
    }
}

__device__ __forceinline__ void fill_row(const CrossDev& c, uint32_t* dom, int nx, int y, Status* st) {
    const size_t row = (size_t)y * nx;
    constexpr int warps = kFillBlock / 32;
    __shared__ uint32_t lastOf[warps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t carry = 0;  // the last mark before this pass (domain + 1, 0: none)
    bool any = false;
    for (int x0 = 0; x0 < nx; x0 += warps * kFillSeg * 32) {
        const int xw = x0 + warp * kFillSeg * 32 + lane;
        uint32_t w[kFillSeg];
#pragma unroll
        for (int j = 0; j < kFillSeg; ++j) {
            const int x = xw + 32 * j;
            w[j] = x >= 1 && x < nx ? c.wDom[row + x] : 0u;
        }
        uint32_t lastMark = 0;
#pragma unroll
        for (int j = 0; j < kFillSeg; ++j) {
            const unsigned bal = __ballot_sync(0xffffffffu, w[j] != 0);
            const uint32_t v = __shfl_sync(0xffffffffu, w[j], bal ? 31 - __clz(bal) : 0);
            if (bal) lastMark = v;
        }
        if (lane == 0) lastOf[warp] = lastMark;
        __syncthreads();
        uint32_t cur = carry;
#pragma unroll
        for (int q = 0; q < warps; ++q) {
            const uint32_t v = lastOf[q];
            if (v) {
                if (q < warp) cur = v;
                carry = v;
                any = true;
            }
        }
#pragma unroll
        for (int j = 0; j < kFillSeg; ++j) {
            const int x = xw + 32 * j;
            const unsigned bal = __ballot_sync(0xffffffffu, w[j] != 0);
            const unsigned own = bal & (0xffffffffu >> (31 - lane));
            const uint32_t v = __shfl_sync(0xffffffffu, w[j], own ? 31 - __clz(own) : lane);
            const uint32_t e = __shfl_sync(0xffffffffu, w[j], bal ? 31 - __clz(bal) : 0);
            const uint32_t mark = own ? v : cur;
            if (x >= 1 && x < nx) {
                dom[row + x] = mark ? mark - 1u : 0u;
                if (w[j]) c.wDom[row + x] = 0;
            }
            if (bal) cur = e;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        c.rowHad[y] = any;
        c.rowNow[y] = 0;
    }
}

void launch_domain_fill(CrossDev& c, uint32_t* dom, int nx, int ny, Status* st, cudaStream_t s, bool gated) {
    launch_pdl(domain_fill_kernel, ny, kFillBlock, 0, s, c, dom, nx, gated ? 1 : 0, st);
}


// ---------------------------------------------------------------------------
// Force list

// st: a step's stage, which a halted step skips (else nullptr).
__global__ void clear_forces_kernel(MembraneDev m, const Status* st) {
    pdl_wait();
    if (st != nullptr && st->halt) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i <= m.topo->M) m.foff[i] = 0;
}

void launch_clear_forces(MembraneDev& m, cudaStream_t s, const Status* st) {
    launch_pdl(clear_forces_kernel, (m.Mcap + 1 + 255) / 256, 256, 0, s, m, st);
}

// Tension renewal when the force list holds only tension pairs: node i gets
// one type-6 record toward each ring neighbour, ordered by the position of the
// contributing connection in the connection vector
// (tutorial_01_BioSolverMembraneTension.cpp:52-73 adds them in that order).
__global__ void tension_pos_kernel(MembraneDev m, int* outPos, int* inPos, const Status* st) {
    pdl_wait();
    if (st->halt) return;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= m.topo->C) return;
    outPos[m.ca[c]] = c;
    inPos[m.cb[c]] = c;
}

__global__ void tension_fill_kernel(MembraneDev m, const int* outPos, const int* inPos, double force,
                                    const Status* st) {
    pdl_wait();
    if (st->halt) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > m.topo->M) return;
    m.foff[i] = 2 * i;
    if (i == m.topo->M) return;
    const int nextNode = m.cb[outPos[i]], prevNode = m.ca[inPos[i]];
    const int first = outPos[i] < inPos[i] ? 0 : 1;
    m.ftype[2 * i + first] = 6;
    m.fpartner[2 * i + first] = nextNode;
    m.ftype[2 * i + 1 - first] = 6;
    m.fpartner[2 * i + 1 - first] = prevNode;
    for (int q = 0; q < 4; ++q) {
        m.fpar[4 * (2 * i) + q] = q == 0 ? force : 0.0;
        m.fpar[4 * (2 * i + 1) + q] = q == 0 ? force : 0.0;
    }
}

void launch_tension_renewal(MembraneDev& m, int* outPos, int* inPos, double force, const Status* st, cudaStream_t s) {
    if (m.Mcap == 0) return;
    launch_pdl(tension_pos_kernel, (m.Ccap + 127) / 128, 128, 0, s, m, outPos, inPos, st);
    launch_pdl(tension_fill_kernel, (m.Mcap + 1 + 127) / 128, 128, 0, s, m, outPos, inPos, force, st);
}

// ---------------------------------------------------------------------------
// Areas (GeometryHandler::computeAreas, shoelace in ring order) and the
// LbibAreaRegulator mass source per domain.
// One block per cell: the terms x_i y_j - x_j y_i are formed in parallel;
// one thread adds them in ring order (the summation order of the shoelace
// sum is part of the result).
constexpr int kAreaMax = 4096;

// beside: launched beside the main sequence (raise_error_beside), whose step counts
// if it got to its domain stages.
__global__ void __launch_bounds__(256) areas_kernel(MembraneDev m, double* area, Status* st, int beside) {
    pdl_wait();
    const int cell = blockIdx.x;
    const int b = m.ringStart[cell], e = m.ringStart[cell + 1];
    const int np = e - b;
    __shared__ double terms[kAreaMax];
    if (np > kAreaMax) {
        if (threadIdx.x == 0 && st) {
            if (!beside) raise_error(st, ERR_CAPACITY, cell, ST_BIO);
            else if (st->domainGo && !st->domainStop) raise_error_beside(st, ERR_CAPACITY, cell, ST_BIO);
        }
        return;
    }
    for (int k = threadIdx.x; k < np; k += blockDim.x) {
        const int i = m.ringNode[b + k];
        const int j = m.ringNode[b + (k + 1 == np ? 0 : k + 1)];
        terms[k] = m.x[i] * m.y[j] - m.x[j] * m.y[i];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int k = 0; k < np; ++k) sum += terms[k];
        area[cell] = sum / 2.0;
    }
}

// ctypeTab == nullptr: LbibAreaRegulator, target = factor x the first area,
// rate strength (target - A) / target.  Otherwise
// tutorial_01_BioSolverAreaRegulator (tutorial_01_BioSolverAreaRegulator.cpp:
// 44-97): target = factor (TARGETAREA), rate strength (target - A) (KP), and
// cells of type 1 get maxsource whatever their area.
// acc != nullptr (FP32-shifted runs): the cell's area is first formed from
// its fixed-point sum, which is reset for the next step (on a halted step too).
__global__ void area_regulator_kernel(MembraneDev m, double* area, double* target, double* massTab,
                                      int nDomains, double factor, double strength, double maxsource,
                                      const uint32_t* ctypeTab, unsigned long long* acc, const Status* st) {
    pdl_wait();
    const int cell = blockIdx.x * blockDim.x + threadIdx.x;
    if (cell >= m.nCells) return;
    int halt = st->halt;
    unsigned long long sum = acc != nullptr ? acc[cell] : 0ull;
    double A = acc != nullptr ? 0.0 : area[cell], tgt = target[cell];
    uint32_t d = m.ringDom[cell];
    read_ahead(halt, d, A, tgt, sum);
    if (acc != nullptr) {
        A = (double)(long long)sum * (1.0 / kAreaFix) / 2.0;
        area[cell] = A;
        acc[cell] = 0ull;
    }
    if (halt) return;
    double r;
    if (ctypeTab == nullptr) {
        if (isnan(tgt)) target[cell] = tgt = factor * A;
        r = strength * (tgt - A) / tgt;
    } else {
        if (isnan(tgt)) target[cell] = tgt = factor;
        r = strength * (tgt - A);
    }
    if (r > maxsource) r = maxsource;
    else if (r < -maxsource) r = -maxsource;
    if (d < (uint32_t)nDomains && d != 0) {
        if (ctypeTab != nullptr && ctypeTab[d] == 1) r = maxsource;
        massTab[d] = r;
    }
}

// tutorial_02_BioSolverGrowth::applyBioProcess (tutorial_02_BioSolverGrowth.cpp:
// 44-80): every node inside a cell gets the mass source MAXSOURCE = 0.001 where
// R^2 L > 1 (THRESHOLD) and MAXSOURCE / 10 elsewhere; R and L are the species'
// getC() after the step (post-collide slot order T, W, S, E, N).  The source is
// per node: FluidSolver::addMass sets the next collide's rhoToAdd.  iR < 0:
// BioSolverGrowth (BioSolverGrowth.cpp:41-62), 0.0025 at every node inside a cell.
template <typename Real>
__global__ void growth_kernel(const Real* g, const uint32_t* dom, size_t L, int iR, int iL, double* massNode,
                              const Status* st) {
    pdl_wait();
    if (st->halt) return;
    const size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= L) return;
    const uint32_t d = dom[n];
    double src = 0.0;
    if (d != 0) {
        auto cOf = [&](int k) {
            const Real* gk = g + (size_t)k * 5 * L;
            double C = 0.0;
            C += (double)gk[0 * L + n];
            C += (double)gk[3 * L + n];
            C += (double)gk[4 * L + n];
            C += (double)gk[1 * L + n];
            C += (double)gk[2 * L + n];
            return C;
        };
        if (iR < 0) {
            src = 0.0025;  // BioSolverGrowth: the same source everywhere inside cells
        } else {
            const double R = cOf(iR), Lc = cOf(iL);
            const double maxsource = 0.001;
            src = R * R * Lc > 1.0 ? maxsource : maxsource / 10.0;
        }
    }
    massNode[n] = src;
}

// The per-domain rates of an area regulator as per-node sources, for runs
// whose host bio solvers change domains after the bio step (a division's
// cureLattice): FluidSolver::addMass gave each node its rate by the domain it
// had at bio time, which the next collide applies whatever the node's domain
// is by then.
__global__ void mass_expand_kernel(const uint32_t* dom, size_t L, const double* massTab, int nDomains,
                                   double* massNode, const Status* st) {
    pdl_wait();
    if (st->halt) return;
    const size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= L) return;
    const uint32_t d = dom[n];
    massNode[n] = (d != 0 && d < (uint32_t)nDomains) ? massTab[d] : 0.0;
}

void launch_mass_expand(const uint32_t* dom, size_t L, const double* massTab, int nDomains, double* massNode,
                        const Status* st, cudaStream_t s) {
    launch_pdl(mass_expand_kernel, (unsigned)((L + 255) / 256), 256, 0, s, dom, L, massTab, nDomains, massNode, st);
}

template <typename Real>
void launch_growth(const Real* g, const uint32_t* dom, size_t L, int iR, int iL, double* massNode, const Status* st,
                   cudaStream_t s) {
    launch_pdl(growth_kernel<Real>, (unsigned)((L + 255) / 256), 256, 0, s, g, dom, L, iR, iL, massNode, st);
}
template void launch_growth<double>(const double*, const uint32_t*, size_t, int, int, double*, const Status*,
                                    cudaStream_t);
template void launch_growth<float>(const float*, const uint32_t*, size_t, int, int, double*, const Status*,
                                   cudaStream_t);

// FP32-shifted runs: the per-cell shoelace sums over the connections in any
// order, each term x_a y_b - x_b y_a (a -> b along the ring) rounded to 64-bit
// fixed point (2^-24), so that the integer sums are exact and independent of
// the order; no ring ranking is needed.  FP64 runs keep the ring-ordered sum.
__global__ void areas_fixed_kernel(MembraneDev m, const int* cellOfDom, int nDomains, unsigned long long* acc) {
    pdl_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = c < m.topo->C;
    area_term_fixed(m, in, in ? m.ca[c] : 0, in ? m.cb[c] : 0, in ? m.cdom[c] : 0u, cellOfDom, nDomains, acc);
}

void launch_areas(const MembraneDev& m, double* area, Status* st, cudaStream_t s) {
    if (m.nCells == 0) return;
    launch_pdl(areas_kernel, m.nCells, 256, 0, s, m, area, st, 0);
}

// The fixed-point sums as areas (the conversion of area_regulator_kernel),
// the sums cleared for their next use.
__global__ void areas_fixed_finish_kernel(int nCells, unsigned long long* acc, double* area) {
    pdl_wait();
    const int cell = blockIdx.x * blockDim.x + threadIdx.x;
    if (cell >= nCells) return;
    area[cell] = (double)(long long)acc[cell] * (1.0 / kAreaFix) / 2.0;
    acc[cell] = 0ull;
}

void launch_areas_fixed(const MembraneDev& m, const int* cellOfDom, int nDomains, unsigned long long* acc,
                        double* area, cudaStream_t s) {
    if (m.nCells == 0) return;
    if (m.Ccap > 0) launch_pdl(areas_fixed_kernel, (m.Ccap + 255) / 256, 256, 0, s, m, cellOfDom, nDomains, acc);
    launch_pdl(areas_fixed_finish_kernel, (m.nCells + 127) / 128, 128, 0, s, m.nCells, acc, area);
}

// The fixed device array of lbib_areas_static: the per-cell sums of one call.
// Every call on a device writes and reads this same array.
static __device__ __align__(256) double g_areaScratch[kStaticAreaCells];

cudaError_t static_area_scratch(double** ptr) {
    return cudaGetSymbolAddress((void**)ptr, g_areaScratch);
}

void launch_area_regulator(const MembraneDev& m, double* area, double* target, double* massTab, int nDomains,
                           double factor, double strength, double maxsource, const uint32_t* ctypeTab,
                           Status* st, cudaStream_t s, bool beside) {
    if (m.nCells == 0) return;
    launch_pdl(areas_kernel, m.nCells, 256, 0, s, m, area, st, beside ? 1 : 0);
    launch_pdl(area_regulator_kernel, (m.nCells + 127) / 128, 128, 0, s, m, area, target, massTab, nDomains, factor,
               strength, maxsource, ctypeTab, (unsigned long long*)nullptr, (const Status*)st);
}

void launch_area_regulator_fixed(const MembraneDev& m, const int* cellOfDom, unsigned long long* acc, double* area,
                                 double* target, double* massTab, int nDomains, double factor, double strength,
                                 double maxsource, const uint32_t* ctypeTab, const Status* st, cudaStream_t s,
                                 bool summed, bool programmatic) {
    if (m.nCells == 0 || m.Ccap == 0) return;
    if (!summed)
        launch_ex(programmatic, areas_fixed_kernel, (m.Ccap + 255) / 256, 256, 0, s, m, cellOfDom, nDomains, acc);
    launch_ex(programmatic || !summed, area_regulator_kernel, (m.nCells + 127) / 128, 128, 0, s, m, area, target, massTab,
              nDomains, factor, strength, maxsource, ctypeTab, acc, st);
}

// ---------------------------------------------------------------------------
// Differentiated runs with moving membrane nodes.  The forward of one step is
// the spread of the node forces from the step-start positions X, the lattice
// step, then X' = X + (the post-collision velocity interpolated at X): the
// reference's distributeForce, collide and collectVelocity + move
// (GeometryNode.cpp:216-254) without the perturbation, whose random jumps
// have no derivative.  The stencil follows from X (stencil_range of the
// position itself: the 4x4 lattice nodes within 2 lu, the set the reference's
// binding holds while the node stays in its unit cell).

// d fast_cos / dx: the derivative of the approximation itself (its two
// parabolas and the 0.225 correction), so that the gradients are those of
// the forward as it is computed.
__device__ __forceinline__ double fast_cos_deriv(const double x) {
    const double halfPi = M_PI / 2.0;
    const double doublePi = 2.0 * M_PI;
    double tempx = x + halfPi;
    if (tempx > M_PI) tempx -= doublePi;
    double c, dc;
    if (tempx < .00) {
        c = 1.27323954 * tempx + 0.405284735 * tempx * tempx;
        dc = 1.27323954 + 2.0 * 0.405284735 * tempx;
    } else {
        c = 1.27323954 * tempx - 0.405284735 * tempx * tempx;
        dc = 1.27323954 - 2.0 * 0.405284735 * tempx;
    }
    // cs = 0.225 (c |c| - c) + c
    return c < 0.0 ? dc * (1.0 + 0.225 * (-2.0 * c - 1.0)) : dc * (1.0 + 0.225 * (2.0 * c - 1.0));
}

// Sixteen lanes per membrane node, one per stencil slot (two nodes per warp):
// a node's 16 scattered lattice reads are issued at once instead of one
// after another, and the sums over the slots are shuffles within the lanes'
// group of 16 (every lane of the warp takes part, in range or not).
constexpr int kMotionBlock = 128;

__device__ __forceinline__ double group16_sum(double v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// A step of such a run is two launches: the lattice step (or its reverse), and
// the nodes' kernel after it, which moves the nodes (or carries dL/dX back
// through the step), clears the fields that the lattice kernel just read, at
// the stencils they were spread from, and spreads the next step's, into the
// other of two buffers.  With a memset and a kernel for each of these (and
// one that rounded the field for FP32-shifted runs) a step of a 256^2 lattice
// with 5,000 nodes took 16.6 us forward and 40 us back (a checkpoint every 5
// steps); now 6.6 and 18.9.

struct NodeSlot {
    size_t n;   // lattice node
    double dl;  // its Dirac weight
    bool ok;
};

// Slot k of the stencil of a node at (x, y).
__device__ __forceinline__ NodeSlot motion_slot(double x, double y, int k, int nx, int ny) {
    NodeSlot s{0, 0.0, false};
    Stencil sc;
    s.ok = stencil_range(x, y, nx, ny, sc);
    if (s.ok) {
        int xk, yk;
        stencil_slot(sc, k, xk, yk);
        s.n = (size_t)yk * nx + xk;
        s.dl = dirac((double)xk - x, (double)yk - y);
    }
    return s;
}

__device__ __forceinline__ void motion_add(const NodeSlot& s, double ax, double ay, size_t L, double* out) {
    atomicAdd(out + s.n, s.dl * ax);
    atomicAdd(out + L + s.n, s.dl * ay);
}

// The fields of a pass's first step: (ax, ay) into out and, when given, (bx, by)
// into out2 (both cleared before).
__global__ void __launch_bounds__(kMotionBlock) motion_spread_kernel(const double* X, const double* Y, const double* ax,
                                                                     const double* ay, const double* bx,
                                                                     const double* by, int M, int nx, int ny, size_t L,
                                                                     double* out, double* out2, Status* st) {
    pdl_wait();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(t >> 4), k = (int)(t & 15);
    if (i >= M) return;
    const NodeSlot s = motion_slot(X[i], Y[i], k, nx, ny);
    if (!s.ok) {
        if (k == 0) raise_error(st, ERR_STENCIL, i, ST_SPREAD);
        return;
    }
    motion_add(s, ax[i], ay[i], L, out);
    if (out2 != nullptr) motion_add(s, bx[i], by[i], L, out2);
}

static unsigned motion_blocks(int M) { return (unsigned)(((long long)M * 16 + kMotionBlock - 1) / kMotionBlock); }

void launch_motion_spread(const double* X, const double* Y, const double* ax, const double* ay, const double* bx,
                          const double* by, int M, int nx, int ny, size_t L, double* out, double* out2, Status* st,
                          cudaStream_t s) {
    if (M <= 0) return;
    launch_pdl(motion_spread_kernel, motion_blocks(M), kMotionBlock, 0, s, X, Y, ax, ay, bx, by, M, nx, ny, L, out, out2,
               st);
}

// After the lattice step from the positions (X0, Y0): the move to (X1, Y1)
// (u != nullptr; else they are known, a recomputed step), and, unless it was the
// last, the field of the forces (fx, fy) at the new positions into `out`, with
// the field just used, `used`, cleared.
template <typename Real>
__global__ void __launch_bounds__(kMotionBlock) motion_next_kernel(const double* X0, const double* Y0, double* X1,
                                                                   double* Y1, int M, const Real* u, const double* fx,
                                                                   const double* fy, double* used, double* out, int nx,
                                                                   int ny, size_t L, Status* st) {
    pdl_wait();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(t >> 4), k = (int)(t & 15);
    double xi = 0.0, yi = 0.0, x1 = 0.0, y1 = 0.0;
    NodeSlot s{0, 0.0, false};
    if (i < M) {
        xi = X0[i];
        yi = Y0[i];
        s = motion_slot(xi, yi, k, nx, ny);
        if (u == nullptr) {
            x1 = X1[i];
            y1 = Y1[i];
        }
    }
    if (u != nullptr) {
        const double vx = group16_sum(s.ok ? (double)u[s.n] * s.dl : 0.0);
        const double vy = group16_sum(s.ok ? (double)u[L + s.n] * s.dl : 0.0);
        x1 = s.ok ? xi + vx : xi;
        y1 = s.ok ? yi + vy : yi;
        if (i < M && k == 0) {
            const double CS = 1 / sqrt(3.0);
            if (!s.ok) raise_error(st, ERR_STENCIL, i, ST_INTERP_MOVE);
            else if (!(((vx * vx) + (vy * vy)) <= CS)) raise_error(st, ERR_SPEED, i, ST_INTERP_MOVE);  // NaN too
            X1[i] = x1;
            Y1[i] = y1;
        }
    }
    if (i >= M || out == nullptr) return;
    if (s.ok) used[s.n] = used[L + s.n] = 0.0;
    const NodeSlot s1 = motion_slot(x1, y1, k, nx, ny);
    if (s1.ok) motion_add(s1, fx[i], fy[i], L, out);
    else if (k == 0) raise_error(st, ERR_STENCIL, i, ST_SPREAD);
}

template <typename Real>
void launch_motion_next(const double* X0, const double* Y0, double* X1, double* Y1, int M, const Real* u,
                        const double* fx, const double* fy, double* used, double* out, int nx, int ny, size_t L,
                        Status* st, cudaStream_t s) {
    if (M <= 0) return;
    launch_pdl(motion_next_kernel<Real>, motion_blocks(M), kMotionBlock, 0, s, X0, Y0, X1, Y1, M, u, fx, fy, used, out, nx,
               ny, L, st);
}
template void launch_motion_next<double>(const double*, const double*, double*, double*, int, const double*,
                                         const double*, const double*, double*, double*, int, int, size_t, Status*,
                                         cudaStream_t);
template void launch_motion_next<float>(const double*, const double*, double*, double*, int, const float*,
                                        const double*, const double*, double*, double*, int, int, size_t, Status*,
                                        cudaStream_t);

// With w(a) = 1 + fast_cos(pi/2 (a - X)) the weight of lattice node (a, b)
// is w(a) w(b) / 16, and d/dX of it is -pi/2 fast_cos'(pi/2 (a - X)) w(b) / 16
// (likewise in Y).  A node whose stencil leaves the lattice was refused by
// the forward (ERR_STENCIL) and contributes nothing here.
// next.out != nullptr: the step before starts from (next.X, next.Y); its fields
// (lambda as it is then, and the forces) are spread from there, and those just
// used are cleared.
__global__ void __launch_bounds__(kMotionBlock) motion_adjoint_kernel(const double* X, const double* Y,
                                                                      const double* fx, const double* fy, double* lx,
                                                                      double* ly, const double* uo, const double* G,
                                                                      double* gfx, double* gfy, MotionNext next, int M,
                                                                      int nx, int ny, size_t L, Status* st) {
    pdl_wait();
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(t >> 4), k = (int)(t & 15);
    double gX = 0.0, gY = 0.0, gx = 0.0, gy = 0.0, lamx = 0.0, lamy = 0.0, Fx = 0.0, Fy = 0.0;
    bool ok = false;
    size_t n = 0;
    if (i < M) {
        const double xi = X[i], yi = Y[i];
        lamx = lx[i];
        lamy = ly[i];
        Fx = fx[i];
        Fy = fy[i];
        Stencil sc;
        ok = stencil_range(xi, yi, nx, ny, sc);
        if (ok) {
            const double halfPi = M_PI / 2.0;
            int xk, yk;
            stencil_slot(sc, k, xk, yk);
            n = (size_t)yk * nx + xk;
            const double ax = halfPi * ((double)xk - xi), ay = halfPi * ((double)yk - yi);
            const double wa = 1.0 + fast_cos(ax), wb = 1.0 + fast_cos(ay);
            const double dl = (wa * wb) / 16.0;
            const double dX = -halfPi * fast_cos_deriv(ax) * wb / 16.0;
            const double dY = -halfPi * wa * fast_cos_deriv(ay) / 16.0;
            const double Gx = G[n], Gy = G[L + n];
            const double c = lamx * uo[n] + lamy * uo[L + n] + Fx * Gx + Fy * Gy;
            gX = dX * c;
            gY = dY * c;
            gx = dl * Gx;
            gy = dl * Gy;
        }
    }
    gX = group16_sum(gX);
    gY = group16_sum(gY);
    gx = group16_sum(gx);
    gy = group16_sum(gy);
    if (i >= M) return;
    if (ok) {
        lamx += gX;
        lamy += gY;
        if (k == 0) {
            lx[i] = lamx;
            ly[i] = lamy;
            gfx[i] += gx;
            gfy[i] += gy;
        }
    }
    if (next.out == nullptr) return;
    if (ok) next.used[n] = next.used[L + n] = next.used2[n] = next.used2[L + n] = 0.0;
    const NodeSlot s = motion_slot(next.X[i], next.Y[i], k, nx, ny);
    if (s.ok) {
        motion_add(s, lamx, lamy, L, next.out);
        motion_add(s, Fx, Fy, L, next.out2);
    } else if (k == 0) {
        raise_error(st, ERR_STENCIL, i, ST_SPREAD);
    }
}

void launch_motion_adjoint(const double* X, const double* Y, const double* fx, const double* fy, double* lx,
                           double* ly, const double* uo, const double* G, double* gfx, double* gfy,
                           const MotionNext& next, int M, int nx, int ny, size_t L, Status* st, cudaStream_t s) {
    if (M <= 0) return;
    launch_pdl(motion_adjoint_kernel, motion_blocks(M), kMotionBlock, 0, s, X, Y, fx, fy, lx, ly, uo, G, gfx, gfy, next, M,
               nx, ny, L, st);
}

}  // namespace lbib

namespace lbib {

void init_kernel_attributes() {
    init_kernel_attributes_topology();
}

}  // namespace lbib
