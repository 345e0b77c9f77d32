// k_topology.cu — membrane topology edits on the device.
//
//   remesh    GeometryHandler::remeshBoundary (GeometryHandler.cpp:385-431) as
//             count (with the crossings' ties, remesh.cuh), apply and commit:
//             every connection longer than MAXLENGTH gets a new node at its
//             midpoint; the new node ids continue from the largest id in
//             connection order (Geometry::addGeometryNode,
//             Geometry.cpp:382-400); the split connection leaves the vector and
//             its two halves are appended (Geometry::eraseConnection /
//             addConnection, Geometry.cpp:433-452).  One pass runs on the
//             device (SimulationRunner.cpp:190-199 repeats until nothing is
//             split); a second that would still split, or a full buffer, hands
//             the step to the host; a new node that needs the random
//             perturbation waits for it before the commit.
//   coarsen   GeometryHandler::coarsenBoundary (GeometryHandler.cpp:433-461):
//             nodes are visited in id order and removed when their neighbours
//             are closer than MAXLENGTH; a removal erases the node's two
//             connections and appends one from its predecessor to its successor
//             (Geometry::removeGeometryNode, Geometry.cpp:402-431).  Removals
//             only interact along a ring, so one thread per cell runs the
//             id-ordered visit over that cell's candidates (a node is a
//             candidate if it is one at the start or a smaller-id neighbour
//             was removed); the new connections are appended in removal order.
//   rings     the node order of GeometryHandler::computeAreas (first connection
//             of each domain in vector order, then the second node's outgoing
//             connection) by pointer jumping, one block per cell.
#include <algorithm>

#include <cub/cub.cuh>

#include "kernels.cuh"
#include "remesh.cuh"

namespace lbib {

// Position of the n-th (from 0) set bit of w; w has more than n set bits.
__device__ __forceinline__ int nth_set_bit(unsigned w, int n) {
    int base = 0;
#pragma unroll
    for (int sh = 16; sh > 0; sh >>= 1) {
        const unsigned low = (1u << sh) - 1u;
        const int c = __popc(w & low);
        if (n >= c) {
            n -= c;
            w >>= sh;
            base += sh;
        } else {
            w &= low;
        }
    }
    return base;
}

// |d| < MAXLENGTH for a squared length d2 (longer_than_max's other side).
__device__ __forceinline__ bool shorter_than_max(double d2) {
    constexpr double m2 = kMAXLENGTH * kMAXLENGTH;
    if (d2 < m2 * (1.0 - 1e-12)) return true;
    if (d2 >= m2) return false;
    return sqrt(d2) < kMAXLENGTH;
}
// Warp-aggregated atomics: lanes with the same key share one atomic.
__device__ __forceinline__ int agg_add(int* addr, int key) {
    const unsigned act = __activemask();
    const unsigned grp = __match_any_sync(act, key);
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(grp) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(addr, __popc(grp));
    base = __shfl_sync(grp, base, leader);
    return base + __popc(grp & ((1u << lane) - 1u));
}

// Minimum of v per key, where v increases with the lane (a warp's
// connection indices): the group's lowest lane holds the group's minimum.
__device__ __forceinline__ void agg_min(int* addr, int key, int v) {
    const unsigned act = __activemask();
    const unsigned grp = __match_any_sync(act, key);
    if ((int)(threadIdx.x & 31) == __ffs(grp) - 1) atomicMin(addr, v);
}

// ---------------------------------------------------------------------------
// Remesh

// The pass was counted with the crossings' ties (remesh_count_block): K
// connections to split.  It runs unless it would overflow a buffer (the host
// runs it then; so it does a second pass, remesh_commit_kernel).  New nodes that
// need the random perturbation are made on the device all the same and listed
// for the host, which perturbs them before the pass is committed.
__device__ __forceinline__ bool remesh_fits(const MembraneDev& m, int K, int M, int C) {
    return M + K <= m.Mcap && C + K <= m.Ccap;
}

// Applies the pass: connection c's rank among the split ones is the sum of the
// block counts before its block plus the split connections before it in the
// block (the same test on the same positions as the count).
__global__ void __launch_bounds__(kRemeshBlock) remesh_apply_kernel(MembraneDev m, TopoDev t, Status* st) {
    pdl_wait();
    Topo* T = m.topo;
    int halt = st->halt, K = T->K;
    read_ahead(halt, K);
    if (halt || K == 0) return;
    const int C = T->C, M = T->M;
    if (!remesh_fits(m, K, M, C)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) raise_halt(st, ST_REMESH);
        return;
    }
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    bool rng = false;
    const bool f = c < C && remesh_split(m, c, rng);
    const unsigned bal = __ballot_sync(0xffffffffu, f);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __shared__ int wsum[kRemeshBlock / 32], wbefore[kRemeshBlock / 32];
    int before = 0;
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += kRemeshBlock) before += t.flag[b];
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) {
        wsum[w] = __popc(bal);
        wbefore[w] = before;
    }
    __syncthreads();
    if (c >= C) return;
    int r = __popc(bal & ((1u << lane) - 1u));
    for (int i = 0; i < w; ++i) r += wsum[i];
#pragma unroll
    for (int i = 0; i < kRemeshBlock / 32; ++i) r += wbefore[i];
    if (!f) {
        const int dst = c - r;
        t.ca2[dst] = m.ca[c]; t.cb2[dst] = m.cb[c]; t.cdom2[dst] = m.cdom[c]; t.cdesc2[dst] = m.cdesc[c];
        return;
    }
    const int a = m.ca[c], b = m.cb[c];
    const int j = M + r;
    const double x = (m.x[a] + m.x[b]) / 2, y = (m.y[a] + m.y[b]) / 2;
    m.x[j] = x; m.y[j] = y;
    m.ox[j] = x - 5.0; m.oy[j] = y - 5.0;   // GeometryNode.cpp:98-103
    m.bx[j] = x; m.by[j] = y;               // bound at once (remesh_commit_kernel tests the edges)
    m.vx[j] = 0.0; m.vy[j] = 0.0; m.fx[j] = 0.0; m.fy[j] = 0.0;
    m.id[j] = T->maxId + 1 + (unsigned)r;
    m.next[a] = j; m.prev[j] = a; m.next[j] = b; m.prev[b] = j;
    m.foff[j + 1] = m.foff[M];              // new nodes carry no forces
    // GeometryNode's constructor perturbs a node made on a lattice line or
    // diagonal (GeometryNode.cpp:98-117): the host draws it, in id order
    if (rng) t.rngList[atomicAdd(&T->rngFill, 1)] = j;
    const int base = C - K + 2 * r;
    t.ca2[base] = a; t.cb2[base] = j; t.cdom2[base] = m.cdom[c]; t.cdesc2[base] = m.cdesc[c];
    t.ca2[base + 1] = j; t.cb2[base + 1] = b; t.cdom2[base + 1] = m.cdom[c]; t.cdesc2[base + 1] = m.cdesc[c];
}

// Commits the pass: copies the new connection list back (the last block to
// finish updates the counts; every block has read K, C and M before any block
// counts itself done), and checks what comes next in the reference:
//  - a connection of the new list still longer than MAXLENGTH (a split half
//    of one longer than 2 * MAXLENGTH) needs another pass
//    (SimulationRunner.cpp:190-199 repeats the remeshing); that rare case goes
//    to the host;
//  - the new nodes are bound to the lattice at once (GeometryHandler.cpp:
//    427-428): their old position is 5 lu away, so they are never in their
//    old unit cell, take their binding from the current position (perturbed
//    by the host where needed) and the edge test of connectGeometryNodesToPhysicalNodes
//    (GeometryHandler.cpp:618-644).  The nodes that existed before the pass
//    were bound, and tested, by the crossing stage from the same positions.
// areaAcc != nullptr (FP32-shifted steps without coarsening): the kernel also
// adds the shoelace terms of the final connection list to the cells'
// fixed-point sums (a kernel of its own otherwise: 3.9 us at 150k connections).
__global__ void __launch_bounds__(256) remesh_commit_kernel(MembraneDev m, TopoDev t, int nx, int ny, Status* st,
                                                            unsigned long long* areaAcc) {
    pdl_wait();
    Topo* T = m.topo;
    const int cn = blockIdx.x * blockDim.x + threadIdx.x, cc = min(cn, m.Ccap - 1);
    int K = T->K, halt = st->halt, haltStage = st->haltStage, C0 = T->C, a0 = 0, b0 = 0;
    uint32_t d0 = 0;
    if (areaAcc != nullptr) {
        a0 = m.ca[cc];
        b0 = m.cb[cc];
        d0 = m.cdom[cc];
    }
    read_ahead(K, halt, haltStage, C0, a0, b0, d0);
    const int stage = halt ? haltStage : 0;
    if (K == 0) {
        if (areaAcc != nullptr && stage == 0)
            area_term_fixed(m, cn < C0, a0, b0, d0, t.cellOfDom, t.nDomains, areaAcc);
        return;
    }
    if ((stage != 0 && stage < ST_REMESH) || !remesh_fits(m, K, T->M, T->C)) {
        // halted before the pass was applied, or handed to the host: not run
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            T->K = 0;
            T->nRng = 0;
        }
        return;
    }
    if (T->nRng > 0) {
        // new nodes wait for the host's perturbation; the step resumes here
        if (blockIdx.x == 0 && threadIdx.x == 0) raise_halt(st, ST_REMESH_RNG);
        return;
    }
    const int C = T->C, M = T->M;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < C + K) {
        const int a = t.ca2[c], b = t.cb2[c];
        m.ca[c] = a; m.cb[c] = b; m.cdom[c] = t.cdom2[c]; m.cdesc[c] = t.cdesc2[c];
        const double x1 = m.x[a], y1 = m.y[a], x2 = m.x[b], y2 = m.y[b];
        if (longer_than_max((x1 - x2) * (x1 - x2) + (y1 - y2) * (y1 - y2))) raise_halt(st, ST_REMESH);
    }
    if (c < K) {
        const int i = M + c;
        const double X = m.x[i], Y = m.y[i];
        m.bx[i] = X;  // bound at its (perturbed) position
        m.by[i] = Y;
        if (X - 2.0 < 0) raise_error(st, ERR_EDGE_W, i, ST_REMESH);
        else if (Y - 2.0 < 0) raise_error(st, ERR_EDGE_S, i, ST_REMESH);
        else if (X + 2.0 > nx) raise_error(st, ERR_EDGE_E, i, ST_REMESH);
        else if (Y + 2.0 > ny) raise_error(st, ERR_EDGE_N, i, ST_REMESH);
    }
    if (areaAcc != nullptr) {
        const bool in = c < C + K;
        area_term_fixed(m, in, in ? t.ca2[c] : 0, in ? t.cb2[c] : 0, in ? t.cdom2[c] : 0u, t.cellOfDom, t.nDomains, areaAcc);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&T->done, 1u) == gridDim.x - 1) {
            T->M += K;
            T->C += K;
            T->maxId += K;
            T->changed = 1;
            T->K = 0;
            T->done = 0;
        }
    }
}

int launch_remesh(MembraneDev& m, TopoDev& t, int nx, int ny, Status* st, cudaStream_t s, bool commitOnly,
                  unsigned long long* areaAcc) {
    if (m.Ccap == 0) return 0;
    int n = 0;
    if (!commitOnly) {
        // the count and the apply kernel partition the connections alike
        launch_pdl(remesh_apply_kernel, (m.Ccap + kRemeshBlock - 1) / kRemeshBlock, kRemeshBlock, 0, s, m, t, st);
        n = 1;
    }
    // a pass runs only when C + K <= Ccap: this grid covers the new list
    launch_pdl(remesh_commit_kernel, (m.Ccap + 255) / 256, 256, 0, s, m, t, nx, ny, st, areaAcc);
    return n + 1;
}

// ---------------------------------------------------------------------------
// Coarsen

// Clears the force list; node -> its incoming / outgoing connection; candidates.
// (A halted step leaves the list alone: the steps between the one that halted and
// this one, queued behind it, have yet to use it.)
__global__ void coarsen_begin_kernel(MembraneDev m, TopoDev t, Status* st) {
    pdl_wait();
    if (st->halt) return;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int M = m.topo->M;
    if (i <= M) m.foff[i] = 0;
    if (i < m.topo->C) {
        t.outConn[m.ca[i]] = i;
        t.inConn[m.cb[i]] = i;
        t.connAlive[i] = 1;
    }
    if (i >= M) return;
    t.removed[i] = 0;
    t.ncAlive[i] = 0;
    const int p = m.prev[i], q = m.next[i];
    const double dx = m.x[q] - m.x[p], dy = m.y[q] - m.y[p];
    const bool cand = shorter_than_max(dx * dx + dy * dy);
    const unsigned bal = __ballot_sync(__activemask(), cand);
    if (cand && (threadIdx.x & 31) == __ffs(bal) - 1) atomicAdd(&m.topo->nCand, __popc(bal));
}

constexpr int kCoarsenMax = 2048;  // nodes of one ring held in shared memory
constexpr size_t kCoarsenSmem = (size_t)kCoarsenMax * (2 * sizeof(double) + sizeof(unsigned long long) +
                                                       7 * sizeof(int) + 2) +
                                 (size_t)kCoarsenMax / 32 * sizeof(unsigned);

// One block per cell.  The ring (in ring order, rebuilt just before) is
// loaded into shared memory as a circular list; thread 0 then visits the
// ring's nodes in id order like GeometryHandler::coarsenBoundary, testing
// only nodes whose span is short at the start or whose neighbour was removed
// (every other node keeps a span >= MAXLENGTH and stays).
// Handles: h < Ccap is connection index h; h >= Ccap is the connection made by
// removing node h - Ccap.
__global__ void __launch_bounds__(256) coarsen_cell_kernel(MembraneDev m, TopoDev t, Status* st) {
    pdl_wait();
    // (the block as one: a ring that is too long raises an error here)
    if (__syncthreads_or(st->halt) || m.topo->nCand == 0) return;
    const int cell = blockIdx.x;
    const int b = m.ringStart[cell], len = m.ringStart[cell + 1] - b;
    if (len > kCoarsenMax) {
        if (threadIdx.x == 0) raise_error(st, ERR_CAPACITY, cell, ST_COARSEN);
        return;
    }
    extern __shared__ __align__(16) unsigned char smem[];
    double* sx = (double*)smem;
    double* sy = sx + kCoarsenMax;
    unsigned long long* ord = (unsigned long long*)(sy + kCoarsenMax);
    int* node = (int*)(ord + kCoarsenMax);
    int* pl = node + kCoarsenMax;
    int* nl = pl + kCoarsenMax;
    int* hin = nl + kCoarsenMax;
    int* hout = hin + kCoarsenMax;
    // boundary descriptor of each position's incoming connection, and the
    // ring's domain (one per cell), so that the serial visit below reads no
    // global memory (it does where a ring mixes domains)
    int* inDesc = hout + kCoarsenMax;
    __shared__ uint32_t ringDomS;
    __shared__ int mixedDom;
    int* rankOf = inDesc + kCoarsenMax;                 // ring position -> place in id order
    unsigned* visit = (unsigned*)(rankOf + kCoarsenMax); // bit j: the node at place j is a candidate
    unsigned char* dirty = (unsigned char*)(visit + kCoarsenMax / 32);
    unsigned char* gone = dirty + kCoarsenMax;
    __shared__ int anyDirty;
    if (threadIdx.x == 0) {
        anyDirty = 0;
        mixedDom = 0;
        ringDomS = len > 0 ? m.cdom[t.inConn[m.ringNode[b]]] : 0u;
    }
    int p2 = 1;
    while (p2 < len) p2 <<= 1;
    __syncthreads();
    for (int k = threadIdx.x; k < p2; k += blockDim.x) {
        if (k < len) {
            const int i = m.ringNode[b + k];
            node[k] = i;
            sx[k] = m.x[i];
            sy[k] = m.y[i];
            pl[k] = k == 0 ? len - 1 : k - 1;
            nl[k] = k == len - 1 ? 0 : k + 1;
            hin[k] = t.inConn[i];
            if (m.cdom[hin[k]] != ringDomS) mixedDom = 1;
            inDesc[k] = m.cdesc[hin[k]];
            hout[k] = t.outConn[i];
            ord[k] = ((unsigned long long)i << 32) | (unsigned)k;
            gone[k] = 0;
        } else {
            ord[k] = ~0ull;
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < len; k += blockDim.x) {
        const int p = pl[k], q = nl[k];
        const double dx = sx[q] - sx[p], dy = sy[q] - sy[p];
        dirty[k] = shorter_than_max(dx * dx + dy * dy);
        if (dirty[k]) anyDirty = 1;
    }
    __syncthreads();
    if (!anyDirty) {
        for (int k = threadIdx.x; k < len; k += blockDim.x) t.removed[node[k]] = 0;
        return;
    }
    // id order of the ring's nodes
    for (int size = 2; size <= p2; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int k = threadIdx.x; k < p2; k += blockDim.x) {
                const int j = k ^ stride;
                if (j > k) {
                    const bool up = (k & size) == 0;
                    const unsigned long long x = ord[k], y = ord[j];
                    if ((x > y) == up) { ord[k] = y; ord[j] = x; }
                }
            }
            __syncthreads();
        }
    }
    // the candidates as bits in id order, so that the visit below jumps from
    // one to the next instead of stepping over every node
    const int nw = (len + 31) >> 5;
    for (int j = threadIdx.x; j < nw * 32; j += blockDim.x) {
        const bool cand = j < len && dirty[(int)(ord[j] & 0xffffffffu)];
        if (j < len) rankOf[(int)(ord[j] & 0xffffffffu)] = j;
        const unsigned bits = __ballot_sync(0xffffffffu, cand);
        if ((threadIdx.x & 31) == 0) visit[j >> 5] = bits;
    }
    __shared__ unsigned wantBits[kCoarsenMax / 32];
    for (int w = threadIdx.x; w < kCoarsenMax / 32; w += blockDim.x) wantBits[w] = 0u;
    __syncthreads();
    if (threadIdx.x < 32) {
        // The visit in id order, 32 candidates per round.  Each lane takes the
        // next candidate place and tests it against the state at the start of
        // the round.  The round keeps the places before T, where T is the
        // first place whose outcome an earlier removal of the round changes:
        // a candidate next to a removed node (its neighbour link changes), or
        // a node that a removal makes a candidate at a later place (the id
        // order visits it there).  The kept removals touch disjoint links, so
        // they are applied together, and the next round starts at T.  The
        // result is the one of the one-by-one visit.
        const int lane = threadIdx.x;
        const int Ccap = m.Ccap;
        int removedHere = 0;
        int j0 = 0;
        while (j0 < len) {
            // the places of the next (up to) 32 candidates at or after j0
            const int w0 = j0 >> 5;
            unsigned word = w0 + lane < nw ? visit[w0 + lane] : 0u;
            if (lane == 0) word &= ~0u << (j0 & 31);
            const int cnt = __popc(word);
            int incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            const int total = __shfl_sync(0xffffffffu, incl, 31);
            if (total == 0) {
                j0 = (w0 + 32) << 5;
                continue;
            }
            // lane l takes candidate l: the word holding it, then its bit
            int src = 0;
#pragma unroll
            for (int st2 = 16; st2 > 0; st2 >>= 1)
                if (__shfl_sync(0xffffffffu, incl, src + st2 - 1) <= lane) src += st2;
            const bool valid = lane < total;
            const int srcS = valid ? src : 31;
            const unsigned srcWord = __shfl_sync(0xffffffffu, word, srcS);
            const int before = __shfl_sync(0xffffffffu, incl - cnt, srcS);
            const int P = valid ? ((w0 + srcS) << 5) + nth_set_bit(srcWord, lane - before) : 0x7fffffff;
            int k = 0, p = 0, q = 0;
            bool want = false;
            if (valid) {
                k = (int)(ord[P] & 0xffffffffu);
                p = pl[k];
                q = nl[k];
                if (dirty[k]) {
                    const double dx = sx[q] - sx[p], dy = sy[q] - sy[p];
                    want = shorter_than_max(dx * dx + dy * dy);
                }
            }
            const int rp = valid ? rankOf[p] : 0, rq = valid ? rankOf[q] : 0;
            if (want) atomicOr(&wantBits[P >> 5], 1u << (P & 31));
            __syncwarp();
            // a removal before this place takes away this node's neighbour
            const bool conflict = valid && ((rp < P && ((wantBits[rp >> 5] >> (rp & 31)) & 1u)) ||
                                            (rq < P && ((wantBits[rq >> 5] >> (rq & 31)) & 1u)));
            int T = 0x7fffffff;
            if (conflict) T = P;
            if (want) {  // the neighbours become candidates at their places
                if (rp > P) T = min(T, rp);
                if (rq > P) T = min(T, rq);
            }
            T = (int)__reduce_min_sync(0xffffffffu, (unsigned)T);
            const int lastP = __shfl_sync(0xffffffffu, P, min(total, 32) - 1);
            if (T > lastP) T = lastP + 1;
            __syncwarp();
            if (want) atomicAnd(&wantBits[P >> 5], ~(1u << (P & 31)));
            if (want && P < T) {
                gone[k] = 1;
                ++removedHere;
                const int i = node[k];
                const int h1 = hin[k], h2 = hout[k];
                uint32_t dom = ringDomS;
                const int desc = inDesc[k];
                if (h1 < Ccap) {
                    t.connAlive[h1] = 0;
                    if (mixedDom) dom = m.cdom[h1];
                } else {
                    t.ncAlive[h1 - Ccap] = 0;
                    if (mixedDom) dom = t.ncDom[h1 - Ccap];
                }
                if (h2 < Ccap) t.connAlive[h2] = 0;
                else t.ncAlive[h2 - Ccap] = 0;
                t.ncA[i] = node[p]; t.ncB[i] = node[q]; t.ncDom[i] = dom; t.ncDesc[i] = desc; t.ncAlive[i] = 1;
                nl[p] = q; pl[q] = p;
                hout[p] = Ccap + i; hin[q] = Ccap + i;
                inDesc[q] = desc;
                dirty[p] = 1; dirty[q] = 1;
                atomicOr(&visit[rp >> 5], 1u << (rp & 31));
                atomicOr(&visit[rq >> 5], 1u << (rq & 31));
            }
            __syncwarp();
            j0 = T;
        }
        removedHere = __reduce_add_sync(0xffffffffu, removedHere);
        if (lane == 0 && removedHere) atomicAdd(&m.topo->removed, removedHere);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < len; k += blockDim.x) {
        const int i = node[k];
        t.removed[i] = gone[k];
        if (!gone[k]) {
            m.prev[i] = node[pl[k]];
            m.next[i] = node[nl[k]];
        }
    }
}

// ---------------------------------------------------------------------------
// Rings

constexpr int kRingPerThread = 16;  // 256 threads x 16 = 4096 nodes per ring
constexpr int kRingMax = 256 * kRingPerThread;

// All blocks of the launch meet (a cooperative launch: they are resident).
// The wait is bounded; a block that gives up raises the error, and false is
// returned: the block then leaves, since what the others were to write may be
// missing.  The arrivals no longer tell where a launch stands after that, so
// later launches that would meet do nothing (ringMeet[2]).
// stage: that of the main sequence, which the error halts; 0: beside it.
#ifndef LBIB_MEET_TRIES
#define LBIB_MEET_TRIES 4000000u
#endif
__device__ bool ring_barrier(const TopoDev& t, unsigned& meet, Status* st, int stage) {
    __syncthreads();
    int late = 0;
    if (threadIdx.x == 0) {
        meet += gridDim.x;
        __threadfence();
        atomicAdd(t.ringMeet, 1u);
        unsigned tries = 0;
        while ((int)(*(volatile unsigned*)t.ringMeet - meet) < 0) {
            __nanosleep(64);
            if (++tries > LBIB_MEET_TRIES) {
                t.ringMeet[2] = 1u;
                if (stage != 0) raise_error(st, ERR_STATE, (int)blockIdx.x, stage);
                else raise_error_beside(st, ERR_STATE, (int)blockIdx.x, ST_BIO);
                late = 1;
                break;
            }
        }
        __threadfence();
    }
    return __syncthreads_or(late) == 0;
}

// The ring order after a topology change, in one launch: a step whose topology
// did not change (the usual one) costs one short kernel (1.1 us) instead of
// seven and two memsets (14 us of an FP64 step).  The ranks are formed in
// shared memory, over the cell's own places; with the links in global memory a
// change cost 75 us at 390 cells of 380 nodes (the seven launches 25 us), now
// 26 us.  Values that other blocks wrote in this launch are read past the L1
// cache.
// beside: launched beside the main sequence (raise_error_beside).
// A remeshing pass that is applied but not committed (it waits for the host; the
// step is halted) has linked nodes into the rings that the counts and the
// connections do not hold yet: the ranking waits for the commit.  No kernel that
// may run beside this one changes K.
__global__ void __launch_bounds__(256) rings_kernel(MembraneDev m, TopoDev t, int nCells, Status* st, int beside) {
    if (!m.topo->changed || m.topo->K != 0) return;
    if (__syncthreads_or((int)t.ringMeet[2])) return;
    const int stage = beside ? 0 : ST_BIO;
    const int M = m.topo->M, C = m.topo->C;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, all = gridDim.x * blockDim.x;
    unsigned meet = *(volatile unsigned*)&t.ringMeet[1];  // arrivals of the launches before this one
    for (int c = tid; c <= nCells; c += all) {
        t.cellCount[c] = 0;
        if (c < nCells) t.cellFill[c] = 0;
    }
    // a node's outgoing connection, and each domain's first connection
    for (int c0 = blockIdx.x * blockDim.x; c0 < C; c0 += all) {
        const int c = c0 + threadIdx.x;
        if (c < C) {
            t.outConn[m.ca[c]] = c;
            agg_min(&t.firstConn[m.cdom[c]], (int)m.cdom[c], c);
        }
    }
    if (!ring_barrier(t, meet, st, stage)) return;
    for (int i0 = blockIdx.x * blockDim.x; i0 < M; i0 += all) {
        const int i = i0 + threadIdx.x;
        if (i < M) {
            const int cell = t.cellOfDom[m.cdom[__ldcg(&t.outConn[i])]];
            agg_add(&t.cellCount[cell], cell);
        }
    }
    if (!ring_barrier(t, meet, st, stage)) return;
    if (blockIdx.x == 0) {  // the cells' places: an exclusive prefix of their counts
        typedef cub::BlockScan<int, 256> Scan;
        __shared__ typename Scan::TempStorage tmp;
        const int per = (nCells + 1 + 255) / 256;
        const int beg = min((int)threadIdx.x * per, nCells + 1), end = min(beg + per, nCells + 1);
        int local = 0, ex;
        for (int c = beg; c < end; ++c) local += __ldcg(&t.cellCount[c]);
        Scan(tmp).ExclusiveSum(local, ex);
        for (int c = beg; c < end; ++c) {
            t.cellStart[c] = ex;
            ex += __ldcg(&t.cellCount[c]);
        }
    }
    if (!ring_barrier(t, meet, st, stage)) return;
    for (int i0 = blockIdx.x * blockDim.x; i0 < M; i0 += all) {
        const int i = i0 + threadIdx.x;
        if (i < M) {
            const uint32_t d = m.cdom[__ldcg(&t.outConn[i])];
            const int cell = t.cellOfDom[d];
            const int k = agg_add(&t.cellFill[cell], cell);
            t.members[__ldcg(&t.cellStart[cell]) + k] = i;
            const int start = m.cb[__ldcg(&t.firstConn[d])];
            // break the ring before its start node: the node whose successor is the start is last
            t.succ[i] = m.next[i] == start ? -1 : m.next[i];
            t.dist[i] = k;  // the node's place among its cell's members
        }
    }
    if (!ring_barrier(t, meet, st, stage)) return;
    // each ring's ranks by pointer jumping, one block per cell
    __shared__ int sNext[kRingMax], sDist[kRingMax];  // by place: the next node's place (-1: none), the links to the end
    for (int cell = blockIdx.x; cell < nCells; cell += gridDim.x) {
        const int b = __ldcg(&t.cellStart[cell]), len = __ldcg(&t.cellCount[cell]);
        if (len > kRingMax) {
            if (threadIdx.x == 0) {
                if (beside) raise_error_beside(st, ERR_CAPACITY, cell, ST_BIO);
                else raise_error(st, ERR_CAPACITY, cell, ST_BIO);
            }
            continue;
        }
        __syncthreads();
        for (int p = threadIdx.x; p < len; p += 256) {
            const int next = __ldcg(&t.succ[__ldcg(&t.members[b + p])]);
            const int q = next >= 0 ? __ldcg(&t.dist[next]) : -1;
            // a ring that leaves its cell has no order: its nodes' ranks fall outside and are reported
            const bool own = next < 0 || t.cellOfDom[m.cdom[__ldcg(&t.outConn[next])]] == cell;
            sNext[p] = own && q < len ? q : -1;
            sDist[p] = own ? (next >= 0 ? 1 : 0) : kRingMax;
        }
        __syncthreads();
        for (int round = 0; (1 << round) < len; ++round) {
            int ns[kRingPerThread], nd[kRingPerThread];
#pragma unroll
            for (int k = 0; k < kRingPerThread; ++k) {
                const int p = threadIdx.x + k * 256;
                if (p >= len) break;
                const int q = sNext[p];
                nd[k] = sDist[p] + (q >= 0 ? sDist[q] : 0);
                ns[k] = q >= 0 ? sNext[q] : -1;
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < kRingPerThread; ++k) {
                const int p = threadIdx.x + k * 256;
                if (p >= len) break;
                sNext[p] = ns[k];
                sDist[p] = nd[k];
            }
            __syncthreads();
        }
        for (int p = threadIdx.x; p < len; p += 256) {
            const int i = __ldcg(&t.members[b + p]);
            const int d = sDist[p];
            if (d >= 0 && d < len) m.ringNode[b + (len - 1 - d)] = i;
            else if (beside) raise_error_beside(st, ERR_STATE, i, ST_BIO);
            else raise_error(st, ERR_STATE, i, ST_BIO);
        }
        if (threadIdx.x == 0) m.ringStart[cell] = b;
        if (threadIdx.x == 0 && cell == nCells - 1) m.ringStart[cell + 1] = b + len;
    }
    for (int d = tid; d < t.nDomains; d += all) t.firstConn[d] = 0x7fffffff;
    if (tid == 0) {
        t.ringMeet[1] = meet;
        m.topo->changed = 0;  // every block has read it: it met the others since
    }
}

// The listed connections to perturb (crossings_kernel, t.rngList), each
// with its place in its cell's ring walk (the rings are current: the host
// rebuilds them first when the topology changed).  The walk visits the
// connection leaving the ring's last node first (the domain's first
// connection), then those leaving ranks 0, 1, ..., len - 2.
__global__ void conn_perturb_gather_kernel(MembraneDev m, TopoDev t, int n, ConnPerturbRec* out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int c = t.rngList[k];
    ConnPerturbRec r{};
    r.a = m.ca[c];
    r.b = m.cb[c];
    r.dom = (int)m.cdom[c];
    r.xa = m.x[r.a]; r.ya = m.y[r.a]; r.xb = m.x[r.b]; r.yb = m.y[r.b];
    r.walk = -1;
    r.z = -1;
    const int cell = (uint32_t)r.dom < (uint32_t)t.nDomains ? t.cellOfDom[r.dom] : -1;
    if (cell >= 0 && cell < m.nCells) {
        const int s0 = m.ringStart[cell], len = m.ringStart[cell + 1] - s0;
        int rank = -1;
        for (int j = 0; j < len; ++j)
            if (m.ringNode[s0 + j] == r.a) { rank = j; break; }
        if (rank >= 0 && len >= 2) {
            r.len = len;
            r.walk = rank == len - 1 ? 0 : rank + 1;
            r.z = m.ringNode[s0 + len - 2];
            r.xz = m.x[r.z];
            r.yz = m.y[r.z];
        }
    }
    out[k] = r;
}

void launch_conn_perturb_gather(const MembraneDev& m, const TopoDev& t, int n, ConnPerturbRec* out, cudaStream_t s) {
    if (n <= 0) return;
    conn_perturb_gather_kernel<<<(n + 127) / 128, 128, 0, s>>>(m, t, n, out);
}

// Blocks that meet at ring_barrier: two per SM at most, never more than are
// resident together (meet_blocks).  A launch that the device refuses leaves its
// error for the caller's cudaGetLastError.
static void launch_meeting(void (*kernel)(MembraneDev, TopoDev, int, Status*, int), int blocks, const MembraneDev& m,
                           const TopoDev& t, int arg, Status* st, int arg2, cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)std::min(t.meetBlocks, blocks));
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, m, t, arg, st, arg2);
}

int launch_rings(MembraneDev& m, TopoDev& t, Status* st, cudaStream_t s, bool beside) {
    const int nCells = t.nCellsCap;
    if (m.Mcap == 0 || nCells == 0) return 0;
    launch_meeting(rings_kernel, std::max(nCells, (std::max(m.Mcap, m.Ccap) + 255) / 256), m, t, nCells, st,
                   beside ? 1 : 0, s);
    return 1;
}

// ---------------------------------------------------------------------------
// Compaction after the removals

// Exclusive place of this thread's three flags among the block's, and their sums.
__device__ __forceinline__ void block_places(const bool (&flag)[3], int (&place)[3], int (&sum)[3], int (*warpCnt)[8]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const unsigned bal = __ballot_sync(0xffffffffu, flag[k]);
        place[k] = __popc(bal & ((1u << lane) - 1u));
        if (lane == 0) warpCnt[k][warp] = __popc(bal);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        sum[k] = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            const int c = warpCnt[k][w];
            if (w < warp) place[k] += c;
            sum[k] += c;
        }
    }
    __syncthreads();
}

// Drops the removed nodes and the dead connections and appends the alive new
// connections in removal (= id) order, in one launch.  Each block counts its
// stretch of the kept nodes, alive connections and alive new connections, places
// them after the blocks before it, and moves them by way of the scratch copies.
// Bound by latency: the three meetings and the reads between them (39 us for 150k
// nodes), or, when nothing was removed (the usual coarsening of a small
// simulation), by its launch (1.4 us).  In eleven launches (flags, three library
// scans over the capacity, gather, scatter, counts) it was 55 and 17 us.  Steps,
// averaged over ten: 200^2 FP32 25.0 -> 23.8 us, FP64 31.4 -> 30.4, 337x521 FP32
// 49.2 -> 46.8, 1024^2 FP64 178 -> 172 (FP32 111 -> 110).
__global__ void __launch_bounds__(256, 2) coarsen_compact_kernel(MembraneDev m, TopoDev t, int, Status* st, int) {
    Topo* T = m.topo;
    // (the block as one: a meeting that fails raises an error here)
    if (__syncthreads_or(st->halt | (int)t.ringMeet[2])) return;
    if (T->removed == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) T->nCand = 0;
        return;
    }
    const int M = T->M, C = T->C;
    unsigned meet = *(volatile unsigned*)&t.ringMeet[1];  // arrivals of the launches before this one
    const int nb = gridDim.x;
    const int chunk = ((max(M, C) + nb * 256 - 1) / (nb * 256)) * 256;
    const int beg = blockIdx.x * chunk, end = min(beg + chunk, max(M, C));
    __shared__ int warpCnt[3][8], before[3], all[3];
    if (threadIdx.x < 3) before[threadIdx.x] = all[threadIdx.x] = 0;
    int cnt[3] = {0, 0, 0};
    for (int i0 = beg; i0 < end; i0 += 256) {
        const int i = i0 + threadIdx.x;
        cnt[0] += __syncthreads_count(i < M && !t.removed[i]);
        cnt[1] += __syncthreads_count(i < C && t.connAlive[i]);
        cnt[2] += __syncthreads_count(i < M && t.ncAlive[i]);
    }
    if (threadIdx.x < 3) t.blockSum[threadIdx.x * nb + blockIdx.x] = cnt[threadIdx.x];
    if (!ring_barrier(t, meet, st, ST_COARSEN)) return;
    for (int k = 0; k < 3; ++k) {
        int lo = 0, sum = 0;
        for (int b = threadIdx.x; b < nb; b += 256) {
            const int c = __ldcg(&t.blockSum[k * nb + b]);
            sum += c;
            if (b < (int)blockIdx.x) lo += c;
        }
        lo = __reduce_add_sync(0xffffffffu, lo);
        sum = __reduce_add_sync(0xffffffffu, sum);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&before[k], lo);
            atomicAdd(&all[k], sum);
        }
    }
    __syncthreads();
    int at[3] = {before[0], before[1], before[2]};
    const int Mn = all[0], Ca = all[1], Cn = all[1] + all[2];
    const size_t cap = (size_t)m.Mcap;
    double* a = t.dalt;
    for (int i0 = beg; i0 < end; i0 += 256) {
        const int i = i0 + threadIdx.x;
        const bool flag[3] = {i < M && !t.removed[i], i < C && t.connAlive[i] != 0, i < M && t.ncAlive[i] != 0};
        int place[3], sum[3];
        block_places(flag, place, sum, warpCnt);
        if (flag[0]) {
            const int d = at[0] + place[0];
            t.nrank[i] = d;
            a[0 * cap + d] = m.x[i]; a[1 * cap + d] = m.y[i]; a[2 * cap + d] = m.ox[i]; a[3 * cap + d] = m.oy[i];
            a[4 * cap + d] = m.vx[i]; a[5 * cap + d] = m.vy[i]; a[6 * cap + d] = m.fx[i]; a[7 * cap + d] = m.fy[i];
            a[8 * cap + d] = m.bx[i]; a[9 * cap + d] = m.by[i];
            t.id2[d] = m.id[i];
        }
        if (flag[1]) t.rank[i] = at[1] + place[1];
        if (flag[2]) t.succ[i] = Ca + at[2] + place[2];
#pragma unroll
        for (int k = 0; k < 3; ++k) at[k] += sum[k];
    }
    if (!ring_barrier(t, meet, st, ST_COARSEN)) return;
    const int tid = blockIdx.x * blockDim.x + threadIdx.x, stride = nb * blockDim.x;
    for (int i0 = beg; i0 < end; i0 += 256) {
        const int i = i0 + threadIdx.x;
        if (i < M && !t.removed[i]) {
            const int d = t.nrank[i];
            t.prev2[d] = __ldcg(&t.nrank[m.prev[i]]);
            t.next2[d] = __ldcg(&t.nrank[m.next[i]]);
        }
        if (i < C && t.connAlive[i]) {
            const int d = t.rank[i];
            t.ca2[d] = __ldcg(&t.nrank[m.ca[i]]); t.cb2[d] = __ldcg(&t.nrank[m.cb[i]]);
            t.cdom2[d] = m.cdom[i]; t.cdesc2[d] = m.cdesc[i];
        }
        if (i < M && t.ncAlive[i]) {
            const int d = t.succ[i];
            t.ca2[d] = __ldcg(&t.nrank[t.ncA[i]]); t.cb2[d] = __ldcg(&t.nrank[t.ncB[i]]);
            t.cdom2[d] = t.ncDom[i]; t.cdesc2[d] = t.ncDesc[i];
        }
    }
    for (int i = tid; i < Mn; i += stride) {  // (their last readers were before the barrier)
        m.x[i] = __ldcg(&a[0 * cap + i]); m.y[i] = __ldcg(&a[1 * cap + i]);
        m.ox[i] = __ldcg(&a[2 * cap + i]); m.oy[i] = __ldcg(&a[3 * cap + i]);
        m.vx[i] = __ldcg(&a[4 * cap + i]); m.vy[i] = __ldcg(&a[5 * cap + i]);
        m.fx[i] = __ldcg(&a[6 * cap + i]); m.fy[i] = __ldcg(&a[7 * cap + i]);
        m.bx[i] = __ldcg(&a[8 * cap + i]); m.by[i] = __ldcg(&a[9 * cap + i]);
        m.id[i] = __ldcg(&t.id2[i]);
        if (i == Mn - 1) T->maxId = __ldcg(&t.id2[i]);
    }
    if (!ring_barrier(t, meet, st, ST_COARSEN)) return;
    for (int i = tid; i < Mn; i += stride) {
        m.prev[i] = __ldcg(&t.prev2[i]);
        m.next[i] = __ldcg(&t.next2[i]);
    }
    for (int i = tid; i < Cn; i += stride) {
        m.ca[i] = __ldcg(&t.ca2[i]); m.cb[i] = __ldcg(&t.cb2[i]);
        m.cdom[i] = __ldcg(&t.cdom2[i]); m.cdesc[i] = __ldcg(&t.cdesc2[i]);
    }
    if (tid == 0) {
        t.ringMeet[1] = meet;
        T->M = Mn;
        T->C = Cn;
        T->changed = 1;
        T->removed = 0;
        T->nCand = 0;
    }
}

cudaError_t meet_blocks(int* blocks) {
    int device = 0, sms = 0, rings = 0, compact = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&rings, rings_kernel, 256, 0);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&compact, coarsen_compact_kernel, 256, 0);
    *blocks = std::max(1, sms * std::min(2, std::min(rings, compact)));
    return e;
}

int launch_coarsen(MembraneDev& m, TopoDev& t, Status* st, cudaStream_t s) {
    const int nCells = t.nCellsCap;
    if (m.Mcap == 0 || nCells == 0) {
        launch_clear_forces(m, s, st);
        return 1;
    }
    const int blocks = (std::max(m.Mcap, m.Ccap) + 1 + 255) / 256;
    launch_pdl(coarsen_begin_kernel, blocks, 256, 0, s, m, t, st);
    const int n = launch_rings(m, t, st, s);  // ring order after this step's remeshing
    launch_pdl(coarsen_cell_kernel, nCells, 256, kCoarsenSmem, s, m, t, st);
    launch_meeting(coarsen_compact_kernel, blocks, m, t, 0, st, 0, s);
    return n + 3;
}

}  // namespace lbib

namespace lbib {

void init_kernel_attributes_topology() {
    cudaFuncSetAttribute(coarsen_cell_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCoarsenSmem);
    // loaded now rather than at a host event's first use (modules load lazily)
    cudaFuncAttributes fa;
    cudaFuncGetAttributes(&fa, conn_perturb_gather_kernel);
}

}  // namespace lbib
