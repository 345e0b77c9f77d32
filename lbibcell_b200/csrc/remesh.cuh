// remesh.cuh — the remeshing pass's tests, shared by the kernel that counts the
// connections to split (with the crossings' ties, k_membrane.cu) and the pass
// itself (k_topology.cu).
#pragma once

#include "kernels.cuh"

namespace lbib {

constexpr int kRemeshBlock = 256;  // connections per block of the count and apply kernels

// |d| > MAXLENGTH for a squared length d2, as the reference tests it (the
// correctly rounded sqrt, Connection::getLength, Connection.cpp:389-394), with
// the root taken only within a few ulps of MAXLENGTH^2: the rounded root is
// monotonic, so well above it is above MAXLENGTH and at or below it is not.
__device__ __forceinline__ bool longer_than_max(double d2) {
    constexpr double m2 = kMAXLENGTH * kMAXLENGTH;
    if (d2 > m2 * (1.0 + 1e-12)) return true;
    if (d2 <= m2) return false;
    return sqrt(d2) > kMAXLENGTH;
}

// Perturbation tests of a new node (GeometryNode.cpp:160, 174, 189, 202).
__device__ __forceinline__ bool new_node_needs_rng(double X, double Y) {
    if (fabs((double)(int)X - X) <= kEPSILON) return true;
    if (fabs((double)(int)Y - Y) <= kEPSILON) return true;
    if (fabs(Y - floor(Y) - (X - floor(X))) <= kEPSILON) return true;
    if (fabs(ceil(Y) - Y - (X - floor(X))) <= kEPSILON) return true;
    return false;
}

// Connection c is split: longer than MAXLENGTH (Connection::getLength,
// Connection.cpp:389-394).  `rng`: its new node needs the random perturbation.
__device__ __forceinline__ bool remesh_split(const MembraneDev& m, int c, bool& rng) {
    const int a = m.ca[c], b = m.cb[c];
    const double x1 = m.x[a], y1 = m.y[a], x2 = m.x[b], y2 = m.y[b];
    const bool split = longer_than_max((x1 - x2) * (x1 - x2) + (y1 - y2) * (y1 - y2));
    rng = split && new_node_needs_rng((x1 + x2) / 2, (y1 + y2) / 2);
    return split;
}

// This block's share of the pass's count: its connections to split
// (t.flag[block]), their total (T->K) and the new nodes that need the random
// generator (T->nRng).  Every thread of the block takes part.
__device__ __forceinline__ void remesh_count_block(const MembraneDev& m, const TopoDev& t) {
    Topo* T = m.topo;
    const int c = blockIdx.x * kRemeshBlock + threadIdx.x;
    bool f = false, rng = false;
    if (c < T->C) f = remesh_split(m, c, rng);
    const int cnt = __syncthreads_count(f);
    if (cnt == 0) {
        if (threadIdx.x == 0 && (long long)blockIdx.x * kRemeshBlock < m.Ccap) t.flag[blockIdx.x] = 0;
        return;
    }
    const int nr = __syncthreads_count(rng);
    if (threadIdx.x == 0) {
        t.flag[blockIdx.x] = cnt;
        atomicAdd(&T->K, cnt);
        if (nr) atomicAdd(&T->nRng, nr);
    }
}

// A connection's (a -> b along the ring, of domain d) shoelace term x_a y_b -
// x_b y_a, rounded to fixed point (2^-24), into its cell's sum
// (areas_fixed_kernel's comment, k_membrane.cu).  Every lane of the warp takes
// part; `in`: the lane has a connection.
constexpr double kAreaFix = 16777216.0;  // 2^24: the fixed-point scale of the shoelace terms
__device__ __forceinline__ void area_term_fixed(const MembraneDev& m, bool in, int a, int b, uint32_t d,
                                                const int* cellOfDom, int nDomains, unsigned long long* acc) {
    int cell = -1;
    long long v = 0;
    if (in) {
        if (d < (uint32_t)nDomains) cell = cellOfDom[d];
        v = __double2ll_rn((m.x[a] * m.y[b] - m.x[b] * m.y[a]) * kAreaFix);
    }
    // one atomic per run of equal cells in the warp (connections of a cell are mostly contiguous)
    const int first = __shfl_sync(0xffffffffu, cell, 0);
    if (__all_sync(0xffffffffu, cell == first)) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (cell >= 0 && (threadIdx.x & 31) == 0) atomicAdd(acc + cell, (unsigned long long)v);
        return;
    }
    const unsigned peers = __match_any_sync(0xffffffffu, cell);
    long long sum = 0;
    for (int l = 0; l < 32; ++l) {
        const long long t = __shfl_sync(0xffffffffu, v, l);
        if ((peers >> l) & 1u) sum += t;
    }
    if (cell >= 0 && (int)(threadIdx.x & 31) == __ffs(peers) - 1)
        atomicAdd(acc + cell, (unsigned long long)sum);
}

}  // namespace lbib
