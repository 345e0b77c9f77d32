// k_readout.cu — the state in the host's layouts.  Compiled with --fmad=false.
//
// A read-out is a sequence of host arrays (parts); one thread forms one
// element of a part from the device's planes: the transposition to the
// reference's slot layout, the widening of FP32-shifted values (f = h + w) and
// the gather of ids and cell types run here, so that the bytes that cross the
// bus are the caller's arrays as they stand.  The host used to do it one value
// at a time, after copying each group of planes to pageable memory: 91 ms for
// the lattice of 1024^2 nodes with two species (200 MB), 13.2 ms this way, bound
// by the first touch of the caller's arrays (the bus takes 4 ms).
#include "kernels.cuh"

namespace lbib {

__device__ __constant__ int kInv9[9] = {0, 3, 4, 1, 2, 7, 8, 5, 6};
__device__ __constant__ double kW9[9] = {4.0 / 9.0,  1.0 / 9.0,  1.0 / 9.0,  1.0 / 9.0, 1.0 / 9.0,
                                         1.0 / 36.0, 1.0 / 36.0, 1.0 / 36.0, 1.0 / 36.0};

// Elements [e0, e0 + n) of part `p` into out[0..n).  Consecutive threads read
// four or so consecutive nodes of each plane: whole 32-byte sectors in FP64.
template <typename Real>
__global__ void __launch_bounds__(256) readout_kernel(ReadoutArgs a, int p, size_t e0, size_t n, void* out) {
    const size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const size_t e = e0 + j, L = a.L;
    double* od = (double*)out + j;
    uint32_t* oi = (uint32_t*)out + j;
    switch (p) {
        case RO_F: {  // f[L][9]: the stored slot of a direction is its inverse's
            const size_t node = e / 9;
            const int q = kInv9[e - node * 9];
            const double v = (double)((const Real*)a.f)[(size_t)q * L + node];
            *od = sizeof(Real) == 8 ? v : v + kW9[q];
            break;
        }
        case RO_G: {  // g[S][L][5]
            const size_t row = e / 5;  // k L + node
            const size_t k = row / L, node = row - k * L;
            *od = (double)((const Real*)a.g)[(k * 5 + (size_t)kInv9[e - row * 5]) * L + node];
            break;
        }
        case RO_C: {  // c[S][L]: the slots of g[S][L][5] added in their order
            const size_t k = e / L, node = e - k * L;
            const Real* g = (const Real*)a.g + k * 5 * L + node;
            double C = 0.0;
#pragma unroll
            for (int d = 0; d < 5; ++d) C += (double)g[(size_t)kInv9[d] * L];
            *od = C;
            break;
        }
        case RO_VEL:  // vel[L][2]
            *od = (double)((const Real*)a.u)[(e & 1) * L + (e >> 1)];
            break;
        case RO_FORCE: {  // force[L][2]: zero where no membrane stencil wrote it
            const size_t node = e >> 1;
            const int x = (int)(node % (size_t)a.nx), y = (int)(node / (size_t)a.nx);
            const bool act = a.tileCount[(y / kTile) * a.tilesX + x / kTile] > 0;
            *od = act ? (double)((const Real*)a.force)[(e & 1) * L + node] : 0.0;
            break;
        }
        case RO_DOM:
            *oi = a.dom[e];
            break;
        case RO_CTYPE: {
            const uint32_t d = a.dom[e];
            *oi = a.cellTypesCopied ? (d < (uint32_t)a.nDomains ? a.ctypeTab[d] : 1u) : 0u;
            break;
        }
        case RO_STATE: {  // state[M][6] = x, y, vx, vy, fx, fy
            const size_t i = e / 6;
            const int c = (int)(e - i * 6);
            const double* const v[6] = {a.m.x, a.m.y, a.m.vx, a.m.vy, a.m.fx, a.m.fy};
            *od = v[c][i];
            break;
        }
        case RO_IDS:
            *oi = a.m.id[e];
            break;
        default: {  // RO_CONN: conn[C][3] = id1, id2, domain
            const size_t c = e / 3;
            const int w = (int)(e - c * 3);
            *oi = w == 2 ? a.m.cdom[c] : a.m.id[w == 0 ? a.m.ca[c] : a.m.cb[c]];
            break;
        }
    }
}

void launch_readout(const ReadoutArgs& a, int part, size_t e0, size_t n, void* out, cudaStream_t s) {
    if (n == 0) return;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (a.fp64) readout_kernel<double><<<blocks, 256, 0, s>>>(a, part, e0, n, out);
    else readout_kernel<float><<<blocks, 256, 0, s>>>(a, part, e0, n, out);
}

}  // namespace lbib
