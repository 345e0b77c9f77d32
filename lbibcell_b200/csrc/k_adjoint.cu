// k_adjoint.cu — reverse-mode (adjoint) step of the FP64 lattice.
//
// One launch runs the adjoint of one time step of the differentiated lattice
// run: pull streaming, FluidSolver::collide with the Luo force term
// (FluidSolver.cpp:103-183, Luo1993ForceModel.cpp:29-70), the D2Q5 species
// collide with their reaction source (CDESolverD2Q5.cpp:75-107,
// tutorial_01_CDESolverD2Q5_SIGNAL.cpp:102-135) and the box outlet rescale
// (MassSolverBoxOutlet.cpp:42-72).  The geometry is frozen: the spread force
// field, the domain ids and the per-domain mass table are constants of the run.
//
// Notation (per lattice node x, step t):
//   A_t        stored state after step t (fluid planes, then species planes),
//   f_q(x)   = A_{t-1,q}(x - c_q)     the pulled inputs of step t,
//   P_t(q, x)  dL/d f_q(x) of step t  (the adjoint of the pulled inputs).
// The adjoint of the state stored after step t is then
//   dL/dA_{t,q}(y) = P_{t+1}(q, y + c_q),
// a gather in the direction opposite to the forward pull, so the kernel reads
// P_{t+1} at shifted positions, recomputes step t's collision from A_{t-1},
// runs the chain rule backwards through it node by node and writes P_t.
// At the final step the adjoint of the stored state is the seed dL/dC_k(x)
// (C_k = sum of the species' five values) for every species direction.
//
// Parameter gradients, accumulated without contended atomics:
//   part[b][0], part[b][1 + k]  dL/d(1/tauF), dL/d(1/tau_k) summed by thread
//                               block b (each block owns its slots; the same
//                               blocks cover the same nodes every step),
//   racc[k][x]                  dL/d source_k at node x (RX_LINEAR species),
//   macc[x]                     dL/d rhoToAdd at node x (FluidSolver::addMass's
//                               per-domain mass source, when the run has one),
//   G[x]                        dL/dF(x) of the force field,
// all summed over the steps; launch_adjoint_finish reduces part, racc and macc
// into grad[0..S], grad[1 + S + k*nDomains + domain] and
// grad[1 + S + S*nDomains + domain].  A seed for the fluid (seedF, the
// gradient of the loss with respect to the final stored distributions) joins
// the species' seed at the final step.
#include <type_traits>

#include "kernels.cuh"

namespace lbib {

namespace {

// Directions and weights as constants of the unrolled loops (T,E,N,W,S,NE,NW,SW,SE).
__host__ __device__ constexpr int cX(int q) {
    return q == 1 || q == 5 || q == 8 ? 1 : (q == 3 || q == 6 || q == 7 ? -1 : 0);
}
__host__ __device__ constexpr int cY(int q) {
    return q == 2 || q == 5 || q == 6 ? 1 : (q == 4 || q == 7 || q == 8 ? -1 : 0);
}
__host__ __device__ constexpr double weight9(int q) { return q == 0 ? 4.0 / 9.0 : (q < 5 ? 1.0 / 9.0 : 1.0 / 36.0); }

// acc + c v for a direction component c of -1, 0 or 1 (v rounded already).
__device__ __forceinline__ double plus(int c, double v, double acc) { return c > 0 ? acc + v : (c < 0 ? acc - v : acc); }
// c_x x + c_y y of direction q
__device__ __forceinline__ double along(int q, double x, double y) {
    const double X = cX(q) < 0 ? -x : x;
    if (cY(q) == 0) return cX(q) == 0 ? 0.0 : X;
    const double Y = cY(q) < 0 ? -y : y;
    return cX(q) == 0 ? Y : X + Y;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Adds v into grad[key] once per group of lanes with the same key (lanes with
// key < 0 add nothing).  Every lane of the warp calls it.
__device__ __forceinline__ void warp_keyed_add(double* grad, int key, double v) {
    const int key0 = __shfl_sync(0xffffffffu, key, 0);
    if (__all_sync(0xffffffffu, key == key0)) {  // the usual case: one domain per warp
        const double sum = warp_sum(v);
        if ((threadIdx.x & 31) == 0 && key0 >= 0 && sum != 0.0) atomicAdd(grad + key0, sum);
        return;
    }
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    double sum = 0.0;
#pragma unroll 4
    for (int l = 0; l < 32; ++l) {
        const double t = __shfl_sync(0xffffffffu, v, l);
        if ((peers >> l) & 1u) sum += t;
    }
    const int lane = threadIdx.x & 31;
    if (key >= 0 && lane == __ffs(peers) - 1 && sum != 0.0) atomicAdd(grad + key, sum);
}

}  // namespace

// NS = number of species (compile-time, so that the species' inputs are
// loaded together with the fluid state).  Grid (ceil(nx / kAdjBlock), ny).
//
// The directions are constants of the unrolled loops: read from constant memory,
// each c_q v was a conversion and a multiply-add, zeros included, and a node took
// 1,270 instructions.  Everything a node reads is under way before the first value
// is used: the adjoint planes wait as the FP32 values they are, the accumulators
// ride along, and the relaxation-time sums leave by reductions that nothing waits
// for.  The step of 512^2 nodes with one species: 23 -> 14.7 us.  The arithmetic is
// what it was, to the last bit: products that a direction's factor kept from being
// contracted into an addition are kept apart by __dmul_rn (the adjoint planes are
// rounded to FP32 every step, and a last bit that differs grows over the steps into
// a difference of the size of those roundings).
//
// Blocks per SM the register budget is sized for: five (96 registers, 90 B of
// spills) with up to one species, four (128) with more.  512^2 reverse pass per
// step with its recomputation, one species: 3 blocks 25.8 us, 4 23.8, 5 23.7, 6 31.0;
// two species: 35.0, 35.4, 38.7, 45.3; 1024^2, one species: 113.7, 102.6, 98.2, 115.2.
constexpr int adjoint_min_blocks(int species) { return species <= 1 ? 5 : 4; }
// Threads per block (nodes of one row segment).
#ifndef LBIB_ADJOINT_BLOCK
#define LBIB_ADJOINT_BLOCK 128
#endif
constexpr int kAdjBlock = LBIB_ADJOINT_BLOCK;
// Real: the precision the states are stored in.  An FP32-shifted run stores
// f_q - w_q in FP32 (and its species as they are); the reverse step reads
// them back as f and runs its arithmetic in FP64 all the same.
// MOT: the motion form of a run with moving membrane nodes: the step's
// velocity output has its own adjoint input a.gu (the nodes interpolate it),
// the post-collision velocity is written to a.uo, and G holds this step's
// dL/dF alone (the force field changes every step).
// SEED: the final step, whose adjoint inputs are the caller's (FP64).
template <int NS, typename Real, bool MOT, bool SEED>
__global__ void __launch_bounds__(kAdjBlock, adjoint_min_blocks(NS)) adjoint_step64(AdjointArgs a) {
    typedef typename std::conditional<SEED, double, float>::type Adj;
    constexpr int NSA = NS > 0 ? NS : 1;
    const int nx = a.nx, ny = a.ny;
    const size_t L = a.L;
    const int xr = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = xr < nx;
    const int x = valid ? xr : nx - 1, y = blockIdx.y;
    const int xm = x == 0 ? nx - 1 : x - 1, xp = x == nx - 1 ? 0 : x + 1;
    const int ym = y == 0 ? ny - 1 : y - 1, yp = y == ny - 1 ? 0 : y + 1;
    const unsigned rC = (unsigned)y * nx, rM = (unsigned)ym * nx, rP = (unsigned)yp * nx;
    const unsigned n = rC + x;
    // forward pull sources x - c_q and adjoint gather sources x + c_q (offsets
    // within a plane), formed where they are used
    auto pull = [&](int q) -> unsigned {
        const unsigned row = cY(q) > 0 ? rM : (cY(q) < 0 ? rP : rC);
        return row + (cX(q) > 0 ? xm : (cX(q) < 0 ? xp : x));
    };
    auto push = [&](int q) -> unsigned {
        const unsigned row = cY(q) > 0 ? rP : (cY(q) < 0 ? rM : rC);
        return row + (cX(q) > 0 ? xp : (cX(q) < 0 ? xm : x));
    };

    // ---- the inputs of the forward recomputation and of the species ------
    // The stored state, the domain ids, the force field and the mass table
    // are written by no kernel of the reverse pass, and every kernel before
    // the previous launch has completed (the previous launch, an adjoint step
    // of the same pass with a.chained, let this one start only after its own
    // wait): they are loaded before the wait, during the previous step's last
    // wave.  The adjoint planes and the accumulators are read after it.
    const Real* __restrict__ fprev = (const Real*)a.fprev;
    Real fr[9], gr[NSA][5];
#pragma unroll
    for (int q = 0; q < 9; ++q) fr[q] = fprev[(size_t)q * L + pull(q)];
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        const Real* gp = (const Real*)a.gprev + (size_t)k * 5 * L;
#pragma unroll
        for (int q = 0; q < 5; ++q) gr[k][q] = gp[(size_t)q * L + pull(q)];
    }
    const uint32_t dom = a.dom[n];
    // The force field of a differentiated run is zero outside the force tiles,
    // so it and G are read and written everywhere: no load waits on another.
    // (With moving nodes the launch before spread it: read after the wait.)
    double fx = 0.0, fy = 0.0;
    if (!MOT) {
        fx = a.force[n];
        fy = a.force[L + n];
    }
    double rta = 0.0;
    if (a.massTab != nullptr && dom < (uint32_t)a.nDomains) rta = a.massTab[dom];
    pdl_wait();
    pdl_launch_dependents();
    if (MOT) {
        fx = a.force[n];
        fy = a.force[L + n];
    }
    Adj lr[9], mr[NSA][5];
#pragma unroll
    for (int k = 0; k < NS; ++k) {
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            if constexpr (SEED) mr[k][q] = a.seed[(size_t)k * L + n];
            else mr[k][q] = a.pg[((size_t)k * 5 + q) * L + push(q)];
        }
    }
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        if constexpr (SEED) lr[q] = a.seedF ? a.seedF[(size_t)q * L + n] : 0.0;
        else lr[q] = a.pf[(size_t)q * L + push(q)];
    }
    double G0 = 0.0, G1 = 0.0, racc[NSA] = {};
    if (!MOT) {
        G0 = a.G[n];
        G1 = a.G[L + n];
    }
#pragma unroll
    for (int k = 0; k < NS; ++k)
        if (a.sp[k].kind == RX_LINEAR) racc[k] = a.racc[(size_t)k * L + n];
    const bool hasMass = a.macc != nullptr && a.massTab != nullptr && dom < (uint32_t)a.nDomains && isfinite(rta);
    if (!isfinite(rta)) rta = 0.0;

    // ---- forward recomputation of the fluid collision --------------------
    double f[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) f[q] = sizeof(Real) == 8 ? (double)fr[q] : (double)fr[q] + weight9(q);
    const double tauI = a.tauIF;
    double rhoF = 0.0;
#pragma unroll
    for (int q = 0; q < 9; ++q) rhoF += f[q];
    const double rho = rhoF + rta;
    double jx = 0.0, jy = 0.0;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        jx = plus(cX(q), f[q], jx);
        jy = plus(cY(q), f[q], jy);
    }
    const double rhoI = 1.0 / rho;
    const double ux = __dmul_rn(jx, rhoI), uy = __dmul_rn(jy, rhoI);
    const double lastTerm = 1.5 * (ux * ux + uy * uy);
    // equilibrium and post-collision value of direction q
    auto feqw = [&](int q) {
        const double cu = along(q, ux, uy);
        return weight9(q) * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - lastTerm);
    };
    auto fs = [&](int q) {
        const double v = f[q] - f[q] * tauI + feqw(q) * tauI;
        return q == 0 ? v : v + 3.0 * weight9(q) * rhoF * along(q, fx, fy);
    };
    double jox = 0.0, joy = 0.0;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const double v = fs(q);
        jox = plus(cX(q), v, jox);
        joy = plus(cY(q), v, joy);
    }
    const double uox = jox * rhoI, uoy = joy * rhoI;  // FluidSolver::velocity_ after collide
    // box outlet: node-local rescale(s) by 1/sum(f) on x = 0 and y = 0 (corner twice)
    const int passes = a.outlet ? (x == 0) + (y == 0) : 0;
    double s1 = 1.0, s2 = 1.0;
    if (passes >= 1) {
        double r = 0.0;
#pragma unroll
        for (int q = 0; q < 9; ++q) r += fs(q);
        s1 = 1.0 / r;
    }
    if (passes == 2) {
        double r = 0.0;
#pragma unroll
        for (int q = 0; q < 9; ++q) r += fs(q) * s1;
        s2 = 1.0 / r;
    }

    // ---- species, backwards (their velocity and outlet terms feed the fluid)
    double D1 = 0.0, D2 = 0.0;      // dL/ds1, dL/ds2 from the species
    double muox = 0.0, muoy = 0.0;  // dL/d(post-collision velocity)
    double gTauK[NSA];
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        const SpeciesConst& sp = a.sp[k];
        const double tauIk = a.tauI[k];
        double g[5], mu[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            g[q] = (double)gr[k][q];
            mu[q] = (double)mr[k][q];
        }
        const double C = g[0] + g[1] + g[2] + g[3] + g[4];
        const double C3 = C * (1.0 / 3.0), C6 = C * (1.0 / 6.0);
        double temp[5];
        temp[0] = C3;
        temp[1] = C6 * (1.0 + 3.0 * uox);
        temp[2] = C6 * (1.0 + 3.0 * uoy);
        temp[3] = C6 * (1.0 - 3.0 * uox);
        temp[4] = C6 * (1.0 - 3.0 * uoy);
        // dR/dC; the reaction value R itself only enters the outlet terms
        double dRdC = 0.0;
        if (sp.kind == RX_LINEAR) dRdC = -sp.decay;
        else if (sp.kind == RX_SIGNAL && !(dom == 1 && a.iteration < 5000u)) dRdC = -0.00001;
        const bool react = sp.kind != RX_NONE;
        auto reaction = [&]() {
            if (sp.kind == RX_LINEAR) {
                double src = 0.0;
                if (a.srcTab != nullptr && dom < (uint32_t)a.nDomains) src = a.srcTab[(size_t)k * a.nDomains + dom];
                return src - sp.decay * C;
            }
            if (sp.kind == RX_SIGNAL) return (dom == 1 && a.iteration < 5000u) ? 0.0001 : -0.00001 * C;
            return 0.0;
        };
        const double R = passes ? reaction() : 0.0;
        auto gs = [&](int q) {
            return g[q] - g[q] * tauIk + temp[q] * tauIk + (react ? R * (q == 0 ? (1.0 / 3.0) : (1.0 / 6.0)) : 0.0);
        };
        // outlet rescales of the species (same factors as the fluid)
        if (passes == 2) {
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                D2 += mu[q] * (gs(q) * s1);
                mu[q] *= s2;
            }
        }
        if (passes >= 1) {
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                D1 += mu[q] * gs(q);
                mu[q] *= s1;
            }
        }
        // collide, backwards
        double gTau = 0.0;
#pragma unroll
        for (int q = 0; q < 5; ++q) gTau += mu[q] * (temp[q] - g[q]);
        const double mR = react ? (mu[0] * (1.0 / 3.0) + (mu[1] + mu[2] + mu[3] + mu[4]) * (1.0 / 6.0)) : 0.0;
        const double mC = tauIk * (mu[0] * (1.0 / 3.0) +
                                   (mu[1] * (1.0 + 3.0 * uox) + mu[2] * (1.0 + 3.0 * uoy) +
                                    mu[3] * (1.0 - 3.0 * uox) + mu[4] * (1.0 - 3.0 * uoy)) * (1.0 / 6.0)) +
                          dRdC * mR;
        muox += tauIk * C * 0.5 * (mu[1] - mu[3]);
        muoy += tauIk * C * 0.5 * (mu[2] - mu[4]);
        if (valid) {
            float* qg = a.qg + (size_t)k * 5 * L;
#pragma unroll
            for (int q = 0; q < 5; ++q) qg[(size_t)q * L + n] = (float)((1.0 - tauIk) * mu[q] + mC);
        }
        gTauK[k] = valid ? gTau : 0.0;
        if (valid && sp.kind == RX_LINEAR) a.racc[(size_t)k * L + n] = racc[k] + mR;
    }

    // ---- fluid: outlet, velocity output and collide, backwards -----------
    double lf[9];
#pragma unroll
    for (int q = 0; q < 9; ++q) lf[q] = (double)lr[q];
    if (passes == 2) {
        double d = D2;
#pragma unroll
        for (int q = 0; q < 9; ++q) d += lf[q] * (fs(q) * s1);
#pragma unroll
        for (int q = 0; q < 9; ++q) lf[q] = s2 * lf[q] - s2 * s2 * d;
    }
    if (passes >= 1) {
        double d = D1;
#pragma unroll
        for (int q = 0; q < 9; ++q) d += lf[q] * fs(q);
#pragma unroll
        for (int q = 0; q < 9; ++q) lf[q] = s1 * lf[q] - s1 * s1 * d;
    }
    // post-collision velocity uo = (sum c_q fs_q) / rho
    if (MOT) {
        muox += a.gu[n];
        muoy += a.gu[L + n];
        if (valid) {
            a.uo[n] = uox;
            a.uo[L + n] = uoy;
        }
    }
    double mrho = -(uox * muox + uoy * muoy) * rhoI;
    const double mjox = __dmul_rn(muox, rhoI), mjoy = __dmul_rn(muoy, rhoI);
#pragma unroll
    for (int q = 1; q < 9; ++q) lf[q] += along(q, mjox, mjoy);

    double gTauF = 0.0, mrhoF = 0.0, mfx = 0.0, mfy = 0.0, mux = 0.0, muy = 0.0, mlast = 0.0;
#pragma unroll
    for (int q = 0; q < 9; ++q) {
        const double w = weight9(q);
        gTauF += lf[q] * (feqw(q) - f[q]);
        const double mfeq = lf[q] * tauI;
        const double cu = along(q, ux, uy);
        if (q > 0) {
            mrhoF += lf[q] * 3.0 * w * along(q, fx, fy);
            const double mf = __dmul_rn(lf[q] * 3.0 * w, rhoF);
            mfx = plus(cX(q), mf, mfx);
            mfy = plus(cY(q), mf, mfy);
        }
        mrho += mfeq * w * (1.0 + 3.0 * cu + 4.5 * cu * cu - lastTerm);
        if (q > 0) {
            const double mcu = __dmul_rn(mfeq * w * rho, 3.0 + 9.0 * cu);
            mux = plus(cX(q), mcu, mux);
            muy = plus(cY(q), mcu, muy);
        }
        mlast -= mfeq * w * rho;
    }
    mux += mlast * 3.0 * ux;
    muy += mlast * 3.0 * uy;
    const double mjx = __dmul_rn(mux, rhoI), mjy = __dmul_rn(muy, rhoI);
    mrho -= (ux * mux + uy * muy) * rhoI;
    mrhoF += mrho;
    // rho = sum f + rhoToAdd: dL/d rhoToAdd = dL/d rho
    if (valid && hasMass) a.macc[n] += mrho;
    if (valid) {
#pragma unroll
        for (int q = 0; q < 9; ++q)
            a.qf[(size_t)q * L + n] = (float)plus(cY(q), mjy, plus(cX(q), mjx, (1.0 - tauI) * lf[q] + mrhoF));
        a.G[n] = G0 + mfx;
        a.G[L + n] = G1 + mfy;
    }
    // relaxation-time gradients: block sums into this block's own slots (the
    // same slots every step), reduced over blocks once at the end of the pass
    __shared__ double red[kAdjBlock / 32][1 + kMaxSpecies];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const double v0 = warp_sum(valid ? gTauF : 0.0);
    if (lane == 0) red[warp][0] = v0;
#pragma unroll
    for (int k = 0; k < NS; ++k) {
        const double v = warp_sum(gTauK[k]);
        if (lane == 0) red[warp][1 + k] = v;
    }
    __syncthreads();
    if (threadIdx.x <= NS) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < kAdjBlock / 32; ++w) t += red[w][threadIdx.x];
        // (no other block adds here: a reduction only so as not to wait for the old sum)
        atomicAdd(a.part + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * (1 + NS) + threadIdx.x, t);
    }
}

// Sums the per-block relaxation-time partials (nBlocks x width) into grad[0..width).
__global__ void adjoint_part_reduce(const double* part, int nBlocks, int width, double* grad) {
    pdl_wait();
    __shared__ double red[8];
    for (int j = 0; j < width; ++j) {
        double t = 0.0;
        for (int b = threadIdx.x; b < nBlocks; b += blockDim.x) t += part[(size_t)b * width + j];
        t = warp_sum(t);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
        __syncthreads();
        if (threadIdx.x == 0) {
            double s = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
            grad[j] = s;
        }
        __syncthreads();
    }
}

// Sums the per-node source-rate partials into grad[1 + S + k*nDomains + dom].
__global__ void adjoint_rate_reduce(const double* racc, const uint32_t* dom, size_t L, int S, int nDomains,
                                    double* grad) {
    pdl_wait();
    const size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = n < L;
    const uint32_t d = valid ? dom[n] : 0u;
    for (int k = 0; k < S; ++k) {
        const int key = (valid && d < (uint32_t)nDomains) ? 1 + S + k * nDomains + (int)d : -1;
        warp_keyed_add(grad, key, valid ? racc[(size_t)k * L + n] : 0.0);
    }
}

__global__ void set_iteration_kernel(Status* st, unsigned it) {
    pdl_wait(); st->iteration = it; }

int adjoint_blocks(int nx, int ny) { return ((nx + kAdjBlock - 1) / kAdjBlock) * ny; }

template <bool MOT>
static void launch_step(const AdjointArgs& a, bool programmatic, cudaStream_t s) {
    const dim3 grid((unsigned)((a.nx + kAdjBlock - 1) / kAdjBlock), (unsigned)a.ny);
    switch ((a.S < 3 ? a.S : 3) + (a.fp32 ? 4 : 0) + (a.seed != nullptr ? 8 : 0)) {
#define LBIB_ADJ_CASE(I, N, R, SD) \
    case I: launch_ex(programmatic, adjoint_step64<N, R, MOT, SD>, grid, kAdjBlock, 0, s, a); break;
        LBIB_ADJ_CASE(0, 0, double, false) LBIB_ADJ_CASE(1, 1, double, false)
        LBIB_ADJ_CASE(2, 2, double, false) LBIB_ADJ_CASE(3, 3, double, false)
        LBIB_ADJ_CASE(4, 0, float, false) LBIB_ADJ_CASE(5, 1, float, false)
        LBIB_ADJ_CASE(6, 2, float, false) LBIB_ADJ_CASE(7, 3, float, false)
        LBIB_ADJ_CASE(8, 0, double, true) LBIB_ADJ_CASE(9, 1, double, true)
        LBIB_ADJ_CASE(10, 2, double, true) LBIB_ADJ_CASE(11, 3, double, true)
        LBIB_ADJ_CASE(12, 0, float, true) LBIB_ADJ_CASE(13, 1, float, true)
        LBIB_ADJ_CASE(14, 2, float, true) LBIB_ADJ_CASE(15, 3, float, true)
#undef LBIB_ADJ_CASE
    }
}

void launch_adjoint_step64(const AdjointArgs& a, cudaStream_t s) { launch_step<false>(a, a.chained != 0, s); }

void launch_adjoint_step64_motion(const AdjointArgs& a, cudaStream_t s) { launch_step<true>(a, true, s); }

__global__ void to_float_kernel(const double* in, float* out, size_t n) {
    pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (float)in[i];
}

void launch_to_float(const double* in, float* out, size_t n, cudaStream_t s) {
    launch_pdl(to_float_kernel, (unsigned)((n + 255) / 256), 256, 0, s, in, out, n);
}

// Sums the per-node mass-source partials into grad[base + dom].
__global__ void adjoint_mass_reduce(const double* macc, const uint32_t* dom, size_t L, int nDomains, int base,
                                    double* grad) {
    pdl_wait();
    const size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = n < L;
    const uint32_t d = valid ? dom[n] : 0u;
    const int key = (valid && d < (uint32_t)nDomains) ? base + (int)d : -1;
    warp_keyed_add(grad, key, valid ? macc[n] : 0.0);
}

void launch_adjoint_finish(const AdjointArgs& a, cudaStream_t s) {
    launch_pdl(adjoint_part_reduce, 1, 256, 0, s, a.part, adjoint_blocks(a.nx, a.ny), 1 + a.S, a.grad);
    if (a.S > 0 && a.srcTab != nullptr)
        launch_pdl(adjoint_rate_reduce, (unsigned)((a.L + 255) / 256), 256, 0, s, a.racc, a.dom, a.L, a.S, a.nDomains,
                                                                          a.grad);
    if (a.macc != nullptr && a.massTab != nullptr)
        launch_pdl(adjoint_mass_reduce, (unsigned)((a.L + 255) / 256), 256, 0, s, a.macc, a.dom, a.L, a.nDomains,
                   1 + a.S + a.S * a.nDomains, a.grad);
}

void launch_set_iteration(Status* st, unsigned it, cudaStream_t s) { launch_pdl(set_iteration_kernel, 1, 1, 0, s, st, it); }

}  // namespace lbib
