// Device kernels of the GPE solver path (templated on the working precision R).
//
// Field layout (device):
//   psi, psii, bnd : cplx<R>[nx*ny*nz], row-major (i*ny + j)*nz + k, z fastest
//   V, phi         : R[nx*ny*nz]
//   S              : cplx<R>[nx * 2ny * nz], index (i*2ny + ky)*nz + (kz - 1): the
//                    dipolar half spectrum with the x axis still in real space and
//                    pruned to the nx planes that are non-zero; the kz = 0 plane is
//                    not stored (V_dd is zero there).
//
// The dipolar convolution of the reference (src/solver/fft_solvers/cpu/
// fftw_poisson_solver.cpp:51-96: zero-pad w|psi|^2 into (2nx,2ny,2nz), R2C,
// multiply by kz^2/k^2, C2R, keep the first octant, scale 1/(8N)) is evaluated
// exactly, but the transforms are pruned: a pass along z, y or x reads only the
// non-zero half of its padded lines, and the inverse passes keep only the first
// octant (general.cuh, fused.cuh).
#pragma once

#include "fft_block.cuh"

namespace gpe {

// Per-iteration coefficients of the nonlinear phase (real-time half steps).
struct StepCoef {
    double g3w;  // (ggp11 - cdd/3) * n_atoms
    double gw15; // gamma * w_15
};

template <class R> __device__ __forceinline__ void sincos_r(R x, R *s, R *c);
template <> __device__ __forceinline__ void sincos_r<float>(float x, float *s, float *c) {
    sincosf(x, s, c);
}
template <> __device__ __forceinline__ void sincos_r<double>(double x, double *s, double *c) {
    sincos(x, s, c);
}

struct StepIdx {
    const StepCoef *coef; // per-iteration coefficients of this call
    const int *base;      // device counter: index of the chunk's first iteration
    int local;            // iteration within the chunk
};

// What the z passes of an iteration work on (k2_z, k4_yz, k5_yz_pair[_it], g_z).
struct ZArgs {
    // fields
    void *psi_in;        // RT: the kinetic increment's yz spectrum (psi in RT_PRO); IT: psi
    void *psi_out;       // RT: same as psi_in; IT: the next psi buffer
    void *psi_r;         // RT: psi in real space after the last phase step (read, then rewritten)
    const void *bnd;     // IT: boundary values (last loaded psi)
    void *S;             // dipolar spectrum
    const void *V;
    void *phi;
    // norms (IT)
    double *norm_state;  // [0] xnorma, [1] divisor of psi_in (read), [2] power-of-two scale of the
                         // spectrum of an undivided psi (g_z, read by g_x); written by the last CTA
    double *partial;     // per-CTA partial sums of |psi_out|^2
    unsigned *ticket;    // CTA completion counter (reset by the last CTA)
    int *status;
    double dV;
    // coefficients
    StepIdx step;
    double half_dt, cdd, w_atoms;
    double cx, cy, cz, dtau; // IT stencil
    int nx, ny;
};

extern __shared__ __align__(16) unsigned char g_smem[];

// Sum of v over the block in a fixed order, valid in thread 0; red: 32 doubles that no thread
// still reads.
__device__ __forceinline__ double block_sum(double v, double *red) {
    const int tid = threadIdx.x, nw = blockDim.x >> 5;
    for (int off = 16; off > 0; off >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, off);
    if ((tid & 31) == 0)
        red[tid >> 5] = v;
    __syncthreads();
    double x = 0;
    if (tid == 0)
        for (int w = 0; w < nw; ++w)
            x += red[w];
    return x;
}

// Norm of the psi an imaginary-time z pass has written, from every thread's sum of
// |psi|^2 over part `slot` of `slots`: the parts' sums, added in their order by the last block
// to finish, into norm_state[0] and [1], 1 into [2] (status[0] on a non-finite or non-positive
// one).  At most 1024 threads; all of them call.
__device__ __forceinline__ void norm_by_last_block(double acc, const ZArgs &a, int slot, int slots) {
    __shared__ double red[32];
    __shared__ bool last;
    const int tid = threadIdx.x;
    const double mine = block_sum(acc, red);
    if (tid == 0) {
        a.partial[slot] = mine;
        __threadfence();
        last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last)
        return;
    __threadfence();
    // 16 loads in flight (one behind the other: 19 us for 8192 parts); zeros change nothing
    double v = 0;
    for (int b = tid; b < slots; b += 16 * blockDim.x) {
        double t[16];
#pragma unroll
        for (int n = 0; n < 16; ++n) {
            const int q = b + n * blockDim.x;
            t[n]        = q < slots ? __ldcg(&a.partial[q]) : 0.0;
        }
#pragma unroll
        for (int n = 0; n < 16; ++n)
            v += t[n];
    }
    const double x = block_sum(v, red) * a.dV;
    if (tid == 0) {
        a.norm_state[0] = x;
        a.norm_state[1] = x;
        a.norm_state[2] = 1.0;
        if (!(x > 0.0) || !isfinite(x))
            a.status[0] = 1;
        *a.ticket = 0u;
    }
}
__device__ __forceinline__ void norm_by_last_block(double acc, const ZArgs &a) {
    norm_by_last_block(acc, a, blockIdx.x, gridDim.x);
}

// Unit-modulus factor applied as v + v*w with w = exp(i theta) - 1 given to
// full relative precision: the factor's modulus error is then ~eps*theta^2
// instead of ~eps, so repeated application does not bias the norm.
template <class C> __device__ __forceinline__ C apply_wm1(C v, C w) {
    return C{v.x + (v.x * w.x - v.y * w.y), v.y + (v.x * w.y + v.y * w.x)};
}

// psi *= 1/sqrt(norm_state[0]) (materialise the lazy normalisation).
template <class R>
__global__ void __launch_bounds__(256)
    k_scale(cplx<R> *__restrict__ psi, size_t N, const double *__restrict__ norm_state) {
    const R s = (R)(1.0 / sqrt(norm_state[0]));
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < N;
         q += (size_t)gridDim.x * blockDim.x)
        psi[q] = cscale(psi[q], s);
}

// ---------------------------------------------------------------------------
// Energies (cpu_solver.cpp:137-194): the five FP64 sums over the interior, as block
// partials [5][blocks] that the last block to finish adds up in block order into out[5]
// (a second launch of one block that walked 5 x 1184 partials took 16 us, at any grid).
// ---------------------------------------------------------------------------
template <class R>
__global__ void __launch_bounds__(256)
    k_energy(const cplx<R> *__restrict__ pin, const R *__restrict__ V,
                     const R *__restrict__ phi, const double *__restrict__ norm_state, int lazy,
                     double *__restrict__ partial, unsigned *ticket, double *out, int nx, int ny, int nz, double idx2, double idy2,
                     double idz2, double ggp11, double cdd, double n_atoms, double gamma) {
    const double s     = lazy ? 1.0 / sqrt(norm_state[0]) : 1.0;
    const size_t N     = (size_t)nx * ny * nz;
    const size_t plane = (size_t)ny * nz;
    double e[5]        = {0, 0, 0, 0, 0};
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < N;
         q += (size_t)gridDim.x * blockDim.x) {
        // grids hold at most 2^30 points: 32-bit index arithmetic
        const unsigned q32 = (unsigned)q, row = q32 / (unsigned)nz;
        const int k = (int)(q32 - row * (unsigned)nz);
        const int i = (int)(row / (unsigned)ny);
        const int j = (int)(row - (unsigned)i * (unsigned)ny);
        if (i < 1 || i >= nx - 1 || j < 1 || j >= ny - 1 || k < 1 || k >= nz - 1)
            continue;
        auto ld = [&](size_t t) {
            const cplx<R> v = pin[t];
            return double2{(double)v.x * s, (double)v.y * s};
        };
        const double2 c0 = ld(q), xm = ld(q - plane), xp = ld(q + plane), ym = ld(q - nz),
                      yp = ld(q + nz), zm = ld(q - 1), zp = ld(q + 1);
        const double gr = -((xp.x + xm.x) - 2. * c0.x) * idx2 - ((yp.x + ym.x) - 2. * c0.x) * idy2 -
                          ((zp.x + zm.x) - 2. * c0.x) * idz2;
        const double gi = -((xp.y + xm.y) - 2. * c0.y) * idx2 - ((yp.y + ym.y) - 2. * c0.y) * idy2 -
                          ((zp.y + zm.y) - 2. * c0.y) * idz2;
        const double nrm = c0.x * c0.x + c0.y * c0.y;
        e[0] += gr * c0.x + gi * c0.y;
        e[1] += (double)V[q] * nrm;
        e[2] += 0.5 * ggp11 * nrm * nrm;
        e[3] += 0.5 * cdd * (double)phi[q] * nrm * n_atoms -
                cdd / 3. * (nrm * nrm) / 2. * (n_atoms * n_atoms);
        e[4] += 2. / 5. * gamma * (nrm * nrm * sqrt(nrm));
    }
    __shared__ double red[5][8];
    __shared__ bool last;
    const int tid = threadIdx.x;
    auto block_sums = [&] { // e[t] of all threads -> thread t < 5
#pragma unroll
        for (int t = 0; t < 5; ++t) {
            for (int off = 16; off > 0; off >>= 1)
                e[t] += __shfl_down_sync(0xffffffffu, e[t], off);
            if ((tid & 31) == 0)
                red[t][tid >> 5] = e[t];
        }
        __syncthreads();
        double v = 0;
        if (tid < 5)
            for (int w = 0; w < 8; ++w)
                v += red[tid][w];
        return v;
    };
    const double mine = block_sums();
    if (tid < 5) {
        partial[(size_t)tid * gridDim.x + blockIdx.x] = mine;
        __threadfence();
    }
    __syncthreads();
    if (tid == 0)
        last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last)
        return;
    __threadfence();
#pragma unroll
    for (int t = 0; t < 5; ++t) {
        e[t] = 0;
        for (int b = tid; b < (int)gridDim.x; b += 256)
            e[t] += ((volatile double *)partial)[(size_t)t * gridDim.x + b];
    }
    const double total = block_sums();
    if (tid < 5)
        out[tid] = total;
    if (tid == 0)
        *ticket = 0u;
}

// ---------------------------------------------------------------------------
// Host-format conversion: FP64 staging <-> working precision.
// ---------------------------------------------------------------------------
template <class R>
__global__ void k_from_f64(const double *__restrict__ src, R *__restrict__ dst, size_t n) {
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n;
         q += (size_t)gridDim.x * blockDim.x)
        dst[q] = (R)src[q];
}

// dst = scale * src (scale = 1/sqrt(norm_state[0]) when lazy), widened to FP64.
template <class R>
__global__ void k_to_f64(const R *__restrict__ src, double *__restrict__ dst, size_t n,
                         const double *__restrict__ norm_state, int lazy) {
    const double s = lazy ? 1.0 / sqrt(norm_state[0]) : 1.0;
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n;
         q += (size_t)gridDim.x * blockDim.x)
        dst[q] = (double)src[q] * s;
}

__global__ void k_advance(int *counter, int by);

} // namespace gpe
