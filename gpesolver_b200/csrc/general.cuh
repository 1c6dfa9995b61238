// The iteration for every grid and both precisions: line lengths at run time.
//
// The grids that fused.cuh has compiled line lengths for take its kernels; all
// others, complex128, and the interface's single steps take these.  One iteration is four
// kernels, each a batch of 1D lines with the elementwise physics in its loads
// and stores, the kinetic and the dipolar lines of a pass in one launch:
//
//   g_x  lines along x, forward, factor, inverse: kinetic FFT(nx), exp(i(-dt/2m)k^2) / N;
//        dipolar FFT(2nx) of nx non-zero planes, V_dd(k) * scale, nx planes kept
//   g_y  lines along y, inverse: kinetic FFT(ny); dipolar FFT(2ny), ny rows kept
//   g_z  rows along z: dipolar C2R (row pairs) -> phi; kinetic inverse; the last half
//        step of one iteration and the first of the next, or the imaginary-time
//        Euler step with its norm; rho; kinetic forward; dipolar R2C (row pairs)
//   g_y  forward
//
// (Before: one kernel per axis pass, 12 launches a real-time iteration, one real
// row per complex line along z, a division per index.)
//
// Spectrum of the dipolar convolution: S[i][ky][kz - 1], 1 <= kz <= nz: V_dd is
// kz^2/k^2, zero on the kz = 0 plane, which is not stored
// (fftw_poisson_solver.cpp:39-45).
//
// A line transform is as few Stockham stages of radix <= 16 as its factors allow (two for
// most lengths up to 256, three for 125, 200, 216, 250 and the like) between two shared-memory
// buffers; the first stage of a line along x or y reads global memory and the last one stores
// there, so a two-stage transform crosses shared memory once.  All transforms run forward: an inverse one swaps re and im at both ends.
// Twiddles are those of plan.hpp, in complex64 hi + lo (compensated).
//
// Bound by the chain of dependent instructions on small grids (one or two warps per
// scheduler; 30 x 20 x 12: 20 us an iteration, 5 a launch), by instruction issue on large ones
// (100 x 90 x 30: 44-54% of the slots).  Real time, us an iteration, one kernel per
// axis pass -> now: 100 x 90 x 30 145 -> 46; complex128 128 x 128 x 32 213 -> 80; imaginary
// time, complex128 64 x 64 x 16: 37 -> 28.
#pragma once

#include "kernels.cuh"

namespace gpe {

template <class R> struct GTwid;
template <> struct GTwid<float> { using T = float4; };   // hi.re, hi.im, lo.re, lo.im
template <> struct GTwid<double> { using T = double2; };
__device__ __forceinline__ float2 g_twmul(float2 v, float4 w) {
    return twmul<-1>(v, float2{w.x, w.y}, float2{w.z, w.w});
}
__device__ __forceinline__ double2 g_twmul(double2 v, double2 w) { return cmul(v, w); }
template <class C> __device__ __forceinline__ C g_swap(C v, bool s) { return s ? C{v.y, v.x} : v; }

constexpr int kGStages = 6;
struct GStage {
    int r, ns, nr, step; // radix, product of the radices before, L / r, L / (ns r)
    unsigned m;          // ceil(2^32 / ns): j / ns = umulhi(j, m) for ns > 1
};
struct GPlan {
    int L, n;
    GStage f[kGStages]; // radices in order
    GStage v[kGStages]; // in reverse order (the inverse along x)
    const void *tw;     // GTwid<R>::T[L], exp(-2 pi i m / L)
};

__device__ __forceinline__ int g_div(int x, int d, unsigned m) { return d == 1 ? x : (int)__umulhi((unsigned)x, m); }

#define GPE_RADICES(M) M(1) M(2) M(3) M(4) M(5) M(6) M(7) M(8) M(9) M(10) M(12) M(14) M(15) M(16)

// Inputs of item j (line b) of a stage, twiddled, from the tile: element t of line
// b at s[t TS + b]; elements from nin on are zero and not read.
template <int RAD, class R>
__device__ __forceinline__ void g_load(cplx<R> (&a)[RAD], const cplx<R> *s, const GStage &st, int jm, int j, int b,
                                       int TS, int nin, const void *tw) {
    using T     = typename GTwid<R>::T;
    const T *tb = reinterpret_cast<const T *>(tw);
#pragma unroll
    for (int k = 0; k < RAD; ++k) {
        const int t = j + k * st.nr;
        a[k]        = t < nin ? s[t * TS + b] : cplx<R>{(R)0, (R)0};
    }
    if (st.ns > 1) {
        const int t0 = jm * st.step;
#pragma unroll
        for (int k = 1; k < RAD; ++k)
            a[k] = g_twmul(a[k], __ldg(&tb[t0 * k]));
    }
}

// One stage from tile src to tile dst (offsets in g_smem, complex elements) of
// 2^lb lines of stride 1 and element stride TS.
template <int RAD, class R>
__device__ __forceinline__ void g_mid_r(const GStage &st, const void *tw, unsigned src, unsigned dst, int lb, int TS,
                                        int nin, int tid, int nt) {
    using C         = cplx<R>;
    C *sm           = reinterpret_cast<C *>(g_smem);
    const int items = st.nr << lb;
    for (int it = tid; it < items; it += nt) {
        const int b = it & ((1 << lb) - 1), j = it >> lb;
        const int d = g_div(j, st.ns, st.m), jm = j - d * st.ns;
        C a[RAD];
        g_load<RAD, R>(a, sm + src, st, jm, j, b, TS, nin, tw);
        DFTPart<RAD, -1, R, true>::run(a);
        C *o         = sm + dst + (d * st.ns * RAD + jm) * TS + b;
        const int os = st.ns * TS;
#pragma unroll
        for (int q = 0; q < RAD; ++q)
            o[q * os] = a[q];
    }
}
template <class R>
__device__ __noinline__ void g_mid(GStage st, const void *tw, unsigned src, unsigned dst, int lb, int TS, int nin,
                                   int tid, int nt) {
    switch (st.r) {
#define GPE_M(N)                                                                                   \
    case N: g_mid_r<N, R>(st, tw, src, dst, lb, TS, nin, tid, nt); break;
        GPE_RADICES(GPE_M)
#undef GPE_M
    }
}

// First stage: the lines' columns from global memory (element t of line b at
// p[t rs + b], t < nin, b < cnt; the rest is zero) into the tile at dst.
template <int RAD, class R>
__device__ __forceinline__ void g_first_r(const GStage &st, const cplx<R> *__restrict__ p, size_t rs, int nin, int cnt,
                                          bool swap, unsigned dst, int lb, int TS, int tid, int nt) {
    using C         = cplx<R>;
    C *sm           = reinterpret_cast<C *>(g_smem) + dst;
    const int items = st.nr << lb;
    for (int it = tid; it < items; it += nt) {
        const int b = it & ((1 << lb) - 1), j = it >> lb;
        C a[RAD];
#pragma unroll
        for (int k = 0; k < RAD; ++k) {
            const int t = j + k * st.nr;
            a[k]        = t < nin && b < cnt ? p[(size_t)t * rs + b] : C{(R)0, (R)0};
        }
#pragma unroll
        for (int k = 0; k < RAD; ++k)
            a[k] = g_swap(a[k], swap);
        DFTPart<RAD, -1, R, true>::run(a);
#pragma unroll
        for (int q = 0; q < RAD; ++q)
            sm[(j * RAD + q) * TS + b] = a[q];
    }
}
// Last stage: from the tile at src to global memory, elements t < nout.
template <int RAD, class R>
__device__ __forceinline__ void g_last_r(const GStage &st, const void *tw, cplx<R> *__restrict__ p, size_t rs, int nout,
                                         int cnt, bool swap, unsigned src, int lb, int TS, int tid, int nt) {
    using C         = cplx<R>;
    const C *sm     = reinterpret_cast<const C *>(g_smem) + src;
    const int items = st.nr << lb;
    for (int it = tid; it < items; it += nt) {
        const int b = it & ((1 << lb) - 1), j = it >> lb;
        C a[RAD];
        g_load<RAD, R>(a, sm, st, j, j, b, TS, st.nr * RAD, tw);
        DFTPart<RAD, -1, R, true>::run(a);
#pragma unroll
        for (int q = 0; q < RAD; ++q) {
            const int t = j + q * st.nr;
            if (t < nout && b < cnt)
                p[(size_t)t * rs + b] = g_swap(a[q], swap);
        }
    }
}

// Whole transform of the columns p -> p, with tiles at elements 0 and L << lb of shared
// memory; the second one only for three stages and more.
template <class R>
__device__ __forceinline__ void g_lines(const GPlan &pl, cplx<R> *p, size_t rs, int nin, int nout, int cnt, bool swap,
                                        int lb, int tid, int nt) {
    using C       = cplx<R>;
    const int TS  = 1 << lb;
    unsigned cur  = 0, oth = (unsigned)(pl.L * TS);
    switch (pl.f[0].r) {
#define GPE_M(N)                                                                                   \
    case N: g_first_r<N, R>(pl.f[0], p, rs, nin, cnt, swap, cur, lb, TS, tid, nt); break;
        GPE_RADICES(GPE_M)
#undef GPE_M
    }
    __syncthreads();
    for (int s = 1; s < pl.n - 1; ++s) {
        g_mid<R>(pl.f[s], pl.tw, cur, oth, lb, TS, pl.L, tid, nt);
        __syncthreads();
        const unsigned t = cur;
        cur = oth, oth = t;
    }
    if (pl.n == 1) { // the first stage was the whole line
        const C *sm = reinterpret_cast<const C *>(g_smem);
        for (int e = tid; e < nout << lb; e += nt) {
            const int b = e & (TS - 1), t = e >> lb;
            if (b < cnt)
                p[(size_t)t * rs + b] = g_swap(sm[e], swap);
        }
        return;
    }
    switch (pl.f[pl.n - 1].r) {
#define GPE_M(N)                                                                                   \
    case N: g_last_r<N, R>(pl.f[pl.n - 1], pl.tw, p, rs, nout, cnt, swap, cur, lb, TS, tid, nt); break;
        GPE_RADICES(GPE_M)
#undef GPE_M
    }
}

// g_x and g_y hold a radix's inputs in registers (g_x twice over, for the pair of
// transforms): MB = 3 CTAs of 256 threads per SM (80 registers) in complex64 up to radix 15,
// 2 (128 registers) for radix 16, where 3 would spill more, and in complex128.  Measured with 3
// against 2: real time 100 x 90 x 30 45.3 against 50.6 us an iteration, 144 x 144 x 40
// 106 against 123; the field at 128 x 128 x 32 (radix 16) 65.6 against 60.7 us.
template <class R> constexpr int g_blocks(int most_radix) { return sizeof(R) == 4 && most_radix <= 15 ? 3 : 2; }

// ---------------------------------------------------------------------------
// y lines: one x plane per blockIdx.y, tiles of 2^lb z columns along blockIdx.x,
// first the kinetic ones (tk), then the dipolar ones
// ---------------------------------------------------------------------------
struct GYArgs {
    void *psi, *S;
    int ny, nz, tk, inverse;
    int lb;
    GPlan k, d;
};
template <class R, int MB> __global__ void __launch_bounds__(256, MB) g_y(const __grid_constant__ GYArgs a) {
    using C        = cplx<R>;
    const bool kin = (int)blockIdx.x < a.tk;
    const int k0   = (kin ? blockIdx.x : blockIdx.x - a.tk) << a.lb;
    const int cnt  = min(1 << a.lb, a.nz - k0);
    const size_t plane = (size_t)blockIdx.y * a.ny * a.nz;
    C *p = kin ? reinterpret_cast<C *>(a.psi) + plane + k0 : reinterpret_cast<C *>(a.S) + 2 * plane + k0;
    const int nin  = kin || !a.inverse ? a.ny : 2 * a.ny;
    const int nout = kin || a.inverse ? a.ny : 2 * a.ny;
    g_lines<R>(kin ? a.k : a.d, p, a.nz, nin, nout, cnt, a.inverse, a.lb, threadIdx.x, blockDim.x);
}

// ---------------------------------------------------------------------------
// x lines: forward, factor, inverse; tiles of 2^lb (y, z) columns, the kinetic
// ones first
// ---------------------------------------------------------------------------
struct GXArgs {
    void *psi, *S;
    const void *ex, *ey, *ez;     // exp(i theta) - 1 per axis (kinetic)
    double inv;                   // 1 / N
    const void *vk;               // V_dd(|kx|, |ky|, kz), kz = 1..nz
    const double *divisor;        // [0] norm the spectrum is still to be divided by, [1] its power-of-two
                                  // scale (g_spectrum_scale); or null
    double dip_scale;
    int nx, ny, nz, tk, lb;
    GPlan k, d;
};

// The forward transform's last stage, the factor and the inverse's first stage
// (radices reversed: it reads exactly the outputs the item holds).
template <int RAD, class R>
__device__ __forceinline__ void g_xmid_r(const GXArgs &a, const GPlan &pl, bool kin, int c0, int cnt, R scale,
                                         unsigned src, unsigned dst, int tid, int nt) {
    using C         = cplx<R>;
    C *sm           = reinterpret_cast<C *>(g_smem);
    const GStage st = pl.f[pl.n - 1];
    const int TS = 1 << a.lb, items = st.nr << a.lb;
    for (int it = tid; it < items; it += nt) {
        const int b = it & (TS - 1), j = it >> a.lb;
        const int c = c0 + min(b, cnt - 1), y = c / a.nz, z = c - y * a.nz;
        C v[RAD];
        g_load<RAD, R>(v, sm + src, st, j, j, b, TS, pl.L, pl.tw);
        C in[sizeof(R) == 4 ? RAD : 1];
        if constexpr (sizeof(R) == 4)
#pragma unroll
            for (int q = 0; q < RAD; ++q)
                in[q] = v[q];
        DFTPart<RAD, -1, R, true>::run(v);
        if (kin) {
            const C *ex = reinterpret_cast<const C *>(a.ex);
            const C wy = __ldg(reinterpret_cast<const C *>(a.ey) + y), wz = __ldg(reinterpret_cast<const C *>(a.ez) + z);
            const C wyz = cadd(cadd(wy, wz), cmul(wy, wz)); // (1+wy)(1+wz) - 1
            const R ih  = (R)a.inv; // one word: a common factor of up to 6e-8 on the increment alone
#pragma unroll
            for (int q = 0; q < RAD; ++q) {
                const C wx = __ldg(&ex[j + q * st.nr]);
                const C w  = cadd(cadd(wx, wyz), cmul(wx, wyz)); // exp(i theta) - 1
                const C u  = sizeof(R) == 4 ? cmul(v[q], w) : apply_wm1(v[q], w);
                v[q]       = C{u.y * ih, u.x * ih}; // swapped: inverse
            }
        } else {
            const int iy = y <= a.ny ? y : 2 * a.ny - y;
            const R *vk  = reinterpret_cast<const R *>(a.vk) + (size_t)iy * a.nz + z;
            const size_t xs = (size_t)(a.ny + 1) * a.nz;
#pragma unroll
            for (int q = 0; q < RAD; ++q) {
                const int t = j + q * st.nr, ix = t <= a.nx ? t : pl.L - t;
                const R f   = __ldg(&vk[ix * xs]) * scale;
                v[q]        = C{v[q].y * f, v[q].x * f};
            }
        }
        DFTPart<RAD, -1, R, true>::run(v);
        // complex64: the transform pair carries the kinetic factor's change of psi,
        // exp(i theta) - 1, and psi itself, RAD / N times the pair's inputs, is added
        // here.  Their rounding then scales with |theta|: done directly, the sums in
        // this most concentrated space (few populated k) drift the norm the most.
        if constexpr (sizeof(R) == 4)
            if (kin) {
                const double f = a.inv * RAD;
                const R fh = (R)f, fl = (R)(f - (double)fh);
#pragma unroll
                for (int q = 0; q < RAD; ++q)
                    v[q] = C{fma(in[q].y, fh, fma(in[q].y, fl, v[q].x)), fma(in[q].x, fh, fma(in[q].x, fl, v[q].y))};
            }
#pragma unroll
        for (int q = 0; q < RAD; ++q)
            sm[dst + (j * RAD + q) * TS + b] = v[q];
    }
}

template <class R, int MB> __global__ void __launch_bounds__(256, MB) g_x(const __grid_constant__ GXArgs a) {
    using C         = cplx<R>;
    const int tid = threadIdx.x, nt = blockDim.x;
    const bool kin  = (int)blockIdx.x < a.tk;
    const GPlan &pl = kin ? a.k : a.d;
    const int cols  = (kin ? 1 : 2) * a.ny * a.nz;
    const int c0    = (kin ? blockIdx.x : blockIdx.x - a.tk) << a.lb;
    const int cnt   = min(1 << a.lb, cols - c0);
    C *p            = (kin ? reinterpret_cast<C *>(a.psi) : reinterpret_cast<C *>(a.S)) + c0;
    const int TS    = 1 << a.lb;
    const R scale   = (R)(a.divisor && !kin ? a.dip_scale / (a.divisor[0] * a.divisor[1]) : a.dip_scale);
    unsigned cur = 0, oth = (unsigned)(pl.L * TS);
    auto flip = [&] {
        __syncthreads();
        const unsigned t = cur;
        cur = oth, oth = t;
    };
    if (pl.n == 1) { // one stage: the columns as they are
        C *sm = reinterpret_cast<C *>(g_smem);
        for (int e = tid; e < pl.L << a.lb; e += nt) {
            const int b = e & (TS - 1), t = e >> a.lb;
            sm[oth + e] = t < a.nx && b < cnt ? p[(size_t)t * cols + b] : C{(R)0, (R)0};
        }
    } else {
        switch (pl.f[0].r) {
#define GPE_M(N)                                                                                   \
    case N: g_first_r<N, R>(pl.f[0], p, cols, a.nx, cnt, false, oth, a.lb, TS, tid, nt); break;
            GPE_RADICES(GPE_M)
#undef GPE_M
        }
    }
    flip();
    for (int s = 1; s < pl.n - 1; ++s) {
        g_mid<R>(pl.f[s], pl.tw, cur, oth, a.lb, TS, pl.L, tid, nt);
        flip();
    }
    switch (pl.f[pl.n - 1].r) {
#define GPE_M(N)                                                                                   \
    case N: g_xmid_r<N, R>(a, pl, kin, c0, cnt, scale, cur, oth, tid, nt); break;
        GPE_RADICES(GPE_M)
#undef GPE_M
    }
    flip();
    for (int s = 1; s < pl.n - 1; ++s) {
        g_mid<R>(pl.v[s], pl.tw, cur, oth, a.lb, TS, pl.L, tid, nt);
        flip();
    }
    if (pl.n == 1) {
        const C *sm = reinterpret_cast<const C *>(g_smem) + cur;
        for (int e = tid; e < a.nx << a.lb; e += nt) {
            const int b = e & (TS - 1), t = e >> a.lb;
            if (b < cnt)
                p[(size_t)t * cols + b] = g_swap(sm[e], true);
        }
        return;
    }
    switch (pl.v[pl.n - 1].r) {
#define GPE_M(N)                                                                                   \
    case N: g_last_r<N, R>(pl.v[pl.n - 1], pl.tw, p, cols, a.nx, cnt, true, cur, a.lb, TS, tid, nt); break;
        GPE_RADICES(GPE_M)
#undef GPE_M
    }
}

// ---------------------------------------------------------------------------
// z rows
// ---------------------------------------------------------------------------
enum {
    GZ_RT_PRO = 0, // first half step of a call, forward
    GZ_RT_MID,     // inverse, both half steps, forward
    GZ_RT_EPI,     // inverse, last half step; psi and phi stored
    GZ_IT_PRO,     // rho of psi, forward
    GZ_IT_MID,     // dipolar inverse, Euler step and norm, forward
    GZ_DIP_INV,    // spectrum -> phi
    GZ_KIN_FWD, GZ_KIN_INV,
    GZ_MODES
};
// The interface's single steps (GZ_DIP_INV and after, g_half_step, g_euler_step, g_norm) run
// the iterations' arithmetic, the norm in their order too, so both sequences agree to the
// last bits.

// The pointwise arithmetic with its roundings written out: the compiler then contracts
// it alike in every kernel.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
template <class C> __device__ __forceinline__ auto g_abs2(C v) { return fma(v.x, v.x, mul_rn(v.y, v.y)); }

// Potential half step (cpu_solver.cpp:99-131):
//   v exp(i theta), theta = -dt/2 [V + cdd phi + g3 |v|^2 + gw |v|^3],
// applied as v + v (exp(i theta) - 1), exp(i theta) - 1 = (-2 sin^2(theta/2), sin theta)
template <class R>
__device__ __forceinline__ cplx<R> g_turn(cplx<R> v, R V, R phi, R cdd, R hdt, R g3, R gw) {
    const R dens  = g_abs2(v), am = sqrt(dens);
    const R total = add_rn(fma(cdd, phi, V), fma(g3, dens, mul_rn(gw, mul_rn(mul_rn(am, am), am))));
    R s, c;
    sincos_r<R>(mul_rn(mul_rn((R)-0.5, hdt), total), &s, &c);
    const R wx = mul_rn(mul_rn((R)-2, s), s), wy = mul_rn(mul_rn((R)2, s), c);
    return cplx<R>{add_rn(v.x, fma(v.x, wx, -mul_rn(v.y, wy))), add_rn(v.y, fma(v.x, wy, mul_rn(v.y, wx)))};
}

// Euler step (cpu_solver.cpp:50-97) of the interior point at psi, held times 1 / sc:
//   psi' = psi - dtau [cx Lx psi - cy Ly psi - cz Lz psi + (V + cdd phi + g3 |psi|^2 + gw |psi|^3) psi]
template <class R>
__device__ __forceinline__ cplx<R> g_euler(const cplx<R> *psi, ptrdiff_t plane, int nz, R sc, R V, R phi, R cdd, R g3,
                                           R gw, R cx, R cy, R cz, R dtau) {
    using C    = cplx<R>;
    const C c0 = cscale(psi[0], sc);
    const C xm = cscale(psi[-plane], sc), xp = cscale(psi[plane], sc);
    const C ym = cscale(psi[-nz], sc), yp = cscale(psi[nz], sc);
    const C zm = cscale(psi[-1], sc), zp = cscale(psi[1], sc);
    const R dens = g_abs2(c0), am = sqrt(dens);
    const R h    = add_rn(fma(cdd, phi, V), fma(g3, dens, mul_rn(gw, mul_rn(mul_rn(am, am), am))));
    auto step    = [&](R c, R xa, R xb, R ya, R yb, R za, R zb) {
        const R dx = fma((R)-2, c, add_rn(xa, xb)), dy = fma((R)-2, c, add_rn(ya, yb)),
                dz = fma((R)-2, c, add_rn(za, zb));
        return fma(-dtau, fma(cx, dx, fma(-cy, dy, fma(-cz, dz, mul_rn(c, h)))), c);
    };
    return C{step(c0.x, xm.x, xp.x, ym.x, yp.x, zm.x, zp.x), step(c0.y, xm.y, xp.y, ym.y, yp.y, zm.y, zp.y)};
}

// A psi of norm d that is still to be divided by sqrt(d) enters rho as psi 2^-h: |psi|^2 N
// and its transforms stay in range for any d that psi itself has room for (complex64, 1e13
// times a normalised state and more: without it 1/d underflows and rho overflows).  Returns h
// such that d 2^-2h is about 1; 0 for d within 2^+-32, where nothing needs it and every
// rounding stays as it is.
template <class R> __device__ __forceinline__ int g_spectrum_scale(double d) {
    const int e = ((__double2hiint(d) >> 20) & 0x7ff) - 1023, most = sizeof(R) == 4 ? 120 : 500;
    return abs(e) <= 32 ? 0 : min(max(e >> 1, -most), most);
}

struct GZArgs {
    ZArgs z;
    int write_phi, nz, lb; // 2^lb rows per CTA
    unsigned mz;           // ceil(2^32 / nz)
    unsigned buf;          // elements of one of the four tiles
    GPlan k, d;
};

// The kinetic rows in tile K and the dipolar pair lines in tile D (offsets in g_smem)
// transformed, stage by stage side by side: each by half of the warps (all of them where only
// one runs), so that a warp executes one of them and they share the
// synchronisations.  The results are left in the tiles that K and D name on return.
template <class R, bool KIN, bool DIP>
__device__ __forceinline__ void g_tiles(const GPlan &pk, unsigned &K, unsigned &K2, int lk, int TK, const GPlan &pd,
                                        unsigned &D, unsigned &D2, int ld, int TD, int nin) {
    const int nt    = KIN && DIP ? blockDim.x >> 1 : blockDim.x;
    const bool kin  = KIN && (!DIP || (int)threadIdx.x < nt);
    const int tid   = KIN && DIP && !kin ? threadIdx.x - nt : threadIdx.x;
    const GPlan &pl = kin ? pk : pd;
    unsigned cur = kin ? K : D, oth = kin ? K2 : D2;
    const int lb = kin ? lk : ld, TS = kin ? TK : TD;
    const int ns = KIN && DIP ? max(pk.n, pd.n) : pl.n;
    for (int s = 0; s < ns; ++s) {
        if (s < pl.n) {
            g_mid<R>(pl.f[s], pl.tw, cur, oth, lb, TS, s == 0 && !kin ? nin : pl.L, tid, nt);
            const unsigned t = cur;
            cur = oth, oth = t;
        }
        __syncthreads();
    }
    if (KIN && (pk.n & 1)) {
        const unsigned t = K;
        K = K2, K2 = t;
    }
    if (DIP && (pd.n & 1)) {
        const unsigned t = D;
        D = D2, D2 = t;
    }
}

template <class R, int MODE> __global__ void __launch_bounds__(256, sizeof(R) == 4 ? 3 : 2) g_z(const __grid_constant__ GZArgs g) {
    using C            = cplx<R>;
    constexpr bool RT  = MODE <= GZ_RT_EPI;
    constexpr bool IT  = MODE == GZ_IT_MID;
    constexpr bool KIN_I = MODE == GZ_RT_MID || MODE == GZ_RT_EPI || MODE == GZ_KIN_INV;
    constexpr bool KIN_F = MODE == GZ_RT_PRO || MODE == GZ_RT_MID || MODE == GZ_KIN_FWD;
    constexpr bool DIP_I = MODE == GZ_RT_MID || MODE == GZ_RT_EPI || MODE == GZ_IT_MID || MODE == GZ_DIP_INV;
    constexpr bool DIP_F = MODE == GZ_RT_PRO || MODE == GZ_RT_MID || MODE == GZ_IT_PRO || MODE == GZ_IT_MID;
    const ZArgs &a = g.z;
    const int tid = threadIdx.x, nt = blockDim.x, nz = g.nz, nx = a.nx, ny = a.ny;
    const int RW = 1 << g.lb, lp = g.lb > 0 ? g.lb - 1 : 0, NP = 1 << lp; // rows, row pairs
    const int TK = RW >= 4 ? RW + 1 : RW, TD = NP >= 2 ? NP + 1 : NP;     // odd tile strides
    const int rows = nx * ny, r0 = blockIdx.x << g.lb, cnt = min(RW, rows - r0);
    // kinetic rows and dipolar pair lines, two tiles each
    C *sm      = reinterpret_cast<C *>(g_smem);
    unsigned D = 0, D2 = g.buf, K = 2 * g.buf, K2 = 3 * g.buf;
    const size_t base = (size_t)r0 * nz;
    C *psi      = reinterpret_cast<C *>(a.psi_in) + base;
    C *out      = reinterpret_cast<C *>(a.psi_out) + base;
    C *S        = reinterpret_cast<C *>(a.S) - 1; // bins from 1
    R *phi      = reinterpret_cast<R *>(a.phi) + base;
    const R *V  = reinterpret_cast<const R *>(a.V) + base;
    // x plane and y of the tile's row; its spectrum row i 2ny + j
    const int i0 = r0 / ny, j0 = r0 - i0 * ny;
    auto place = [&](int row, int &i, int &j) {
        i = i0;
        j = j0 + row;
        while (j >= ny) {
            j -= ny;
            ++i;
        }
    };
    auto srow = [&](int row) {
        int i, j;
        place(row, i, j);
        return (size_t)(2 * i * ny + j) * nz;
    };

    // ---- in: psi rows (inverse: swapped) and the pair lines of the spectrum ------
    if (KIN_I || MODE == GZ_KIN_FWD) {
        for (int e = tid; e < RW * nz; e += nt) {
            const int row = g_div(e, nz, g.mz), k = e - row * nz;
            sm[K + k * TK + row] = row < cnt ? g_swap(psi[e], KIN_I) : C{(R)0, (R)0};
        }
    }
    // step coefficients, this iteration's and the next one's: two dependent reads, by one
    // thread and behind the others' loads
    __shared__ R cf[4];
    if ((RT || IT) && tid == nt - 1) {
        const int it      = RT ? *a.step.base + a.step.local : 0;
        const StepCoef c0 = a.step.coef[it], c1 = a.step.coef[MODE == GZ_RT_MID ? it + 1 : it];
        cf[0] = (R)c0.g3w, cf[1] = (R)c0.gw15;
        cf[2] = (R)c1.g3w, cf[3] = (R)c1.gw15;
    }
    if (DIP_I) {
        // line z[m] = xa[m] + i xb[m] over the full 2nz-point spectrum: bin 0 is
        // zero, bins > nz by symmetry; stored swapped (inverse transform)
        for (int e = tid; e < NP * nz; e += nt) {
            const int p = g_div(e, nz, g.mz), m = e - p * nz + 1;
            const C xa = 2 * p < cnt ? S[srow(2 * p) + m] : C{(R)0, (R)0};
            const C xb = 2 * p + 1 < cnt ? S[srow(2 * p + 1) + m] : C{(R)0, (R)0};
            if (m == nz) {
                sm[D + m * TD + p] = C{xb.x, xa.x}; // self-conjugate bin: real parts only
                sm[D + p]          = C{(R)0, (R)0};
            } else {
                sm[D + m * TD + p]            = C{xa.y + xb.x, xa.x - xb.y};
                sm[D + (2 * nz - m) * TD + p] = C{xb.x - xa.y, xa.x + xb.y};
            }
        }
    }
    __syncthreads();
    if (KIN_I || DIP_I)
        g_tiles<R, KIN_I, DIP_I>(g.k, K, K2, g.lb, TK, g.d, D, D2, lp, TD, 2 * nz);

    // ---- the step on row pairs: element k of rows 2p and 2p + 1 ----------------
    double acc = 0.0;
    if (MODE == GZ_KIN_INV) {
        for (int e = tid; e < cnt * nz; e += nt) {
            const int row = g_div(e, nz, g.mz), k = e - row * nz;
            out[e]        = g_swap(sm[K + k * TK + row], true);
        }
        return;
    }
    if (MODE != GZ_KIN_FWD) {
        const R g3 = cf[0], gw = cf[1], g3n = cf[2], gwn = cf[3];
        const R sc   = (R)(IT ? 1.0 / sqrt(a.norm_state[1]) : 1.0);
        const R wat  = (R)a.w_atoms;
        R fold       = (R)1;
        if (MODE == GZ_IT_PRO && a.norm_state) {
            const int h = g_spectrum_scale<R>(a.norm_state[1]);
            fold        = (R)scalbn(1.0, -h);
            if (blockIdx.x == 0 && tid == 0)
                a.norm_state[2] = scalbn(1.0, -2 * h);
        }
        const R hdt = (R)a.half_dt, cdd = (R)a.cdd;
        const R cx = (R)a.cx, cy = (R)a.cy, cz = (R)a.cz, dtau = (R)a.dtau;
        const ptrdiff_t plane = (ptrdiff_t)ny * nz;
        for (int e = tid; e < NP * nz; e += nt) {
            const int p = g_div(e, nz, g.mz), k = e - p * nz;
            C z{(R)0, (R)0};
            if (DIP_I)
                z = sm[D + k * TD + p]; // swapped: (row 2p + 1, row 2p)
            R rho[2] = {(R)0, (R)0};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = 2 * p + h;
                if (row >= cnt)
                    break;
                const int q = row * nz + k;
                R f         = h == 0 ? z.y : z.x;
                if (MODE == GZ_RT_PRO)
                    f = phi[q];
                if (MODE == GZ_DIP_INV || MODE == GZ_RT_EPI || (MODE == GZ_IT_MID && g.write_phi))
                    phi[q] = f;
                if (MODE == GZ_DIP_INV)
                    continue;
                int i, j;
                place(row, i, j);
                const bool in = i >= 1 && i < nx - 1 && j >= 1 && j < ny - 1 && k >= 1 && k < nz - 1;
                C v;
                if (RT) {
                    v = MODE == GZ_RT_PRO ? psi[q] : g_swap(sm[K + k * TK + row], true);
                    if (in) {
                        v = g_turn<R>(v, V[q], f, cdd, hdt, g3, gw);
                        if (MODE == GZ_RT_MID) // the next iteration's first half step
                            v = g_turn<R>(v, V[q], f, cdd, hdt, g3n, gwn);
                    }
                    if (MODE == GZ_RT_EPI)
                        out[q] = v;
                    else
                        sm[K + k * TK + row] = v;
                } else if (MODE == GZ_IT_PRO) {
                    v = cscale(psi[q], fold);
                } else { // the Euler step of psi_in / sqrt(divisor)
                    if (!in) {
                        v = reinterpret_cast<const C *>(a.bnd)[base + q];
                    } else {
                        v = g_euler<R>(psi + q, plane, nz, sc, V[q], f, cdd, g3, gw, cx, cy, cz, dtau);
                    }
                    out[q] = v;
                    acc    = add_rn(acc, g_abs2(double2{(double)v.x, (double)v.y}));
                }
                rho[h] = mul_rn(wat, g_abs2(v));
            }
            if (DIP_F)
                sm[D + k * TD + p] = C{rho[0], rho[1]};
        }
        if (!DIP_F)
            return;
        if (KIN_F) // rows beyond the grid's last
            for (int e = cnt * nz + tid; e < RW * nz; e += nt) {
                const int row = g_div(e, nz, g.mz), k = e - row * nz;
                sm[K + k * TK + row] = C{(R)0, (R)0};
            }
        __syncthreads();
    }

    // ---- out: kinetic spectrum, then bins 1..nz of the row pairs -----------------
    if (KIN_F || DIP_F) // the pair lines' padding half is not read
        g_tiles<R, KIN_F, DIP_F>(g.k, K, K2, g.lb, TK, g.d, D, D2, lp, TD, nz);
    if (KIN_F) {
        for (int e = tid; e < cnt * nz; e += nt) {
            const int row = g_div(e, nz, g.mz), k = e - row * nz;
            out[e]        = sm[K + k * TK + row];
        }
    }
    if (DIP_F) {
        for (int e = tid; e < NP * nz; e += nt) {
            const int p = g_div(e, nz, g.mz), m = e - p * nz + 1;
            const C zm = sm[D + m * TD + p], zc = sm[D + (2 * nz - m) * TD + p];
            if (2 * p < cnt) // (Z_m + conj(Z_{L-m}))/2
                S[srow(2 * p) + m] = C{(R)0.5 * (zm.x + zc.x), (R)0.5 * (zm.y - zc.y)};
            if (2 * p + 1 < cnt) // (Z_m - conj(Z_{L-m}))/(2i)
                S[srow(2 * p + 1) + m] = C{(R)0.5 * (zm.y + zc.y), (R)0.5 * (zc.x - zm.x)};
        }
    }

    // ---- norm of psi' (imaginary time): deterministic two-level reduction --------
    if (MODE == GZ_IT_MID)
        norm_by_last_block(acc, a);
}

// ---------------------------------------------------------------------------
// The interface's pointwise steps
// ---------------------------------------------------------------------------
// One potential half step of psi in place, phi in memory: a thread per point.  Bound by DRAM
// on large grids, by the launch on small ones: 256 x 256 x 64 24.8 us, 4 x 4 x 1600 3.7 (6.4 as
// a pass over rows, a CTA per 32 of them: long rows leave most SMs idle).
template <class R>
__global__ void __launch_bounds__(256)
    g_half_step(cplx<R> *__restrict__ psi, const __grid_constant__ ZArgs a, int nz) {
    const unsigned q = blockIdx.x * 256u + threadIdx.x, row = q / (unsigned)nz, i = row / (unsigned)a.ny;
    const int j = (int)(row - i * a.ny), k = (int)(q - row * nz);
    if (i < 1 || (int)i >= a.nx - 1 || j < 1 || j >= a.ny - 1 || k < 1 || k >= nz - 1)
        return;
    const StepCoef c = a.step.coef[0];
    psi[q] = g_turn<R>(psi[q], reinterpret_cast<const R *>(a.V)[q], reinterpret_cast<const R *>(a.phi)[q], (R)a.cdd,
                       (R)a.half_dt, (R)c.g3w, (R)c.gw15);
}

// The Euler step from psi / sqrt(divisor) into `out`, phi in memory; the boundary takes the
// values last loaded.  Bound by DRAM on large grids.  Exactly the CTAs that are resident at once
// (6 an SM, 5 in complex128) walk through the points together, so that a plane's neighbours
// meet in the L2: 256 x 256 x 64 37.6 us, 47 with 8 an SM, 46 with a thread per point, 64 as a pass
// over rows; complex128 49, 56, 68 and 82.
template <class R> constexpr int g_euler_blocks() { return sizeof(R) == 4 ? 6 : 5; }
template <class R>
__global__ void __launch_bounds__(256, g_euler_blocks<R>())
    g_euler_step(const cplx<R> *__restrict__ psi, cplx<R> *__restrict__ out, const cplx<R> *__restrict__ bnd,
                 const R *__restrict__ V, const R *__restrict__ phi, const __grid_constant__ ZArgs a, int nz) {
    const StepCoef c      = a.step.coef[0];
    const R sc            = (R)(1.0 / sqrt(a.norm_state[1]));
    const ptrdiff_t plane = (ptrdiff_t)a.ny * nz;
    const unsigned n      = (unsigned)a.nx * a.ny * nz;
    for (unsigned q = blockIdx.x * 256u + threadIdx.x; q < n; q += gridDim.x * 256u) {
        const unsigned row = q / (unsigned)nz, i = row / (unsigned)a.ny;
        const int j = (int)(row - i * a.ny), k = (int)(q - row * nz);
        const bool in = i >= 1 && (int)i < a.nx - 1 && j >= 1 && j < a.ny - 1 && k >= 1 && k < nz - 1;
        out[q] = in ? g_euler<R>(psi + q, plane, nz, sc, V[q], phi[q], (R)a.cdd, (R)c.g3w, (R)c.gw15, (R)a.cx,
                                 (R)a.cy, (R)a.cz, (R)a.dtau)
                    : bnd[q];
    }
}

// The norm of psi, summed in the order of g_z's imaginary-time step (parts of 2^lb rows, row
// pairs, the same threads).  Bound by DRAM, and by the parts' sums where they are small; so a
// resident CTA takes several parts and one fence and ticket for all of them: 300 x 300 x 100
// 22.1 us, 512 x 512 x 8 16.6 (27.1 and 31.0 with a CTA and a ticket per part).
template <class R> constexpr int g_norm_blocks() { return sizeof(R) == 4 ? 6 : 5; }
template <class R>
__global__ void __launch_bounds__(256, g_norm_blocks<R>())
    g_norm(const cplx<R> *__restrict__ psi, const __grid_constant__ ZArgs a, int nz, unsigned mz, int lb) {
    using C         = cplx<R>;
    constexpr int U = 2; // pairs of loads in flight
    __shared__ double red[2][32];
    const int nt = blockDim.x, rows = a.nx * a.ny, parts = (rows + (1 << lb) - 1) >> lb;
    const int dp = g_div(nt, nz, mz), dk = nt - dp * nz; // items nt apart: row pairs, elements
    const int p0 = g_div(threadIdx.x, nz, mz);
    for (int part = blockIdx.x, odd = 0;; part += gridDim.x, odd ^= 1) {
        const int r0 = part << lb, cnt = min(1 << lb, rows - r0), n = ((cnt + 1) >> 1) * nz;
        const C *src = psi + (size_t)r0 * nz;
        double acc   = 0.0;
        int p = p0, k = threadIdx.x - p0 * nz; // row 2p and 2p + 1, element k
        while (p * nz + k < n) {
            C v[U][2];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const C *x = src + 2 * p * nz + k;
                v[u][0]    = 2 * p < cnt ? x[0] : C{(R)0, (R)0};
                v[u][1]    = 2 * p + 1 < cnt ? x[nz] : C{(R)0, (R)0};
                p += dp, k += dk;
                if (k >= nz)
                    k -= nz, ++p;
            }
#pragma unroll
            for (int u = 0; u < 2 * U; ++u) // (zeros change nothing)
                acc = add_rn(acc, g_abs2(double2{(double)v[u >> 1][u & 1].x, (double)v[u >> 1][u & 1].y}));
        }
        if (part + (int)gridDim.x >= parts) {
            norm_by_last_block(acc, a, part, parts);
            return;
        }
        const double sum = block_sum(acc, red[odd]);
        if (threadIdx.x == 0)
            a.partial[part] = sum;
    }
}

} // namespace gpe
