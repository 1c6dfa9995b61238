// Fused iteration pipeline (compile-time line lengths).
//
// One imaginary- or real-time iteration is four kernels, each a batch of 1D
// FFT lines along one axis with the elementwise physics fused into its loads
// and stores:
//
//   X  pencils along x: kinetic  fwd FFT(nx) * (exp(i(-dt/2m)k^2) - 1)/N * inv FFT(nx)
//                       dipolar  fwd FFT(2nx, upper half zero) * V_dd(k) * scale
//                                * inv FFT(2nx), first nx kept
//   Yi lines along y, inverse:   kinetic iFFT(ny); dipolar iFFT(2ny), first ny kept
//   Z  rows along z:   dipolar C2R (pairs of rows packed in one complex FFT of
//                      2nz) -> phi; kinetic iFFT(nz) -> the kinetic increment,
//                      added to the kept real-space psi (psi_r); the real-time phases
//                      of two consecutive half steps merged into one rotation
//                      (they see the same |psi|, V and phi); rho = w|psi|^2;
//                      kinetic FFT(nz); dipolar R2C (pairs) -> spectrum
//                      (imaginary time: the Euler stencil update instead of the
//                      kinetic transforms, with the norm reduced on the fly)
//   Yf lines along y, forward:   kinetic FFT(ny); dipolar FFT(2ny, upper half zero)
//
// Dipolar spectrum layout: S[i][ky][kz-1], i < nx (x in real space between the
// X passes), ky < 2ny, 1 <= kz <= nz.  The kz = 0 plane is not stored: V_dd is
// kz^2/k^2, exactly 0 on that plane (fftw_poisson_solver.cpp:39-45), so it adds
// nothing to phi.
#pragma once

#include "ct_fft.cuh"
#include "kernels.cuh"
#include "rfft.cuh"

namespace gpe {

struct Twid {
    const void *tw;
    const void *lo;
};

enum { ZM_RT_PRO = 0, ZM_RT_MID, ZM_RT_EPI, ZM_IT_PRO, ZM_IT_MID };

// Asynchronous global -> shared copies (cp.async, completion per thread; a
// barrier after the wait makes the data visible to the block).
__device__ __forceinline__ void cp_async8(void *smem, const void *g) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *g) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// wait until at most N of this thread's committed groups are pending
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One-dimensional bulk copies (global -> this CTA's shared memory) completing
// on an mbarrier: one thread arms the barrier with the byte count and issues
// the copies, every thread waits for the barrier's phase.  Addresses and sizes
// must be multiples of 16 bytes.  No multicast: each CTA copies into its own
// shared memory.
__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
    // make the initialised barrier visible to the async proxy (the bulk copies)
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_g2s(void *smem, const void *g, unsigned bytes, unsigned long long *bar) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const unsigned b = (unsigned)__cvta_generic_to_shared(bar);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(s),
                 "l"(g), "r"(bytes), "r"(b)
                 : "memory");
}
// Waits for phase `parity` of the barrier, at most `tries` polls (each poll may
// suspend the thread for a while); false when it gave up.
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity, int tries) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
    for (int t = 0; t < tries; ++t) {
        unsigned done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(a), "r"(parity)
                     : "memory");
        if (done)
            return true;
    }
    return false;
}


// ---------------------------------------------------------------------------
// X pencils
// ---------------------------------------------------------------------------
// Lines per CTA of the x passes: 8 or 16 (64 / 128-byte row segments per x),
// picked per grid by the solver's autotuner (Solver::autotune_x).

// Kinetic x pencils, increment form: psi(x, ky, kz) -> FFT_x ->
// (exp(i(-dt/2m)k^2) - 1) / N -> iFFT_x, i.e. the change the kinetic step makes
// to psi, which the z / plane kernel adds to the real-space psi it kept from the
// previous phase step (ZArgs::psi_r).  In exact arithmetic this is the kinetic
// step itself; in FP32 the rounding of the transforms scales with |e^{i theta} -
// 1| instead of with |psi|, so the per-step error is about one rounding of the
// sum instead of that of a forward and an inverse 3D FFT.  The forward transform
// ends and the inverse one starts in registers, with the factor applied in
// between.
template <class R, int NX, int CNT, int NT>
__global__ void __launch_bounds__(NT)
    k3_x_kin(cplx<R> *__restrict__ psi, const cplx<R> *__restrict__ ex, const cplx<R> *__restrict__ ey,
             const cplx<R> *__restrict__ ez, R inv_hi, R inv_lo, int ny, int nz, Twid tk) {
    using C  = cplx<R>;
    using Fw = LinePass<-1, R, NX, CNT, CNT, NT, true, false>;
    using Iv = LinePass<+1, R, NX, CNT, CNT, NT, true, true>;
    static_assert(Fw::RL == Iv::R0 && Fw::ROUNDSL == Iv::ROUNDS0 && Fw::ITEMSL == Iv::ITEMS0,
                  "paired transforms share the register layout");
    const int tid  = threadIdx.x;
    C *buf         = reinterpret_cast<C *>(g_smem);
    const C *tw    = (const C *)tk.tw, *tl = (const C *)tk.lo;
    const int cols = ny * nz;
    const int c0   = blockIdx.x * CNT;
    const int cnt  = min(CNT, cols - c0);
    // the line's (1+wy)(1+wz) - 1, read before the transform so that its L2
    // reads land behind the line loads
    const int b = Fw::line_of(tid);
    C wyz       = C{(R)0, (R)0};
    if (b < cnt) {
        const int c = c0 + b, j = c / nz, k = c - j * nz;
        const C wy = __ldg(&ey[j]), wz = __ldg(&ez[k]);
        wyz        = cadd(cadd(wy, wz), cmul(wy, wz));
    }
    C a[Fw::ROUNDSL][Fw::RL];
    Fw::run_to_regs(
        buf, [&](int b, int t) { return b < cnt ? psi[(size_t)t * cols + c0 + b] : C{(R)0, (R)0}; }, a, tw, tl,
        tid);
    {
#pragma unroll
        for (int rd = 0; rd < Fw::ROUNDSL; ++rd) {
            if (!Fw::template valid<Fw::ITEMSL>(rd * NT + tid))
                break;
#pragma unroll
            for (int q = 0; q < Fw::RL; ++q) {
                const C wx = __ldg(&ex[Fw::last_index(tid, rd, q)]);
                const C w  = cadd(cadd(wx, wyz), cmul(wx, wyz)); // (1+wx)(1+wyz) - 1
                const C v  = cmul(a[rd][q], w);
                a[rd][q]   = C{fma(v.x, inv_hi, v.x * inv_lo), fma(v.y, inv_hi, v.y * inv_lo)};
            }
        }
    }
    __syncthreads();
    Iv::run_from_regs(
        buf, a,
        [&](int b, int t, C v) {
            if (b < cnt)
                psi[(size_t)t * cols + c0 + b] = v;
        },
        tw, tl, tid);
}

// Dipolar x pencils: S(x, ky, kz) -> FFT_2nx (upper half zero) -> V_dd(k) * scale
// -> iFFT_2nx, lower half kept.  scale = 1/(8N) (C2R normalisation) and, in
// imaginary time, 1/xnorma (the spectrum was built from the unnormalised psi).
// The twiddle table and the V_dd(k) values of the CTA's lines (|kx| = 0..nx) are
// copied into shared memory (cp.async) at kernel start, behind the forward
// transform's global loads, instead of being gathered from L2 after it.
template <class R, int NX, int CNT> constexpr size_t x_dip_smem() {
    return sizeof(cplx<R>) * (CNT * 2 * NX + 2 * NX) + sizeof(R) * (NX + 1) * CNT;
}

template <class R, int NX, int CNT, int NT>
__global__ void __launch_bounds__(NT, NX >= 256 ? 2 : 3) // 512-point lines: two CTAs per SM; 256: three
    k3_x_dip(cplx<R> *__restrict__ S, const R *__restrict__ vk, const double *__restrict__ divisor,
             double dip_scale, int ny, int nz, Twid td) {
    using C          = cplx<R>;
    constexpr int L  = 2 * NX;
    // two-stage lines (radix pairs) take their twiddles from the shared copy;
    // longer radix chains (nx = 96) keep the global table in the middle stages
    constexpr bool TW2 = radices_of(L).n == 2;
    using Fw         = LinePass<-1, R, L, CNT, CNT, NT, false, false, true, false, TW2>;
    using Iv         = LinePass<+1, R, L, CNT, CNT, NT, false, true, false, true, TW2>;
    static_assert(Fw::RL == Iv::R0 && Fw::ROUNDSL == Iv::ROUNDS0 && Fw::ITEMSL == Iv::ITEMS0,
                  "paired transforms share the register layout");
    const int tid  = threadIdx.x;
    C *buf         = reinterpret_cast<C *>(g_smem);
    C *tws         = buf + CNT * L;                    // twiddles exp(-2 pi i m / L)
    R *vs          = reinterpret_cast<R *>(tws + L);   // V_dd of |kx| = 0..NX, line b: vs[|kx| CNT + b]
    const C *tw    = (const C *)td.tw;
    const C *twu   = TW2 ? tws : tw;                   // the table the stages read
    const int cols = 2 * ny * nz;
    const int c0   = blockIdx.x * CNT;
    const int cnt  = min(CNT, cols - c0);
    const size_t xs = (size_t)(ny + 1) * nz;
    for (int m = tid; m < L; m += NT)
        cp_async8(&tws[m], &tw[m]);
    for (int e = tid; e < (NX + 1) * CNT; e += NT) {
        const int ix = e / CNT, b = e - ix * CNT;
        const int c  = min(c0 + b, cols - 1);
        const int ky = c / nz, kz = c - ky * nz;
        const int iy = ky <= ny ? ky : 2 * ny - ky;
        cp_async4(&vs[e], &vk[(size_t)ix * xs + (size_t)iy * nz + kz]);
    }
    cp_async_commit();
    // the spectrum's scale (imaginary time: over the norm of the psi it was
    // built from), read before the transform
    const R scale = (R)(divisor ? dip_scale / divisor[0] : dip_scale);
    auto ld = [&](int b, int t) { return b < cnt ? S[(size_t)t * cols + c0 + b] : C{(R)0, (R)0}; };
    C a[Fw::ROUNDSL][Fw::RL];
    Fw::stage0_to_tile(buf, ld, tid);
    cp_async_wait<0>();
    __syncthreads();
    Fw::template middle<1>(buf, twu, nullptr, tid);
#pragma unroll
    for (int rd = 0; rd < Fw::ROUNDSL; ++rd) {
        const int it = rd * NT + tid;
        if (!Fw::template valid<Fw::ITEMSL>(it))
            break;
        const int j = it / CNT, b = it - j * CNT;
        Fw::loadL(buf, a[rd], j, b, twu, nullptr);
    }
    {
        const int b   = Fw::line_of(tid);
#pragma unroll
        for (int rd = 0; rd < Fw::ROUNDSL; ++rd) {
            if (!Fw::template valid<Fw::ITEMSL>(rd * NT + tid))
                break;
#pragma unroll
            for (int q = 0; q < Fw::RL; ++q) {
                const int t  = Fw::last_index(tid, rd, q);
                const int ix = t <= NX ? t : L - t;
                a[rd][q]     = cscale(a[rd][q], vs[ix * CNT + b] * scale);
            }
        }
    }
    __syncthreads();
    Iv::run_from_regs(
        buf, a,
        [&](int b, int t, C v) {
            if (b < cnt)
                S[(size_t)t * cols + c0 + b] = v;
        },
        twu, nullptr, tid);
}

// Dipolar x pencils of 2nx = 512 points as two transforms of nx = 256 each: the even
// bins are FFT_nx(S), the odd ones FFT_nx(S w^x), w = exp(-2 pi i / 2nx), and the kept
// half of the inverse is iFFT_nx(even) + w^-x iFFT_nx(odd).  256 points are two stages of
// radix 16 where 512 were three of radix 8: fewer synchronisations, and one butterfly a
// thread needs 32 registers for its points instead of 64.  The instructions stay (46.4 ->
// 46.1 M): the second half's twiddles and the sums take what the third stage gave back.  A
// tile holds CNT even and CNT odd lines; both of a column lie in one warp, read the same
// addresses and are added by a shuffle.
// Bound by instruction issue (62%).  256 x 256 x 64: 79 -> 72 us, the iteration 253 ->
// 248 us (2%) against k3_x_dip with 8 lines, 267 against its 16 (spilled).  16 lines spill here
// too (248 bytes); the autotuner times both widths.
template <class R, int NX, int CNT> constexpr size_t x_dip_eo_smem() {
    return sizeof(cplx<R>) * (2 * CNT * NX + 3 * NX) + sizeof(R) * (NX + 1) * CNT;
}

template <class R, int NX, int CNT>
__global__ void __launch_bounds__(CNT * NX / 8, CNT == 8 ? 3 : 1)
    k3_x_dip_eo(cplx<R> *__restrict__ S, const R *__restrict__ vk, const double *__restrict__ divisor,
                double dip_scale, int ny, int nz, Twid td, Twid tk) {
    using C          = cplx<R>;
    constexpr int NT = CNT * NX / 8, LN = 2 * CNT, L = 2 * NX;
    using Fw = LinePass<-1, R, NX, LN, LN, NT, false, false, false, false, true>;
    using Iv = LinePass<+1, R, NX, LN, LN, NT, false, true, false, false, true>;
    static_assert(Fw::NSTG == 2 && Fw::RL == Iv::R0 && Fw::ROUNDSL == 1 && Fw::ROUNDS0 == 1 && Fw::ITEMS0 == NT &&
                      Fw::ITEMSL == NT && 32 % LN == 0,
                  "one butterfly a thread, both lines of a column in one warp");
    const int tid  = threadIdx.x;
    C *buf         = reinterpret_cast<C *>(g_smem);
    C *w2          = buf + LN * NX;                  // exp(-2 pi i m / 2nx), m < 2nx
    C *tws         = w2 + L;                         // exp(-2 pi i m / nx)
    R *vs          = reinterpret_cast<R *>(tws + NX); // V_dd of |kx| = 0..NX, column b: vs[|kx| CNT + b]
    const int cols = 2 * ny * nz;
    const int c0   = blockIdx.x * CNT;
    const int cnt  = min(CNT, cols - c0);
    const size_t xs = (size_t)(ny + 1) * nz;
    // w2 is read by the first stage's loader: its own group, waited for there
    for (int m = tid; m < L; m += NT)
        cp_async8(&w2[m], reinterpret_cast<const C *>(td.tw) + m);
    cp_async_commit();
    for (int m = tid; m < NX; m += NT)
        cp_async8(&tws[m], reinterpret_cast<const C *>(tk.tw) + m);
    for (int e = tid; e < (NX + 1) * CNT; e += NT) {
        const int ix = e / CNT, b = e - ix * CNT;
        const int c  = min(c0 + b, cols - 1);
        const int ky = c / nz, kz = c - ky * nz;
        const int iy = ky <= ny ? ky : 2 * ny - ky;
        cp_async4(&vs[e], &vk[(size_t)ix * xs + (size_t)iy * nz + kz]);
    }
    cp_async_commit();
    const R scale = (R)(divisor ? dip_scale / divisor[0] : dip_scale);
    const int j = tid / LN, b2 = tid - j * LN, b = b2 % CNT, odd = b2 / CNT;
    C a[1][Fw::R0];
#pragma unroll
    for (int k = 0; k < Fw::R0; ++k)
        a[0][k] = b < cnt ? S[(size_t)(j + k * Fw::NR0) * cols + c0 + b] : C{(R)0, (R)0};
    cp_async_wait<1>();
    __syncthreads();
    if (odd) {
#pragma unroll
        for (int k = 0; k < Fw::R0; ++k)
            a[0][k] = cmul(a[0][k], w2[j + k * Fw::NR0]);
    }
    DFT<Fw::R0, -1, R, false>::run(a[0]);
    Fw::store0(buf, a[0], j, b2);
    cp_async_wait<0>();
    __syncthreads();
    Fw::loadL(buf, a[0], j, b2, tws, nullptr);
#pragma unroll
    for (int q = 0; q < Fw::RL; ++q) {
        const int t  = 2 * (j + q * Fw::NSL) + odd; // bin of the 2nx points
        const int ix = 2 * q < Fw::RL ? t : L - t;
        a[0][q]      = cscale(a[0][q], vs[ix * CNT + b] * scale);
    }
    __syncthreads();
    DFT<Iv::R0, +1, R, false>::run(a[0]);
    Iv::store0(buf, a[0], j, b2);
    __syncthreads();
    Iv::loadL(buf, a[0], j, b2, tws, nullptr);
#pragma unroll
    for (int q = 0; q < Iv::RL; ++q) {
        const int t = j + q * Iv::NSL;
        C v         = a[0][q];
        if (odd)
            v = cmulc(v, w2[t]);
        const C o{__shfl_xor_sync(0xffffffffu, v.x, CNT), __shfl_xor_sync(0xffffffffu, v.y, CNT)};
        if (b < cnt && odd == (q & 1)) // the two lanes of a column share its stores
            S[(size_t)t * cols + c0 + b] = cadd(v, o);
    }
}

// ---------------------------------------------------------------------------
// Y lines (one x plane per blockIdx.y; z-column tiles along blockIdx.x)
// ---------------------------------------------------------------------------
template <class R, int NY, int SIGN, int CNT, int NT>
__global__ void __launch_bounds__(NT) k3_y_kin(cplx<R> *__restrict__ psi, int nz, Twid tk) {
    using C       = cplx<R>;
    using P       = LinePass<SIGN, R, NY, CNT, CNT, NT, true, false>;
    const int k0  = blockIdx.x * CNT;
    const int cnt = min(CNT, nz - k0);
    C *plane      = psi + (size_t)blockIdx.y * NY * nz + k0;
    P::run(
        reinterpret_cast<C *>(g_smem),
        [&](int b, int t) { return b < cnt ? plane[(size_t)t * nz + b] : C{(R)0, (R)0}; },
        [&](int b, int t, C v) {
            if (b < cnt)
                plane[(size_t)t * nz + b] = v;
        },
        (const C *)tk.tw, (const C *)tk.lo, threadIdx.x);
}

// Dipolar y lines of length 2ny: forward (SIGN < 0) with the upper half of the
// input zero, inverse (SIGN > 0) with only the lower half of the output kept.
template <class R, int NY, int SIGN, int CNT, int NT>
__global__ void __launch_bounds__(NT) k3_y_dip(cplx<R> *__restrict__ S, int nz, Twid td) {
    using C         = cplx<R>;
    constexpr int L = 2 * NY;
    using P         = LinePass<SIGN, R, L, CNT, CNT, NT, false, (SIGN > 0), (SIGN < 0), (SIGN > 0)>;
    const int k0    = blockIdx.x * CNT;
    const int cnt   = min(CNT, nz - k0);
    C *plane        = S + (size_t)blockIdx.y * L * nz + k0;
    P::run(
        reinterpret_cast<C *>(g_smem),
        [&](int b, int t) { return b < cnt ? plane[(size_t)t * nz + b] : C{(R)0, (R)0}; },
        [&](int b, int t, C v) {
            if (b < cnt)
                plane[(size_t)t * nz + b] = v;
        },
        (const C *)td.tw, (const C *)td.lo, threadIdx.x);
}

// Shared memory of the x / y passes (one tile of COUNT lines).
template <class R, int L, int CNT> constexpr size_t xy_smem() { return sizeof(cplx<R>) * CNT * L; }

// y pass for ny = N with CNT z columns per tile.
template <class R, int N, int CNT> struct YShape {
    static constexpr int NTK = pass_threads<N, CNT>(), NTD = pass_threads<2 * N, CNT>();
    static constexpr size_t SK = xy_smem<R, N, CNT>(), SD = xy_smem<R, 2 * N, CNT>();
};

} // namespace gpe
