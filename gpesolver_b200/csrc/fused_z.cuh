// Z rows of the four-kernel schedule (grids whose y-z planes do not fit one SM).
//
// One CTA per 32 rows of an x plane: dipolar C2R (row pairs packed in one complex
// line of 2nz) -> V + cdd phi, kinetic iFFT(nz) + kept psi, the merged phase step, rho,
// FFT(nz) and R2C (imaginary time: the Euler stencil step in place of the
// kinetic transforms, with the norm).  The stages are those of the plane kernels
// (fused_yz.cuh): dipolar and kinetic lines side by side, the inverse z transform
// handing over to the phase and the forward one in registers, rho read by the R2C's
// first stage, inputs brought in by cp.async behind the transforms, twiddles staged in
// shared memory.
//
// Bound by instruction issue, then DRAM (218 MB an iteration at 256 x 256 x 64, 33
// us).  With a pass of its own over the tiles for the pair lines, phi, the phase and rho, and
// every bin of the spectrum read twice, it executed 472 instructions a point there: 90 us.
#pragma once

#include "fused_yz.cuh"

namespace gpe {

constexpr int kZRows = 32;

// Shared memory: K, RP (rows of complex, odd stride), DP (pair lines), FP, twiddles.
template <class R, int NZ> struct ZShape {
    using C                    = cplx<R>;
    using G                    = YZShape<R, kZRows, NZ>;
    static constexpr size_t K_B   = sizeof(C) * kZRows * G::PS;
    static constexpr size_t DP_B  = sizeof(C) * G::LD * G::TD;
    static constexpr size_t FP_B  = sizeof(R) * G::FPN;
    static constexpr size_t TW_B  = sizeof(C) * (G::LD + 2 * NZ);
    static constexpr size_t OFF_FP = DP_B, OFF_TW = OFF_FP + FP_B, OFF_K = OFF_TW + TW_B, OFF_RP = OFF_K + K_B;
    static_assert(FP_B % 16 == 0, "aligned tiles");
};
template <class R, int NZ> constexpr size_t z_smem() { return ZShape<R, NZ>::OFF_RP + ZShape<R, NZ>::K_B; }

template <class R, int NZ, int MODE>
__global__ void __launch_bounds__(256, 3) k2_z(ZArgs a, Twid tk, Twid td) {
    using C          = cplx<R>;
    using G          = YZShape<R, kZRows, NZ>;
    using Z          = ZShape<R, NZ>;
    constexpr int NT = 256, RW = kZRows, PS = G::PS, NP = G::NP, LD = G::LD, TD = G::TD;
    constexpr bool RT      = MODE <= ZM_RT_EPI;
    constexpr bool KEPT    = MODE == ZM_RT_MID || MODE == ZM_RT_EPI;
    constexpr bool HAS_INV = KEPT || MODE == ZM_IT_MID;
    using DW  = DipolarPlane<R, RW, NZ, NT, 0, true>;
    using C2R = PlanePass<+1, R, LD, NP, 1, TD, NT, false, true, false, true, 0, true>;
    using R2C = PlanePass<-1, R, LD, NP, 1, TD, NT, false, false, true, false, 0, true>;
    using ZI  = PlanePass<+1, R, NZ, RW, PS, 1, NT, true, false, false, false, 0, true>;
    using ZF  = PlanePass<-1, R, NZ, RW, PS, 1, NT, true, true, false, false, 0, true>;
    static_assert(ZI::Last::RADIX == ZF::First::RADIX && ZI::Last::ROUNDS == ZF::First::ROUNDS &&
                      ZI::Last::ITEMS == ZF::First::ITEMS,
                  "paired z transforms share the register layout");
    // short lines (nz = 8, 16: one stage, a thread per row) take the phase step from the
    // tile, a thread per point; longer ones from the transform's registers
    constexpr bool FLAT = ZI::Last::ITEMS < NT / 2;
    const int tid = threadIdx.x;
    const int nx = a.nx, ny = a.ny; // ny is a multiple of 32: a tile lies in one x plane
    const int r0 = blockIdx.x * RW, i = r0 / ny, j0 = r0 - i * ny;
    const size_t base = (size_t)r0 * NZ;

    C *DP = reinterpret_cast<C *>(g_smem);
    R *FP = reinterpret_cast<R *>(g_smem + Z::OFF_FP);
    C *dzt = reinterpret_cast<C *>(g_smem + Z::OFF_TW), *kzt = dzt + LD, *kzl = kzt + NZ;
    const C *dzl = nullptr; // the dipolar transforms apply plain twiddles
    C *K  = reinterpret_cast<C *>(g_smem + Z::OFF_K);
    C *RP = reinterpret_cast<C *>(g_smem + Z::OFF_RP);
    C *S_g       = reinterpret_cast<C *>(a.S) + ((size_t)i * 2 * ny + j0) * NZ;
    const R *V_g = reinterpret_cast<const R *>(a.V) + base;
    R *phi_g     = reinterpret_cast<R *>(a.phi) + base;
    const C *pin = reinterpret_cast<const C *>(a.psi_in) + base;
    C *pout      = reinterpret_cast<C *>(a.psi_out) + base;
    C *Pr_g      = reinterpret_cast<C *>(a.psi_r) + base;
    const R cdd  = (R)a.cdd;
    const bool xin = i >= 1 && i < nx - 1;

    // twiddles and the increment's rows, then V and the kept psi
    for (int e = tid; e < LD; e += NT)
        cp_async8(&dzt[e], reinterpret_cast<const C *>(td.tw) + e);
    if (RT && tid < 2 * NZ)
        cp_async8(&kzt[tid], reinterpret_cast<const C *>(tid < NZ ? tk.tw : tk.lo) + tid % NZ);
    if (KEPT)
        plane_in_async<C, RW, NZ, PS, NT>(K, pin, tid);
    cp_async_commit();
    if (MODE != ZM_IT_PRO) {
#pragma unroll 4
        for (int e = tid; e < RW * NZ; e += NT)
            cp_async4(&FP[G::fpi(e / NZ, e % NZ)], &V_g[e]);
    }
    if (KEPT)
        plane_in_async<C, RW, NZ, PS, NT>(RP, Pr_g, tid);
    cp_async_commit();
    // step coefficients (real time: the sum of two consecutive half steps in the middle)
    R g3, gw;
    {
        const int it      = RT ? *a.step.base + a.step.local : 0;
        const StepCoef c0 = a.step.coef[it];
        g3 = (R)c0.g3w, gw = (R)c0.gw15;
        if (MODE == ZM_RT_MID) {
            const StepCoef c1 = a.step.coef[it + 1];
            g3 = (R)(c0.g3w + c1.g3w), gw = (R)(c0.gw15 + c1.gw15);
        }
    }
    typename ZI::Last::Regs zr;
    if (HAS_INV) {
        // pair lines z[m] = X_a[m] + i X_b[m] over the full 2nz-point spectrum: bin 0 is
        // zero, bins > nz by symmetry; every bin is read once
#pragma unroll 4
        for (int e = tid; e < NP * NZ; e += NT) {
            const int p = e / NZ, m = e % NZ + 1;
            const C xa = S_g[(2 * p) * NZ + m - 1], xb = S_g[(2 * p + 1) * NZ + m - 1];
            if (m == NZ) {
                DP[p + m * TD] = C{xa.x, xb.x}; // self-conjugate bin: real parts only
                DP[p]          = C{(R)0, (R)0};
            } else {
                DP[p + m * TD]        = C{xa.x - xb.y, xa.y + xb.x};
                DP[p + (LD - m) * TD] = C{xa.x + xb.y, xb.x - xa.y};
            }
        }
        cp_async_wait<1>();
        __syncthreads();
        // C2R || kinetic iFFT_z, all stages but the last
        joint_stages<C2R, 0, C2R::NSTG - 1, ZI, 0, RT ? ZI::NSTG - 1 : 0>(DP, dzt, dzl, K, kzt, kzl, tid);
        typename C2R::Last::Regs ca;
        C2R::Last::read(DP, ca, dzt, dzl, tid);
        if (RT)
            ZI::Last::read(K, zr, kzt, kzl, tid);
        cp_async_wait<0>();
        __syncthreads(); // V
        if (RT && FLAT)
            ZI::Last::write(K, zr, tid);
#pragma unroll
        for (int rd = 0; rd < C2R::Last::ROUNDS; ++rd) {
            if (!C2R::Last::valid(rd * NT + tid))
                break;
            const int p = C2R::Last::line(tid, rd);
#pragma unroll
            for (int q = 0; q < C2R::Last::RADIX; ++q) {
                if (2 * q >= C2R::Last::RADIX) // pruned: z >= nz is not kept
                    continue;
                const int k = C2R::Last::elem(tid, rd, q);
                const C v   = ca[rd][q];
                if (MODE != ZM_RT_MID) { // read after a call's last iteration only
                    phi_g[(2 * p) * NZ + k]     = v.x;
                    phi_g[(2 * p + 1) * NZ + k] = v.y;
                }
                FP[G::fpi(2 * p, k)] += cdd * v.x;
                FP[G::fpi(2 * p + 1, k)] += cdd * v.y;
            }
        }
    } else {
        cp_async_wait<0>();
        if (RT) { // prologue: phi of the previous calc_fi3d (its own elements of V)
#pragma unroll 4
            for (int e = tid; e < RW * NZ; e += NT)
                FP[G::fpi(e / NZ, e % NZ)] += cdd * phi_g[e];
        }
    }
    __syncthreads(); // FP = V + cdd phi

    double acc = 0.0;
    const R wat = (R)a.w_atoms;
    if (RT) {
        // theta = -dt/2 [cV (V + cdd phi) + g3 |psi|^2 + gw |psi|^3]
        const R cV = MODE == ZM_RT_MID ? (R)2 : (R)1, hdt = (R)a.half_dt;
        auto phase = [&](C p, int y, int z) -> C {
            const int f = G::fpi(y, z);
            if (xin && j0 + y >= 1 && j0 + y < ny - 1 && z >= 1 && z < NZ - 1) {
                const R dens  = p.x * p.x + p.y * p.y;
                const R am    = sqrt(dens);
                const R total = cV * FP[f] + g3 * dens + gw * (am * am * am);
                R s, c;
                sincos_r<R>((R)-0.5 * hdt * total, &s, &c);
                p = apply_wm1(p, C{(R)-2 * s * s, (R)2 * s * c});
            }
            FP[f] = wat * (p.x * p.x + p.y * p.y); // rho for the next dipolar spectrum
            return p;
        };
        if (MODE == ZM_RT_PRO) {
            for (int e = tid; e < RW * NZ; e += NT) {
                const int r = e / NZ, k = e % NZ;
                const C v     = phase(pin[e], r, k);
                K[r * PS + k] = v;
                Pr_g[e]       = v;
            }
        } else if (FLAT) {
            for (int e = tid; e < RW * NZ; e += NT) {
                const int r = e / NZ, k = e % NZ;
                const C v = phase(cadd(K[r * PS + k], RP[r * PS + k]), r, k); // kept psi + increment
                K[r * PS + k] = RP[r * PS + k] = v;
            }
        } else {
#pragma unroll
            for (int rd = 0; rd < ZI::Last::ROUNDS; ++rd) {
                if (!ZI::Last::valid(rd * NT + tid))
                    break;
                const int y = ZI::Last::line(tid, rd);
#pragma unroll
                for (int q = 0; q < ZI::Last::RADIX; ++q) {
                    const int z    = ZI::Last::elem(tid, rd, q);
                    zr[rd][q]      = phase(cadd(zr[rd][q], RP[y * PS + z]), y, z); // kept psi + increment
                    RP[y * PS + z] = zr[rd][q];
                }
            }
        }
        __syncthreads(); // rho, and RP complete
        if (MODE == ZM_RT_EPI) {
            plane_out<R, RW, NZ, PS, NT>(pout, RP, tid);
            return;
        }
        if (MODE == ZM_RT_PRO) {
            for (int e = tid; e < NP * NZ; e += NT)
                DP[e / NZ + (e % NZ) * TD] = DW::rho_pair(FP, e / NZ, e % NZ);
            __syncthreads();
            joint_stages<R2C, 0, R2C::NSTG, ZF, 0, ZF::NSTG>(DP, dzt, dzl, K, kzt, kzl, tid);
        } else {
            plane_out<R, RW, NZ, PS, NT>(Pr_g, RP, tid); // kept psi for the next iteration
            // first FFT_z stage from the registers (or the tile) || first R2C stage from rho
            if (FLAT) {
                ZF::First::read(K, zr, kzt, kzl, tid);
                __syncthreads();
            } else {
#pragma unroll
                for (int rd = 0; rd < ZF::First::ROUNDS; ++rd) {
                    if (!ZF::First::valid(rd * NT + tid))
                        break;
                    DFT<ZF::First::RADIX, -1, R, true>::run(zr[rd]);
                }
            }
            ZF::First::write(K, zr, tid);
            {
                auto ldr = [&](int p, int m) { return DW::rho_pair(FP, p, m); };
                typename R2C::First::Regs ra;
                R2C::First::read_ld(ldr, ra, tid);
                R2C::First::write(DP, ra, tid);
            }
            __syncthreads();
            joint_stages<R2C, 1, R2C::NSTG, ZF, 1, ZF::NSTG>(DP, dzt, dzl, K, kzt, kzl, tid);
        }
        plane_out<R, RW, NZ, PS, NT>(pout, K, tid);
    } else {
        // imaginary time: psi_in / sqrt(divisor)
        const R sc             = (R)(1.0 / sqrt(a.norm_state[1]));
        const ptrdiff_t plane  = (ptrdiff_t)ny * NZ;
        const C *__restrict__ bnd = reinterpret_cast<const C *>(a.bnd) + base;
        const R cx = (R)a.cx, cy = (R)a.cy, cz = (R)a.cz, dtau = (R)a.dtau;
#pragma unroll 2
        for (int e = tid; e < RW * NZ; e += NT) {
            const int r = e / NZ, k = e % NZ, j = j0 + r;
            C o;
            if (MODE == ZM_IT_PRO) {
                o = pin[e];
            } else {
                if (!xin || j < 1 || j >= ny - 1 || k < 1 || k >= NZ - 1) {
                    o = bnd[e];
                } else {
                    const C c0 = cscale(pin[e], sc);
                    const C xm = cscale(pin[e - plane], sc), xp = cscale(pin[e + plane], sc);
                    const C ym = cscale(pin[e - NZ], sc), yp = cscale(pin[e + NZ], sc);
                    const C zm = cscale(pin[e - 1], sc), zp = cscale(pin[e + 1], sc);
                    const R vv   = FP[G::fpi(r, k)];
                    const R dens = c0.x * c0.x + c0.y * c0.y;
                    const R am   = sqrt(dens);
                    const R nl   = g3 * dens + gw * (am * am * am);
                    const R lr   = cx * ((xm.x + xp.x) - 2 * c0.x) - cy * ((ym.x + yp.x) - 2 * c0.x) -
                                 cz * ((zm.x + zp.x) - 2 * c0.x) + c0.x * vv + nl * c0.x;
                    const R li = cx * ((xm.y + xp.y) - 2 * c0.y) - cy * ((ym.y + yp.y) - 2 * c0.y) -
                                 cz * ((zm.y + zp.y) - 2 * c0.y) + c0.y * vv + nl * c0.y;
                    o = C{c0.x - dtau * lr, c0.y - dtau * li};
                }
                pout[e] = o;
                acc += (double)o.x * o.x + (double)o.y * o.y;
            }
            FP[G::fpi(r, k)] = wat * (o.x * o.x + o.y * o.y);
        }
        __syncthreads(); // rho
        auto ldr = [&](int p, int m) { return DW::rho_pair(FP, p, m); };
        typename R2C::First::Regs ra;
        R2C::First::read_ld(ldr, ra, tid);
        R2C::First::write(DP, ra, tid);
        __syncthreads();
        R2C::template stages<1, R2C::NSTG>(DP, dzt, dzl, tid);
    }
    // bins 1..nz of the rows
#pragma unroll 4
    for (int e = tid; e < RW * NZ; e += NT)
        S_g[e] = DW::rho_bin(DP, e / NZ, e % NZ + 1);
    if (MODE == ZM_IT_MID)
        norm_by_last_block(acc, a);
}

} // namespace gpe
