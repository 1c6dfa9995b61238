// gpe_calc_fi3d_noalloc: the dipolar potential without any device allocation.
//
// Some callers cannot call cudaMalloc: a host framework that owns all device
// memory through its own allocator (a caching allocator or a pre-reserved
// pool), or a time-critical loop that must not add the device-wide
// synchronisation cudaMalloc/cudaFree can cause.  For them this entry point
// computes phi = calc_fi3d(psi) (same kernels as the handle-based path) with
// every intermediate in one file-scope __device__ array of fixed size.  The
// caller passes device pointers to psi (complex64) and phi (float); nothing
// else is allocated, on the device or in pinned host memory.
//
// Limits and sharing:
//  * scratch holds the pruned dipolar spectrum (nx * 2ny * nz complex64, room for
//    nz+1 bins), the V_dd(k) table ((nx+1) * (ny+1) * nz floats, likewise) and three
//    twiddle tables with their rounding remainders; grids whose room exceeds
//    GPE_NOALLOC_SCRATCH_BYTES are rejected with GPE_ERR_SIZE (128 x 128 x 32 takes about
//    10.9 MB).  The kz = 0 bin is not stored; its room keeps the limit where callers know it;
//   * the array lives on every GPU that loads the library until the process
//    exits, and every call on a GPU shares it: calls that overlap on that GPU
//    (other streams, other threads) race.  Every call rebuilds the twiddle and
//    V_dd(k) tables it needs before its passes (a few microseconds): no state
//    carries over from one call to the next, whatever stream or grid the
//    previous call used;
//  * the first call on each device does a one-time set-up on the host (looks
//    up the array's device address with cudaGetSymbolAddress and raises the
//    kernels' shared-memory limit to the device's opt-in maximum); make that
//    first call before any stream capture on that device.
#include "../../include/gpe_b200.h"
#include "general_plan.hpp"

#include <cuda_runtime.h>

#include <cstring>
#include <mutex>
#include <string>

namespace gpe {
namespace {

static __device__ __align__(256) unsigned char g_noalloc_scratch[GPE_NOALLOC_SCRATCH_BYTES];

constexpr int kMaxDevices = 64;

struct NoallocSlot {
    bool ready          = false;
    unsigned char *base = nullptr; // device address of g_noalloc_scratch
    size_t smem_max     = 0;       // dynamic shared memory the kernels may use on this device
};

std::mutex g_noalloc_mu;
NoallocSlot g_noalloc_slots[kMaxDevices];

size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

// The tables of a grid in one launch: twiddles exp(-2 pi i m / L) of the three
// doubled axes (FP64, hi rounded to float and lo the rounding remainder) and V_dd(k) =
// kz^2 / k^2 on the (2nx, 2ny, 2nz) box for kz = 1..nz, reduced by |kx|, |ky| symmetry
// (fftw_poisson_solver.cpp:12-49), FP64 then rounded to float.
__global__ void k_na_tables(float4 *twx, float4 *twy, float4 *twz, float *vk, int nx, int ny, int nz, double dx,
                            double dy, double dz) {
    const int first = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    auto tw = [&](float4 *t, int L) {
        for (int m = first; m < L; m += step) {
            double s, c;
            sincospi(2.0 * (double)m / (double)L, &s, &c);
            const float ch = (float)c, sh = (float)-s;
            t[m]           = make_float4(ch, sh, (float)(c - (double)ch), (float)(-s - (double)sh));
        }
    };
    tw(twx, 2 * nx);
    tw(twy, 2 * ny);
    tw(twz, 2 * nz);
    const int px = 2 * nx, py = 2 * ny, pz = 2 * nz;
    const double dkx = 2. * M_PI / (px * dx), dky = 2. * M_PI / (py * dy), dkz = 2. * M_PI / (pz * dz);
    const size_t total = (size_t)(nx + 1) * (ny + 1) * nz;
    for (size_t q = first; q < total; q += step) {
        const unsigned r = (unsigned)(q / nz);
        const int k = (int)(q - (size_t)r * nz) + 1, i = (int)(r / (ny + 1)), j = (int)(r - (unsigned)i * (ny + 1));
        const double kx = i * dkx, ky = j * dky, kz = k * dkz;
        const double k2 = __dadd_rn(__dadd_rn(__dmul_rn(kx, kx), __dmul_rn(ky, ky)), __dmul_rn(kz, kz));
        vk[q]           = (k2 > 1e-30) ? (float)__ddiv_rn(__dmul_rn(kz, kz), k2) : 0.0f;
    }
}

struct Layout {
    size_t a_off, vk_off, twx_off, twy_off, twz_off, total;
    // twiddle regions: (hi, lo) pairs
};

Layout layout(int nx, int ny, int nz) {
    Layout l{};
    const int H = nz + 1; // the limit's count of bins, one more than is stored
    size_t off = 0;
    l.a_off    = off;
    off += align256(sizeof(float2) * (size_t)nx * 2 * ny * H);
    l.vk_off = off;
    off += align256(sizeof(float) * (size_t)(nx + 1) * (ny + 1) * H);
    l.twx_off = off;
    off += align256(sizeof(float2) * 2 * 2 * (size_t)nx);
    l.twy_off = off;
    off += align256(sizeof(float2) * 2 * 2 * (size_t)ny);
    l.twz_off = off;
    off += align256(sizeof(float2) * 2 * 2 * (size_t)nz);
    l.total = off;
    return l;
}

int fail(int code, const std::string &msg) {
    last_error() = msg;
    return code;
}

} // namespace
} // namespace gpe

extern "C" int gpe_calc_fi3d_noalloc(const void *psi_c64_dev, float *fi3d_dev, int nx, int ny, int nz,
                                     double dx, double dy, double dz, double n_atoms,
                                     void *cuda_stream) {
    using namespace gpe;
    if (!psi_c64_dev || !fi3d_dev)
        return fail(GPE_ERR_ARG, "gpe_calc_fi3d_noalloc: null device pointer");
    if (nx < 1 || ny < 1 || nz < 1 || !(dx > 0) || !(dy > 0) || !(dz > 0))
        return fail(GPE_ERR_ARG, "gpe_calc_fi3d_noalloc: grid dimensions and spacings must be positive");
    const Layout lay = layout(nx, ny, nz);
    if (lay.total > (size_t)GPE_NOALLOC_SCRATCH_BYTES)
        return fail(GPE_ERR_SIZE, "gpe_calc_fi3d_noalloc: a " + std::to_string(nx) + "x" +
                                      std::to_string(ny) + "x" + std::to_string(nz) + " grid needs " +
                                      std::to_string(lay.total) + " bytes of scratch, above the " +
                                      std::to_string((size_t)GPE_NOALLOC_SCRATCH_BYTES) +
                                      "-byte limit");
    GPlan lx, ly, lz;
    GShape sh;
    try {
        for (int n : {nx, ny, nz})
            factor_line(2 * n); // rejects unsupported lengths
        lx = g_plan(2 * nx, nullptr);
        ly = g_plan(2 * ny, nullptr);
        lz = g_plan(2 * nz, nullptr);
        sh = g_shape<float>(nx, ny, nz, false);
    } catch (const Error &e) {
        return fail(e.code, std::string("gpe_calc_fi3d_noalloc: ") + e.what());
    }
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess)
        return fail(GPE_ERR_CUDA, std::string("cudaGetDevice: ") + cudaGetErrorString(err));
    if (dev < 0 || dev >= kMaxDevices)
        return fail(GPE_ERR_ARG, "gpe_calc_fi3d_noalloc: device ordinal out of range");
    cudaStream_t s = (cudaStream_t)cuda_stream;

    NoallocSlot &slot = g_noalloc_slots[dev];
    {
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!slot.ready) {
            // One-time set-up on this device: the host-side name of the array is
            // not its device address, so look the address up.
            void *p = nullptr;
            err     = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (err != cudaSuccess)
                return fail(GPE_ERR_CUDA, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(err));
            int optin = 0;
            err       = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
            if (err != cudaSuccess)
                return fail(GPE_ERR_CUDA, std::string("cudaDeviceGetAttribute: ") + cudaGetErrorString(err));
            const void *kern[] = {(const void *)g_z<float, GZ_IT_PRO>, (const void *)g_z<float, GZ_DIP_INV>,
                                  (const void *)g_y<float, 2>, (const void *)g_y<float, 3>,
                                  (const void *)g_x<float, 2>, (const void *)g_x<float, 3>};
            int fixed = 0; // the most that a kernel holds statically
            for (const void *f : kern) {
                cudaFuncAttributes fa{};
                err = cudaFuncGetAttributes(&fa, f);
                if (err == cudaSuccess)
                    err = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               optin - (int)fa.sharedSizeBytes);
                if (err != cudaSuccess)
                    return fail(GPE_ERR_CUDA, std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(err));
                fixed = std::max(fixed, (int)fa.sharedSizeBytes);
            }
            slot.base     = static_cast<unsigned char *>(p);
            slot.smem_max = (size_t)(optin - fixed);
            slot.ready    = true;
        }
    }
    if (std::max({sh.smx, sh.smy, sh.smz}) > slot.smem_max)
        return fail(GPE_ERR_SIZE, "gpe_calc_fi3d_noalloc: the line tiles of this grid need more shared memory "
                                  "than the device allows per block");
    // An error left by earlier, unrelated work would be reported as this call's:
    // refuse to start instead (the error stays pending for its owner).
    err = cudaPeekAtLastError();
    if (err != cudaSuccess)
        return fail(GPE_ERR_CUDA, std::string("gpe_calc_fi3d_noalloc: a CUDA error from earlier work is pending: ") +
                                      cudaGetErrorString(err));
    unsigned char *base = slot.base;
    float2 *S           = reinterpret_cast<float2 *>(base + lay.a_off);
    float *vk           = reinterpret_cast<float *>(base + lay.vk_off);
    float4 *twx         = reinterpret_cast<float4 *>(base + lay.twx_off);
    float4 *twy         = reinterpret_cast<float4 *>(base + lay.twy_off);
    float4 *twz         = reinterpret_cast<float4 *>(base + lay.twz_off);
    lx.tw = twx, ly.tw = twy, lz.tw = twz;

    // the tables of this grid, rebuilt by every call (in stream order before the
    // passes that read them)
    k_na_tables<<<592, 256, 0, s>>>(twx, twy, twz, vk, nx, ny, nz, dx, dy, dz);
    // The pruned dipolar convolution (general.cuh): every element of S that a pass
    // reads was written by the pass before it in this call, so nothing needs clearing.
    GZArgs z{};
    z.z.psi_in  = const_cast<void *>(psi_c64_dev);
    z.z.S       = S;
    z.z.phi     = fi3d_dev;
    z.z.w_atoms = n_atoms;
    z.z.nx = nx, z.z.ny = ny;
    z.nz = nz, z.mz = g_magic(nz), z.lb = sh.lbz, z.buf = sh.buf;
    z.d = lz;
    GYArgs y{};
    y.S = S, y.ny = ny, y.nz = nz, y.lb = sh.lby, y.d = ly;
    GXArgs x{};
    x.S = S, x.vk = vk, x.dip_scale = 1.0 / (8.0 * (double)nx * ny * nz);
    x.nx = nx, x.ny = ny, x.nz = nz, x.lb = sh.lbx, x.d = lx;
    const int wx = 1 << sh.lbx, zt = (nx * ny + (1 << sh.lbz) - 1) >> sh.lbz;
    const dim3 yt((nz + (1 << sh.lby) - 1) >> sh.lby, nx);
    g_z<float, GZ_IT_PRO><<<zt, sh.ntz, sh.smz, s>>>(z);
    g_with_y<float>(sh.mby, [&](auto k) { k<<<yt, sh.nty, sh.smy, s>>>(y); });
    g_with_x<float>(sh.mbx, [&](auto k) { k<<<(2 * ny * nz + wx - 1) / wx, sh.ntx, sh.smx, s>>>(x); });
    y.inverse = 1;
    g_with_y<float>(sh.mby, [&](auto k) { k<<<yt, sh.nty, sh.smy, s>>>(y); });
    g_z<float, GZ_DIP_INV><<<zt, sh.ntz, sh.smz, s>>>(z);
    err = cudaGetLastError();
    if (err != cudaSuccess)
        return fail(GPE_ERR_CUDA, std::string("gpe_calc_fi3d_noalloc launch: ") + cudaGetErrorString(err));
    return GPE_OK;
}
