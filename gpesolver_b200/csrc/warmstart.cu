// Learned warm start for imaginary time: a small network maps the physical
// parameters (edd, n_atoms, omega_r, omega_z) to a ground-state amplitude
// |psi_0| on the solver grid; imaginary time then refines that guess instead of
// starting from a Gaussian.  The reference has no counterpart (it always starts
// from its initialisers); plain Gaussian-start imaginary time stays the
// fallback and the reference answer the prediction is measured against.
//
// Network (weights BF16, arithmetic FP32):
//   dense 4 -> H, SiLU;  dense H -> C0 * X0 * Y0 * Z0 (the latent volume), SiLU
//   `levels` stages of: nearest-neighbour upsampling x2 in x, y, z, 3x3x3
//   convolution (zero padding) C_s -> C_{s+1}, SiLU
//   a last 3x3x3 convolution C_L -> 1 at full resolution: the amplitude
//   (linear: a saturating output such as softplus stalls at zero, where the
//   targets are zero over most of the box)
// Volumes are [channel][x][y][z] with z fastest, the solver's layout.
//
// Training minimises the mean squared amplitude error against ground states
// that imaginary time produced, with Adam on FP32 master weights; the BF16
// copies are refreshed after every step.  All of it is memory- and
// latency-bound (few channels, large volumes): the kernels are plain SIMT with
// FP32 accumulation, and none of the products is a dense contraction worth a
// tensor-core tile.
#include "../../include/gpe_b200.h"
#include "plan.hpp"

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <memory>
#include <random>
#include <type_traits>
#include <string>
#include <vector>

namespace gpe {
namespace {

#define WS_CUDA(call)                                                                              \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            throw Error(e_ == cudaErrorMemoryAllocation ? GPE_ERR_NOMEM : GPE_ERR_CUDA,            \
                        std::string(#call) + ": " + cudaGetErrorString(e_));                      \
    } while (0)

template <class T> struct Buf {
    T *p     = nullptr;
    size_t n = 0;
    void alloc(size_t k) {
        if (p)
            cudaFree(p);
        p = nullptr;
        n = k;
        if (k)
            WS_CUDA(cudaMalloc(&p, sizeof(T) * k));
    }
    ~Buf() {
        if (p)
            cudaFree(p);
    }
};

__device__ __forceinline__ float silu(float y) { return y / (1.f + __expf(-y)); }
__device__ __forceinline__ float silu_grad(float y) {
    const float s = 1.f / (1.f + __expf(-y));
    return s * (1.f + y * (1.f - s));
}

// ---------------------------------------------------------------------------
// dense layers: Y[b][o] = sum_i W[o][i] X[b][i] + bias[o]
// ---------------------------------------------------------------------------
// One warp per output row: the row is read once, coalesced, for up to eight
// samples at a time (one thread per output walked its row alone: 25 us for 4096 x
// 256, now bound by the 2 MB of weights and the launch).
__global__ void __launch_bounds__(128)
    k_dense_fwd(const float *__restrict__ X, const __nv_bfloat16 *__restrict__ W,
                const __nv_bfloat16 *__restrict__ bias, float *__restrict__ Ypre, float *__restrict__ Y, int B, int I,
                int O) {
    const int o = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (o >= O)
        return;
    const __nv_bfloat16 *w = W + (size_t)o * I;
    for (int b0 = 0; b0 < B; b0 += 8) {
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int i = lane; i < I; i += 32) {
            const float wi = __bfloat162float(w[i]);
#pragma unroll
            for (int b = 0; b < 8; ++b)
                if (b0 + b < B)
                    acc[b] = fmaf(wi, __ldg(&X[(size_t)(b0 + b) * I + i]), acc[b]);
        }
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            float v = acc[b];
            for (int off = 16; off > 0; off >>= 1)
                v += __shfl_xor_sync(0xffffffffu, v, off);
            if (lane == b && b0 + b < B) {
                v += __bfloat162float(bias[o]);
                Ypre[(size_t)(b0 + b) * O + o] = v;
                Y[(size_t)(b0 + b) * O + o]    = silu(v);
            }
        }
    }
}

// dW[o][i] = sum_b G[b][o] X[b][i];  db[o] = sum_b G[b][o]
__global__ void k_dense_wgrad(const float *__restrict__ G, const float *__restrict__ X, float *__restrict__ dW,
                              float *__restrict__ db, int B, int I, int O) {
    const size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (e >= (size_t)O * I)
        return;
    const int o = (int)(e / I), i = (int)(e % I);
    float acc = 0.f;
    for (int b = 0; b < B; ++b)
        acc = fmaf(G[(size_t)b * O + o], X[(size_t)b * I + i], acc);
    dW[e] = acc;
    if (i == 0) {
        float s = 0.f;
        for (int b = 0; b < B; ++b)
            s += G[(size_t)b * O + o];
        db[o] = s;
    }
}

// dX[b][i] = sum_o W[o][i] G[b][o], times SiLU'(pre[b][i]): the rows o in chunks
// (blockIdx.y), eight samples at a time, coalesced along i; then the chunks'
// sums.  (One thread per (b, i) over all rows: 381 us at 4096 x 256, 8 samples,
// 16 CTAs with one serial chain each.)  Chunks of 32 rows, longer ones where that
// would make more than 4096 (blockIdx.y ends at 65535, and so do the sums).
int xg_rows(int O) { return std::max(32, (O + 4095) / 4096); }
__global__ void __launch_bounds__(128)
    k_dense_xgrad_part(const float *__restrict__ G, const __nv_bfloat16 *__restrict__ W, float *__restrict__ part,
                       int B, int I, int O, int rows) {
    const int i = blockIdx.x * 128 + threadIdx.x;
    if (i >= I)
        return;
    const int o0 = blockIdx.y * rows, o1 = min(o0 + rows, O);
    for (int b0 = 0; b0 < B; b0 += 8) {
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int o = o0; o < o1; ++o) {
            const float w = __bfloat162float(W[(size_t)o * I + i]);
#pragma unroll
            for (int b = 0; b < 8; ++b)
                if (b0 + b < B)
                    acc[b] = fmaf(w, __ldg(&G[(size_t)(b0 + b) * O + o]), acc[b]);
        }
        for (int b = 0; b < 8 && b0 + b < B; ++b)
            part[((size_t)blockIdx.y * B + b0 + b) * I + i] = acc[b];
    }
}
__global__ void k_dense_xgrad_sum(const float *__restrict__ part, const float *__restrict__ pre,
                                  float *__restrict__ dX, int n, int nparts) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n)
        return;
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    int p      = 0;
    for (; p + 3 < nparts; p += 4)
#pragma unroll
        for (int k = 0; k < 4; ++k)
            s[k] += part[(size_t)(p + k) * n + e];
    for (; p < nparts; ++p)
        s[0] += part[(size_t)p * n + e];
    dX[e] = ((s[0] + s[1]) + (s[2] + s[3])) * silu_grad(pre[e]);
}

// ---------------------------------------------------------------------------
// 3x3x3 convolution of the (optionally x2 nearest-upsampled) input
// ---------------------------------------------------------------------------
struct ConvGeom {
    int cin, cout;
    int X, Y, Z;    // output (fine) grid
    int up;         // 1: input is (X/2, Y/2, Z/2), read through nearest upsampling
};

constexpr int kMaxCout = 32;

// acc[n] += w[n] u: two channels per instruction (packed FP32x2, each with the scalar
// rounding)
template <int N> __device__ __forceinline__ void axpy(float (&acc)[N], const float *w, float u) {
    if constexpr (N % 2 == 0) {
#pragma unroll
        for (int n = 0; n < N; n += 2) {
            const float2 a = __ffma2_rn(float2{w[n], w[n + 1]}, float2{u, u}, float2{acc[n], acc[n + 1]});
            acc[n]         = a.x;
            acc[n + 1]     = a.y;
        }
    } else {
#pragma unroll
        for (int n = 0; n < N; ++n)
            acc[n] = fmaf(w[n], u, acc[n]);
    }
}

// Folded weights of the upsampling convolutions, refreshed whenever the BF16
// weights change.  Of the 27 fine taps an output voxel reads, the nearest
// upsampling makes 1, 2, 4 or 8 meet in one coarse voxel: per axis an output of
// parity p sees the coarse voxels v + p - 1 + t, t = 0, 1, with the FP32 sums
//   k = fold_k(p, t):  0 the tap +1;  1 taps 0 and +1;  2 taps -1 and 0;  3 the tap -1
// fwd[px py][c][tx ty pz tz][o] for the forward pass, bwd[o][kx ky kz][c] for the
// input gradient.
struct FoldArgs {
    int n;
    struct {
        int cin, cout;
        size_t w, f; // offsets of the layer's weights and of its folded weights
    } L[8];
};

// position of the (parity, coarse tap) pair among the four folded taps of an axis
__host__ __device__ __forceinline__ int fold_k(int p, int t) { return p == 0 ? (t == 0 ? 3 : 1) : (t == 0 ? 2 : 0); }

__global__ void k_fold(const __nv_bfloat16 *__restrict__ wb, float *__restrict__ fwd, float *__restrict__ bwd,
                       FoldArgs a) {
    const auto L = a.L[blockIdx.y];
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < L.cin * L.cout * 64; e += gridDim.x * blockDim.x) {
        const int c = e % L.cin, k = (e / L.cin) & 63, o = e / (L.cin * 64);
        // first tap and number of taps per axis
        auto lo = [](int q) { return q == 0 ? 2 : (q == 1 ? 1 : 0); };
        auto nt = [](int q) { return q == 0 || q == 3 ? 1 : 2; };
        const int kx = k >> 4, ky = (k >> 2) & 3, kz = k & 3;
        const __nv_bfloat16 *w = wb + L.w + ((size_t)o * L.cin + c) * 27;
        float v = 0.f;
        for (int i = lo(kx); i < lo(kx) + nt(kx); ++i)
            for (int j = lo(ky); j < lo(ky) + nt(ky); ++j)
                for (int l = lo(kz); l < lo(kz) + nt(kz); ++l)
                    v += __bfloat162float(w[(i * 3 + j) * 3 + l]);
        bwd[L.f + e] = v;
        // k -> (parity, tap): 3 (0, 0), 1 (0, 1), 2 (1, 0), 0 (1, 1)
        auto par = [](int q) { return q == 0 || q == 2; };
        auto tap = [](int q) { return q == 0 || q == 1; };
        const int pxy = par(kx) * 2 + par(ky), t = tap(kx) * 8 + tap(ky) * 4 + par(kz) * 2 + tap(kz);
        fwd[L.f + (((size_t)pxy * L.cin + c) * 16 + t) * L.cout + o] = v;
    }
}

// Forward upsampling convolution with the folded weights: 8 multiply-adds per
// fine voxel and channel pair instead of 27.  A block has one (x, y) parity and
// one group of OT output channels (blockIdx.y); a thread makes both z parities
// of VX coarse voxels along x, so that a step's weights (shared memory, warp-uniform
// 16-byte reads) serve 2 VX x OT sums and its u (L1) all of them; lanes run along z and
// store 8 bytes each.  Bound by FP32 issue at <8, 2>; small volumes take fewer
// channels a thread, so that the layer fills the SMs, and the smallest split the input
// channels over KS groups of 128 threads, summed in order through shared memory: there a
// thread's chain of loads is the time.  pre may be null (prediction).
// Measured: 32 -> 32 channels to 16 x 16 x 4, 1 sample, 190 -> 18 (KS = 1) -> 8.8 us; 8 -> 8 to
// 128 x 128 x 32, 8 samples, 747 -> 176 us.
template <int OT, int VX, int KS>
__global__ void __launch_bounds__(128 * KS)
    k_up_fwd(const float *__restrict__ in, const float *__restrict__ fwd, const __nv_bfloat16 *__restrict__ bias,
             float *__restrict__ pre, float *__restrict__ out, ConvGeom g, size_t in_stride, size_t out_stride) {
    extern __shared__ __align__(16) float uf_ws[]; // [c][16][OT], then the other groups' sums [KS - 1][2 VX OT][128]
    const int pxy = blockIdx.y & 3, px = pxy >> 1, py = pxy & 1, o0 = (blockIdx.y >> 2) * OT;
    for (int e = threadIdx.x; e < g.cin * 16 * OT; e += 128 * KS)
        uf_ws[e] = fwd[((size_t)pxy * g.cin * 16 + e / OT) * g.cout + o0 + e % OT];
    __syncthreads();
    const int Xi = g.X >> 1, Yi = g.Y >> 1, Zi = g.Z >> 1;
    const int grp = KS > 1 ? threadIdx.x / 128 : 0, lane = threadIdx.x - grp * 128;
    const int idx = blockIdx.x * 128 + lane;
    const bool live = idx < Xi / VX * Yi * Zi;
    if (KS == 1 && !live)
        return;
    const int zi = idx % Zi, yi = idx / Zi % Yi, xi = idx / Zi / Yi * VX;
    const size_t ni  = (size_t)Xi * Yi * Zi;
    const float *inb = in + blockIdx.z * in_stride + zi;
    float acc[VX][2][OT];
#pragma unroll
    for (int v = 0; v < VX; ++v)
#pragma unroll
        for (int o = 0; o < OT; ++o)
            acc[v][0][o] = acc[v][1][o] = grp ? 0.f : __bfloat162float(bias[o0 + o]);
    const bool zl = zi > 0, zr = zi + 1 < Zi;
#pragma unroll 2
    for (int c = live ? grp : g.cin; c < g.cin; c += KS) {
        float u[VX + 1][2][3];
#pragma unroll
        for (int a = 0; a <= VX; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const int x = xi + px - 1 + a, y = yi + py - 1 + b;
                u[a][b][0] = u[a][b][1] = u[a][b][2] = 0.f;
                if (x >= 0 && x < Xi && y >= 0 && y < Yi) {
                    const float *r = inb + c * ni + ((size_t)x * Yi + y) * Zi;
                    u[a][b][1]     = __ldg(r);
                    if (zl)
                        u[a][b][0] = __ldg(r - 1);
                    if (zr)
                        u[a][b][2] = __ldg(r + 1);
                }
            }
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int tx = k >> 3, ty = (k >> 2) & 1, pz = (k >> 1) & 1, tz = k & 1;
            const float *w = uf_ws + (size_t)(c * 16 + k) * OT;
            float wo[OT];
#pragma unroll
            for (int o = 0; o < OT; ++o)
                wo[o] = w[o];
#pragma unroll
            for (int v = 0; v < VX; ++v)
                axpy(acc[v][pz], wo, u[v + tx][ty][pz + tz]);
        }
    }
    if constexpr (KS > 1) {
        float *red = uf_ws + g.cin * 16 * OT + lane;
        if (grp) {
#pragma unroll
            for (int j = 0; j < 2 * VX * OT; ++j)
                red[((grp - 1) * 2 * VX * OT + j) * 128] = acc[j / (2 * OT)][j / OT & 1][j % OT];
        }
        __syncthreads();
        if (grp || !live)
            return;
#pragma unroll
        for (int k = 0; k < KS - 1; ++k)
#pragma unroll
            for (int j = 0; j < 2 * VX * OT; ++j)
                acc[j / (2 * OT)][j / OT & 1][j % OT] += red[(k * 2 * VX * OT + j) * 128];
    }
#pragma unroll
    for (int v = 0; v < VX; ++v)
#pragma unroll
        for (int o = 0; o < OT; ++o) {
            const size_t q = blockIdx.z * out_stride +
                             (((size_t)(o0 + o) * g.X + 2 * (xi + v) + px) * g.Y + 2 * yi + py) * g.Z + 2 * zi;
            const float2 y = make_float2(acc[v][0][o], acc[v][1][o]);
            if (pre)
                *reinterpret_cast<float2 *>(pre + q) = y;
            *reinterpret_cast<float2 *>(out + q) = make_float2(silu(y.x), silu(y.y));
        }
}

// The last convolution (cin -> 1, no upsampling, linear).  One thread: 4 voxels
// along x, whose windows share their loads (L1); lanes take neighbouring (y, z)
// columns.  Bound by the L1 reads (54 per 108 multiply-adds): 448 -> 145 us at 8
// channels, 128 x 128 x 32, 8 samples (one voxel a thread, staged tiles, before).
__global__ void __launch_bounds__(128, 8)
    k_last_fwd(const float *__restrict__ in, const __nv_bfloat16 *__restrict__ W,
               const __nv_bfloat16 *__restrict__ bias, float *__restrict__ out, ConvGeom g, size_t in_stride) {
    constexpr int RX = 4;
    __shared__ float ws[kMaxCout * 27];
    for (int e = threadIdx.x; e < g.cin * 27; e += 128)
        ws[e] = __bfloat162float(W[e]);
    __syncthreads();
    // blockIdx.x = column block + column blocks * x block
    const int cols = g.Y * g.Z, ncb = (cols + 127) / 128, xb = blockIdx.x / ncb;
    const int col  = (blockIdx.x - xb * ncb) * 128 + threadIdx.x;
    if (col >= cols)
        return;
    const int y = col / g.Z, z = col - y * g.Z, x0 = xb * RX;
    const float *inb = in + blockIdx.z * in_stride + col;
    float acc[RX];
#pragma unroll
    for (int r = 0; r < RX; ++r)
        acc[r] = __bfloat162float(bias[0]);
    bool ok[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int yy = y + k / 3 - 1, zz = z + k % 3 - 1;
        ok[k] = yy >= 0 && yy < g.Y && zz >= 0 && zz < g.Z;
    }
    for (int c = 0; c < g.cin; ++c) {
        const float *u = inb + (size_t)c * g.X * cols;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            float uv[RX + 2];
#pragma unroll
            for (int r = 0; r < RX + 2; ++r) {
                const int x = x0 + r - 1;
                uv[r] = ok[k] && x >= 0 && x < g.X ? __ldg(u + (size_t)x * cols + (k / 3 - 1) * g.Z + k % 3 - 1) : 0.f;
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const float w = ws[c * 27 + d * 9 + k];
#pragma unroll
                for (int r = 0; r < RX; ++r)
                    acc[r] = fmaf(w, uv[r + d], acc[r]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < RX; ++r)
        if (x0 + r < g.X)
            out[(blockIdx.z * (size_t)g.X + x0 + r) * cols + col] = acc[r];
}

// Weight and bias gradients of an upsampling convolution, folded taps.
//
// The gradient is gathered for the 4 x 4 x 4 products of (parity, coarse tap)
// pairs of fold_k,
//   dK[o][c][kx ky kz] = sum_v gy[o][2v + p] u[c][v + p - 1 + t],
// and the 27 tap gradients are sums of 8 of them (k_up_wgrad_reduce): 8
// multiply-adds per fine voxel and channel pair instead of 27.
//
// Bound by FP32 issue (FMA pipe) in the inner loop.  A CTA takes 8 input
// channels x OT output channels (blockIdx.y) and strides over tiles of at most
// 128 coarse voxels.  A warp holds one (x, y) parity (warp & 3) and its lanes 8
// input channels x the 4 (x, y) taps, so gy comes as warp-uniform 16-byte loads
// and a new u as one load per z step: 32 multiply-adds per 5 shared-memory
// wavefronts, with the 4 x OT sums in registers.  The pitches put the 32 lanes'
// u values in 32 banks.  Two halves of the warps split a tile's rows and are
// added in shared memory at the end.
// Measured at 8 -> 8 channels, 128 x 128 x 32, 8 samples: 30.8 ms (one thread per
// tap over 2048 voxels) -> 212 us.
constexpr int kWgVox = 128; // coarse voxels per tile, at most

struct WgTile {
    int tx, ty, tz;        // tile edges (coarse voxels)
    int ys, xs, cs;        // u pitches: row, x plane, channel
    int nx, ny, nz, ntile; // tiles per axis, tiles over all samples
    int ncg;               // groups of 8 input channels
};

template <int OT>
__global__ void __launch_bounds__(256, 3)
    k_up_wgrad(const float *__restrict__ in, const float *__restrict__ gy, float *__restrict__ partial,
               float *__restrict__ bpartial, ConvGeom g, WgTile w, size_t in_stride, size_t g_stride) {
    extern __shared__ __align__(16) float wg_smem[];
    float *us = wg_smem;                                   // 8 channels of u with halo
    const int un = (8 * w.cs + 3) & ~3;
    float *gs = wg_smem + un;                              // [pxy][voxel][pz][OT]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cg = blockIdx.y % w.ncg, og = blockIdx.y / w.ncg;
    const int c0 = cg * 8, o0 = og * OT;
    const int Xi = g.X >> 1, Yi = g.Y >> 1, Zi = g.Z >> 1;
    const int nvox = w.tx * w.ty * w.tz;
    const int pxy = warp & 3, half = warp >> 2, px = pxy >> 1, py = pxy & 1;
    const int cl = lane & 7, tx = lane >> 4, ty = (lane >> 3) & 1;
    float acc[4][OT]; // (pz, tz), output channel
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int o = 0; o < OT; ++o)
            acc[k][o] = 0.f;
    float bsum = 0.f; // of this thread's staged gy (channel lane % OT)
    for (int tile = blockIdx.x; tile < w.ntile; tile += gridDim.x) {
        int r         = tile;
        const int bz = r % w.nz;
        r /= w.nz;
        const int by = r % w.ny;
        r /= w.ny;
        const int bx = r % w.nx, smp = r / w.nx;
        const int x0 = bx * w.tx, y0 = by * w.ty, z0 = bz * w.tz;
        const float *inb = in + smp * in_stride, *gyb = gy + smp * g_stride;
        __syncthreads(); // the previous tile's reads
        // u: a channel per warp, one row of z per step
        {
            const bool cok   = c0 + warp < g.cin;
            const float *src = inb + ((size_t)(c0 + warp) * Xi + x0 - 1) * Yi * Zi + (ptrdiff_t)(y0 - 1) * Zi + z0 - 1;
            const bool zok   = z0 + lane - 1 >= 0 && z0 + lane - 1 < Zi; // tz + 2 <= 18 lanes
            float *dst       = us + warp * w.cs + lane;
            for (int xl = 0; xl < w.tx + 2; ++xl)
#pragma unroll 2
                for (int yl = 0; yl < w.ty + 2; ++yl) {
                    const bool ok = cok && zok && (unsigned)(x0 + xl - 1) < (unsigned)Xi &&
                                    (unsigned)(y0 + yl - 1) < (unsigned)Yi;
                    if (lane < w.tz + 2)
                        dst[xl * w.xs + yl * w.ys] = ok ? __ldg(&src[(xl * Yi + yl) * Zi + lane]) : 0.f;
                }
        }
        // gy: an (x, y) parity per pair of warps; lanes take the output channels first
        // (conflict-free stores)
        {
            const int o      = lane % OT, f0 = lane / OT;
            const float *src = gyb + ((size_t)(o0 + o) * g.X + 2 * x0 + px) * g.Y * g.Z + (size_t)(2 * y0 + py) * g.Z +
                               2 * z0;
            float *dst = gs + (size_t)pxy * nvox * 2 * OT + o;
            for (int xl = 0; xl < w.tx; ++xl)
                for (int yl = half; yl < w.ty; yl += 2) {
                    const bool ok  = 2 * (x0 + xl) < g.X && 2 * (y0 + yl) < g.Y;
                    const float *r = src + (size_t)(2 * xl * g.Y + 2 * yl) * g.Z;
                    float *d       = dst + (xl * w.ty + yl) * w.tz * 2 * OT;
#pragma unroll 4
                    for (int fz = f0; fz < 2 * w.tz; fz += 32 / OT) {
                        const float v = ok && 2 * z0 + fz < g.Z ? __ldg(&r[fz]) : 0.f;
                        d[fz * OT]    = v;
                        bsum += v;
                    }
                }
        }
        __syncthreads();
        for (int row = half; row < w.tx * w.ty; row += 2) {
            const int xl = row / w.ty, yl = row - xl * w.ty;
            const float *u = us + cl * w.cs + (xl + px + tx) * w.xs + (yl + py + ty) * w.ys;
            const float *gr = gs + (size_t)(pxy * nvox + row * w.tz) * 2 * OT;
            float u0 = u[0], u1 = u[1];
#pragma unroll 4
            for (int z = 0; z < w.tz; ++z) {
                const float u2 = u[z + 2];
                alignas(16) float ga[2 * OT];
                if constexpr (OT % 2 == 0) {
#pragma unroll
                    for (int k = 0; k < 2 * OT; k += 4)
                        *reinterpret_cast<float4 *>(ga + k) = *reinterpret_cast<const float4 *>(gr + z * 2 * OT + k);
                } else {
                    ga[0] = gr[z * 2], ga[1] = gr[z * 2 + 1];
                }
                axpy(acc[0], ga, u0);
                axpy(acc[1], ga, u1);
                axpy(acc[2], ga + OT, u1);
                axpy(acc[3], ga + OT, u2);
                u0 = u1;
                u1 = u2;
            }
        }
    }
    // the two halves, then this CTA's part: [c][kx ky][kz][o]
    __syncthreads();
    if (half == 1)
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int o = 0; o < OT; ++o)
                gs[(k * OT + o) * 128 + (tid & 127)] = acc[k][o];
    __syncthreads();
    float *dst = partial + ((size_t)blockIdx.x * gridDim.y + blockIdx.y) * (8 * 64 * OT);
    if (half == 0) {
        const int kxy = fold_k(px, tx) * 4 + fold_k(py, ty);
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int o = 0; o < OT; ++o)
                dst[(cl * 64 + kxy * 4 + fold_k(k >> 1, k & 1)) * OT + o] = acc[k][o] + gs[(k * OT + o) * 128 + tid];
    }
    if (cg == 0) {
        __syncthreads();
        gs[tid] = bsum;
        __syncthreads();
        if (tid < OT) {
            float s = 0.f;
            for (int t = tid; t < 256; t += OT)
                s += gs[t];
            bpartial[(size_t)blockIdx.x * g.cout + o0 + tid] = s;
        }
    }
}

// First level of the parts' sum where there are many: parts p = blockIdx.y, blockIdx.y +
// gridDim.y, ... of every element into out[blockIdx.y] (one block per channel alone walked 444
// parts in 44 us).
__global__ void __launch_bounds__(256)
    k_sum_parts(const float *__restrict__ partial, float *__restrict__ out, int n, int nparts) {
    const int e = blockIdx.x * 256 + threadIdx.x;
    if (e >= n)
        return;
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    int p      = blockIdx.y;
    for (; p + 3 * (int)gridDim.y < nparts; p += 4 * gridDim.y)
#pragma unroll
        for (int k = 0; k < 4; ++k)
            s[k] += partial[(size_t)(p + k * gridDim.y) * n + e];
    for (; p < nparts; p += gridDim.y)
        s[0] += partial[(size_t)p * n + e];
    out[(size_t)blockIdx.y * n + e] = (s[0] + s[1]) + (s[2] + s[3]);
}

// Sums the CTAs' parts of one input channel (blockIdx.x) and output-channel
// group (blockIdx.y), then unfolds the 64 products into the 27 tap gradients:
// tap -1 of an axis collects k = 2, 3, tap 0 k = 1, 2, tap 1 k = 0, 1.
// 64 x OT threads per slice of the parts, 1024 / (64 OT) slices (at most 4).
template <int OT> constexpr int up_reduce_slices() { return 1024 / (64 * OT) > 4 ? 4 : 1024 / (64 * OT); }
template <int OT>
__global__ void __launch_bounds__(64 * OT * up_reduce_slices<OT>())
    k_up_wgrad_reduce(const float *__restrict__ partial, const float *__restrict__ bpartial, float *__restrict__ dW,
                      float *__restrict__ db, int cout, int cin, int ncg, int nparts, int nbparts) {
    constexpr int SL = up_reduce_slices<OT>();
    __shared__ float red[SL][64 * OT];
    const int c = blockIdx.x, og = blockIdx.y, tid = threadIdx.x;
    const int sl = tid / (64 * OT), e = tid % (64 * OT);
    const int pair      = og * ncg + c / 8, npair = gridDim.y * ncg;
    const float *src    = partial + (size_t)pair * (8 * 64 * OT) + (c % 8) * 64 * OT + e;
    const size_t stride = (size_t)npair * (8 * 64 * OT);
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    int p      = sl;
    for (; p + 3 * SL < nparts; p += 4 * SL)
#pragma unroll
        for (int k = 0; k < 4; ++k)
            s[k] += src[(size_t)(p + k * SL) * stride];
    for (; p < nparts; p += SL)
        s[0] += src[(size_t)p * stride];
    red[sl][e] = (s[0] + s[1]) + (s[2] + s[3]);
    __syncthreads();
    for (int q = tid; q < 27 * OT; q += blockDim.x) {
        const int o = q % OT, t = q / OT;
        float v = 0.f;
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int k = ((2 - t / 9 + (m >> 2)) * 4 + (2 - (t / 3) % 3 + ((m >> 1) & 1))) * 4 + (2 - t % 3 + (m & 1));
#pragma unroll
            for (int l = 0; l < SL; ++l)
                v += red[l][k * OT + o];
        }
        dW[((size_t)(og * OT + o) * cin + c) * 27 + t] = v;
    }
    if (c == 0 && tid < 32)
        for (int o = 0; o < OT; ++o) {
            float b = 0.f;
            for (int q = tid; q < nbparts; q += 32)
                b += bpartial[(size_t)q * cout + og * OT + o];
            for (int off = 16; off > 0; off >>= 1)
                b += __shfl_down_sync(0xffffffffu, b, off);
            if (tid == 0)
                db[og * OT + o] = b;
        }
}

// Weight and bias gradients of the last convolution (cin -> 1, no upsampling).
// Lanes take neighbouring (y, z) columns and walk along x over a segment of sx
// planes, holding the 3 x 9 window of one input channel (blockIdx.y) and the 27
// sums in registers: 9 loads (L1) and 27 multiply-adds per voxel.  The block's
// sums meet in shared memory.  8 channels, 128 x 128 x 32, 8 samples: 4.2 ms -> 143 us.
//  blockIdx.x = column block x segment, z = sample.
__global__ void __launch_bounds__(256, 3)
    k_last_wgrad(const float *__restrict__ in, const float *__restrict__ gy, float *__restrict__ partial,
                 ConvGeom g, int sx, int nseg, size_t in_stride, size_t g_stride) {
    __shared__ float red[28][257];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cols = g.Y * g.Z;
    const int cb = blockIdx.x / nseg, seg = blockIdx.x - cb * nseg;
    const int col = cb * 256 + tid, y = col / g.Z, z = col - y * g.Z;
    const float *u   = in + blockIdx.z * in_stride + (size_t)blockIdx.y * g.X * cols;
    const float *gyb = gy + blockIdx.z * g_stride;
    const int x0 = seg * sx, x1 = min(x0 + sx, g.X);
    float acc[3][9], w[3][9], gsum = 0.f;
    bool ok[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int yy = y + k / 3 - 1, zz = z + k % 3 - 1;
        ok[k] = col < cols && yy >= 0 && yy < g.Y && zz >= 0 && zz < g.Z;
        acc[0][k] = acc[1][k] = acc[2][k] = 0.f;
        const int off = (k / 3 - 1) * g.Z + k % 3 - 1;
        w[0][k] = ok[k] && x0 > 0 ? __ldg(&u[(size_t)(x0 - 1) * cols + col + off]) : 0.f;
        w[1][k] = ok[k] && x0 < g.X ? __ldg(&u[(size_t)x0 * cols + col + off]) : 0.f;
    }
    // sx is a multiple of 3: the window's planes rotate by renaming
    const float *r[3], *gp = gyb + (size_t)x0 * cols + col;
#pragma unroll
    for (int d = 0; d < 3; ++d)
        r[d] = u + (size_t)(x0 + 1) * cols + col + (d - 1) * g.Z;
#pragma unroll 1
    for (int xb = x0; xb < x1; xb += 3) {
#pragma unroll
        for (int s = 0; s < 3; ++s) {
            const int x    = xb + s;
            const bool in  = x + 1 < g.X;
            const float gv = col < cols && x < x1 ? __ldg(gp) : 0.f;
            gsum += gv;
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                w[(s + 2) % 3][k] = ok[k] && in ? __ldg(r[k / 3] + k % 3 - 1) : 0.f;
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    acc[d][k] = fmaf(gv, w[(s + d) % 3][k], acc[d][k]);
            }
            gp += cols;
#pragma unroll
            for (int d = 0; d < 3; ++d)
                r[d] += cols;
        }
    }
#pragma unroll
    for (int t = 0; t < 27; ++t)
        red[t][tid] = acc[t / 9][t % 9];
    red[27][tid] = gsum;
    __syncthreads();
    float *dst = partial + (((size_t)blockIdx.z * gridDim.x + blockIdx.x) * g.cin + blockIdx.y) * 28;
    for (int t = warp; t < 28; t += 8) {
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            v += red[t][lane + 32 * k];
        for (int off = 16; off > 0; off >>= 1)
            v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane == 0)
            dst[t] = v;
    }
}

// dW[c][t] and db of the last convolution: one warp per (c, t), lanes over the parts
__global__ void __launch_bounds__(256)
    k_last_wgrad_reduce(const float *__restrict__ partial, float *__restrict__ dW, float *__restrict__ db, int cin,
                        int nparts) {
    const int lane = threadIdx.x & 31, e = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (e >= cin * 28)
        return;
    const int c = e / 28, t = e - c * 28;
    float v = 0.f;
    for (int p = lane; p < nparts; p += 32)
        v += partial[(size_t)p * cin * 28 + e];
    for (int off = 16; off > 0; off >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, off);
    if (lane == 0) {
        if (t < 27)
            dW[c * 27 + t] = v;
        else if (c == 0)
            db[0] = v;
    }
}

// Input gradient of an upsampling convolution, on the coarse grid, times
// SiLU'(pre) of the layer below (its dL/d(pre-activation)).  A coarse voxel v
// collects from the fine voxels 2v - 1 .. 2v + 2 per axis with the folded
// weights: 64 multiply-adds per channel pair instead of 8 x 27.  One thread: VX
// coarse voxels along x and CT input channels (blockIdx.y: channel group), the
// weights of a step shared by its voxels; lanes run along z (8-byte loads).
// Bound by FP32 issue and the shared-memory weight reads (VX = 2 halves them);
// small volumes take CT = 2, VX = 1 so that the layer fills the SMs, the smallest with
// the output channels over KS groups of 128 threads.  8 -> 8
// channels at 128 x 128 x 32, 8 samples: 1086 + 2 x 70 (SiLU' pass) -> 170 us.
template <int CT, int VX, int KS>
__global__ void __launch_bounds__(128 * KS)
    k_up_xgrad(const float *__restrict__ gy, const float *__restrict__ bwd, const float *__restrict__ pre_in,
               float *__restrict__ dx, ConvGeom g, size_t g_stride, size_t dx_stride) {
    extern __shared__ __align__(16) float xg_ws[]; // [o][64][CT], then the other groups' sums [KS - 1][VX CT][128]
    const int c0 = blockIdx.y * CT;
    for (int e = threadIdx.x; e < g.cout * 64 * CT; e += 128 * KS)
        xg_ws[e] = bwd[(size_t)(e / CT) * g.cin + c0 + e % CT];
    __syncthreads();
    const int Xi = g.X >> 1, Yi = g.Y >> 1, Zi = g.Z >> 1;
    const int grp = KS > 1 ? threadIdx.x / 128 : 0, lane = threadIdx.x - grp * 128;
    const int idx = blockIdx.x * 128 + lane;
    const bool live = idx < Xi / VX * Yi * Zi;
    if (KS == 1 && !live)
        return;
    const int zi = idx % Zi, yi = idx / Zi % Yi, xi = idx / Zi / Yi * VX;
    const size_t nv = (size_t)g.X * g.Y * g.Z;
    const float *gyb = gy + blockIdx.z * g_stride + 2 * zi;
    float acc[VX][CT];
#pragma unroll
    for (int v = 0; v < VX; ++v)
#pragma unroll
        for (int c = 0; c < CT; ++c)
            acc[v][c] = 0.f;
    const bool zl = zi > 0, zr = zi + 1 < Zi;
    for (int o = live ? grp : g.cout; o < g.cout; o += KS) {
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int y = 2 * yi - 1 + b;
            if (y < 0 || y >= g.Y)
                continue;
            float gv[2 * VX + 2][4];
#pragma unroll
            for (int a = 0; a < 2 * VX + 2; ++a) {
                const int x = 2 * xi - 1 + a;
                gv[a][0] = gv[a][1] = gv[a][2] = gv[a][3] = 0.f;
                if (x >= 0 && x < g.X) {
                    const float *r = gyb + o * nv + ((size_t)x * g.Y + y) * g.Z;
                    const float2 m = __ldg(reinterpret_cast<const float2 *>(r));
                    gv[a][1]       = m.x;
                    gv[a][2]       = m.y;
                    if (zl)
                        gv[a][0] = __ldg(r - 1);
                    if (zr)
                        gv[a][3] = __ldg(r + 2);
                }
            }
#pragma unroll
            for (int kx = 0; kx < 4; ++kx)
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    const float *w = xg_ws + (size_t)(o * 64 + (kx * 4 + b) * 4 + d) * CT;
                    float wc[CT];
#pragma unroll
                    for (int c = 0; c < CT; ++c)
                        wc[c] = w[c];
#pragma unroll
                    for (int v = 0; v < VX; ++v)
                        axpy(acc[v], wc, gv[2 * v + kx][d]);
                }
        }
    }
    if constexpr (KS > 1) {
        float *red = xg_ws + g.cout * 64 * CT + lane;
        if (grp) {
#pragma unroll
            for (int j = 0; j < VX * CT; ++j)
                red[((grp - 1) * VX * CT + j) * 128] = acc[j / CT][j % CT];
        }
        __syncthreads();
        if (grp || !live)
            return;
#pragma unroll
        for (int k = 0; k < KS - 1; ++k)
#pragma unroll
            for (int j = 0; j < VX * CT; ++j)
                acc[j / CT][j % CT] += red[(k * VX * CT + j) * 128];
    }
#pragma unroll
    for (int v = 0; v < VX; ++v)
#pragma unroll
        for (int c = 0; c < CT; ++c) {
            const size_t q = blockIdx.z * dx_stride + (((size_t)(c0 + c) * Xi + xi + v) * Yi + yi) * Zi + zi;
            dx[q]          = acc[v][c] * silu_grad(pre_in[q]);
        }
}

// Input gradient of the last convolution (cin -> 1), times SiLU'(pre) of the
// layer below.  One thread: 4 voxels along x and CT input channels; lanes take
// neighbouring (y, z) columns.  A step's window of gy and its weights serve
// 4 x CT sums.  Bound by the stores and the reads of `pre` (DRAM) at CT = 8.
template <int CT>
__global__ void __launch_bounds__(128)
    k_last_xgrad(const float *__restrict__ gy, const __nv_bfloat16 *__restrict__ W, const float *__restrict__ pre_in,
                 float *__restrict__ dx, ConvGeom g, size_t g_stride, size_t dx_stride) {
    constexpr int RX = 4;
    __shared__ __align__(16) float ws[27 * CT]; // [tap, mirrored][CT]
    // blockIdx.x = column block + column blocks * (channel group + groups * x block)
    const int cols = g.Y * g.Z, ncb = (cols + 127) / 128, row = blockIdx.x / ncb;
    const int ngrp = g.cin / CT, c0 = (row % ngrp) * CT;
    for (int e = threadIdx.x; e < 27 * CT; e += 128)
        ws[e] = __bfloat162float(W[(size_t)(c0 + e % CT) * 27 + 26 - e / CT]);
    __syncthreads();
    const int col = (blockIdx.x - row * ncb) * 128 + threadIdx.x;
    if (col >= cols)
        return;
    const int y = col / g.Z, z = col - y * g.Z, x0 = row / ngrp * RX;
    const float *gyb = gy + blockIdx.z * g_stride + col;
    float acc[RX][CT];
#pragma unroll
    for (int r = 0; r < RX; ++r)
#pragma unroll
        for (int c = 0; c < CT; ++c)
            acc[r][c] = 0.f;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        const int yy = y + k / 3 - 1, zz = z + k % 3 - 1;
        if (yy < 0 || yy >= g.Y || zz < 0 || zz >= g.Z)
            continue;
        float gv[RX + 2];
#pragma unroll
        for (int r = 0; r < RX + 2; ++r) {
            const int x = x0 + r - 1;
            gv[r] = x >= 0 && x < g.X ? __ldg(gyb + (size_t)x * cols + (k / 3 - 1) * g.Z + k % 3 - 1) : 0.f;
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            float wc[CT];
#pragma unroll
            for (int c = 0; c < CT; ++c)
                wc[c] = ws[(d * 9 + k) * CT + c];
#pragma unroll
            for (int r = 0; r < RX; ++r)
                axpy(acc[r], wc, gv[r + d]);
        }
    }
    // SiLU' of four channels' voxels at a time: their reads of `pre` together
    constexpr int CB = CT < 4 ? CT : 4;
#pragma unroll
    for (int cb = 0; cb < CT; cb += CB) {
        float pv[CB][RX];
        const size_t q0 = blockIdx.z * dx_stride + ((size_t)(c0 + cb) * g.X + x0) * cols + col;
#pragma unroll
        for (int c = 0; c < CB; ++c)
#pragma unroll
            for (int r = 0; r < RX; ++r)
                pv[c][r] = x0 + r < g.X ? __ldg(&pre_in[q0 + ((size_t)c * g.X + r) * cols]) : 0.f;
#pragma unroll
        for (int c = 0; c < CB; ++c)
#pragma unroll
            for (int r = 0; r < RX; ++r)
                if (x0 + r < g.X)
                    dx[q0 + ((size_t)c * g.X + r) * cols] = acc[r][cb + c] * silu_grad(pv[c][r]);
    }
}

// loss partials of (u - target)^2 per block and gu = dL/du = 2 (u - t) / (B n)
__global__ void k_loss(const float *__restrict__ u, const float *__restrict__ t, float *__restrict__ gu,
                       double *__restrict__ part, size_t n_total, float inv_n) {
    double acc = 0.;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n_total; e += (size_t)gridDim.x * blockDim.x) {
        const float d = u[e] - t[e];
        acc += (double)d * d;
        gu[e] = 2.f * d * inv_n;
    }
    __shared__ double red[256];
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s)
            red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        part[blockIdx.x] = red[0];
}


// Adam (Kingma and Ba, 2015) on the FP32 master weights, then the BF16 copy.
__global__ void k_adam(float *__restrict__ w, float *__restrict__ m, float *__restrict__ v,
                       const float *__restrict__ g, __nv_bfloat16 *__restrict__ wb, size_t n, float lr, float b1,
                       float b2, float eps, float c1, float c2) {
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const float ge = g[e];
        const float me = b1 * m[e] + (1.f - b1) * ge;
        const float ve = b2 * v[e] + (1.f - b2) * ge * ge;
        m[e]           = me;
        v[e]           = ve;
        const float we = w[e] - lr * (me / c1) / (sqrtf(ve / c2) + eps);
        w[e]           = we;
        wb[e]          = __float2bfloat16_rn(we);
    }
}

__global__ void k_to_bf16(const float *__restrict__ w, __nv_bfloat16 *__restrict__ wb, size_t n) {
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
        wb[e] = __float2bfloat16_rn(w[e]);
}

int grid_for(size_t n, int bs = 256) { return (int)std::min<size_t>((n + bs - 1) / bs, 148 * 16); }

// channel counts the kernels are compiled for
bool channels_ok(int c) { return c == 1 || c == 2 || c == 4 || c == 8 || c == 16 || c == 32; }

// output channels per thread of the folded kernels (channel counts are powers of two)
template <class F> void by_ot(int ot, F &&f) {
    switch (ot) {
    case 1: f(std::integral_constant<int, 1>{}); break;
    case 2: f(std::integral_constant<int, 2>{}); break;
    case 4: f(std::integral_constant<int, 4>{}); break;
    default: f(std::integral_constant<int, 8>{}); break;
    }
}
} // namespace
} // namespace gpe

using gpe::Buf;

struct gpe_warm {
    gpe_warm_config cfg{};
    int device = 0;
    cudaStream_t stream = nullptr;
    // parameter layout (offsets into the flat weight vector)
    struct Layer {
        size_t w = 0, b = 0; // offsets
        size_t f = 0;        // offset of the folded weights (upsampling layers)
        int cin = 0, cout = 0;
        gpe::ConvGeom g{};
    };
    size_t d1w = 0, d1b = 0, d2w = 0, d2b = 0, nweights = 0;
    int latent = 0;
    std::vector<Layer> conv; // levels upsampling stages + the last one
    Buf<float> w, m, v, grad;
    Buf<__nv_bfloat16> wb;
    Buf<float> fold; // folded weights of the upsampling layers, as wb
    // activations (max_batch samples)
    Buf<float> x, h1pre, h1, h2pre, h2, gh1, gh2;
    std::vector<Buf<float>> pre, act, gact; // per conv layer output
    Buf<float> partial, target_scratch;
    Buf<double> lpart;
    long step = 0;

    size_t vox(int l) const { return (size_t)conv[l].g.X * conv[l].g.Y * conv[l].g.Z; }
};

namespace {

int wbad(const char *msg) {
    gpe::last_error() = msg;
    return GPE_ERR_ARG;
}

template <class F> int wguard(F &&f) {
    try {
        f();
        return GPE_OK;
    } catch (const gpe::Error &e) {
        gpe::last_error() = e.what();
        return e.code;
    } catch (const std::exception &e) {
        gpe::last_error() = e.what();
        return GPE_ERR_CUDA;
    }
}

using gpe::Error;

// the folded weights follow every change of the BF16 weights
void refold(gpe_warm *W) {
    gpe::FoldArgs a{};
    for (const auto &L : W->conv)
        if (L.g.up) {
            a.L[a.n].cin  = L.cin;
            a.L[a.n].cout = L.cout;
            a.L[a.n].w    = L.w;
            a.L[a.n++].f  = L.f;
        }
    if (a.n)
        gpe::k_fold<<<dim3(64, a.n), 256, 0, W->stream>>>(W->wb.p, W->fold.p, W->fold.p + W->fold.n / 2, a);
    WS_CUDA(cudaGetLastError());
}

// the amplitudes of W->x into amp; the backward pass's values are kept when training
void forward(gpe_warm *W, int B, float *amp, bool training) {
    using namespace gpe;
    const auto &c = W->cfg;
    cudaStream_t s = W->stream;
    const __nv_bfloat16 *wb = W->wb.p;
    k_dense_fwd<<<(c.hidden + 3) / 4, 128, 0, s>>>(W->x.p, wb + W->d1w, wb + W->d1b, W->h1pre.p, W->h1.p, B,
                                                   c.n_inputs, c.hidden);
    k_dense_fwd<<<(W->latent + 3) / 4, 128, 0, s>>>(W->h1.p, wb + W->d2w, wb + W->d2b, W->h2pre.p, W->h2.p, B,
                                                    c.hidden, W->latent);
    const float *in  = W->h2.p;
    size_t in_stride = W->latent;
    for (const auto &L : W->conv) {
        const size_t l = &L - W->conv.data();
        if (!L.g.up) {
            k_last_fwd<<<dim3((L.g.Y * L.g.Z + 127) / 128 * ((L.g.X + 3) / 4), 1, B), 128, 0, s>>>(
                in, wb + L.w, wb + L.b, amp, L.g, in_stride);
            break;
        }
        const int Xi = L.g.X / 2, nvox = Xi * (L.g.Y / 2) * (L.g.Z / 2);
        const size_t n = W->vox((int)l) * L.cout;
        auto go = [&](auto O, auto V, auto K) {
            constexpr int OT = decltype(O)::value, VX = decltype(V)::value, KS = decltype(K)::value;
            k_up_fwd<OT, VX, KS><<<dim3((nvox / VX + 127) / 128, 4 * (L.cout / OT), B), 128 * KS,
                                   sizeof(float) * (L.cin * 16 * OT + (KS - 1) * 2 * VX * OT * 128), s>>>(
                in, W->fold.p + L.f, wb + L.b, training ? W->pre[l].p : nullptr, W->act[l].p, L.g, in_stride, n);
        };
        using I1 = std::integral_constant<int, 1>;
        using I2 = std::integral_constant<int, 2>;
        using I4 = std::integral_constant<int, 4>;
        // two voxels and eight channels a thread where that still leaves 512 threads
        // per SM, one voxel and four channels where that does, else two (or one); with
        // the input channels split over four groups where all CTAs are resident at once
        // (two per SM: 64 CTAs 18.2 -> 8.8 us, 256 CTAs 19.4 -> 11.1, 512 CTAs 19.4 -> 19.9)
        const size_t small = (size_t)((nvox + 127) / 128) * 4 * (L.cout / 2) * B;
        if (Xi % 2 == 0 && L.cout >= 8 && (size_t)nvox / 2 * 4 * (L.cout / 8) * B >= 148 * 512)
            go(std::integral_constant<int, 8>{}, I2{}, I1{});
        else if (L.cout >= 4 && (size_t)nvox * 4 * (L.cout / 4) * B >= 148 * 512)
            go(I4{}, I1{}, I1{});
        else if (L.cout >= 2 && L.cin >= 8 && small <= 148 * 2)
            go(I2{}, I1{}, I4{});
        else if (L.cout >= 2)
            go(I2{}, I1{}, I1{});
        else
            go(I1{}, I1{}, I1{});
        in        = W->act[l].p;
        in_stride = n;
    }
    WS_CUDA(cudaGetLastError());
}

constexpr size_t kWgSmem = 96 * 1024; // the weight-gradient kernel's limit
int wg_ot(const gpe_warm::Layer &L) { return std::min(L.cout, 8); }
size_t wg_smem(const gpe::WgTile &w, int ot) {
    const size_t gs = (size_t)8 * w.tx * w.ty * w.tz * ot;
    return sizeof(float) * (((size_t)8 * w.cs + 3) / 4 * 4 + std::max<size_t>(gs, (size_t)512 * ot));
}
// tile of the folded weight gradient for a coarse volume: at most 128 voxels, fewer along x
// where the volume is thin (ty tz <= 2: a plane of u then takes 48 floats a channel with its
// halo, and 128 of them do not fit into shared memory)
gpe::WgTile wg_tile(const gpe_warm::Layer &L, int B) {
    gpe::WgTile w{};
    const int Xi = L.g.X / 2, Yi = L.g.Y / 2, Zi = L.g.Z / 2;
    auto pow2 = [](int n, int most) {
        int p = 1;
        while (2 * p <= most && p < n)
            p *= 2;
        return p;
    };
    w.tz = pow2(Zi, 16);
    w.ty = pow2(Yi, std::min(gpe::kWgVox / w.tz, 4));
    w.tx = pow2(Xi, gpe::kWgVox / (w.tz * w.ty));
    auto up = [](int v, int rem, int mod) { // smallest value >= v that is rem modulo mod
        return v + ((rem - v) % mod + mod) % mod;
    };
    w.ys = up(w.tz + 2, 8, 16);
    w.xs = up((w.ty + 2) * w.ys, 16, 32);
    auto fits = [&] {
        w.cs = up((w.tx + 2) * w.xs, 1, 32);
        return wg_smem(w, wg_ot(L)) <= kWgSmem;
    };
    while (!fits())
        w.tx /= 2;
    w.nx = (Xi + w.tx - 1) / w.tx;
    w.ny = (Yi + w.ty - 1) / w.ty;
    w.nz = (Zi + w.tz - 1) / w.tz;
    w.ntile = w.nx * w.ny * w.nz * B;
    w.ncg   = (L.cin + 7) / 8;
    return w;
}
// CTAs along the tiles: up to three per SM (all resident) over all channel groups
int wg_parts(const gpe::WgTile &w, int pairs) { return std::min(w.ntile, std::max(1, 148 * 3 / pairs)); }
// planes per segment of the last layer's gradient (a multiple of 3) and segments
int last_segments(const gpe_warm::Layer &L) { return (L.g.X + 32) / 33; }
int last_segment(const gpe_warm::Layer &L) {
    const int n = last_segments(L);
    return ((L.g.X + n - 1) / n + 2) / 3 * 3;
}
constexpr int kSumSlices = 16; // of the parts, in their sum's first level
// floats of partial sums that layer l's weight gradient needs
size_t wg_partial(const gpe_warm::Layer &L, int B) {
    if (!L.g.up)
        return (size_t)B * last_segments(L) * (((size_t)L.g.Y * L.g.Z + 255) / 256) * L.cin * 28;
    const gpe::WgTile w = wg_tile(L, B);
    const int ot = wg_ot(L), pairs = w.ncg * (L.cout / ot);
    return (size_t)wg_parts(w, pairs) * ((size_t)pairs * 512 * ot + L.cout) + (size_t)kSumSlices * pairs * 512 * ot;
}

// weight and bias gradients of layer l from its input and dL/d(pre-activation)
void conv_wgrad(gpe_warm *W, int l, int B, const float *in, size_t in_stride, const float *gy, size_t g_stride) {
    const auto &L  = W->conv[l];
    cudaStream_t s = W->stream;
    if (!L.g.up) {
        const int nseg = last_segments(L), nb = (L.g.Y * L.g.Z + 255) / 256 * nseg;
        gpe::k_last_wgrad<<<dim3(nb, L.cin, B), 256, 0, s>>>(in, gy, W->partial.p, L.g, last_segment(L), nseg,
                                                             in_stride, g_stride);
        gpe::k_last_wgrad_reduce<<<(L.cin * 28 + 7) / 8, 256, 0, s>>>(W->partial.p, W->grad.p + L.w,
                                                                      W->grad.p + L.b, L.cin, nb * B);
        return;
    }
    const gpe::WgTile w = wg_tile(L, B);
    gpe::by_ot(wg_ot(L), [&](auto O) {
        constexpr int OT = decltype(O)::value;
        const int nog = L.cout / OT, pairs = w.ncg * nog, parts = wg_parts(w, pairs);
        float *bp = W->partial.p + (size_t)parts * pairs * 512 * OT;
        gpe::k_up_wgrad<OT><<<dim3(parts, pairs), 256, wg_smem(w, OT), s>>>(in, gy, W->partial.p, bp, L.g, w,
                                                                            in_stride, g_stride);
        const int n   = pairs * 512 * OT, lvl = parts > 4 * kSumSlices ? kSumSlices : parts;
        float *sums   = lvl < parts ? bp + (size_t)parts * L.cout : W->partial.p;
        if (lvl < parts)
            gpe::k_sum_parts<<<dim3((n + 255) / 256, lvl), 256, 0, s>>>(W->partial.p, sums, n, parts);
        gpe::k_up_wgrad_reduce<OT><<<dim3(L.cin, nog), 64 * OT * gpe::up_reduce_slices<OT>(), 0, s>>>(
            sums, bp, W->grad.p + L.w, W->grad.p + L.b, L.cout, L.cin, w.ncg, lvl, parts);
    });
}

// dL/d(pre-activation) of the layer below l, from layer l's
void conv_xgrad(gpe_warm *W, int l, int B, const float *gy, size_t g_stride, const float *pre_in, float *dx,
                size_t dx_stride) {
    const auto &L  = W->conv[l];
    cudaStream_t s = W->stream;
    if (!L.g.up) {
        gpe::by_ot(std::min(L.cin, 8), [&](auto C) {
            constexpr int CT = decltype(C)::value;
            gpe::k_last_xgrad<CT><<<dim3((L.g.Y * L.g.Z + 127) / 128 * ((L.g.X + 3) / 4 * (L.cin / CT)), 1, B), 128, 0,
                                    s>>>(
                gy, W->wb.p + L.w, pre_in, dx, L.g, g_stride, dx_stride);
        });
        return;
    }
    const int Xi = L.g.X / 2, nvox = Xi * (L.g.Y / 2) * (L.g.Z / 2);
    auto go = [&](auto C, auto V, auto K) {
        constexpr int CT = decltype(C)::value, VX = decltype(V)::value;
        constexpr int KS = decltype(K)::value;
        gpe::k_up_xgrad<CT, VX, KS><<<dim3((nvox / VX + 127) / 128, L.cin / CT, B), 128 * KS,
                                      sizeof(float) * (L.cout * 64 * CT + (KS - 1) * VX * CT * 128), s>>>(
            gy, W->fold.p + W->fold.n / 2 + L.f, pre_in, dx, L.g, g_stride, dx_stride);
    };
    using I1 = std::integral_constant<int, 1>;
    using I2 = std::integral_constant<int, 2>;
    using I4 = std::integral_constant<int, 4>;
    // two voxels and eight channels a thread where that still leaves 256 threads
    // per SM, one voxel and four channels where that does, else two (or one); with the
    // output channels split over four groups where all CTAs are resident at once (two
    // per SM: 128 CTAs 49.6 -> 25.1 us; 512 CTAs of four channels 52.8 -> 54.3)
    if (Xi % 2 == 0 && L.cin >= 8 && (size_t)nvox / 2 * (L.cin / 8) * B >= 148 * 256)
        go(std::integral_constant<int, 8>{}, I2{}, I1{});
    else if (L.cin >= 4 && (size_t)nvox * (L.cin / 4) * B >= 148 * 256)
        go(I4{}, I1{}, I1{});
    else if (L.cin >= 2 && L.cout >= 8 && (size_t)((nvox + 127) / 128) * (L.cin / 2) * B <= 148 * 2)
        go(I2{}, I1{}, I4{});
    else if (L.cin >= 2)
        go(I2{}, I1{}, I1{});
    else
        go(I1{}, I1{}, I1{});
}

// gradients of the mean squared amplitude error against `targets` (device,
// B x N floats); returns the loss (host)
double backward(gpe_warm *W, int B, const float *targets) {
    using namespace gpe;
    const auto &c   = W->cfg;
    cudaStream_t s  = W->stream;
    const __nv_bfloat16 *wb = W->wb.p;
    const int nl    = (int)W->conv.size();
    const size_t N  = W->vox(nl - 1);
    const int lb    = 148 * 4;
    k_loss<<<lb, 256, 0, s>>>(W->pre[nl - 1].p, targets, W->gact[nl - 1].p, W->lpart.p, (size_t)B * N,
                              1.f / (float)((size_t)B * N));
    for (int l = nl - 1; l >= 0; --l) {
        const auto &L  = W->conv[l];
        const size_t n   = W->vox(l) * L.cout;
        const float *gy  = W->gact[l].p; // dL/d(pre-activation)
        const float *in  = l == 0 ? W->h2.p : W->act[l - 1].p;
        const size_t ins = l == 0 ? (size_t)W->latent : W->vox(l - 1) * W->conv[l - 1].cout;
        conv_wgrad(W, l, B, in, ins, gy, n);
        conv_xgrad(W, l, B, gy, n, l == 0 ? W->h2pre.p : W->pre[l - 1].p, l == 0 ? W->gh2.p : W->gact[l - 1].p, ins);
    }
    // dense 2 and dense 1 (gh2 and gh1 are gradients of the pre-activations)
    k_dense_wgrad<<<(int)(((size_t)W->latent * c.hidden + 255) / 256), 256, 0, s>>>(
        W->gh2.p, W->h1.p, W->grad.p + W->d2w, W->grad.p + W->d2b, B, c.hidden, W->latent);
    const int rows = xg_rows(W->latent), chunks = (W->latent + rows - 1) / rows;
    k_dense_xgrad_part<<<dim3((c.hidden + 127) / 128, chunks), 128, 0, s>>>(W->gh2.p, wb + W->d2w, W->partial.p, B,
                                                                            c.hidden, W->latent, rows);
    k_dense_xgrad_sum<<<(B * c.hidden + 63) / 64, 64, 0, s>>>(W->partial.p, W->h1pre.p, W->gh1.p, B * c.hidden,
                                                              chunks);
    k_dense_wgrad<<<(int)(((size_t)c.hidden * c.n_inputs + 255) / 256), 256, 0, s>>>(
        W->gh1.p, W->x.p, W->grad.p + W->d1w, W->grad.p + W->d1b, B, c.n_inputs, c.hidden);
    WS_CUDA(cudaGetLastError());
    std::vector<double> lp(lb);
    WS_CUDA(cudaMemcpyAsync(lp.data(), W->lpart.p, sizeof(double) * lb, cudaMemcpyDeviceToHost, s));
    WS_CUDA(cudaStreamSynchronize(s));
    double loss = 0.;
    for (double v : lp)
        loss += v;
    return loss / (double)((size_t)B * N);
}

// Whether a kernel of W may store floats at p: memory of its own device, aligned.  Memory of
// another device, the host's, or at an odd address is left to the copy engine, which takes
// them all or returns an error.
bool kernel_may_store(const gpe_warm *W, const void *p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice && a.device == W->device && (uintptr_t)p % alignof(float) == 0;
}

void upload_inputs(gpe_warm *W, const float *params_host, int B) {
    WS_CUDA(cudaMemcpyAsync(W->x.p, params_host, sizeof(float) * B * W->cfg.n_inputs, cudaMemcpyHostToDevice,
                            W->stream));
}

} // namespace

extern "C" {

int gpe_warm_create(const gpe_warm_config *cfg, int device, gpe_warm **out) {
    if (!cfg || !out)
        return wbad("null argument");
    *out = nullptr;
    const auto &c = *cfg;
    if (c.levels < 0 || c.levels > 6 || c.hidden <= 0 || c.n_inputs <= 0 || c.max_batch <= 0)
        return wbad("bad network configuration");
    const int f = 1 << c.levels;
    if (c.nx % f || c.ny % f || c.nz % f)
        return wbad("grid sizes must be divisible by 2^levels");
    for (int s = 0; s <= c.levels; ++s)
        if (!gpe::channels_ok(c.channels[s]))
            return wbad("channels must be 1, 2, 4, 8, 16 or 32");
    return wguard([&] {
        auto W    = std::make_unique<gpe_warm>();
        W->cfg    = c;
        W->device = device;
        WS_CUDA(cudaSetDevice(device));
        WS_CUDA(cudaStreamCreateWithFlags(&W->stream, cudaStreamNonBlocking));
        const int X0 = c.nx / f, Y0 = c.ny / f, Z0 = c.nz / f;
        W->latent    = c.channels[0] * X0 * Y0 * Z0;
        size_t off   = 0;
        W->d1w = off, off += (size_t)c.hidden * c.n_inputs;
        W->d1b = off, off += c.hidden;
        W->d2w = off, off += (size_t)W->latent * c.hidden;
        W->d2b = off, off += W->latent;
        int X = X0, Y = Y0, Z = Z0;
        for (int s = 0; s <= c.levels; ++s) {
            gpe_warm::Layer L;
            L.cin  = c.channels[s];
            L.cout = s < c.levels ? c.channels[s + 1] : 1;
            const int up = s < c.levels;
            if (up)
                X *= 2, Y *= 2, Z *= 2;
            L.g = gpe::ConvGeom{L.cin, L.cout, X, Y, Z, up};
            L.w = off, off += (size_t)L.cout * L.cin * 27;
            L.b = off, off += L.cout;
            W->conv.push_back(L);
        }
        W->nweights = off;
        size_t foff = 0;
        for (auto &L : W->conv)
            if (L.g.up)
                L.f = foff, foff += (size_t)L.cin * L.cout * 64;
        W->fold.alloc(2 * foff); // forward, then backward
        W->w.alloc(off);
        W->m.alloc(off);
        W->v.alloc(off);
        W->grad.alloc(off);
        W->wb.alloc(off);
        WS_CUDA(cudaMemset(W->w.p, 0, sizeof(float) * off));
        WS_CUDA(cudaMemset(W->m.p, 0, sizeof(float) * off));
        WS_CUDA(cudaMemset(W->v.p, 0, sizeof(float) * off));
        const int B = c.max_batch;
        W->x.alloc((size_t)B * c.n_inputs);
        W->h1pre.alloc((size_t)B * c.hidden);
        W->h1.alloc((size_t)B * c.hidden);
        W->gh1.alloc((size_t)B * c.hidden);
        W->h2pre.alloc((size_t)B * W->latent);
        W->h2.alloc((size_t)B * W->latent);
        W->gh2.alloc((size_t)B * W->latent);
        // partial sums: the weight gradients' and dense 2's input gradient's
        const int xr   = gpe::xg_rows(W->latent);
        size_t maxpart = (size_t)((W->latent + xr - 1) / xr) * B * c.hidden;
        W->pre.resize(W->conv.size());
        W->act.resize(W->conv.size());
        W->gact.resize(W->conv.size());
        for (size_t l = 0; l < W->conv.size(); ++l) {
            const size_t n = W->vox((int)l) * W->conv[l].cout * B;
            W->pre[l].alloc(n);
            W->act[l].alloc(n);
            W->gact[l].alloc(n);
            maxpart = std::max(maxpart, wg_partial(W->conv[l], B));
        }
        W->partial.alloc(maxpart);
        W->lpart.alloc(148 * 4);
        // folded weights staged in shared memory, up to 32 channels
        WS_CUDA(cudaFuncSetAttribute((const void *)gpe::k_up_xgrad<8, 2, 1>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(float) * gpe::kMaxCout * 64 * 8));
        for (int ot : {1, 2, 4, 8})
            gpe::by_ot(ot, [&](auto O) {
                WS_CUDA(cudaFuncSetAttribute((const void *)gpe::k_up_wgrad<decltype(O)::value>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWgSmem));
            });
        *out = W.release();
    });
}

int gpe_warm_destroy(gpe_warm *W) {
    if (!W)
        return GPE_OK;
    cudaSetDevice(W->device);
    cudaStreamSynchronize(W->stream);
    cudaStream_t s = W->stream;
    delete W;
    cudaStreamDestroy(s);
    return GPE_OK;
}

int gpe_warm_num_weights(gpe_warm *W, size_t *n) {
    if (!W || !n)
        return wbad("null argument");
    *n = W->nweights;
    return GPE_OK;
}

int gpe_warm_set_weights(gpe_warm *W, const float *host, size_t n) {
    if (!W || !host || n != W->nweights)
        return wbad("weight count mismatch");
    return wguard([&] {
        WS_CUDA(cudaSetDevice(W->device));
        WS_CUDA(cudaMemcpyAsync(W->w.p, host, sizeof(float) * n, cudaMemcpyHostToDevice, W->stream));
        gpe::k_to_bf16<<<gpe::grid_for(n), 256, 0, W->stream>>>(W->w.p, W->wb.p, n);
        refold(W);
        WS_CUDA(cudaMemsetAsync(W->m.p, 0, sizeof(float) * n, W->stream));
        WS_CUDA(cudaMemsetAsync(W->v.p, 0, sizeof(float) * n, W->stream));
        WS_CUDA(cudaStreamSynchronize(W->stream));
        W->step = 0;
    });
}

int gpe_warm_get_weights(gpe_warm *W, float *host, size_t n) {
    if (!W || !host || n != W->nweights)
        return wbad("weight count mismatch");
    return wguard([&] {
        WS_CUDA(cudaSetDevice(W->device));
        WS_CUDA(cudaMemcpyAsync(host, W->w.p, sizeof(float) * n, cudaMemcpyDeviceToHost, W->stream));
        WS_CUDA(cudaStreamSynchronize(W->stream));
    });
}

int gpe_warm_init_weights(gpe_warm *W, unsigned long long seed) {
    if (!W)
        return wbad("null network");
    // He-style uniform initialisation scaled by fan-in, zero biases
    std::vector<float> h(W->nweights, 0.f);
    std::mt19937_64 rng(seed);
    auto fill = [&](size_t off, size_t n, int fan_in) {
        const float a = std::sqrt(3.f / (float)fan_in);
        std::uniform_real_distribution<float> U(-a, a);
        for (size_t e = 0; e < n; ++e)
            h[off + e] = U(rng);
    };
    const auto &c = W->cfg;
    fill(W->d1w, (size_t)c.hidden * c.n_inputs, c.n_inputs);
    fill(W->d2w, (size_t)W->latent * c.hidden, c.hidden);
    for (const auto &L : W->conv)
        fill(L.w, (size_t)L.cout * L.cin * 27, L.cin * 27);
    return gpe_warm_set_weights(W, h.data(), h.size());
}

int gpe_warm_forward(gpe_warm *W, const float *params_host, int B, float *amp_dev) {
    if (!W || !params_host || !amp_dev || B <= 0 || B > W->cfg.max_batch)
        return wbad("bad forward arguments");
    return wguard([&] {
        WS_CUDA(cudaSetDevice(W->device));
        upload_inputs(W, params_host, B);
        const bool direct = kernel_may_store(W, amp_dev);
        forward(W, B, direct ? amp_dev : W->pre.back().p, false);
        if (!direct)
            WS_CUDA(cudaMemcpyAsync(amp_dev, W->pre.back().p, sizeof(float) * B * W->vox((int)W->conv.size() - 1),
                                    cudaMemcpyDeviceToDevice, W->stream));
        WS_CUDA(cudaStreamSynchronize(W->stream));
    });
}

int gpe_warm_gradients(gpe_warm *W, const float *params_host, const float *targets_dev, int B, float *grad_host,
                       double *loss) {
    if (!W || !params_host || !targets_dev || B <= 0 || B > W->cfg.max_batch)
        return wbad("bad gradient arguments");
    return wguard([&] {
        WS_CUDA(cudaSetDevice(W->device));
        upload_inputs(W, params_host, B);
        forward(W, B, W->pre.back().p, true);
        const double l = backward(W, B, targets_dev);
        if (loss)
            *loss = l;
        if (grad_host) {
            WS_CUDA(cudaMemcpyAsync(grad_host, W->grad.p, sizeof(float) * W->nweights, cudaMemcpyDeviceToHost,
                                    W->stream));
            WS_CUDA(cudaStreamSynchronize(W->stream));
        }
    });
}

int gpe_warm_train_step(gpe_warm *W, const float *params_host, const float *targets_dev, int B, float lr,
                        double *loss) {
    if (!W || !params_host || !targets_dev || B <= 0 || B > W->cfg.max_batch || !(lr > 0))
        return wbad("bad training arguments");
    return wguard([&] {
        WS_CUDA(cudaSetDevice(W->device));
        upload_inputs(W, params_host, B);
        forward(W, B, W->pre.back().p, true);
        const double l = backward(W, B, targets_dev);
        if (loss)
            *loss = l;
        ++W->step;
        const float b1 = 0.9f, b2 = 0.999f;
        const float c1 = 1.f - std::pow(b1, (float)W->step), c2 = 1.f - std::pow(b2, (float)W->step);
        gpe::k_adam<<<gpe::grid_for(W->nweights), 256, 0, W->stream>>>(W->w.p, W->m.p, W->v.p, W->grad.p, W->wb.p,
                                                                        W->nweights, lr, b1, b2, 1e-8f, c1, c2);
        WS_CUDA(cudaGetLastError());
        refold(W);
    });
}

} // extern "C"
