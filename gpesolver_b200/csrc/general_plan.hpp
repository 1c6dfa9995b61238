// Host side of general.cuh: plans, twiddle tables and launch shapes.
#pragma once

#include "general.cuh"
#include "plan.hpp"

#include <algorithm>

namespace gpe {

inline unsigned g_magic(int d) { return d <= 1 ? 0u : (unsigned)((0x100000000ULL + (unsigned)d - 1) / (unsigned)d); }

inline GPlan g_plan(int L, const void *tw) {
    GPlan p{};
    p.L  = L;
    p.tw = tw;
    const std::vector<int> r = general_radices(L);
    p.n                      = (int)r.size();
    if (p.n > kGStages)
        throw Error(2, "FFT length " + std::to_string(L) + " needs more than " + std::to_string(kGStages) + " stages");
    auto fill = [&](GStage *st, bool rev) {
        int ns = 1;
        for (int s = 0; s < p.n; ++s) {
            const int q = r[rev ? p.n - 1 - s : s];
            st[s]       = GStage{q, ns, L / q, L / (ns * q), g_magic(ns)};
            ns *= q;
        }
    };
    fill(p.f, false);
    fill(p.v, true);
    return p;
}

// Launch shapes for a grid.
struct GShape {
    int lbx, lby, lbz;    // log2 of the lines per CTA
    int ntx, nty, ntz;    // threads
    size_t smx, smy, smz; // shared memory
    int mbx, mby;         // CTAs per SM the x and y kernels are compiled for
    unsigned buf;         // elements of one of the z pass's four tiles
};

// Tiles as wide as a 128-byte row of columns (z: 32 rows), halved while a tile takes
// more than 72 KB (three CTAs per SM) or the pass has fewer than two CTAs per SM;
// below 32 bytes a row, or 8 rows, only the shared memory of one CTA counts.
template <class R> GShape g_shape(int nx, int ny, int nz, bool kinetic) {
    const size_t c = sizeof(cplx<R>);
    const int row  = (int)(128 / c), least = (int)(32 / c);
    const size_t want = 72 * 1024;
    const long long enough = 2 * 148;
    auto lg = [](int v) {
        int l = 0;
        while ((2 << l) <= v)
            ++l;
        return l;
    };
    auto threads = [](const GPlan &p, int lb) {
        int n = 1;
        for (int s = 0; s < p.n; ++s)
            n = std::max(n, p.f[s].nr << lb);
        return std::min(256, std::max(64, (n + 31) / 32 * 32));
    };
    auto most = [](const GPlan &p) {
        int r = 0;
        for (int s = 0; s < p.n; ++s)
            r = std::max(r, p.f[s].r);
        return r;
    };
    GShape g{};
    const GPlan px = g_plan(2 * nx, nullptr), py = g_plan(2 * ny, nullptr);
    {
        const long long cols = (long long)(kinetic ? 3 : 2) * ny * nz;
        auto sm = [&](int lb) { return 2 * c * ((size_t)(2 * nx) << lb); };
        g.lbx   = lg(row);
        while (g.lbx > 0 && (sm(g.lbx) > want || (cols >> g.lbx) < enough) && (g.lbx > lg(least) || sm(g.lbx) > want))
            --g.lbx;
        g.smx = sm(g.lbx);
        g.ntx = threads(px, g.lbx);
        g.mbx = g_blocks<R>(most(px));
    }
    {
        auto sm = [&](int lb) { return (py.n > 2 ? 2 : 1) * c * ((size_t)(2 * ny) << lb); };
        auto ctas = [&](int lb) { return (long long)(kinetic ? 2 : 1) * nx * ((nz + (1 << lb) - 1) >> lb); };
        g.lby   = lg(row);
        while (g.lby > 0 && ((1 << g.lby) >= 2 * nz || sm(g.lby) > want ||
                             (ctas(g.lby) < enough && g.lby > lg(least))))
            --g.lby;
        g.smy = sm(g.lby);
        g.nty = threads(py, g.lby);
        g.mby = g_blocks<R>(most(py));
    }
    {
        const int rows = nx * ny;
        auto buf = [&](int lb) {
            const int rw = 1 << lb, np = std::max(1, rw / 2);
            return (size_t)nz * std::max(rw >= 4 ? rw + 1 : rw, 2 * (np >= 2 ? np + 1 : np));
        };
        g.lbz = 5;
        while (g.lbz > 0 && (4 * c * buf(g.lbz) > want || ((rows >> g.lbz) < enough && g.lbz > 3)))
            --g.lbz;
        g.buf = (unsigned)buf(g.lbz);
        g.smz = 4 * c * (size_t)g.buf;
        g.ntz = ((size_t)nz << g.lbz) < 1024 ? 128 : 256;
    }
    return g;
}

// f(kernel): the x or y kernel for `mb` CTAs per SM
template <class R, class F> void g_with_x(int mb, F &&f) {
    if constexpr (sizeof(R) == 4)
        if (mb == 3)
            return f(g_x<R, 3>);
    f(g_x<R, 2>);
}
template <class R, class F> void g_with_y(int mb, F &&f) {
    if constexpr (sizeof(R) == 4)
        if (mb == 3)
            return f(g_y<R, 3>);
    f(g_y<R, 2>);
}

} // namespace gpe
