// Column walk of the kernels that take a lattice of any shape straight from global memory.
#pragma once

#include <cstdint>

#include "tipt_internal.h"

namespace tipt {

// Quotient of a number below 2^31 by a divisor fixed at launch: n / d = (n m) >>
// (31 + l) with l = ceil(log2 d) and m = floor(2^(31 + l) / d) + 1 < 2^32 (Granlund
// and Montgomery, "Division by invariant integers using multiplication", PLDI
// 1994: exact because n (m d - 2^(31 + l)) <= n d < 2^(31 + l)).
struct FastDiv {
    uint32_t d, m, s;
    FastDiv() = default;
    explicit FastDiv(uint32_t div) : d(div), m(0), s(0) {
        if (div <= 1) return;
        uint32_t l = 0;
        while ((1ull << l) < div) ++l;
        m = (uint32_t)((1ull << (31 + l)) / div + 1);
        s = l - 1;
    }
    __device__ __forceinline__ uint32_t div(uint32_t n) const {
        return d <= 1 ? n : __umulhi(n, m) >> s;
    }
};

// A thread walks one column of an i-chunk: it reads its own site of plane i + 1 and the
// j and k neighbours of plane i straight from global memory through L1, and keeps its
// values of planes i - 1 and i, so a site takes five reads instead of seven.  Blocks of
// 256 consecutive in-plane sites; items (chunk, block of sites), sites innermost, round
// robin over the resident blocks.
struct ColumnGeom {
    int n0, n1, n2;
    FastDiv d2;       // by the row length
    FastDiv dt;       // by the blocks of sites
    int i_begin, i_end;
    int ci;           // planes per item
    uint32_t items;
};

// Planes [i_begin, i_end) on `resident` blocks; `blocks` receives the grid.
inline ColumnGeom column_geom(int n0, int n1, int n2, int i_begin, int i_end, int64_t resident,
                              unsigned& blocks) {
    ColumnGeom g;
    g.n0 = n0;
    g.n1 = n1;
    g.n2 = n2;
    const uint32_t tiles = (uint32_t)(((int64_t)n1 * n2 + 255) / 256);
    g.d2 = FastDiv((uint32_t)n2);
    g.dt = FastDiv(tiles);
    g.i_begin = i_begin;
    g.i_end = i_end;
    // planes per item: 16 (two prologue reads in 82), fewer until every resident block
    // has two items
    const int planes = i_end - i_begin;
    const auto items = [&](int ci) { return (int64_t)tiles * ((planes + ci - 1) / ci); };
    g.ci = 16;
    while (g.ci > 1 && items(g.ci) < 2 * resident) g.ci /= 2;
    while (items(g.ci) > 0x7FFFFFFF) g.ci *= 2;
    g.items = (uint32_t)items(g.ci);
    blocks = (unsigned)(g.items < resident ? g.items : resident);
    return g;
}
inline bool column_wide(int n1, int n2) { return (int64_t)n1 * n2 >= 0x7FFFFF00; }

// Calls body(s, nb) for every site s of the planes, nb[v] = value v at the stencil sites
// (centre, ip, im, jp, jm, kp, km); value(s, v) fills the NV values of site s.
// I: the type of an in-plane site, int, or int64_t for planes of 2^31 sites and more
// (column_wide).
template <typename E, int NV, typename I, typename Value, typename Body>
__device__ __forceinline__ void walk_columns(const ColumnGeom& g, Value value, Body body) {
    const int n1 = g.n1, n2 = g.n2;
    const I n12 = (I)n1 * n2;
    const int64_t N = (int64_t)g.n0 * n12;
    for (uint32_t item = blockIdx.x; item < g.items; item += gridDim.x) {
        const uint32_t ic = g.dt.div(item);
        const I q = (I)(item - ic * g.dt.d) * 256 + (I)threadIdx.x;
        if (q >= n12) continue;
        const int j = sizeof(I) == 4 ? (int)g.d2.div((uint32_t)q) : (int)(q / n2);
        const int k = (int)(q - (I)j * n2);
        const I jp = j + 1 < n1 ? q + n2 : (I)k, jm = j > 0 ? q - n2 : q + (I)(n1 - 1) * n2;
        const I kp = k + 1 < n2 ? q + 1 : q - k, km = k > 0 ? q - 1 : q + (n2 - 1);
        int i = g.i_begin + (int)ic * g.ci;
        const int ie = min(i + g.ci, g.i_end);
        int64_t pl = (int64_t)i * n12;   // plane i
        E cur[NV], prev[NV];
        value((i > 0 ? pl : N) - n12 + q, prev);
        value(pl + q, cur);
        for (; i < ie; ++i) {
            const int64_t pn = i + 1 < g.n0 ? pl + n12 : 0;
            E nb[NV][7], v[NV];
            const auto neighbour = [&](int64_t s, int at) {
                value(s, v);
#pragma unroll
                for (int u = 0; u < NV; ++u) nb[u][at] = v[u];
            };
            neighbour(pn + q, 1);
            neighbour(pl + jp, 3);
            neighbour(pl + jm, 4);
            neighbour(pl + kp, 5);
            neighbour(pl + km, 6);
#pragma unroll
            for (int u = 0; u < NV; ++u) {
                nb[u][0] = cur[u];
                nb[u][2] = prev[u];
                prev[u] = cur[u];
                cur[u] = nb[u][1];
            }
            body(pl + q, nb);
            pl = pn;
        }
    }
}

}  // namespace tipt
