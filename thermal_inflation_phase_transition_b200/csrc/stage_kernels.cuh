// The generic stage kernel: the per-site update (stage_site.cuh) for every shape and
// storage.
#pragma once

#include "stage_site.cuh"
#include "tipt_internal.h"

namespace tipt {

__device__ __forceinline__ F32CConst stage_consts(const RealStageParams& p) { return f32c_const(p); }
__device__ __forceinline__ F32CConst stage_consts(const ComplexStageParams&) { return F32CConst{}; }
inline int stage_begin(const RealStageParams& p) { return p.i_begin; }
inline int stage_end(const RealStageParams& p) { return p.i_end; }
inline int stage_begin(const ComplexStageParams&) { return 0; }
inline int stage_end(const ComplexStageParams& p) { return p.n0; }

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
// values of planes i - 1 and i, so a site takes five reads (and float32 storage five
// midpoint conversions) instead of seven.  Blocks of 256 consecutive in-plane sites;
// items (chunk, block of sites), sites innermost, round robin over the resident blocks,
// which stage a table row once each.
//
// Bound: the latency of the loads and of the FP64 chains (64 registers a thread, four
// blocks an SM; five or six blocks spill), then issue and, in float32 storage, the
// conversions.  256^3 float32 script loop 337 -> 303 us against one site per thread with
// seven reads, complex 512x512x64 647 -> 583 us, 126x131x98 FP64 driver 1050 -> 1003 us.
// (A block walking the planes with the midpoint field in shared
// memory measured 251 us for the float32 stage, and slower on odd rows.)
struct GenericGeom {
    FastDiv d2;       // by the row length
    FastDiv dt;       // by the blocks of sites
    int i_begin, i_end;
    int ci;           // planes per item
    uint32_t items;
};

// I: the type of an in-plane site, int, or int64_t for planes of 2^31 sites and more.
template <class M, typename I>
__global__ void __launch_bounds__(256, 4) stage_generic(typename M::Params p_in, GenericGeom g) {
    typename M::Params p = p_in;
    M::prepare(p);
    using E = typename M::E;
    constexpr int NV = M::NV, NR = M::NR;
    RangeAcc racc;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (p.table_in_smem) M::stage(p, smem_raw);
    const F32CConst kc = stage_consts(p);
    const int n1 = p.n1, n2 = p.n2;
    const I n12 = (I)n1 * n2;
    const int64_t N = (int64_t)p.n0 * n12;
    const auto value = [&](int64_t s, E (&v)[NV]) {
        E raw[NR];
        M::load(p, s, N, raw);
        M::values(p, raw, v);
    };
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
            const int64_t pn = i + 1 < p.n0 ? pl + n12 : 0;
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
            M::update(p, kc, smem_raw, nb, pl + q, N, racc);
            pl = pn;
        }
    }
    if constexpr (M::RG) racc.flush(p.range);
}

// ----------------------------------------------------------------- launch ---
template <class M>
static int launch_stage_generic(const typename M::Params& p, int64_t smem, cudaStream_t st) {
    const int64_t n12 = (int64_t)p.n1 * p.n2;
    auto kern = n12 < 0x7FFFFF00 ? stage_generic<M, int> : stage_generic<M, int64_t>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return fail_cuda(e, "stage_generic smem attribute");
    }
    GenericGeom g;
    const uint32_t tiles = (uint32_t)((n12 + 255) / 256);
    g.d2 = FastDiv((uint32_t)p.n2);
    g.dt = FastDiv(tiles);
    g.i_begin = stage_begin(p);
    g.i_end = stage_end(p);
    // planes per item: 16 (two prologue reads in 82), fewer until every resident block
    // has two items
    const int planes = g.i_end - g.i_begin;
    const int64_t resident = 4 * (int64_t)num_sms();
    const auto items = [&](int ci) { return (int64_t)tiles * ((planes + ci - 1) / ci); };
    g.ci = 16;
    while (g.ci > 1 && items(g.ci) < 2 * resident) g.ci /= 2;
    while (items(g.ci) > 0x7FFFFFFF) g.ci *= 2;
    g.items = (uint32_t)items(g.ci);
    const int64_t blocks = g.items < resident ? g.items : resident;
    kern<<<(unsigned)blocks, 256, (size_t)smem, st>>>(p, g);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TIPT_OK : fail_cuda(e, "stage_generic launch");
}

}  // namespace tipt
