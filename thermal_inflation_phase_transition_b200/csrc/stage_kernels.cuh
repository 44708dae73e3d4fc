// The generic stage kernel: the per-site update (stage_site.cuh) for every shape and
// storage.
#pragma once

#include "column_walk.cuh"
#include "stage_site.cuh"

namespace tipt {

__device__ __forceinline__ F32CConst stage_consts(const RealStageParams& p) { return f32c_const(p); }
__device__ __forceinline__ F32CConst stage_consts(const ComplexStageParams&) { return F32CConst{}; }
inline int stage_begin(const RealStageParams& p) { return p.i_begin; }
inline int stage_end(const RealStageParams& p) { return p.i_end; }
inline int stage_begin(const ComplexStageParams&) { return 0; }
inline int stage_end(const ComplexStageParams& p) { return p.n0; }

// Walks columns (column_walk.cuh); float32 storage keeps the midpoint values along the
// column too, five conversions and back a site instead of seven.  V' rows are read in
// place through L1, a 2-D table's two rows blended at each lookup.
//
// Bound: the latency of the loads and of the FP64 chains (64 registers a thread, four
// blocks an SM; five or six blocks spill), then issue and, in float32 storage, the
// conversions.  256^3 float32 script loop 337 -> 303 us against one site per thread with
// seven reads, complex 512x512x64 647 -> 583 us, 126x131x98 FP64 driver 1050 -> 1003 us.
// (A block walking the planes with the midpoint field in shared memory measured 251 us
// for the float32 stage alone, and slower on odd rows.)
template <class M, typename I>
__global__ void __launch_bounds__(256, 4) stage_generic(typename M::Params p_in, ColumnGeom g) {
    typename M::Params p = p_in;
    M::prepare(p);
    using E = typename M::E;
    RangeAcc racc;
    const auto row = M::row(p);
    const F32CConst kc = stage_consts(p);
    const int64_t N = (int64_t)p.n0 * p.n1 * p.n2;
    walk_columns<E, M::NV, I>(
        g,
        [&](int64_t s, E (&v)[M::NV]) {
            E raw[M::NR];
            M::load(p, s, N, raw);
            M::values(p, raw, v);
        },
        [&](int64_t s, const E (&nb)[M::NV][7]) { M::update(p, kc, row, nb, s, N, racc); });
    if constexpr (M::RG) racc.flush(p.range);
}

// ----------------------------------------------------------------- launch ---
template <class M>
static int launch_stage_generic(const typename M::Params& p, cudaStream_t st) {
    auto kern = column_wide(p.n1, p.n2) ? stage_generic<M, int64_t> : stage_generic<M, int>;
    unsigned blocks;
    const ColumnGeom g = column_geom(p.n0, p.n1, p.n2, stage_begin(p), stage_end(p),
                                     4 * (int64_t)num_sms(), blocks);
    kern<<<blocks, 256, 0, st>>>(p, g);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TIPT_OK : fail_cuda(e, "stage_generic launch");
}

}  // namespace tipt
