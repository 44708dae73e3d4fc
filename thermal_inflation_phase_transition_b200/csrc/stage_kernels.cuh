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

// One site per thread (grid stride): the stencil straight from global memory through
// L1.  Bound: the latency of the loads and of the FP64 chains (64 registers a thread,
// four blocks an SM; five or six blocks spill), then issue and, in float32 storage, the
// conversions.  Coordinates by two multiplications and 32-bit site indices instead of
// 64-bit divisions and addresses: a 256^3 float32 stage with noise array, 16384-point
// table and range 283 -> 210 us, the complex one at 512x512x64 534 -> 420 us.  (A tile
// walking the planes with the midpoint field in shared memory measured 251 us, and
// slower on odd rows.)
struct GenericGeom {
    FastDiv d1, d2;
    int i_begin, i_end;
};

// I: the type of a site index, int (sites < 2^31: coordinates by multiplication, one
// instruction per address) or int64_t.
template <class M, typename I>
__global__ void __launch_bounds__(256, 4) stage_generic(typename M::Params p_in, GenericGeom g) {
    typename M::Params p = p_in;
    M::prepare(p);
    using E = typename M::E;
    RangeAcc racc;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (p.table_in_smem) M::stage(p, smem_raw);
    const F32CConst kc = stage_consts(p);
    const int64_t N = (int64_t)p.n0 * p.n1 * p.n2;
    const I n12 = (I)((int64_t)p.n1 * p.n2);
    const int64_t s_end = (int64_t)g.i_end * n12;
    for (int64_t sl = (int64_t)g.i_begin * n12 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
         sl < s_end; sl += (int64_t)gridDim.x * blockDim.x) {
        const I s = (I)sl;
        int i, j, k;
        if constexpr (sizeof(I) == 4) {
            const uint32_t r = g.d2.div((uint32_t)s);
            k = (int)((uint32_t)s - r * (uint32_t)p.n2);
            i = (int)g.d1.div(r);
            j = (int)(r - (uint32_t)i * (uint32_t)p.n1);
        } else {
            const I r = s / p.n2;
            k = (int)(s - r * p.n2);
            i = (int)(r / p.n1);
            j = (int)(r - (I)i * p.n1);
        }
        const I idx[7] = {
            s,
            s + ((i + 1 < p.n0) ? n12 : -(I)(p.n0 - 1) * n12),
            s + ((i > 0) ? -n12 : (I)(p.n0 - 1) * n12),
            s + ((j + 1 < p.n1) ? (I)p.n2 : -(I)(p.n1 - 1) * p.n2),
            s + ((j > 0) ? -(I)p.n2 : (I)(p.n1 - 1) * p.n2),
            s + ((k + 1 < p.n2) ? (I)1 : -(I)(p.n2 - 1)),
            s + ((k > 0) ? (I)-1 : (I)(p.n2 - 1))};
        E nb[M::NR][7];
#pragma unroll
        for (int q = 0; q < 7; ++q) {
            E raw[M::NR];
            M::load(p, idx[q], N, raw);
#pragma unroll
            for (int u = 0; u < M::NR; ++u) nb[u][q] = raw[u];
        }
        M::update(p, kc, smem_raw, nb, sl, N, racc);
    }
    if constexpr (M::RG) racc.flush(p.range);
}

// ----------------------------------------------------------------- launch ---
template <class M>
static int launch_stage_generic(const typename M::Params& p, int64_t smem, cudaStream_t st) {
    const bool small = (int64_t)p.n0 * p.n1 * p.n2 < (1ll << 31);
    auto kern = small ? stage_generic<M, int> : stage_generic<M, int64_t>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return fail_cuda(e, "stage_generic smem attribute");
    }
    GenericGeom g;
    g.d1 = FastDiv((uint32_t)p.n1);
    g.d2 = FastDiv((uint32_t)p.n2);
    g.i_begin = stage_begin(p);
    g.i_end = stage_end(p);
    const int64_t n = (int64_t)(g.i_end - g.i_begin) * p.n1 * p.n2;
    int64_t blocks = (n + 255) / 256;
    const int64_t cap = (int64_t)num_sms() * 8;
    if (blocks > cap) blocks = cap;
    kern<<<(unsigned)blocks, 256, (size_t)smem, st>>>(p, g);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TIPT_OK : fail_cuda(e, "stage_generic launch");
}

}  // namespace tipt
