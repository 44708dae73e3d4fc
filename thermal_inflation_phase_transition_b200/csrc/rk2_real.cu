// Real-field fused midpoint RK2 stage kernels.
//
//  * stage_generic (stage_kernels.cuh): threads walk columns, any lattice shape and storage;
//    loads the stencil of phi and pi straight from HBM through L1 and reads V' tables in place.
//  * rk2_stage_march (rk2_march.cuh): rows by bulk copies into a shared-memory ring, n2 % 4
//    == 0; taken where march_pays.
#include "rk2_real.cuh"
#include "rk2_march.cuh"
#include "stage_kernels.cuh"
#include "tipt_internal.h"

namespace tipt {

// Bytes of shared memory the V' row needs for storage S (0 if polynomial).
static int64_t table_smem_bytes(int S, const RealStageParams& p) {
    if (p.vkind == TIPT_VP_POLY || p.vkind == TIPT_VP_THERMAL) return 0;
    return (int64_t)p.npts * (S == TIPT_F32C ? 4 : 8);
}

static int g_num_sms = 0;
int num_sms() {
    if (g_num_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_num_sms <= 0) g_num_sms = 148;
    }
    return g_num_sms;
}

template <int S>
static int launch_generic(const RealStageParams& p, cudaStream_t st) {
    const auto go = [&](auto src) {
        constexpr int SRC = decltype(src)::value;
        return p.range ? launch_stage_generic<RealSite<S, SRC, true>>(p, st)
                       : launch_stage_generic<RealSite<S, SRC, false>>(p, st);
    };
    if (p.vkind == TIPT_VP_THERMAL) return go(std::integral_constant<int, kSrcThermal>{});
    if (p.vkind == TIPT_VP_TABLE2D) return go(std::integral_constant<int, kSrcRow2>{});
    return go(std::integral_constant<int, kSrcRow>{});
}

// Largest V' row staged in shared memory; longer 1-D tables are read from
// global memory (L1/L2 resident), longer 2-D tables are rejected.
constexpr int64_t kMaxTableSmem = 96 * 1024;

// Kernel choice: 0 automatic, 1 generic kernel only, 2 marching kernel only.
static int g_kernel_policy = 0;

int kernel_policy() { return g_kernel_policy; }

// A lattice whose contiguous extent is 1 (the reference's 2-D form nz = 1) is
// relabelled so the contiguous axis is the longest non-trivial one: (nx, ny, 1)
// -> (1, nx, ny) and (nx, 1, 1) -> (1, 1, nx).  Linear site indices, hence the
// noise keys, are unchanged; the neighbour set of every site is the same.
static void canonical_shape(RealStageParams& p) {
    if (p.n2 != 1) return;
    if (p.n1 > 1) {
        p.n2 = p.n1;
        p.n1 = p.n0;
        p.n0 = 1;
    } else {
        p.n2 = p.n0;
        p.n0 = 1;
    }
}

// Whether the marching kernel is the faster one where it applies (march / generic in us, 2-D
// table unless said).  It reads whole rows by bulk copies and runs at most 17 warps an SM
// against the generic kernel's 32:
//  * a lattice has to be large enough to fill its pipeline: FP64 64^3 9.8 / 7.2, 128^3 34.3 /
//    33, 256^3 219 / 235; float32 96^3 19.8 / 17.4, 128^3 34.3 / 36.6, 1024^2 23.2 / 22.5;
//    compensated FP32 64^3 10.2 / 7.6, 200x48x64 16.5 / 13.4, 96^3 16.2 / 16.9;
//  * the row length and the row count decide how many consumer warps a tile has.  FP64 with 10
//    to 13 warps 160^3 78 / 62, 208^3 144 / 139, 320^3 539 / 456, with 15 or 16 240^3 190 /
//    205, 256x100x512 174 / 186; float32 with 9 to 11 144^3 54 / 50, 160^3 81 / 67, 320^3 615
//    / 508, with 12 and more 224^3 173 / 191, 256^3 223 / 259, 384^3 836 / 890;
//  * compensated FP32 halves the instructions of the generic kernel where rows are whole
//    128-byte lines (128^3 25.6 / 36.6, 256^3 134 / 254); other rows are copied one by one
//    (80^3 48 / 12, 112^3 68 / 25, 208^3 178 / 140, 240^3 228 / 210) and have no tile above 256
//    sites (the consumers of such a row's tile would be more than 512);
//  * inline thermal V', long FP64 chains: 256^3, two halves, FP64 1032 / 841, float32 1009 /
//    894; compensated FP32, whose stencil reads four components, 256^3 804 / 853, 96^3 67 / 54;
//  * a noise array in the FP64 and float32 storages, loaded where the hash would be drawn (the
//    script's loop: 256^3 FP64 469 / 316, float32 344 / 337).
static bool march_pays(int storage, const RealStageParams& p, int64_t sites, int warps) {
    if (storage == TIPT_F32C)
        return p.n2 % 32 == 0 && sites >= (p.vkind == TIPT_VP_THERMAL ? 6 << 20 : 3 << 18);
    if (p.vkind == TIPT_VP_THERMAL || p.noise) return false;
    return storage == TIPT_F64 ? sites >= 4 << 20 && warps >= 15 : sites >= 2 << 20 && warps >= 12;
}

int launch_real_stage(int storage, RealStageParams p, cudaStream_t st) {
    if (p.i_end == 0) {
        canonical_shape(p);
        p.i_begin = 0;
        p.i_end = p.n0;
    }
    const int64_t tb = table_smem_bytes(storage, p);
    p.table_in_smem = (tb > 0 && tb <= kMaxTableSmem) ? 1 : 0;
    if (p.vkind == TIPT_VP_TABLE2D && !p.table_in_smem)
        return fail(TIPT_ERR_UNSUPPORTED, "2-D V' table row of %d points exceeds %lld bytes of "
                    "shared memory", p.npts, (long long)kMaxTableSmem);
    const int64_t smem = p.table_in_smem ? tb : 0;
    set_f32c_pairs(p);
    const int64_t sites = (int64_t)p.n1 * p.n2 * (p.i_end - p.i_begin);
    int warps = 0;
    const bool march = g_kernel_policy == 2   ? march_supported(storage, p)
                       : g_kernel_policy == 1 ? false
                       : march_tiles_installed() ? march_supported(storage, p)
                                              : march_pays(storage, p, sites, 16) &&
                                                    march_supported(storage, p, &warps) &&
                                                    march_pays(storage, p, sites, warps);
    if (g_kernel_policy == 2 && !march)
        return fail(TIPT_ERR_UNSUPPORTED, "marching kernel does not cover this shape/storage");
    if (march) return launch_march(storage, p, smem, st);
    switch (storage) {
        case TIPT_F64: return launch_generic<TIPT_F64>(p, st);
        case TIPT_F32: return launch_generic<TIPT_F32>(p, st);
        case TIPT_F32C: return launch_generic<TIPT_F32C>(p, st);
    }
    return fail(TIPT_ERR_STORAGE, "unknown storage %d", storage);
}

}  // namespace tipt

// Selects the real-field stage kernel: 0 automatic (the marching kernel where it
// applies), 1 the generic kernel, 2 the marching kernel or an error.  Results are
// bitwise identical between the two kernels; this exists for tests and tuning.
extern "C" int tipt_set_kernel_policy(int policy) {
    if (policy < 0 || policy > 2) return tipt::fail(TIPT_ERR_ARG, "policy must be 0, 1 or 2");
    tipt::g_kernel_policy = policy;
    return TIPT_OK;
}
