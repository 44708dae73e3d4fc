// Real-field fused midpoint RK2 stage kernels.
//
//  * rk2_stage_generic: one site per thread (grid-stride), any lattice shape
//    and storage; loads the 7-point stencil of phi and pi straight from HBM
//    through L1.  Used for shapes the marching kernel does not cover.
//  * rk2_stage_march (rk2_march.cuh): the bandwidth kernel for n2 % 4 == 0.
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
static int launch_generic(const RealStageParams& p, int64_t smem, cudaStream_t st) {
    const bool th = p.vkind == TIPT_VP_THERMAL;
    if (p.range) return th ? launch_stage_generic<RealSite<S, true, true>>(p, smem, st) : launch_stage_generic<RealSite<S, false, true>>(p, smem, st);
    return th ? launch_stage_generic<RealSite<S, true, false>>(p, smem, st) : launch_stage_generic<RealSite<S, false, false>>(p, smem, st);
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

// Whether the marching kernel is the faster one where it applies.  It runs 17 warps an
// SM against the generic kernel's 32, so it hides latency worse:
//  * the inline thermal V', long FP64 chains (256^3, two halves: FP64 1032 against 841 us,
//    float32 1009 against 894 us), except in compensated FP32 on large lattices, whose
//    stencil reads four components (256^3 804 against 853 us, 96^3 67 against 54 us);
//  * a noise array in the FP64 and float32 storages, loaded where the hash would be
//    drawn (the script's loop: 256^3 FP64 469 against 316 us, float32 344 against 337).
// With hash noise it wins: 256^3 FP64 227 against 259 us, float32 227 against 279 us.
static bool march_pays(int storage, const RealStageParams& p) {
    if (p.vkind == TIPT_VP_THERMAL)
        return storage == TIPT_F32C && (int64_t)p.n0 * p.n1 * p.n2 >= 6 << 20;
    return storage == TIPT_F32C || !p.noise;
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
    const bool march = g_kernel_policy != 1 && march_supported(storage, p) &&
                       (g_kernel_policy == 2 || march_pays(storage, p));
    if (g_kernel_policy == 2 && !march)
        return fail(TIPT_ERR_UNSUPPORTED, "marching kernel does not cover this shape/storage");
    if (march) return launch_march(storage, p, smem, st);
    switch (storage) {
        case TIPT_F64: return launch_generic<TIPT_F64>(p, smem, st);
        case TIPT_F32: return launch_generic<TIPT_F32>(p, smem, st);
        case TIPT_F32C: return launch_generic<TIPT_F32C>(p, smem, st);
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
