// Complex-field fused midpoint RK2 stage (C:2067-2215 rk2_step_table) and
// its entry point.  Same single-launch fusion as the real field: the midpoint
// phi~_a = phi_a + h1*pi_a is pointwise, so both reference passes run on the
// 7-point stencil of (phi1, phi2, pi1, pi2).
#include <cstring>

#include "rk2_complex.cuh"
#include "rk2_march.cuh"
#include "stage_kernels.cuh"
#include "tipt_internal.h"

namespace tipt {

// Longest V' row that the marching kernel stages; longer ones take FP64 lookups.
constexpr int64_t kMaxTableSmemC = 96 * 1024;

template <int S>
static int launch_complex_generic(const ComplexStageParams& p, cudaStream_t st) {
    const bool th = p.vkind == TIPT_VP_THERMAL;
    if (p.range) return th ? launch_stage_generic<ComplexSite<S, true, true>>(p, st) : launch_stage_generic<ComplexSite<S, false, true>>(p, st);
    return th ? launch_stage_generic<ComplexSite<S, true, false>>(p, st) : launch_stage_generic<ComplexSite<S, false, false>>(p, st);
}

int launch_complex_stage(int storage, ComplexStageParams p, cudaStream_t st) {
    set_complex_f32(p);
    const bool no_table = p.vkind == TIPT_VP_POLY || p.vkind == TIPT_VP_THERMAL;
    int64_t tb = no_table ? 0 : (int64_t)p.npts * (storage == TIPT_F32C ? 4 : 8);
    p.table_in_smem = (tb > 0 && tb <= kMaxTableSmemC) ? 1 : 0;
    // The marching kernel needs enough planes of tiles, and more of them where rows are not
    // whole 128-byte lines (march / generic in us: 64^3 13.7 / 13.2, 96^3 27.8 / 27.6, 128^3 49 /
    // 60, 256^3 290 / 580; 80^3 49 / 20, 112^3 75 / 43, 144^3 121 / 82, 208^3 247 / 233, 240^3
    // 322 / 347).
    const int64_t sites = (int64_t)p.n0 * p.n1 * p.n2;
    const bool pays = march_tiles_installed() || march_kseg_installed() ||
                      sites >= (p.n2 % 32 == 0 ? 1 << 20 : 12 << 20);
    if (storage == TIPT_F32C && (kernel_policy() == 2 || (kernel_policy() == 0 && pays))) {
        if (complex_march_supported(p)) return launch_complex_march(p, st);
        if (kernel_policy() == 2)
            return fail(TIPT_ERR_UNSUPPORTED, "the complex marching kernel does not take this "
                        "call (Z_N active, noise arrays, table or shape)");
    }
    switch (storage) {
        case TIPT_F64: return launch_complex_generic<TIPT_F64>(p, st);
        case TIPT_F32: return launch_complex_generic<TIPT_F32>(p, st);
        case TIPT_F32C: return launch_complex_generic<TIPT_F32C>(p, st);
    }
    return fail(TIPT_ERR_STORAGE, "unknown storage %d", storage);
}

}  // namespace tipt

using namespace tipt;

// Checks a complex stage call and fills its parameters (one midpoint stage of
// size dt with the pass-2 hash multiplier; callers adjust the half steps).
static int complex_stage_call(int storage, const void* phi1, const void* phi2, const void* pi1,
                              const void* pi2, void* phi1_out, void* phi2_out, void* pi1_out,
                              void* pi2_out, int64_t nx, int64_t ny, int64_t nz,
                              const tipt_step_params* sp, const tipt_vsource* vp,
                              const tipt_complex_terms* ct, const void* noise1,
                              const void* noise2, ComplexStageParams& p) {
    int rc;
    if ((rc = check_state(storage, phi1, phi2, phi1_out, phi2_out, nx, ny, nz)) ||
        (rc = check_state(storage, pi1, pi2, pi1_out, pi2_out, nx, ny, nz)))
        return rc;
    {
        const int64_t bytes = nx * ny * nz * elem_bytes(storage);
        const void* ins[4] = {phi1, phi2, pi1, pi2};
        const void* outs[4] = {phi1_out, phi2_out, pi1_out, pi2_out};
        for (int a = 0; a < 4; ++a) {
            for (int b = 0; b < 4; ++b)
                if (overlap(outs[a], ins[b], bytes))
                    return fail(TIPT_ERR_ARG, "an output array overlaps an input array");
            for (int b = a + 1; b < 4; ++b)
                if (overlap(outs[a], outs[b], bytes))
                    return fail(TIPT_ERR_ARG, "two output arrays overlap");
        }
    }
    if (!sp) return fail(TIPT_ERR_ARG, "step params are NULL");
    if ((rc = check_vsource(vp, "vp"))) return rc;
    if (vp->kind == TIPT_VP_TABLE2D)
        return fail(TIPT_ERR_UNSUPPORTED, "complex field takes a 1-D V'(rho) table");
    if ((noise1 == nullptr) != (noise2 == nullptr))
        return fail(TIPT_ERR_ARG, "noise1 and noise2 must both be given or both be NULL");
    if (noise1 && ((rc = check_ptr(noise1, storage == TIPT_F32 ? 4 : 8, "noise1")) ||
                   (rc = check_ptr(noise2, storage == TIPT_F32 ? 4 : 8, "noise2"))))
        return rc;
    memset(&p, 0, sizeof(p));
    p.f[0] = phi1;
    p.f[1] = phi2;
    p.f[2] = pi1;
    p.f[3] = pi2;
    p.o[0] = phi1_out;
    p.o[1] = phi2_out;
    p.o[2] = pi1_out;
    p.o[3] = pi2_out;
    p.n0 = (int)nx;
    p.n1 = (int)ny;
    p.n2 = (int)nz;
    p.h1 = 0.5 * sp->dt;
    p.h2 = sp->dt;
    p.inv_dx2 = 1.0 / (sp->dx * sp->dx);
    p.eta = sp->eta_eff;
    p.inv_mu2 = 1.0 / (sp->mu * sp->mu);
    p.inv_a2 = sp->inv_a2;
    p.noise1 = noise1;
    p.noise2 = noise2;
    p.ns_eff = sp->noise_scale;
    p.nfac = 1.0;
    p.step = sp->noise_step;
    p.mul = kPass2Mul;
    p.seed = sp->noise_seed;
    if (ct) {
        p.zn_n = ct->zn_n;
        p.zn_dv = ct->zn_dv;
        p.zn_active = ct->zn_active;
        p.eps4 = ct->eps4;
    }
    p.vkind = vp->kind;
    p.npts = vp->npts;
    p.table = vp->table;
    p.tmin = vp->tmin;
    p.dinv = vp->dinv;
    p.c1 = vp->c1;
    p.c2 = vp->c2;
    p.c3 = vp->c3;
    if (vp->kind == TIPT_VP_THERMAL) p.th = thermal_site(*vp->thermal, vp->T);
    return TIPT_OK;
}


extern "C" int tipt_complex_rk2_step_table(int storage, const void* phi1, const void* phi2,
                                           const void* pi1, const void* pi2, void* phi1_out,
                                           void* phi2_out, void* pi1_out, void* pi2_out, int64_t nx,
                                           int64_t ny, int64_t nz, const tipt_step_params* sp,
                                           const tipt_vsource* vp,
                                           const tipt_complex_terms* ct, const void* noise1,
                                           const void* noise2, void* stream) {
    ComplexStageParams p;
    int rc = complex_stage_call(storage, phi1, phi2, pi1, pi2, phi1_out, phi2_out, pi1_out,
                                pi2_out, nx, ny, nz, sp, vp, ct, noise1, noise2, p);
    if (rc) return rc;
    return launch_complex_stage(storage, p, (cudaStream_t)stream);
}

extern "C" int tipt_complex_rk2_step_table_range(int storage, const void* phi1, const void* phi2,
                                                 const void* pi1, const void* pi2, void* phi1_out,
                                                 void* phi2_out, void* pi1_out, void* pi2_out,
                                                 int64_t nx, int64_t ny, int64_t nz,
                                                 const tipt_step_params* sp,
                                                 const tipt_vsource* vp,
                                                 const tipt_complex_terms* ct, const void* noise1,
                                                 const void* noise2, uint32_t* range,
                                                 uint32_t* range_next, void* stream) {
    ComplexStageParams p;
    int rc = complex_stage_call(storage, phi1, phi2, pi1, pi2, phi1_out, phi2_out, pi1_out,
                                pi2_out, nx, ny, nz, sp, vp, ct, noise1, noise2, p);
    if (rc) return rc;
    if ((rc = check_ptr(range, 4, "range")) || (rc = check_ptr(range_next, 4, "range_next")))
        return rc;
    if (overlap(range, range_next, 12)) return fail(TIPT_ERR_ARG, "range and range_next overlap");
    p.range = reinterpret_cast<unsigned int*>(range);
    p.range_next = reinterpret_cast<unsigned int*>(range_next);
    return launch_complex_stage(storage, p, (cudaStream_t)stream);
}

extern "C" int tipt_complex_rk2_fused_table(int storage, const void* phi1, const void* phi2,
                                            const void* pi1, const void* pi2, void* phi1_out,
                                            void* phi2_out, void* pi1_out, void* pi2_out,
                                            void* mid1, void* mid2, void* mid3, void* mid4,
                                            int64_t nx, int64_t ny, int64_t nz,
                                            const tipt_step_params* sp,
                                            const tipt_vsource* vp_T, const tipt_vsource* vp_Tm,
                                            const tipt_complex_terms* ct, const void* noise1,
                                            const void* noise2, void* stream) {
    ComplexStageParams a, b;
    int rc = complex_stage_call(storage, phi1, phi2, pi1, pi2, mid1, mid2, mid3, mid4, nx, ny, nz,
                                sp, vp_T, ct, noise1, noise2, a);
    if (rc) return rc;
    rc = complex_stage_call(storage, mid1, mid2, mid3, mid4, phi1_out, phi2_out, pi1_out, pi2_out,
                            nx, ny, nz, sp, vp_Tm, ct, noise1, noise2, b);
    if (rc) return rc;
    // first half at T (C:1829-1946), pass-2 multiplier; second at T_mid
    // (C:1948-2064), pass-4 multiplier; 0.5 noise (array or hash) in each
    for (ComplexStageParams* q : {&a, &b}) {
        q->h1 = q->h2 = 0.5 * sp->dt;
        q->nfac = 0.5;
        q->ns_eff = 0.5 * sp->noise_scale;
    }
    b.mul = kPass4Mul;
    if ((rc = launch_complex_stage(storage, a, (cudaStream_t)stream))) return rc;
    return launch_complex_stage(storage, b, (cudaStream_t)stream);
}
