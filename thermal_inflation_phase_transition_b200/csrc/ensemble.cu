// Batched ensemble of independent real-field replicas with uneven lattice
// sizes, seeds and potentials, advanced by one persistent launch per step.
//
// The reference runs one replica per CLI invocation (one numba call per
// step).  Here every replica's state is a slice of one packed buffer (planar
// for the compensated storage: hi plane of all replicas, then the lo plane);
// a work-list of chunks (replica, site range) covers the active replicas and
// persistent CTAs walk it, so a step of 1792 small replicas is one launch
// instead of 1792.  Each site runs the same midpoint arithmetic as the
// single-lattice kernels, with the replica's own extents, noise seed and
// amplitude, and polynomial V'(phi) = c1 phi + c2 phi^2 + c3 phi^3 (the
// potential family's derivative: c1 = 2D(T^2-T0^2), c2 = -3ET, c3 = lam).
// Results are bitwise those of stepping the replica alone with the generic
// kernel.
//
// tipt_ensemble_observe counts, per replica, the
// fraction of sites with phi > thr; the first time it exceeds the stop
// fraction the step is recorded as the replica's first-passage step, and once
// it exceeds the retire fraction (>= the stop fraction) the replica is retired
// (its chunks are skipped from then on).
#include <cooperative_groups.h>

#include <cstring>

#include "rk2_march.cuh"
#include "rk2_real.cuh"
#include "tipt_internal.h"

namespace tipt {

struct EnsParams {
    const void* phi;
    const void* pi;
    void* phi_out;
    void* pi_out;
    int64_t n_total;
    const tipt_replica* reps;
    const tipt_chunk* chunks;
    int n_chunks;
    // a shape class instead of a chunk list: replicas rids[0..*n_rids), kClassChunk sites a
    // chunk, cpr chunks a replica
    const int32_t* rids;
    const int32_t* n_rids;
    int cpr;
    uint32_t m1, m2;                     // tipt_replica's multipliers of the class
    int* status;                         // tipt_device_status's word
    int pieces;                          // blocks that share a chunk
    const int32_t* active;
    double h1, h2, inv_dx2, eta, inv_mu2, inv_a2;
    uint64_t step;                       // hash step = step (+ *ctr + offset)
    const unsigned long long* ctr;       // device step counter or nullptr
    long long offset;
};

// x / d for x < 2^32 / d by a multiply-high with m = ceil(2^32 / d) (exact:
// x m / 2^32 = x/d + x e / (d 2^32) with e = m d - 2^32 < d); m = 0 means d = 1.
__device__ __forceinline__ uint32_t fdiv(uint32_t x, uint32_t m) { return m ? __umulhi(x, m) : x; }

constexpr int kClassChunk = 8192;

// Bound by the latency of the loads: four blocks an SM (at three, with 76 registers, the
// compensated kernel over a chunk list took 219 instead of 155 us for 1024 replicas of 128^2).
template <int S, bool CLASS>
__global__ void __launch_bounds__(256, S == TIPT_F32C ? 4 : 0) ensemble_stage_kernel(EnsParams e) {
    const uint64_t step = e.step + (e.ctr ? *e.ctr + (unsigned long long)e.offset : 0ull);
    // Blocks that share a chunk take its 256-thread passes in turn.
    const int stride = e.pieces * (int)blockDim.x;
    const int n_chunks = CLASS && e.n_rids ? *e.n_rids * e.cpr : e.n_chunks;
    for (int64_t item = blockIdx.x; item < (int64_t)n_chunks * e.pieces; item += gridDim.x) {
        const int c = (int)(item / e.pieces);
        const int t0 = (int)(item - (int64_t)c * e.pieces) * (int)blockDim.x + (int)threadIdx.x;
        tipt_chunk ch;
        if constexpr (CLASS) {
            ch.replica = e.rids[c / e.cpr];
            ch.begin = (int64_t)(c % e.cpr) * kClassChunk;
        } else {
            ch = e.chunks[c];
        }
        if (!e.active[ch.replica]) continue;
        tipt_replica rp = e.reps[ch.replica];
        if constexpr (CLASS) {
            if (rp.offset & 3) {  // as the marching stage: skipped and reported
                if (threadIdx.x == 0) atomicExch(e.status, (int)TIPT_ERR_ALIGN);
                continue;
            }
            const int64_t left = (int64_t)rp.n0 * rp.n1 * rp.n2 - ch.begin;
            ch.count = left < kClassChunk ? (int32_t)left : kClassChunk;
            rp.m1 = e.m1;
            rp.m2 = e.m2;
        }
        // the replica as a single lattice with a polynomial V' and hash noise
        RealStageParams p;
        memset(&p, 0, sizeof(p));
        p.n0 = rp.n0;
        p.n1 = rp.n1;
        p.n2 = rp.n2;
        p.h1 = e.h1;
        p.h2 = e.h2;
        p.inv_dx2 = e.inv_dx2;
        p.eta = e.eta;
        p.inv_mu2 = e.inv_mu2;
        p.inv_a2 = e.inv_a2;
        p.ns_eff = rp.noise_scale;
        p.nfac = 1.0;
        p.step = step;
        p.mul = kPass2Mul;
        p.seed = rp.seed;
        p.vkind = TIPT_VP_POLY;
        p.c1 = rp.c1;
        p.c2 = rp.c2;
        p.c3 = rp.c3;
        const uint32_t n12 = (uint32_t)rp.n1 * (uint32_t)rp.n2;
        set_f32c_pairs(p);
        const F32CConst kc = f32c_const(p);
        if constexpr (S == TIPT_F32C) {
            // Site pairs (s, s + 1) with s even share i and j when n2 is even: one
            // 8-byte load per field plane and neighbour, the stencil sums and the
            // update in the lanes of the packed FP32x2 instructions (bitwise the
            // one-site arithmetic, as in the marching kernel).
            if ((rp.n2 & 1) == 0 && ((ch.begin | ch.count | rp.offset) & 1) == 0) {
                const float* phi = static_cast<const float*>(e.phi);
                const float* pi = static_cast<const float*>(e.pi);
                float* po = static_cast<float*>(e.phi_out);
                float* vo = static_cast<float*>(e.pi_out);
                const int64_t N = e.n_total;
                for (int t = t0; 2 * t < ch.count; t += stride) {
                    const uint32_t s = (uint32_t)(ch.begin + 2 * t);
                    const uint32_t q = fdiv(s, rp.m2);
                    const uint32_t k = s - q * (uint32_t)rp.n2;
                    const uint32_t i = fdiv(q, rp.m1);
                    const uint32_t j = q - i * (uint32_t)rp.n1;
                    const int64_t g = rp.offset + s;
                    const int64_t o4[4] = {
                        (i + 1 < (uint32_t)rp.n0) ? (int64_t)n12 : -(int64_t)(rp.n0 - 1) * n12,
                        (i > 0) ? -(int64_t)n12 : (int64_t)(rp.n0 - 1) * n12,
                        (j + 1 < (uint32_t)rp.n1) ? rp.n2 : -(int64_t)(rp.n1 - 1) * rp.n2,
                        (j > 0) ? -(int64_t)rp.n2 : (int64_t)(rp.n1 - 1) * rp.n2};
                    const int64_t gkr = g + ((k + 2 < (uint32_t)rp.n2) ? 2 : 2 - (int64_t)rp.n2);
                    const int64_t gkl = g + ((k > 0) ? -1 : (int64_t)(rp.n2 - 1));
                    const float* base[4] = {phi, phi + N, pi, pi + N};  // phi hi, lo, pi hi, lo
                    float2 dsum[4], cen[4];
#pragma unroll
                    for (int f = 0; f < 4; ++f) {
                        const float* b = base[f];
                        const float2 cc = __ldg(reinterpret_cast<const float2*>(b + g));
                        float2 nb[6];
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            nb[u] = __ldg(reinterpret_cast<const float2*>(b + g + o4[u]));
                        const float kr = __ldg(b + gkr), kl = __ldg(b + gkl);  // k+1, k-1
                        // the order of stencil_sums_k: i and j terms, then the k pair
                        float2 acc;
                        if ((f & 1) == 0) {  // hi: sum (hi_n - hi_c)
                            acc = v_add(v_sub(nb[0], cc), v_sub(nb[1], cc));
                            acc = v_add(acc, v_sub(nb[2], cc));
                            acc = v_add(acc, v_sub(nb[3], cc));
                            const float2 kk = make_float2(
                                __fadd_rn(__fsub_rn(cc.y, cc.x), __fsub_rn(kl, cc.x)),
                                __fadd_rn(__fsub_rn(kr, cc.y), __fsub_rn(cc.x, cc.y)));
                            acc = v_add(acc, kk);
                        } else {             // lo: fma(-6, lo_c, sum lo_n)
                            acc = v_add(v_add(v_add(nb[0], nb[1]), nb[2]), nb[3]);
                            const float2 kk = make_float2(__fadd_rn(cc.y, kl), __fadd_rn(kr, cc.x));
                            acc = v_fma(vs<float2>(-6.0f), cc, v_add(acc, kk));
                        }
                        dsum[f] = acc;
                        cen[f] = cc;
                    }
                    F32CIn<float2> x;
                    x.dh_phi = dsum[0];
                    x.dl_phi = dsum[1];
                    x.dh_pi = dsum[2];
                    x.dl_pi = dsum[3];
                    x.phh = cen[0];
                    x.phl = cen[1];
                    x.pih = cen[2];
                    x.pil = cen[3];
                    float2 a, b, cc, d;
                    update_f32c<float2, false>(p, kc, static_cast<const float*>(nullptr), x, site_kick_f32c2(p, kc, (uint64_t)s), a, b,
                                        cc, d);
                    *reinterpret_cast<float2*>(po + g) = a;
                    *reinterpret_cast<float2*>(po + N + g) = b;
                    *reinterpret_cast<float2*>(vo + g) = cc;
                    *reinterpret_cast<float2*>(vo + N + g) = d;
                }
                continue;
            }
        }
        for (int t = t0; t < ch.count; t += stride) {
            const uint32_t s = (uint32_t)(ch.begin + t);
            const uint32_t q = fdiv(s, rp.m2);
            const uint32_t k = s - q * (uint32_t)rp.n2;
            const uint32_t i = fdiv(q, rp.m1);
            const uint32_t j = q - i * (uint32_t)rp.n1;
            const int64_t o_ip = (i + 1 < (uint32_t)rp.n0) ? (int64_t)n12 : -(int64_t)(rp.n0 - 1) * n12;
            const int64_t o_im = (i > 0) ? -(int64_t)n12 : (int64_t)(rp.n0 - 1) * n12;
            const int64_t o_jp = (j + 1 < (uint32_t)rp.n1) ? rp.n2 : -(int64_t)(rp.n1 - 1) * rp.n2;
            const int64_t o_jm = (j > 0) ? -(int64_t)rp.n2 : (int64_t)(rp.n1 - 1) * rp.n2;
            const int64_t o_kp = (k + 1 < (uint32_t)rp.n2) ? 1 : -(int64_t)(rp.n2 - 1);
            const int64_t o_km = (k > 0) ? -1 : (int64_t)(rp.n2 - 1);
            const int64_t g = rp.offset + s;
            const int64_t idx[7] = {g, g + o_ip, g + o_im, g + o_jp, g + o_jm, g + o_kp, g + o_km};
            if constexpr (S == TIPT_F64) {
                const double* phi = static_cast<const double*>(e.phi);
                const double* pi = static_cast<const double*>(e.pi);
                double ph[7], pv[7];
#pragma unroll
                for (int u = 0; u < 7; ++u) {
                    ph[u] = __ldg(phi + idx[u]);
                    pv[u] = __ldg(pi + idx[u]);
                }
                double a, b;
                update_f64<false>(p, static_cast<const double*>(nullptr), ph, pv, site_noise<double>(p, (uint64_t)s), a, b);
                static_cast<double*>(e.phi_out)[g] = a;
                static_cast<double*>(e.pi_out)[g] = b;
            } else {
                const float* phi = static_cast<const float*>(e.phi);
                const float* pi = static_cast<const float*>(e.pi);
                const int64_t N = e.n_total;
                float hh[7], hl[7], vh[7], vl[7];
#pragma unroll
                for (int u = 0; u < 7; ++u) {
                    hh[u] = __ldg(phi + idx[u]);
                    hl[u] = __ldg(phi + N + idx[u]);
                    vh[u] = __ldg(pi + idx[u]);
                    vl[u] = __ldg(pi + N + idx[u]);
                }
                F32CIn<float> x;
                stencil_sums_k(hh, hl, x.dh_phi, x.dl_phi);
                stencil_sums_k(vh, vl, x.dh_pi, x.dl_pi);
                x.phh = hh[0];
                x.phl = hl[0];
                x.pih = vh[0];
                x.pil = vl[0];
                float a, b, cc, d;
                update_f32c<float, false>(p, kc, static_cast<const float*>(nullptr), x, site_kick_f32c(p, kc, (uint64_t)s), a, b,
                                   cc, d);
                float* po = static_cast<float*>(e.phi_out);
                float* vo = static_cast<float*>(e.pi_out);
                po[g] = a;
                po[N + g] = b;
                vo[g] = cc;
                vo[N + g] = d;
            }
        }
    }
}

// The blocks of a replica (NC, a cluster) count its sites with phi > thr (a whole number, so
// the order is free) and add the counts up in the first block's shared memory; 16-byte loads
// where the replica's planes are aligned.  Bound by HBM: 112 replicas of 128^2, 64^3 and 96^3
// (23.6 M sites) 970 us with one block of 256 threads a replica and single loads -> 58 us on
// clusters of eight blocks of 512 threads.
struct ObsParams {
    const void* phi;
    int64_t n_total;
    const tipt_replica* reps;
    int32_t n_replicas;
    int32_t* active;
    int32_t* n_active;
    double thr, stop_frac, retire_frac;
    uint64_t step0;
    const unsigned long long* ctr;
    long long offset;
    int64_t* first_step;
    double* frac_out;
};

template <int S, int NC, int NT>
__device__ __forceinline__ void observe_replicas(const ObsParams& o) {
    namespace cg = cooperative_groups;
    using E = typename std::conditional<S == TIPT_F64, double, float>::type;
    using V = typename std::conditional<S == TIPT_F64, double2, float4>::type;
    constexpr int W = 16 / sizeof(E);
    __shared__ unsigned long long s_count;
    const cg::cluster_group cluster = cg::this_cluster();
    const unsigned part = NC > 1 ? cluster.block_rank() : 0;
    const auto meet = [&] {
        if constexpr (NC > 1) cluster.sync();
        else __syncthreads();
    };
    const uint64_t step = o.step0 + (o.ctr ? *o.ctr + (unsigned long long)o.offset : 0ull);
    const int64_t t0 = (int64_t)part * NT + threadIdx.x;
    constexpr int64_t kStride = (int64_t)NC * NT;
    for (int64_t r = blockIdx.x / NC; r < o.n_replicas; r += gridDim.x / NC) {
        if (threadIdx.x == 0) s_count = 0;
        meet();
        const tipt_replica rp = o.reps[r];
        const int64_t n = (int64_t)rp.n0 * rp.n1 * rp.n2;
        const E* hi = static_cast<const E*>(o.phi) + rp.offset;
        const E* lo = hi + o.n_total;  // float32 pairs
        const auto above = [&](E a, E b) {
            return (S == TIPT_F64 ? (double)a : (double)a + (double)b) > o.thr ? 1u : 0u;
        };
        unsigned long long cnt = 0;
        const bool vec = reinterpret_cast<uintptr_t>(hi) % 16 == 0 &&
                         (S == TIPT_F64 || reinterpret_cast<uintptr_t>(lo) % 16 == 0);
        const int64_t nv = vec ? n / W : 0;
        const V* vh = reinterpret_cast<const V*>(hi);
        const V* vl = reinterpret_cast<const V*>(lo);
        int64_t q = t0;
        if constexpr (S == TIPT_F64) {
            // eight loads in flight (unrolled by the compiler four times: 285 instead of 152 us
            // for three replicas of 200x203x199, 8.4 instead of 4.5 us for 64 of 128^2)
            for (; q + 7 * kStride < nv; q += 8 * kStride) {
                V x[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) x[u] = __ldg(vh + q + u * kStride);
#pragma unroll
                for (int u = 0; u < 8; ++u) cnt += above(x[u].x, 0.0) + above(x[u].y, 0.0);
            }
        }
#pragma unroll 4
        for (; q < nv; q += kStride) {
            const V x = __ldg(vh + q);
            if constexpr (S == TIPT_F64) {
                cnt += above(x.x, 0.0) + above(x.y, 0.0);
            } else {
                const V y = __ldg(vl + q);
                cnt += above(x.x, y.x) + above(x.y, y.y) + above(x.z, y.z) + above(x.w, y.w);
            }
        }
        for (q = nv * W + t0; q < n; q += kStride)
            cnt += above(__ldg(hi + q), S == TIPT_F64 ? E(0) : __ldg(lo + q));
#pragma unroll
        for (int m = 16; m > 0; m >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, m);
        if ((threadIdx.x & 31) == 0)
            atomicAdd(NC > 1 ? cluster.map_shared_rank(&s_count, 0) : &s_count, cnt);
        meet();
        if (part == 0 && threadIdx.x == 0) {
            const double frac = (double)s_count / (double)n;
            o.frac_out[r] = frac;
            if (o.active[r]) {
                if (frac > o.stop_frac && o.first_step[r] < 0) o.first_step[r] = (int64_t)step;
                if (frac > o.retire_frac) {
                    o.active[r] = 0;
                    atomicSub(o.n_active, 1);
                }
            }
        }
    }
}
template <int S>
__global__ void __launch_bounds__(256) ensemble_observe_kernel(ObsParams o) {
    observe_replicas<S, 1, 256>(o);
}
template <int S>
__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(512) ensemble_observe_cluster(ObsParams o) {
    observe_replicas<S, 8, 512>(o);
}

// Chunks are shared between blocks until an SM has sixteen blocks (four are resident, the others
// even out the end), but not into less than a pass of the 256 threads each (chunk_sites: a
// chunk's sites on average; two a thread in compensated FP32).  One block a chunk / this, in us:
// 64 replicas of 128^2 17 / 14, 300 of 101 x 97 75 / 54, 1000 163 / 151, 1024 of 128^2 155 / 159,
// one of 64^3 17 / 5.5; 200 of 8^3, cut into eleven 7.9, uncut 4.1.
static int stage_grid(EnsParams& e, int storage, int64_t chunk_sites) {
    const int most = num_sms() * 16;
    const int64_t passes = chunk_sites / (storage == TIPT_F32C ? 512 : 256);
    int64_t per = e.n_chunks < most ? (most + e.n_chunks - 1) / e.n_chunks : 1;
    if (per > 16) per = 16;
    if (per > passes) per = passes > 1 ? passes : 1;
    e.pieces = (int)per;
    const int64_t items = e.n_chunks * per;
    return items < most ? (int)items : most;
}

// Whether the marching stage is the faster one for n_rids replicas of a class: a launch takes
// 60 us however little it has to do, and rows that are not whole 128-byte lines are copied one
// by one (march / work-list kernel in us a step: 64 x 32^3 61 / 31; 4, 16, 64 x 64^3 72 / 18,
// 74 / 71, 145 / 250; 4, 16 x 96^3 61 / 54, 116 / 202; 64 x 48^3 420 / 109, 64 x 80^3 676 / 494).
static bool class_march_pays(int32_t n_rids, int32_t n0, int32_t n1, int32_t n2) {
    const int64_t n = (int64_t)n0 * n1 * n2;
    if (n * (n1 > n2 ? n1 : n2) >= (1ll << 32)) return true;  // 32-bit site decomposition
    return n2 % 32 == 0 && n_rids * n >= 4 << 20;
}

}  // namespace tipt

using namespace tipt;

extern "C" int tipt_ensemble_step(int storage, const void* phi, const void* pi, void* phi_out,
                                  void* pi_out, int64_t n_total, const tipt_replica* replicas,
                                  const tipt_chunk* chunks, int32_t n_chunks,
                                  const int32_t* active, const tipt_step_params* sp,
                                  const uint64_t* counter, int64_t offset, void* stream) {
    int rc;
    if (storage != TIPT_F64 && storage != TIPT_F32C)
        return fail(TIPT_ERR_STORAGE, "the ensemble takes F64 or F32C storage");
    if ((rc = check_state_sites(storage, phi, pi, phi_out, pi_out, n_total))) return rc;
    if (!replicas || !chunks || !active || !sp) return fail(TIPT_ERR_ARG, "NULL argument");
    if (n_chunks < 0) return fail(TIPT_ERR_ARG, "n_chunks < 0");
    if (n_chunks == 0) return TIPT_OK;
    EnsParams e;
    e.phi = phi;
    e.pi = pi;
    e.phi_out = phi_out;
    e.pi_out = pi_out;
    e.n_total = n_total;
    e.reps = replicas;
    e.chunks = chunks;
    e.n_chunks = n_chunks;
    e.active = active;
    e.h1 = 0.5 * sp->dt;
    e.h2 = sp->dt;
    e.inv_dx2 = 1.0 / (sp->dx * sp->dx);
    e.eta = sp->eta_eff;
    e.inv_mu2 = 1.0 / (sp->mu * sp->mu);
    e.inv_a2 = sp->inv_a2;
    e.step = sp->noise_step;
    e.ctr = reinterpret_cast<const unsigned long long*>(counter);
    e.offset = offset;
    e.rids = nullptr;
    e.n_rids = nullptr;
    const int grid = stage_grid(e, storage, n_total / n_chunks);
    cudaStream_t st = (cudaStream_t)stream;
    if (storage == TIPT_F64) ensemble_stage_kernel<TIPT_F64, false><<<grid, 256, 0, st>>>(e);
    else ensemble_stage_kernel<TIPT_F32C, false><<<grid, 256, 0, st>>>(e);
    cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? TIPT_OK : fail_cuda(err, "ensemble_stage launch");
}

extern "C" int tipt_ensemble_observe(int storage, const void* phi, int64_t n_total,
                                     const tipt_replica* replicas, int32_t n_replicas,
                                     int32_t* active, int32_t* n_active, double thr,
                                     double stop_frac, double retire_frac, uint64_t step,
                                     const uint64_t* counter,
                                     int64_t offset, int64_t* first_step, double* frac_out,
                                     void* stream) {
    if (storage != TIPT_F64 && storage != TIPT_F32C)
        return fail(TIPT_ERR_STORAGE, "the ensemble takes F64 or F32C storage");
    if (!phi || !replicas || !active || !n_active || !first_step || !frac_out)
        return fail(TIPT_ERR_ARG, "NULL argument");
    if (!(retire_frac >= stop_frac))
        return fail(TIPT_ERR_ARG, "retire_frac must be >= stop_frac");
    if (n_replicas <= 0) return TIPT_OK;
    cudaStream_t st = (cudaStream_t)stream;
    // A cluster costs 80 ns of a full chip however little it counts, a single block 3 to 6 ns:
    // single blocks for small replicas, and for middling ones (on average) where there are
    // enough of them to fill the SMs.  Single / cluster in us, compensated FP32: 1024 of 128^2
    // 28 / 80, 5000 of 16^2 14 / 275, 300 of 32^3 12 / 27, 400 of 40^3 37 / 58.
    const int64_t sites = n_total / n_replicas;
    const bool single = sites <= 16384 || (sites <= 65536 && n_replicas >= num_sms());
    const ObsParams o{phi, n_total, replicas, n_replicas, active, n_active, thr, stop_frac,
                      retire_frac, step, reinterpret_cast<const unsigned long long*>(counter), offset,
                      first_step, frac_out};
    const unsigned grid = (unsigned)(n_replicas < (1 << 24) ? n_replicas : 1 << 24);
    const bool f64 = storage == TIPT_F64;
    if (single) (f64 ? ensemble_observe_kernel<TIPT_F64> : ensemble_observe_kernel<TIPT_F32C>)<<<grid, 256, 0, st>>>(o);
    else (f64 ? ensemble_observe_cluster<TIPT_F64> : ensemble_observe_cluster<TIPT_F32C>)<<<grid * 8, 512, 0, st>>>(o);
    cudaError_t err = cudaGetLastError();
    return err == cudaSuccess ? TIPT_OK : fail_cuda(err, "ensemble_observe launch");
}

// The replicas of one 3-D shape class in compensated FP32, bitwise the step of
// tipt_ensemble_step for them, on the marching stage (shared-memory tiles, TMA/bulk-copy
// ring) where it pays, else on the work-list kernel over the class (kernel policy 2: always
// the marching stage).
extern "C" int tipt_ensemble_step_march(const void* phi, const void* pi, void* phi_out,
                                        void* pi_out, int64_t n_total,
                                        const tipt_replica* replicas, const int32_t* rids,
                                        int32_t n_rids, const int32_t* n_rids_dev, int32_t n0,
                                        int32_t n1, int32_t n2, const int32_t* active,
                                        const tipt_step_params* sp, const uint64_t* counter,
                                        int64_t offset, void* stream) {
    int rc;
    if ((rc = check_state_sites(TIPT_F32C, phi, pi, phi_out, pi_out, n_total))) return rc;
    if (!replicas || !rids || !active || !sp) return fail(TIPT_ERR_ARG, "NULL argument");
    if (n_rids < 0) return fail(TIPT_ERR_ARG, "n_rids < 0");
    if (n_rids == 0) return TIPT_OK;
    if (!ensemble_march_supported(n0, n1, n2))
        return fail(TIPT_ERR_UNSUPPORTED, "replica shape %d x %d x %d has no marching tiles", n0,
                    n1, n2);
    const uintptr_t a = reinterpret_cast<uintptr_t>(phi) | reinterpret_cast<uintptr_t>(pi) |
                        reinterpret_cast<uintptr_t>(phi_out) | reinterpret_cast<uintptr_t>(pi_out);
    if (a % 16 || (n_total * 4) % 16) return fail(TIPT_ERR_ALIGN, "packed buffers must be 16-byte aligned");
    if (kernel_policy() != 2 && !class_march_pays(n_rids, n0, n1, n2)) {
        const int64_t cpr = ((int64_t)n0 * n1 * n2 + kClassChunk - 1) / kClassChunk;
        if (cpr * n_rids <= 0x7FFFFFFF) {
            const auto magic = [](uint32_t d) {
                return d == 1 ? 0u : (uint32_t)(((1ull << 32) + d - 1) / d);
            };
            EnsParams e;
            memset(&e, 0, sizeof(e));
            e.phi = phi;
            e.pi = pi;
            e.phi_out = phi_out;
            e.pi_out = pi_out;
            e.n_total = n_total;
            e.reps = replicas;
            e.n_chunks = (int)(cpr * n_rids);
            e.rids = rids;
            e.n_rids = n_rids_dev;
            e.cpr = (int)cpr;
            e.m1 = magic((uint32_t)n1);
            e.m2 = magic((uint32_t)n2);
            e.active = active;
            e.h1 = 0.5 * sp->dt;
            e.h2 = sp->dt;
            e.inv_dx2 = 1.0 / (sp->dx * sp->dx);
            e.eta = sp->eta_eff;
            e.inv_mu2 = 1.0 / (sp->mu * sp->mu);
            e.inv_a2 = sp->inv_a2;
            e.step = sp->noise_step;
            e.ctr = reinterpret_cast<const unsigned long long*>(counter);
            e.offset = offset;
            cudaError_t err = device_status_word(&e.status);
            if (err != cudaSuccess) return fail_cuda(err, "device status word");
            const int grid = stage_grid(e, TIPT_F32C, (int64_t)n0 * n1 * n2 / cpr);
            ensemble_stage_kernel<TIPT_F32C, true><<<grid, 256, 0, (cudaStream_t)stream>>>(e);
            err = cudaGetLastError();
            return err == cudaSuccess ? TIPT_OK : fail_cuda(err, "ensemble class launch");
        }
    }
    RealStageParams p;
    memset(&p, 0, sizeof(p));
    p.phi = phi;
    p.pi = pi;
    p.phi_out = phi_out;
    p.pi_out = pi_out;
    p.n0 = n0;
    p.n1 = n1;
    p.n2 = n2;
    p.h1 = 0.5 * sp->dt;
    p.h2 = sp->dt;
    p.inv_dx2 = 1.0 / (sp->dx * sp->dx);
    p.eta = sp->eta_eff;
    p.inv_mu2 = 1.0 / (sp->mu * sp->mu);
    p.inv_a2 = sp->inv_a2;
    p.nfac = 1.0;
    p.step = sp->noise_step;
    return launch_ensemble_march(p, replicas, rids, n_rids, n_rids_dev, active, n_total,
                                 reinterpret_cast<const unsigned long long*>(counter),
                                 (long long)offset, (cudaStream_t)stream);
}

// 1 when replicas of shape n0 x n1 x n2 (n2 contiguous) can step on the marching
// stage (tipt_ensemble_step_march), 0 otherwise.
extern "C" int tipt_ensemble_march_supported(int32_t n0, int32_t n1, int32_t n2) {
    return ensemble_march_supported(n0, n1, n2) ? 1 : 0;
}

// Ordered compaction of a class's replica ids: rids_out[0..*n_out) = the ids
// rids[q] (in order) whose active flag is set.  One block.
__global__ void __launch_bounds__(1024) ensemble_compact_kernel(const int32_t* rids, int32_t n,
                                                                 const int32_t* active,
                                                                 int32_t* rids_out,
                                                                 int32_t* n_out) {
    __shared__ int32_t s_warp[32];
    __shared__ int32_t s_base;
    if (threadIdx.x == 0) s_base = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int b = 0; b < n; b += blockDim.x) {
        const int q = b + (int)threadIdx.x;
        const bool keep = q < n && active[rids[q]] != 0;
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) s_warp[wid] = __popc(m);
        __syncthreads();
        int before = s_base;
        for (int w = 0; w < wid; ++w) before += s_warp[w];
        if (keep) rids_out[before + __popc(m & ((1u << lane) - 1u))] = rids[q];
        __syncthreads();
        if (threadIdx.x == 0) {
            int tot = 0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += s_warp[w];
            s_base += tot;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *n_out = s_base;
}

// The active replicas of a class, compacted in order (for tipt_ensemble_step_march's
// device count): rids_out receives them, *n_out their number.
extern "C" int tipt_ensemble_compact(const int32_t* rids, int32_t n, const int32_t* active,
                                     int32_t* rids_out, int32_t* n_out, void* stream) {
    if (!rids || !active || !rids_out || !n_out) return fail(TIPT_ERR_ARG, "NULL argument");
    if (n < 0) return fail(TIPT_ERR_ARG, "n < 0");
    ensemble_compact_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(rids, n, active, rids_out,
                                                                  n_out);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TIPT_OK : fail_cuda(e, "ensemble_compact launch");
}
