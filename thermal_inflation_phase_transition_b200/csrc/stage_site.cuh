// What a midpoint stage does at one site, for the real and the complex field in
// every storage: what it reads at a site (load), the values its stencil takes there
// (values) and the update from the seven stencil values of each.
//
// Stencil order of nb[v]: centre, ip, im, jp, jm, kp, km (R:1913-1920).
#pragma once

#include <type_traits>

#include "rk2_complex.cuh"

namespace tipt {

// Noise increments of a complex site (FP64): arrays times nfac, or ns_eff z.
template <typename NT>
__device__ __forceinline__ void complex_noise(const ComplexStageParams& p, uint64_t site,
                                              double& n1, double& n2) {
    if (p.noise1) {
        n1 = p.nfac * (double)static_cast<const NT*>(p.noise1)[site];
        n2 = p.nfac * (double)static_cast<const NT*>(p.noise2)[site];
    } else if (p.ns_eff != 0.0) {
        double z1, z2;
        gauss_pair(noise_key(site, p.step, p.mul, p.seed), z1, z2);
        n1 = p.ns_eff * z1;
        n2 = p.ns_eff * z2;
    } else {
        n1 = n2 = 0.0;
    }
}

// ------------------------------------------------------------ real field ---
// What a real stage is compiled for: a 1-D table or the polynomial, a 2-D table, thermal V'.
enum : int { kSrcRow = 0, kSrcRow2, kSrcThermal };

template <int S_, int SRC, bool RG_>
struct RealSite {
    static constexpr bool TH = SRC == kSrcThermal;
    using Params = RealStageParams;
    using E = typename std::conditional<S_ == TIPT_F64, double, float>::type;
    using TT = typename std::conditional<S_ == TIPT_F32C, float, double>::type;  // the row is read in
    static constexpr int S = S_;
    static constexpr bool RG = RG_;
    static constexpr int NR = S == TIPT_F32C ? 4 : 2;  // phi, pi; with F32C each hi, lo
    static constexpr int NV = S == TIPT_F32 ? 3 : NR;  // as read; float32: phi, phi~, pi

    static __device__ __forceinline__ void prepare(Params& p) {
        resolve_schedule(p);
        if constexpr (RG) reset_next_range(p);
    }
    using Row = RowReader<TT, SRC == kSrcRow2>;
    static __device__ __forceinline__ Row row(const Params& p) {
        return row_reader<TT, SRC == kSrcRow2>(p);
    }
    template <typename I>
    static __device__ __forceinline__ void load(const Params& p, I s, int64_t N, E raw[NR]) {
        const E* phi = static_cast<const E*>(p.phi);
        const E* pi = static_cast<const E*>(p.pi);
        if constexpr (S == TIPT_F32C) {
            raw[0] = __ldg(phi + s);
            raw[1] = __ldg(phi + N + s);
            raw[2] = __ldg(pi + s);
            raw[3] = __ldg(pi + N + s);
        } else {
            raw[0] = __ldg(phi + s);
            raw[1] = __ldg(pi + s);
        }
    }
    static __device__ __forceinline__ void values(const Params& p, const E raw[NR], E v[NV]) {
        if constexpr (S == TIPT_F32) {
            v[0] = raw[0];
            v[1] = TH ? midpoint_f32(p, raw[0], raw[1]) : midpoint_f32_bits(p, raw[0], raw[1]);
            v[2] = raw[1];
        } else {
#pragma unroll
            for (int q = 0; q < NV; ++q) v[q] = raw[q];
        }
    }
    static __device__ __forceinline__ void update(const Params& p, const F32CConst& kc,
                                                  const Row& tab, const E nb[NV][7],
                                                  int64_t s, int64_t N, RangeAcc& racc) {
        const uint64_t site = (uint64_t)(s + p.site_offset);
        E* po = static_cast<E*>(p.phi_out);
        E* vo = static_cast<E*>(p.pi_out);
        if constexpr (S == TIPT_F32C) {
            // planar {hi, lo}: hi plane at [0, N), lo plane at [N, 2N)
            F32CIn<float> x;
            stencil_sums_k(nb[0], nb[1], x.dh_phi, x.dl_phi);
            stencil_sums_k(nb[2], nb[3], x.dh_pi, x.dl_pi);
            x.phh = nb[0][0];
            x.phl = nb[1][0];
            x.pih = nb[2][0];
            x.pil = nb[3][0];
            float a, b, c, d;
            update_f32c<float, TH>(p, kc, tab, x,
                                   site_kick_f32c(p, kc, site), a, b, c, d);
            po[s] = a;
            po[N + s] = b;
            vo[s] = c;
            vo[N + s] = d;
            if constexpr (RG) racc.fold_ff(a, b);
        } else {
            E a, b;
            const double noise = site_noise<E>(p, site);
            if constexpr (S == TIPT_F64) {
                update_f64<TH>(p, tab, nb[0], nb[1], noise, a, b);
                if constexpr (RG) racc.fold_d(a);
            } else {
                update_f32_mid<TH>(p, tab, nb[0], nb[1], nb[2][0], noise, a, b);
                if constexpr (RG) racc.fold(a);
            }
            po[s] = a;
            vo[s] = b;
        }
    }
};

// --------------------------------------------------------- complex field ---
template <int S_, bool TH, bool RG_>
struct ComplexSite {
    using Params = ComplexStageParams;
    using E = typename std::conditional<S_ == TIPT_F64, double, float>::type;
    using TT = typename std::conditional<S_ == TIPT_F32C, float, double>::type;
    static constexpr int S = S_;
    static constexpr bool RG = RG_;
    static constexpr int NR = S == TIPT_F32C ? 8 : 4;  // phi1, phi2, pi1, pi2; F32C: hi, lo each
    static constexpr int NV = S == TIPT_F32 ? 6 : NR;  // as read; float32: phi, phi~, pi

    static __device__ __forceinline__ void prepare(Params& p) {
        if constexpr (RG) reset_range_words(p.range_next);
    }
    using Row = RowReader<TT, false>;
    static __device__ __forceinline__ Row row(const Params& p) { return Row{p.table}; }
    template <typename I>
    static __device__ __forceinline__ void load(const Params& p, I s, int64_t N, E raw[NR]) {
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            const E* src = static_cast<const E*>(p.f[f]);
            if constexpr (S == TIPT_F32C) {
                raw[2 * f] = __ldg(src + s);
                raw[2 * f + 1] = __ldg(src + N + s);
            } else {
                raw[f] = __ldg(src + s);
            }
        }
    }
    static __device__ __forceinline__ void values(const Params& p, const E raw[NR], E v[NV]) {
        if constexpr (S == TIPT_F32) {
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                v[a] = raw[a];
                v[2 + a] = TH ? midpoint_f32(p, raw[a], raw[2 + a])
                              : midpoint_f32_bits(p, raw[a], raw[2 + a]);
                v[4 + a] = raw[2 + a];
            }
        } else {
#pragma unroll
            for (int q = 0; q < NV; ++q) v[q] = raw[q];
        }
    }
    static __device__ __forceinline__ void update(const Params& p, const F32CConst&,
                                                  const Row& tab, const E nb[NV][7],
                                                  int64_t s, int64_t N, RangeAcc& racc) {
        if constexpr (S == TIPT_F32C) {
            // planar {hi, lo} fields; FP32 forces, float-float state updates
            CplxIn<float> in;
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                stencil_sums_k(nb[2 * f], nb[2 * f + 1], in.dh[f], in.dl[f]);
                in.ch[f] = nb[2 * f][0];
                in.cl[f] = nb[2 * f + 1][0];
            }
            const float h1 = (float)p.h1;
            // The Z_N force of the reference form (C:2152-2158) grows like 1/rho
            // near the origin and amplifies FP32 rounding, so with Z_N active (or a
            // table too large for shared memory) the force is evaluated in FP64 from
            // the full hi + lo values of the centre or the midpoint.
            const bool fp32_force = !(p.zn_active > 0.5 && p.zn_n > 0.5) &&
                                    (p.table_in_smem || p.vkind == TIPT_VP_POLY);
            auto force = [&](float q1, float q2, int which, float& d1, float& d2) {
                if (fp32_force) {
                    complex_force_v<float>(p, tab, (float)p.tmin, (float)p.dinv, q1, q2, d1, d2);
                } else {
                    double q1d = (double)nb[0][0] + (double)nb[1][0];
                    double q2d = (double)nb[2][0] + (double)nb[3][0];
                    if (which) {
                        q1d = (double)nb[0][0] + ((double)nb[1][0] + (double)h1 * ((double)nb[4][0] + (double)nb[5][0]));
                        q2d = (double)nb[2][0] + ((double)nb[3][0] + (double)h1 * ((double)nb[6][0] + (double)nb[7][0]));
                    }
                    double e1, e2;
                    complex_force<TH>(p, p.table, q1d, q2d, e1, e2);
                    d1 = (float)e1;
                    d2 = (float)e2;
                }
            };
            float kick[2] = {0.0f, 0.0f};
            if (p.noise1) {
                kick[0] = (float)(p.nfac * static_cast<const double*>(p.noise1)[s]);
                kick[1] = (float)(p.nfac * static_cast<const double*>(p.noise2)[s]);
            } else {
                complex_kick_f32c(p, (uint64_t)s, kick[0], kick[1]);
            }
            float oh[4], ol[4];
            complex_update_f32c<float>(p, in, kick, force, oh, ol);
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                float* po = static_cast<float*>(p.o[f]);
                po[s] = oh[f];
                po[N + s] = ol[f];
            }
            if constexpr (RG) fold_rho_ff(racc, oh[0], ol[0], oh[1], ol[1]);
        } else {
            // FP64 arithmetic after the neighbour sums.  The Laplacian of phi~ = phi + h1 pi
            // is lap + h1 lap(pi); float32 storage takes it from the float32 phi~ and rounds
            // the midpoint's pi, as the reference stores them (see update_f32_mid).
            const auto lap_of = [&](const E v[7], double c) {
                const E s6 = v[1] + v[2] + v[3] + v[4] + v[5] + v[6];
                return __dmul_rn(__fma_rn(-6.0, c, (double)s6), p.inv_dx2);
            };
            constexpr int PI = S == TIPT_F32 ? 4 : 2;   // pi1 among the values
            double c[4], lap[2], lapt[2], q[2];         // q: phi~ at the site
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                c[a] = (double)nb[a][0];
                c[2 + a] = (double)nb[PI + a][0];
                lap[a] = lap_of(nb[a], c[a]);
                if constexpr (S == TIPT_F32) {
                    q[a] = (double)nb[2 + a][0];
                    lapt[a] = lap_of(nb[2 + a], q[a]);
                } else {
                    q[a] = __fma_rn(p.h1, c[2 + a], c[a]);
                    lapt[a] = __fma_rn(p.h1, lap_of(nb[2 + a], c[2 + a]), lap[a]);
                }
            }
            double d[2], pt[2], n[2];
            complex_force<TH>(p, p.table, c[0], c[1], d[0], d[1]);
#pragma unroll
            for (int a = 0; a < 2; ++a)
                pt[a] = (double)(E)(c[2 + a] + p.h1 * (p.inv_a2 * lap[a] - p.eta * c[2 + a] -
                                                       d[a] * p.inv_mu2));
            complex_force<TH>(p, p.table, q[0], q[1], d[0], d[1]);
            complex_noise<E>(p, (uint64_t)s, n[0], n[1]);
            E o[2];
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                const double k2 = p.inv_a2 * lapt[a] - p.eta * pt[a] - d[a] * p.inv_mu2;
                o[a] = (E)(c[a] + p.h2 * pt[a]);
                static_cast<E*>(p.o[a])[s] = o[a];
                static_cast<E*>(p.o[2 + a])[s] = (E)(c[2 + a] + (p.h2 * k2 + n[a]));
            }
            if constexpr (RG) {
                if constexpr (S == TIPT_F64) fold_rho_f64(racc, o[0], o[1]);
                else racc.fold(rho_f32(o[0], o[1]));
            }
        }
    }
};

}  // namespace tipt
