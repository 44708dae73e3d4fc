// FP64 Box-Muller transform of the counter-based hash (R:2515-2522), from the
// hash's 53-bit integers m1, m2 (u = m 2^-53):
//   z = sqrt(-2 ln u1) cos(a),  a = fl(2 pi u2) as the reference rounds it.
//
// What bounds it: instruction issue.  CUDA's log, sqrt and cos take any argument;
// the arguments here lie in (1e-12, 1), [2e-16, 56) and [0, 2 pi), so no range
// checks, no slow paths, and the angle's quadrant is in the bits of m2:
//  * -2 ln u1: table-driven (P. T. P. Tang, "Table-driven implementation of the
//    logarithm function in IEEE floating-point arithmetic", ACM TOMS 16, 1990).
//    u1 = 2^k w, w in [0.6875, 1.375) in 128 intervals with reciprocal centres c
//    (low words zero; c = 1 for [1 - 2^-8, 1), so u1 near 1 keeps its relative
//    accuracy), r = w c - 1, |r| < 2^-7:
//      -2 ln u1 = (k L_hi + T_hi) + (-2 r + (r^2 (1 - 2r/3 + ...) + (k L_lo + T_lo))),
//    L = -2 ln 2 and T = 2 ln c split at 2^-40, so k L_hi + T_hi is exact.
//  * cos a = +-sin y with y = a - pi/2 or a - 3 pi/2 (u2 below or above 1/2: bit 52
//    of m2), |y| <= pi/2; sin a = +-sin y with y = a - n pi, n = round(2 u2).  sin y =
//    y + y^3 P(y^2), P interpolating at the eight Chebyshev nodes (relative error
//    below 4e-17).
//  * sqrt: the hardware approximation of 1/sqrt, one first-order step to s, and the
//    residual v - s^2 as a second addend d, so sqrt(v) = s + d to 2^-60 and the
//    product s c + d c rounds once.
// Error against quad precision over 2e6 keys (uniform, and u1 -> 1): 0.53 ulp rms,
// 2.5 ulp at most, 7.9e-17 in the 2-norm relative to z; CUDA's log, sqrt and cos:
// 0.59, 2.8, 8.5e-17.  A 256^3 noise field takes 98 us with it, 142 us with CUDA's
// functions; the FP64 stage at 512^3 1.79 ms instead of 2.19 ms.
// oracle/gauss_tables.py computes the table and the coefficients from these definitions.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace tipt {

constexpr double kTwoPiLit = 6.283185307179586;  // literal of R:2520

// Per interval: T_hi, then the high words of T_lo (upper half) and c (lower half).
static __device__ const ulonglong2 kLogTab[128] = {
    {0x3fe7cc801fb46000, 0x3d52812e3ff734f1}, {0x3fe76fed9b946000, 0x3d5d45773ff71378},
    {0x3fe713e2fa46a000, 0x3d25b9b23ff6f260}, {0x3fe6b85ae0ffa000, 0x3d3d0d753ff6d1a6},
    {0x3fe65d556f4ce000, 0x3cbcd3f53ff6b149}, {0x3fe602cfe4f0a000, 0xbd5dd6be3ff69147},
    {0x3fe5a8ca41bee000, 0xbd2186673ff6719f}, {0x3fe54f447b7be000, 0xbd30fb553ff65250},
    {0x3fe4f638b9baa000, 0xbd5277bc3ff63357}, {0x3fe49da6c5bcc000, 0x3d25644d3ff614b3},
    {0x3fe445914853a000, 0xbd26bcac3ff5f664}, {0x3fe3edf513c16000, 0x3d4d31843ff5d868},
    {0x3fe396cedf9bc000, 0xbd28de4e3ff5babd}, {0x3fe3401e3eaec000, 0x3d5723863ff59d62},
    {0x3fe2e9e2b8e12000, 0x3d342f0c3ff58056}, {0x3fe2941bcb186000, 0x3d54539f3ff56398},
    {0x3fe23ec5e51ec000, 0xbd4790643ff54726}, {0x3fe1e9e06188a000, 0xbd5047e73ff52aff},
    {0x3fe1956d999bc000, 0x3d35aab73ff50f23}, {0x3fe14166c1368000, 0xbd568b0c3ff4f38f},
    {0x3fe0edd128b78000, 0xbd16f64b3ff4d844}, {0x3fe09aa5dce6c000, 0x3d49f1823ff4bd3f},
    {0x3fe047e70cde8000, 0x3d2b7be23ff4a280}, {0x3fdfeb215fea0000, 0x3d3c75d93ff48805},
    {0x3fdf4749cb4e0000, 0xbd4ef6ca3ff46dce}, {0x3fdea4455704c000, 0xbd558fb53ff453da},
    {0x3fde020b92234000, 0x3d5942b03ff43a27}, {0x3fdd60a08b904000, 0xbd47a8003ff420b5},
    {0x3fdcc001f5db4000, 0xbd3434ec3ff40783}, {0x3fdc2026ff180000, 0xbd422e273ff3ee8f},
    {0x3fdb8119f8b80000, 0x3d5c15cd3ff3d5da}, {0x3fdae2cb6b674000, 0xbd5523a53ff3bd61},
    {0x3fda453f12e6c000, 0xbd570bc43ff3a524}, {0x3fd9a878b1ebc000, 0xbd5714933ff38d23},
    {0x3fd90c6ee9fcc000, 0xbd323efb3ff3755c}, {0x3fd8711ebf510000, 0xbd5c83ca3ff35dce},
    {0x3fd7d69264af4000, 0x3d5629a53ff3467a}, {0x3fd73cb9834fc000, 0x3d51109b3ff32f5d},
    {0x3fd6a39786bbc000, 0x3d4c2fab3ff31877}, {0x3fd60b2fe0b08000, 0x3d5331d53ff301c8},
    {0x3fd5737f45018000, 0x3d3ac5103ff2eb4f}, {0x3fd4dc7b817bc000, 0x3d1c75b63ff2d50a},
    {0x3fd4462ea5c9c000, 0xbd55546c3ff2befa}, {0x3fd3b08e53580000, 0xbd55e0843ff2a91d},
    {0x3fd31b96d53a4000, 0x3d42d90f3ff29372}, {0x3fd287523411c000, 0xbd56b3993ff27dfa},
    {0x3fd1f3b5c1f24000, 0x3d51c2063ff268b3}, {0x3fd160c48e4b0000, 0x3d5bc4243ff2539d},
    {0x3fd0ce81adccc000, 0xbd36dd693ff23eb8}, {0x3fd03cdb16520000, 0xbd54db423ff22a01},
    {0x3fcf57c38d900000, 0xbd4315e43ff2157a}, {0x3fce3706ee308000, 0xbd5c025f3ff20120},
    {0x3fcd179428218000, 0x3d3b64673ff1ecf4}, {0x3fcbf962ae9f8000, 0x3d5cad533ff1d8f5},
    {0x3fcadc78265b0000, 0xbd4579d23ff1c523}, {0x3fc9c0bd4d4d0000, 0x3d44063f3ff1b17c},
    {0x3fc8a64602920000, 0xbd5275b03ff19e01}, {0x3fc78d093e3d8000, 0xbd4655b53ff18ab1},
    {0x3fc674ef19368000, 0xbd5347733ff1778a}, {0x3fc55e0b5d0e0000, 0xbd2d4dc73ff1648d},
    {0x3fc4486353dc0000, 0xbd57379c3ff151ba}, {0x3fc333dea0180000, 0x3d5492253ff13f0f},
    {0x3fc220823c780000, 0x3d5e7dc73ff12c8c}, {0x3fc10e4433cb0000, 0xbd48ef693ff11a30},
    {0x3fbffa70d1ac0000, 0xbd5f00dd3ff107fc}, {0x3fbdda8b7c680000, 0xbd31caac3ff0f5ee},
    {0x3fbbbce1dc690000, 0xbd42c0623ff0e406}, {0x3fb9a17d75740000, 0xbd4de42e3ff0d244},
    {0x3fb78867da350000, 0x3d50ca9f3ff0c0a8}, {0x3fb5714e9c040000, 0xbd57f9d73ff0af2f},
    {0x3fb35c96baa10000, 0x3d3386fb3ff09ddc}, {0x3fb149ed24000000, 0x3d514a3b3ff08cac},
    {0x3fae72b508140000, 0xbd3f3f913ff07b9f}, {0x3faa560d88c60000, 0xbd50a85c3ff06ab6},
    {0x3fa63d78d8680000, 0x3d58f12f3ff059ef}, {0x3fa22907dfea0000, 0x3d29d5c63ff0494a},
    {0x3f9c319744c80000, 0xbd4e1b543ff038c7}, {0x3f94192bb9680000, 0x3d295f473ff02865},
    {0x3f8811dc14580000, 0x3d00340d3ff01824}, {0x0000000000000000, 0x000000003ff00000},
    {0xbf7fefeaa2b00000, 0xbd31bc053fefe020}, {0xbf97dc319f800000, 0xbd52807e3fefa11d},
    {0xbfa3ce99a3460000, 0xbd56722e3fef6311}, {0xbfab9fc8e7b00000, 0x3d4935813fef25f6},
    {0xbfb1b0d909240000, 0x3d43381f3feee9c8}, {0xbfb58a63afc90000, 0x3d2656e73feeae80},
    {0xbfb95c7d1ec90000, 0x3d3344433fee741b}, {0xbfbd27739adb0000, 0xbd3b92523fee3a91},
    {0xbfc0759935990000, 0x3d4b0ed03fee01e0}, {0xbfc253f4ff0a0000, 0xbd44cb793fedca02},
    {0xbfc42eddeea68000, 0x3d5c2da23fed92f2}, {0xbfc6065451378000, 0x3d52e6973fed5cad},
    {0xbfc7da73457b0000, 0xbd47c7a43fed272d}, {0xbfc9ab4576200000, 0xbd5c60ae3fecf26e},
    {0xbfcb78c47bb10000, 0x3d3724f03fecbe6e}, {0xbfcd4317066c8000, 0xbd5c38ef3fec8b26},
    {0xbfcf0a2f18118000, 0x3d4bfa7f3fec5895}, {0xbfd0671616ca4000, 0xbd5a763a3fec26b5},
    {0xbfd1478534674000, 0xbd262b453febf584}, {0xbfd22670ed0a4000, 0xbd5e230d3febc4fd},
    {0xbfd303d7e0e48000, 0xbcfbcfa53feb951e}, {0xbfd3dfc22cecc000, 0xbd39b76a3feb65e3},
    {0xbfd4ba38539a4000, 0xbd57c95a3feb3748}, {0xbfd59339c5984000, 0x3d5ea09d3feb094b},
    {0xbfd66acfa272c000, 0x3d4a16423feadbe8}, {0xbfd740f9d9404000, 0x3d3e40993feaaf1d},
    {0xbfd815c229434000, 0xbd5a43173fea82e6}, {0xbfd8e92902888000, 0x3d52ba463fea5741},
    {0xbfd9bb33e27e0000, 0xbd093cb93fea2c2b}, {0xbfda8bed7c884000, 0x3d50a73d3fea01a0},
    {0xbfdb5b52128fc000, 0x3d444e033fe9d79f}, {0xbfdc2967e98c0000, 0xbd58ee333fe9ae25},
    {0xbfdcf6359209c000, 0xbd37b9643fe9852f}, {0xbfddc1bcdcac0000, 0x3d53748f3fe95cbb},
    {0xbfde8c04daaa8000, 0x3d5f37d73fe934c6}, {0xbfdf550ab24b8000, 0x3d329fa43fe90d4f},
    {0xbfe00e6d81ad6000, 0x3d59ae333fe8e652}, {0xbfe071b715cd6000, 0x3d3d00d83fe8bfcf},
    {0xbfe0d46b3d9ac000, 0x3d515f2f3fe899c1}, {0xbfe136865293a000, 0xbd5344be3fe87428},
    {0xbfe1980c8bd42000, 0xbd40f1bd3fe84f01}, {0xbfe1f8ffa248a000, 0xbd37956c3fe82a4a},
    {0xbfe2595ebcdf8000, 0x3d48fbc43fe80602}, {0xbfe2b93114b8a000, 0x3d2681a53fe7e225},
    {0xbfe31870a1544000, 0xbd40c5eb3fe7beb4}, {0xbfe3772786bfe000, 0x3d442bb73fe79baa},
    {0xbfe3d54fd5c20000, 0x3d51bcf23fe77908}, {0xbfe432ee8004e000, 0xbd51eafb3fe756cb},
};

// -2 ln(m1 2^-53), u1 clamped to 1e-12 (R:2336).
__device__ __forceinline__ double neg2_log_m(uint64_t m1) {
    const double um = fmax((double)m1, 9007.199254740992);   // 1e-12 2^53
    const uint32_t hi = (uint32_t)__double2hiint(um);
    // 53 is taken off the exponent together with the offset of [0.6875, 1.375)
    const int32_t t = (int32_t)(hi - (0x3fe60000u + (53u << 20)));
    const ulonglong2 e = __ldg(&kLogTab[(t >> 13) & 127]);
    const double w = __hiloint2double((int)(hi - (53u << 20) - ((uint32_t)t & 0xfff00000u)),
                                      __double2loint(um));
    const double k = (double)(t >> 20);
    const double c = __hiloint2double((int)(uint32_t)e.y, 0);
    const double tl = __hiloint2double((int)(uint32_t)(e.y >> 32), 0);
    const double r = __fma_rn(w, c, -1.0);
    const double head = __fma_rn(k, -0x1.62e42fefa4000p+0, __longlong_as_double((long long)e.x));
    const double tail = __fma_rn(k, 0x1.8432a1b0e2634p-42, tl);
    double p = __fma_rn(r, -2.0 / 7.0, 1.0 / 3.0);
    p = __fma_rn(r, p, -2.0 / 5.0);
    p = __fma_rn(r, p, 0.5);
    p = __fma_rn(r, p, -2.0 / 3.0);
    p = __fma_rn(r, p, 1.0);
    return __dadd_rn(head, __fma_rn(-2.0, r, __fma_rn(__dmul_rn(r, r), p, tail)));
}

// sqrt(v) = s + d for v in [2e-16, 56).
__device__ __forceinline__ void sqrt_parts(double v, double& s, double& d) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
    const double h = __dmul_rn(0.5, y);
    const double m = __dmul_rn(v, y);
    s = __fma_rn(__dmul_rn(v, h), __fma_rn(-m, y, 1.0), m);
    d = __dmul_rn(__fma_rn(-s, s, v), h);
}

// y = 1/sqrt(v) and, with SQ, s = sqrt(v), both to about half an ulp, for v in
// [1e-300, 1e300]: the hardware approximation and one step of third order
// (Householder), (1 - e)^(-1/2) = 1 + e (1/2 + 3 e / 8) with e = 1 - v y0^2 from the
// exact product v y0 = m + l.  Replaces a square root and the divisions by it: 7 to 9
// FP64 operations and no branch.
template <bool SQ>
__device__ __forceinline__ void rsqrt_sqrt(double v, double& y, double& s) {
    double y0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(v));
    const double m = __dmul_rn(v, y0);
    const double l = __fma_rn(v, y0, -m);
    const double e = __fma_rn(-l, y0, __fma_rn(-m, y0, 1.0));
    const double w = __dmul_rn(e, __fma_rn(0.375, e, 0.5));
    y = __fma_rn(y0, w, y0);
    if constexpr (SQ) s = __dadd_rn(m, __fma_rn(m, w, l));
}

// sin y, |y| <= pi/2
__device__ __forceinline__ double sin_half_pi(double y) {
    const double t = __dmul_rn(y, y);
    double p = 0x1.89a4866f527ebp-49;
    p = __fma_rn(t, p, -0x1.ae5138c1216b3p-41);
    p = __fma_rn(t, p, 0x1.6124015b5ee3ap-33);
    p = __fma_rn(t, p, -0x1.ae6455a1d7087p-26);
    p = __fma_rn(t, p, 0x1.71de3a5456716p-19);
    p = __fma_rn(t, p, -0x1.a01a01a018aadp-13);
    p = __fma_rn(t, p, 0x1.1111111111107p-7);
    p = __fma_rn(t, p, -0x1.5555555555555p-3);
    return __fma_rn(__dmul_rn(y, t), p, y);
}

// fl(2 pi u2): the scaling by 2^-53 is exact, so the product rounds as the reference's
__device__ __forceinline__ double angle_m(uint64_t m2) {
    return __dmul_rn((double)m2, kTwoPiLit * 0x1p-53);
}

__device__ __forceinline__ double cos_m(double a, uint64_t m2) {
    const bool up = (m2 >> 52) != 0;   // u2 >= 1/2: a - 3 pi/2, else pi/2 - a
    const double b = up ? a : -a;
    const double y = __dadd_rn(__dadd_rn(b, up ? -0x1.2d97c7f3321d2p+2 : 0x1.921fb54442d18p+0),
                               up ? -0x1.a79394c9e8a0ap-53 : 0x1.1a62633145c07p-54);
    return sin_half_pi(y);
}

__device__ __forceinline__ double sin_m(double a, uint64_t m2) {
    const int n = (int)((m2 + (1ull << 51)) >> 52);
    const double y = __fma_rn(-(double)n, 0x1.1a62633145c07p-53,
                              __fma_rn(-(double)n, 0x1.921fb54442d18p+1, a));
    const double s = sin_half_pi(y);
    return (n & 1) ? -s : s;
}

}  // namespace tipt
