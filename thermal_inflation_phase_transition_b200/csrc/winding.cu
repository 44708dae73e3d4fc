// Plaquette winding numbers: compute_winding_number (C:2683-2744,
// tools/winding.py:15-64) and the string count of C:4661.
//
// The reference sums atan2(sin d, cos d) over the four edges of each
// plaquette and divides by 2 pi.  atan2(sin d, cos d) equals d - 2 pi m with
// m = +1 for d > pi, -1 for d < -pi and 0 otherwise (d itself is a difference
// of two atan2 values in [-pi, pi], so |d| < 2 pi), and the four raw
// differences telescope to zero.  The plaquette winding is therefore the
// integer -(m1 + m2 + m3 + m4), computed here exactly from the four wrap
// decisions instead of from the rounded floating sum.
#include "tipt_device.cuh"
#include "tipt_internal.h"

namespace tipt {

constexpr double kPiD = 3.141592653589793;  // the double nearest pi (numpy's np.pi)

__device__ __forceinline__ int wrap_count(double d) { return d > kPiD ? 1 : (d < -kPiD ? -1 : 0); }

// Site value in FP64; F32C is planar (hi plane, then lo plane N sites later).
template <int S>
__device__ __forceinline__ double load_field(const void* p, int64_t s, int64_t N) {
    if constexpr (S == TIPT_F64) return __ldg(static_cast<const double*>(p) + s);
    else if constexpr (S == TIPT_F32) return (double)__ldg(static_cast<const float*>(p) + s);
    else {
        const float* f = static_cast<const float*>(p);
        return (double)__ldg(f + s) + (double)__ldg(f + N + s);
    }
}

struct WindParams {
    const void* phi1;
    const void* phi2;
    int n0, n1, n2;
    float* w_site;
    int8_t* w3;
    uint32_t* pierced;
    int64_t cap;
    unsigned long long* counts;  // [5]
};

// One site: the FP32 values of (phi1, phi2), and the bias-raised 1-norm
// |phi1| + |phi2| + 1e-18 of them.
struct WindV {
    float x, y, n;
};
__device__ __forceinline__ WindV wind_v(float x, float y) {
    return {x, y, fabsf(x) + fabsf(y) + 1e-18f};
}
template <int S>
__device__ __forceinline__ float load_f32(const void* p, int64_t base, unsigned o, int64_t N) {
    if constexpr (S == TIPT_F64) return (float)__ldg(static_cast<const double*>(p) + base + o);
    else if constexpr (S == TIPT_F32) return __ldg(static_cast<const float*>(p) + base + o);
    else {
        const float* f = static_cast<const float*>(p) + base;
        return __fadd_rn(__ldg(f + o), __ldg(f + N + o));
    }
}

// The wrap decision from the phases themselves: FP64 atan2 of the FP64 field
// values, as the reference computes it on FP64 casts (C:4627-4629).
template <int S>
__device__ __noinline__ int wrap_exact(const void* phi1, const void* phi2, int64_t sa, int64_t sb,
                                       int64_t N) {
    const double ta = atan2(load_field<S>(phi2, sa, N), load_field<S>(phi1, sa, N));
    const double tb = atan2(load_field<S>(phi2, sb, N), load_field<S>(phi1, sb, N));
    return wrap_count(tb - ta);
}

// Wrap of the edge a -> b without the phases.  theta(b) - theta(a) can pass
// +-pi only where the sign bits of phi2 differ (equal bits put both phases into
// [0, pi] or [-pi, 0]), and there it does so exactly when b lies on the far side
// of -a: cross = a.x b.y - a.y b.x has the sign of a.y.  The FP32 cross product
// is off by less than 3e-7 |a|_1 |b|_1 (input rounding included) and the rounded
// phases by less than 1e-14, so the sign decides wherever |cross| > 1e-6 |a|_1
// |b|_1; otherwise (a few edges in a million, and every NaN, infinity,
// underflow, overflow: the comparison then fails) the phases must (wrap_exact).
// Results in bit 31 (the other bits are not defined): wrap where there is one
// (+1 if the sign bit of a.y is set, else -1), `open` accumulates the edges that
// the phases must decide.
__device__ __forceinline__ uint32_t edge_wrap(const WindV& a, const WindV& b, uint32_t& open) {
    const float cr = __fmaf_rn(a.x, b.y, -__fmul_rn(a.y, b.x));
    const float d = __fmaf_rn(__fmul_rn(a.n, b.n), 1e-6f, -fabsf(cr));
    const uint32_t ya = __float_as_uint(a.y), differ = ya ^ __float_as_uint(b.y);
    open |= differ & ~__float_as_uint(d);
    return differ & ~(__float_as_uint(cr) ^ ya);
}

// Marching kernel (contiguous extent >= 24).  With e_i(s) = wrap(theta(s + i) -
// theta(s)), e_j, e_k alike, every plaquette is a signed sum of four edge counts:
// the reference's atan2(sin d, cos d) over an edge traversed backwards is the
// wrap of -d, and IEEE subtraction gives (a - b) = -(b - a) exactly, so
// wrap(-d) = -wrap(d):
//   XY(s) = -(e_i(s) + e_j(s + i) - e_i(s + j) - e_j(s)),  XZ, YZ alike.
// A warp takes 31 columns (lane 31 is the k + 1 halo) of kWR rows and walks np
// planes; a lane keeps its kWR + 1 rows of plane i, loads plane i + 2 while it
// works on plane i + 1, and takes the k + 1 values from the next lane.  The wrap
// bits of a lane's rows and the signs that go with them index a table of the four
// rows' counts, one per byte as the sum of count times 256^r: a plaquette then
// costs one add per term for four sites, a word of plaquettes is zero exactly
// when all four are, and with 8 added per byte every byte is non-negative, hence
// the plaquette plus 8.
//
// Bound: instruction issue (3.5 edges a site, 104 thread instructions), then HBM.
// 256^3 float32: 290 us with one FP64 atan2 per site of a shared-memory tile, 72 us
// here (2.8 TB/s of 12 bytes a site, 0.43 of the copy rate).
constexpr int kWR = 4;    // rows per lane
constexpr int kWP = 32;   // planes per block at most (counts are kept in bytes)

// LIST: the per-orientation windings and the pierced-plaquette list as well.
template <int S, bool LIST>
__global__ void __launch_bounds__(256, 2) winding_march_kernel(WindParams p, int nkt, int tasks, int np) {
    // counts of four rows from their wrap bits (low nibble) and sign bits (high nibble)
    __shared__ uint32_t s_cnt[256];
    {
        const uint32_t w = threadIdx.x & 15u, y = threadIdx.x >> 4;
        uint32_t e = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (w >> r & 1u) e += (y >> r & 1u) ? 1u << (8 * r) : 0u - (1u << (8 * r));
        s_cnt[threadIdx.x] = e;
    }
    __syncthreads();
    const int n0 = p.n0, n1 = p.n1, n2 = p.n2;
    const int64_t n12 = (int64_t)n1 * n2, N = (int64_t)n0 * n12;
    const int lane = threadIdx.x & 31;
    const int task = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (task >= tasks) return;  // whole warps
    const int jg = task / nkt, kt = task - jg * nkt;
    const int k = kt * 31 + lane, j0 = jg * kWR, i0 = blockIdx.y * np;
    const int ni = min(np, n0 - i0);
    unsigned ro[kWR + 1];      // offsets of the rows in a plane (periodic)
    uint32_t rows_live = 0;    // 0xff per row that this lane writes
#pragma unroll
    for (int r = 0; r <= kWR; ++r) {
        ro[r] = (unsigned)((j0 + r) % n1) * (unsigned)n2 + (unsigned)(k % n2);
        if (r < kWR && lane < 31 && k < n2 && j0 + r < n1) rows_live |= 0xffu << (8 * r);
    }
    float nx[kWR + 1], ny[kWR + 1];
    const auto load = [&](int64_t pl) {
#pragma unroll
        for (int r = 0; r <= kWR; ++r) {
            nx[r] = load_f32<S>(p.phi1, pl, ro[r], N);
            ny[r] = load_f32<S>(p.phi2, pl, ro[r], N);
        }
    };
    // offset of the lane's row r, dk columns to the right
    const auto row = [&](int r, int dk) { return (int64_t)((j0 + r) % n1) * n2 + (k + dk) % n2; };
    // (the slow path) wrap bits of rows 0 .. nr - 1 from the phases; edge r joins the
    // sites exact(r, a, b) sets
    const auto settle = [&](uint32_t& w, int nr, auto sites) {
        w = 0;
        for (int r = 0; r < nr; ++r) {
            int64_t a, b;
            sites(r, a, b);
            if (wrap_exact<S>(p.phi1, p.phi2, a, b, N)) w |= 1u << r;
        }
    };
    // sign bits of a plane's rows 0..3 and 1..4 as the table index's high nibble
    uint32_t y0, y1;
    const auto signs = [&](const WindV (&v)[kWR + 1]) {
        uint32_t y = 0;
#pragma unroll
        for (int r = kWR; r >= 0; --r) y = __funnelshift_l(__float_as_uint(v[r].y), y, 1);
        y0 = (y & 15u) << 4;
        y1 = (y << 3) & 0xf0u;
    };
    // e_j (rows 0..3) and e_k (rows 0..3 and 1..4) of the plane at pl (signs y0, y1)
    uint32_t ej, ek, ekj, ejk;
    const auto plane_edges = [&](const WindV (&v)[kWR + 1], int64_t pl) {
        uint32_t wj = 0, wk = 0, open = 0;
#pragma unroll
        for (int r = kWR; r >= 0; --r) {
            const WindV w = wind_v(__shfl_down_sync(0xffffffffu, v[r].x, 1),
                                   __shfl_down_sync(0xffffffffu, v[r].y, 1));
            wk = __funnelshift_l(edge_wrap(v[r], w, open), wk, 1);
            if (r < kWR) wj = __funnelshift_l(edge_wrap(v[r], v[r + 1], open), wj, 1);
        }
        if ((int32_t)open < 0) {
            settle(wj, kWR, [&](int r, int64_t& a, int64_t& b) {
                a = pl + row(r, 0);
                b = pl + row(r + 1, 0);
            });
            settle(wk, kWR + 1, [&](int r, int64_t& a, int64_t& b) {
                a = pl + row(r, 0);
                b = pl + row(r, 1);
            });
        }
        ej = s_cnt[wj | y0];
        ek = s_cnt[(wk & 15u) | y0];
        ekj = s_cnt[(wk >> 1) | y1];
        ejk = __shfl_down_sync(0xffffffffu, ej, 1);
    };

    int64_t pl = (int64_t)i0 * n12;            // plane i
    WindV c[kWR + 1];
    load(pl);
#pragma unroll
    for (int r = 0; r <= kWR; ++r) c[r] = wind_v(nx[r], ny[r]);
    int64_t pn = i0 + 1 < n0 ? pl + n12 : 0;   // plane i + 1
    load(pn);
    signs(c);
    plane_edges(c, pl);
    uint32_t a_xy = 0, a_xz = 0, a_yz = 0, a_str = 0;   // counts per byte (<= kWP)
    for (int q = 0; q < ni; ++q) {
        WindV d[kWR + 1];
#pragma unroll
        for (int r = 0; r <= kWR; ++r) d[r] = wind_v(nx[r], ny[r]);
        const int64_t pd = pn;
        if (q + 1 < ni) {
            pn = i0 + q + 2 < n0 ? pd + n12 : 0;
            load(pn);
        }
        uint32_t wi = 0, open = 0;
#pragma unroll
        for (int r = kWR; r >= 0; --r) wi = __funnelshift_l(edge_wrap(c[r], d[r], open), wi, 1);
        if ((int32_t)open < 0)
            settle(wi, kWR + 1, [&](int r, int64_t& a, int64_t& b) {
                a = pl + row(r, 0);
                b = pd + row(r, 0);
            });
        const uint32_t ei = s_cnt[(wi & 15u) | y0], eij = s_cnt[(wi >> 1) | y1];
        const uint32_t eik = __shfl_down_sync(0xffffffffu, ei, 1);
        uint32_t wxy = eij + ej - ei, wxz = eik + ek - ei;
        const uint32_t wyz = ejk + ek - ej - ekj;
        signs(d);
        plane_edges(d, pd);
        wxy -= ej;
        wxz -= ek;
        const uint32_t ws = wxy + wxz + wyz + 0x18181818u;   // 24 added per byte
        if (p.w_site) {
            float* const o = p.w_site + pl;
#pragma unroll
            for (int r = 0; r < kWR; ++r)      // 2^23 + byte as a float, exactly
                if (rows_live >> (8 * r) & 1u)
                    o[ro[r]] = __uint_as_float(__byte_perm(ws, 0x4B000000u, 0x7550 + r)) -
                               (0x1p23f + 24.0f);
        }
        // pierced plaquettes and string sites (|w| > 0.5), counted per byte over the
        // planes: a biased byte xor its bias is zero exactly where the winding is, and
        // is below 16 (plaquettes) or 64 (their sum)
        const uint32_t bxy = wxy + 0x08080808u, bxz = wxz + 0x08080808u, byz = wyz + 0x08080808u;
        const auto pierced = [&](uint32_t b) {
            return ((b ^ 0x08080808u) + 0x0f0f0f0fu) & 0x10101010u & rows_live;
        };
        const uint32_t z[3] = {pierced(bxy), pierced(bxz), pierced(byz)};
        a_xy += z[0] >> 4;
        a_xz += z[1] >> 4;
        a_yz += z[2] >> 4;
        a_str += (((ws ^ 0x18181818u) + 0x3f3f3f3fu) & 0x40404040u & rows_live) >> 6;
        if constexpr (LIST) {
            // warp-ballot compaction: one atomic per warp and plane, whose latency the walk
            // waits for (one per row and orientation / one: 4x32x156 FP64 35 / 12 us, 2x250000x32
            // float32 1644 / 566 us)
            uint32_t hits[3][kWR], found = 0;
#pragma unroll
            for (int o = 0; o < 3; ++o) {
                const uint32_t w = o == 0 ? bxy : (o == 1 ? bxz : byz);
#pragma unroll
                for (int r = 0; r < kWR; ++r) {
                    if (p.w3 && (rows_live >> (8 * r) & 1u))
                        p.w3[o * N + pl + ro[r]] = (int8_t)((int)(w >> (8 * r) & 0xffu) - 8);
                    hits[o][r] = __ballot_sync(0xffffffffu, z[o] >> (8 * r) & 16u);
                    found += __popc(hits[o][r]);
                }
            }
            if (p.pierced && found) {
                unsigned long long slot = 0;
                if (lane == 0) slot = atomicAdd(&p.counts[4], (unsigned long long)found);
                slot = __shfl_sync(0xffffffffu, slot, 0);
#pragma unroll
                for (int o = 0; o < 3; ++o)
#pragma unroll
                    for (int r = 0; r < kWR; ++r) {
                        const uint32_t m = hits[o][r];
                        const unsigned long long at = slot + __popc(m & ((1u << lane) - 1u));
                        if ((m >> lane & 1u) && (int64_t)at < p.cap)
                            p.pierced[at] = (uint32_t)((pl + ro[r]) * 3 + o);
                        slot += __popc(m);
                    }
            }
        }
        pl = pd;
#pragma unroll
        for (int r = 0; r <= kWR; ++r) c[r] = d[r];
    }
    const auto total = [](uint32_t a) {
        return __reduce_add_sync(0xffffffffu, (a & 0xffu) + (a >> 8 & 0xffu) + (a >> 16 & 0xffu) +
                                                  (a >> 24));
    };
    const unsigned c_xy = total(a_xy), c_xz = total(a_xz), c_yz = total(a_yz), c_str = total(a_str);
    if (lane == 0) {
        if (c_xy) atomicAdd(&p.counts[0], (unsigned long long)c_xy);
        if (c_xz) atomicAdd(&p.counts[1], (unsigned long long)c_xz);
        if (c_yz) atomicAdd(&p.counts[2], (unsigned long long)c_yz);
        if (c_str) atomicAdd(&p.counts[3], (unsigned long long)c_str);
    }
}

// Tiled kernel for short rows (a contiguous extent below 24 would leave most of
// a warp's columns idle).  A block takes a tile of TI x TJ x TK sites and its
// forward halo (one more plane, row and column, periodic): the field values of
// the region into shared memory, then the wrap count of each forward edge and
// the plaquettes as above.
template <int TK>
struct WindTile {
    static constexpr int TJ = TK == 8 ? 16 : 64;
    static constexpr int TI = TK == 8 ? 16 : 32;
    static constexpr int RI = TI + 1, RJ = TJ + 1, RK = TK + 1;
    static constexpr int REGION = RI * RJ * RK;
    static constexpr int INTERIOR = TI * TJ * TK;
};

template <int S, int TK>
__global__ void __launch_bounds__(256) winding_tiled_kernel(WindParams p) {
    using W = WindTile<TK>;
    __shared__ float2 s_v[W::REGION];
    __shared__ int8_t s_e[3][W::REGION];
    const int64_t n12 = (int64_t)p.n1 * p.n2;
    const int64_t N = (int64_t)p.n0 * n12;
    const int nti = (p.n0 + W::TI - 1) / W::TI, ntj = (p.n1 + W::TJ - 1) / W::TJ,
              ntk = (p.n2 + TK - 1) / TK;
    const int64_t tiles = (int64_t)nti * ntj * ntk;
    const unsigned lane = threadIdx.x & 31;
    unsigned long long c_xy = 0, c_xz = 0, c_yz = 0, c_str = 0;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int tk = (int)(tile % ntk);
        const int64_t tr = tile / ntk;
        const int tj = (int)(tr % ntj), ti = (int)(tr / ntj);
        const int i0 = ti * W::TI, j0 = tj * W::TJ, k0 = tk * TK;
        // site of the region's element q (coordinates taken modulo the lattice)
        const auto site = [&](int q) -> int64_t {
            const int c = q % W::RK, rr = q / W::RK;
            const int b = rr % W::RJ, a = rr / W::RJ;
            return (int64_t)((i0 + a) % p.n0) * n12 + (int64_t)((j0 + b) % p.n1) * p.n2 +
                   (k0 + c) % p.n2;
        };
        for (int q = threadIdx.x; q < W::REGION; q += blockDim.x) {
            const int64_t sq = site(q);
            s_v[q] = make_float2(load_f32<S>(p.phi1, sq, 0, N), load_f32<S>(p.phi2, sq, 0, N));
        }
        __syncthreads();
        // forward-edge wrap counts (the far faces are never read)
        for (int q = threadIdx.x; q < W::REGION; q += blockDim.x) {
            const int c = q % W::RK, rr = q / W::RK;
            const int b = rr % W::RJ, a = rr / W::RJ;
            const WindV v = wind_v(s_v[q].x, s_v[q].y);
            const auto count = [&](bool on, int qn) -> int8_t {
                if (!on) return 0;
                uint32_t open = 0;
                const uint32_t w = edge_wrap(v, wind_v(s_v[qn].x, s_v[qn].y), open);
                if ((int32_t)open < 0)
                    return (int8_t)wrap_exact<S>(p.phi1, p.phi2, site(q), site(qn), N);
                return (int32_t)w >= 0 ? 0 : (__float_as_int(v.y) < 0 ? 1 : -1);
            };
            s_e[0][q] = count(a < W::TI, q + W::RJ * W::RK);
            s_e[1][q] = count(b < W::TJ, q + W::RK);
            s_e[2][q] = count(c < TK, q + 1);
        }
        __syncthreads();
        // plaquettes: warp-uniform trip count (the ballots need full warps)
        for (int q0 = threadIdx.x & ~31; q0 < W::INTERIOR; q0 += blockDim.x) {
            const int q = q0 + (int)lane;
            const int c = q % TK, rr = q / TK;
            const int b = rr % W::TJ, a = rr / W::TJ;
            const int i = i0 + a, j = j0 + b, k = k0 + c;
            const bool live = i < p.n0 && j < p.n1 && k < p.n2;
            int wxy = 0, wxz = 0, wyz = 0;
            int64_t s = 0;
            if (live) {
                const int r0 = (a * W::RJ + b) * W::RK + c;
                const int ri = r0 + W::RJ * W::RK, rj = r0 + W::RK, rk = r0 + 1;
                wxy = -(s_e[0][r0] + s_e[1][ri] - s_e[0][rj] - s_e[1][r0]);
                wxz = -(s_e[0][r0] + s_e[2][ri] - s_e[0][rk] - s_e[2][r0]);
                wyz = -(s_e[1][r0] + s_e[2][rj] - s_e[1][rk] - s_e[2][r0]);
                s = (int64_t)i * n12 + (int64_t)j * p.n2 + k;
                const int w = wxy + wxz + wyz;
                if (p.w_site) p.w_site[s] = (float)w;
                if (p.w3) {
                    p.w3[s] = (int8_t)wxy;
                    p.w3[N + s] = (int8_t)wxz;
                    p.w3[2 * N + s] = (int8_t)wyz;
                }
                c_xy += wxy != 0;
                c_xz += wxz != 0;
                c_yz += wyz != 0;
                c_str += w != 0;  // |w| > 0.5 for integer w
            }
            if (p.pierced) {
                // warp-ballot compaction: one atomic per warp and orientation
                const int wo[3] = {wxy, wxz, wyz};
#pragma unroll
                for (int o = 0; o < 3; ++o) {
                    const unsigned m = __ballot_sync(0xffffffffu, live && wo[o] != 0);
                    if (m == 0) continue;
                    unsigned long long b0 = 0;
                    if (lane == 0) b0 = atomicAdd(&p.counts[4], (unsigned long long)__popc(m));
                    b0 = __shfl_sync(0xffffffffu, b0, 0);
                    if (live && wo[o] != 0) {
                        const unsigned long long slot = b0 + __popc(m & ((1u << lane) - 1u));
                        if ((int64_t)slot < p.cap) p.pierced[slot] = (uint32_t)(s * 3 + o);
                    }
                }
            }
        }
        __syncthreads();  // the region buffers are refilled by the next tile
    }
    // warp totals -> one atomic per warp and counter
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        c_xy += __shfl_down_sync(0xffffffffu, c_xy, off);
        c_xz += __shfl_down_sync(0xffffffffu, c_xz, off);
        c_yz += __shfl_down_sync(0xffffffffu, c_yz, off);
        c_str += __shfl_down_sync(0xffffffffu, c_str, off);
    }
    if (lane == 0) {
        if (c_xy) atomicAdd(&p.counts[0], c_xy);
        if (c_xz) atomicAdd(&p.counts[1], c_xz);
        if (c_yz) atomicAdd(&p.counts[2], c_yz);
        if (c_str) atomicAdd(&p.counts[3], c_str);
    }
}

template <int S>
static void launch_winding_march(const WindParams& p, dim3 nb, int nkt, int tasks, int np,
                                 cudaStream_t st) {
    if (p.w3 || p.pierced) winding_march_kernel<S, true><<<nb, 256, 0, st>>>(p, nkt, tasks, np);
    else winding_march_kernel<S, false><<<nb, 256, 0, st>>>(p, nkt, tasks, np);
}

// counts[4] collects the total number of pierced plaquettes found by the
// ballots; clamp it to the list capacity afterwards.
__global__ void winding_clamp_kernel(unsigned long long* counts, int64_t cap) {
    if (counts[4] > (unsigned long long)cap) counts[4] = (unsigned long long)cap;
}

}  // namespace tipt

using namespace tipt;

extern "C" int tipt_compute_winding_number(int storage, const void* phi1, const void* phi2,
                                           int64_t nx, int64_t ny, int64_t nz, float* w_site,
                                           int8_t* w3, uint32_t* pierced, int64_t pierced_cap,
                                           int64_t* counts, void* stream) {
    int rc;
    if ((rc = check_storage(storage)) || (rc = check_dims(nx, ny, nz))) return rc;
    const int eb = elem_align(storage);
    if ((rc = check_ptr(phi1, eb, "phi1")) || (rc = check_ptr(phi2, eb, "phi2")) ||
        (rc = check_ptr(counts, 8, "counts")))
        return rc;
    if (pierced && pierced_cap < 0) return fail(TIPT_ERR_ARG, "pierced_cap < 0");
    if (nx * ny * nz * 3 > 0xFFFFFFFFll && pierced)
        return fail(TIPT_ERR_UNSUPPORTED, "pierced list entries are 32-bit (N*3 < 2^32)");
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e = cudaMemsetAsync(counts, 0, 5 * sizeof(int64_t), st);
    if (e != cudaSuccess) return fail_cuda(e, "winding counts memset");
    WindParams p;
    p.phi1 = phi1;
    p.phi2 = phi2;
    p.n0 = (int)nx;
    p.n1 = (int)ny;
    p.n2 = (int)nz;
    p.w_site = w_site;
    p.w3 = w3;
    p.pierced = pierced;
    p.cap = pierced ? pierced_cap : 0;
    p.counts = reinterpret_cast<unsigned long long*>(counts);
    // rows of at least 24 sites march; shorter ones take 16 x 16 x 8 or 32 x 64 x 1 tiles
    const int tk = nz >= 6 ? 8 : 1;
    const int64_t cap_blocks = (int64_t)num_sms() * 8;
    auto grid = [&](int ti, int tj, int tkk) {
        const int64_t nb = ((nx + ti - 1) / ti) * ((ny + tj - 1) / tj) * ((nz + tkk - 1) / tkk);
        return (unsigned)(nb < cap_blocks ? nb : cap_blocks);
    };
    const int64_t nkt = (nz + 30) / 31, tasks = nkt * ((ny + kWR - 1) / kWR);
    // planes per warp: 32 (1/32 of the loads twice), fewer on lattices that would leave
    // the SMs' 16 resident warps empty: a warp's walk is a serial chain
    int np = kWP;
    while (np > 4 && tasks * ((nx + np - 1) / np) < 16 * (int64_t)num_sms()) np /= 2;
    const int64_t nic = (nx + np - 1) / np;
    // (offsets inside a plane and the grid are 32-bit in the marching kernel)
    if (nz >= 24 && ny * nz < 0x7FFFFFFF && nic <= 65535) {
        const dim3 nb((unsigned)((tasks + 7) / 8), (unsigned)nic);
        if (storage == TIPT_F64)
            launch_winding_march<TIPT_F64>(p, nb, (int)nkt, (int)tasks, np, st);
        else if (storage == TIPT_F32)
            launch_winding_march<TIPT_F32>(p, nb, (int)nkt, (int)tasks, np, st);
        else launch_winding_march<TIPT_F32C>(p, nb, (int)nkt, (int)tasks, np, st);
    } else if (tk == 8) {
        const unsigned nb = grid(WindTile<8>::TI, WindTile<8>::TJ, 8);
        if (storage == TIPT_F64) winding_tiled_kernel<TIPT_F64, 8><<<nb, 256, 0, st>>>(p);
        else if (storage == TIPT_F32) winding_tiled_kernel<TIPT_F32, 8><<<nb, 256, 0, st>>>(p);
        else winding_tiled_kernel<TIPT_F32C, 8><<<nb, 256, 0, st>>>(p);
    } else {
        const unsigned nb = grid(WindTile<1>::TI, WindTile<1>::TJ, 1);
        if (storage == TIPT_F64) winding_tiled_kernel<TIPT_F64, 1><<<nb, 256, 0, st>>>(p);
        else if (storage == TIPT_F32) winding_tiled_kernel<TIPT_F32, 1><<<nb, 256, 0, st>>>(p);
        else winding_tiled_kernel<TIPT_F32C, 1><<<nb, 256, 0, st>>>(p);
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail_cuda(e, "winding launch");
    if (pierced) {
        winding_clamp_kernel<<<1, 1, 0, st>>>(p.counts, p.cap);
        e = cudaGetLastError();
        if (e != cudaSuccess) return fail_cuda(e, "winding clamp launch");
    }
    return TIPT_OK;
}
