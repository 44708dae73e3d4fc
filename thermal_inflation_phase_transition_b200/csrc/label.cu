// Connected-component labelling of thresholded lattice fields: bubbles
// (|phi| > threshold) and string voxels (|winding| > 0.5), the GPU
// replacement of scipy.ndimage.label in the reference's post-processing
// (postprocess/revisualize_snapshots.py:171-214 _identify_bubbles, :360-392
// _identify_strings).
//
// Connectivity is the face-neighbour (6-connected) structure of
// scipy.ndimage.label's default; the lattice is open (non-periodic) like
// scipy's, or periodic on request.  Labels are numbered 1..n in raster order
// of each component's first voxel, which is scipy's numbering, so the label
// array is identical.
//
// Method (union-find with atomic-min hooking, Playne & Hawick, "A new
// algorithm for parallel connected-component labelling on GPUs", IEEE TPDS
// 2018): two masked neighbours unite by hooking the larger root under the
// smaller one with atomicMin, so a component's root ends as its smallest linear
// index.  Tiles of 2048 sites are labelled in shared memory first, where a run of
// masked sites along a row is one entry (its start, from the row's ballot) and
// two rows unite once per overlapping pair of runs; then the pairs across tile
// faces unite in global memory; roots are ranked in index order (per-chunk
// ranks, one scan) and every site gathers its root's rank.  Every chase loop is
// bounded; an exhausted bound sets the status word to TIPT_ERR_TIMEOUT.
//
// Bound: the latency of the chases and the passes over the labels (20 bytes a
// site, L2 resident up to about 2e7 sites).  250x243x237 float32, one label call:
// 819 us with a union per site and direction in global memory and seven passes,
// 218 us here (tiles 88, faces 53, ranks and scan 19, gather 38 of it).
#include "column_walk.cuh"
#include "tipt_device.cuh"
#include "tipt_internal.h"

namespace tipt {

constexpr int kChunk = 8192;        // sites per ranking chunk
constexpr int kChase = 1 << 24;     // bound on any find / unite loop

__device__ int g_label_status = 0;

template <int S>
__device__ __forceinline__ double field_abs(const void* f, int64_t s, int64_t N) {
    if constexpr (S == TIPT_F64) return fabs(__ldg(static_cast<const double*>(f) + s));
    else if constexpr (S == TIPT_F32) return fabs((double)__ldg(static_cast<const float*>(f) + s));
    else {
        const float* p = static_cast<const float*>(f);
        return fabs((double)__ldg(p + s) + (double)__ldg(p + N + s));
    }
}
template <int S>
__device__ __forceinline__ double field_val(const void* f, int64_t s, int64_t N) {
    if constexpr (S == TIPT_F64) return __ldg(static_cast<const double*>(f) + s);
    else if constexpr (S == TIPT_F32) return (double)__ldg(static_cast<const float*>(f) + s);
    else {
        const float* p = static_cast<const float*>(f);
        return (double)__ldg(p + s) + (double)__ldg(p + N + s);
    }
}

// |field| > thr.  float32: thrf is the largest float <= thr, which no float
// separates from thr, so the comparison needs no conversion.
template <int S>
__device__ __forceinline__ bool above(const void* f, int64_t s, int64_t N, double thr, float thrf) {
    if constexpr (S == TIPT_F32) return fabsf(__ldg(static_cast<const float*>(f) + s)) > thrf;
    else return field_abs<S>(f, s, N) > thr;
}

__device__ __forceinline__ int32_t find_root(const int32_t* L, int32_t x, bool& ok) {
    for (int it = 0; it < kChase; ++it) {
        const int32_t y = L[x];
        if (y == x) return x;
        x = y;
    }
    ok = false;
    return x;
}

// find_root that halves the path behind it (each site visited is linked to its
// grandparent).  Only non-roots are written, with an ancestor of theirs; a hook
// that such a store overwrites is not lost, because unite() goes on with the value
// that its atomicMin returned unless it hooked a root.
__device__ __forceinline__ int32_t find_halving(int32_t* L, int32_t x, bool& ok) {
    for (int it = 0; it < kChase; ++it) {
        const int32_t y = L[x];
        if (y == x) return x;
        const int32_t z = L[y];
        if (z == y) return y;
        L[x] = z;
        x = z;
    }
    ok = false;
    return x;
}

__device__ __forceinline__ void unite(int32_t* L, int32_t a, int32_t b, bool& ok) {
    for (int it = 0; it < kChase && ok; ++it) {
        a = find_halving(L, a, ok);
        b = find_halving(L, b, ok);
        if (a == b) return;
        if (a < b) {
            const int32_t old = atomicMin(&L[b], a);
            if (old == b) return;
            b = old;
        } else {
            const int32_t old = atomicMin(&L[a], b);
            if (old == a) return;
            a = old;
        }
    }
    ok = false;
}

// Masks of up to 32 sites: the first column of the run that holds column q, and
// the run that starts at column q.
__device__ __forceinline__ int run_start(uint32_t m, int q) {
    const uint32_t gap = ~m & ((1u << q) - 1u);
    return gap ? 32 - __clz((int)gap) : 0;
}
__device__ __forceinline__ uint32_t run_mask(uint32_t m, int q) {
    const uint32_t end = ~(m >> q);                 // bit 0 is clear
    const int len = end ? __ffs((int)end) - 1 : 32;
    return (len < 32 ? (1u << len) - 1u : 0xffffffffu) << q;
}

// Labels of one tile of TI x TJ lattice rows of KS x TK sites: L[s] = linear index of
// the smallest site of s's component within the tile (-1 where not masked).  A lattice
// row is KS consecutive rows of TK sites here, joined where one ends and the next
// begins.  Warps read rows (8 passes of 32 / TK rows) into masks; then one thread per
// row walks its runs, so that a warp works on 32 rows at once (a lane per site spent 2.5
// times the instructions: most lanes idle in every union); then warps write rows.
template <int S, int TI, int TJ, int KS, int TK>
__global__ void __launch_bounds__(256) label_tile_kernel(const void* f, double thr, float thrf,
                                                         int32_t* L, int n0, int n1, int n2) {
    constexpr int RPW = 32 / TK;  // rows per warp and pass
    constexpr int RS = TK + 1;    // entries per row, odd: rows in different banks
    constexpr int ROWS = TI * TJ * KS, RI = TJ * KS;  // rows of a tile, and of a plane of it
    static_assert(ROWS * TK == 2048 && 32 % TK == 0, "eight warps of eight passes");
    __shared__ int32_t s_l[ROWS * RS];  // union-find over the runs, at their first column
    __shared__ uint32_t s_m[ROWS];      // mask of each row
    const int ntk = (n2 + KS * TK - 1) / (KS * TK), ntj = (n1 + TJ - 1) / TJ;
    const int tk = blockIdx.x % ntk, tr = blockIdx.x / ntk;
    const int ti = tr / ntj, tj = tr - ti * ntj;
    const int lane = threadIdx.x & 31, sub = lane / TK, c = lane % TK;
    const int row0 = (threadIdx.x >> 5) * 8 * RPW + sub;
    const int64_t N = (int64_t)n0 * n1 * n2;
    // the lattice site of column q of a tile's row
    const auto place = [&](int row, int q, int& i, int& j, int& k) {
        i = ti * TI + row / RI;
        j = tj * TJ + row / KS % TJ;
        k = (tk * KS + row % KS) * TK + q;
    };
    bool on[8];
#pragma unroll
    for (int it = 0; it < 8; ++it) {
        int i, j, k;
        place(row0 + it * RPW, c, i, j, k);
        on[it] = i < n0 && j < n1 && k < n2 && above<S>(f, (i * n1 + j) * n2 + k, N, thr, thrf);
    }
#pragma unroll
    for (int it = 0; it < 8; ++it) {
        uint32_t m = __ballot_sync(0xffffffffu, on[it]) >> (sub * TK);
        if constexpr (TK < 32) m &= (1u << TK) - 1u;
        if (c == 0) s_m[row0 + it * RPW] = m;
    }
    __syncthreads();
    const int row = threadIdx.x;
    const bool walks = row < ROWS;
    const uint32_t m = walks ? s_m[row] : 0u;
    const uint32_t mj = walks && row % RI >= KS ? s_m[row - KS] : 0u;  // the row above (j - 1)
    const uint32_t mi = walks && row >= RI ? s_m[row - RI] : 0u;       // the row behind (i - 1)
    const uint32_t mk = KS > 1 && walks && row % KS > 0 ? s_m[row - 1] : 0u;  // the one before
    const bool joined = KS > 1 && (m & 1u) && mk >> (TK - 1) & 1u;
    bool ok = true;
    // a run starts under the first run of the row above that it touches, or else of
    // the row behind: no union needed for that one
    for (uint32_t rest = m; rest;) {
        const int q = __ffs((int)rest) - 1;
        const uint32_t run = run_mask(rest, q);
        rest &= ~run;
        int parent = row * RS + q;
        if (run & mj) parent = (row - KS) * RS + run_start(mj, __ffs((int)(run & mj)) - 1);
        else if (run & mi) parent = (row - RI) * RS + run_start(mi, __ffs((int)(run & mi)) - 1);
        else if (q == 0 && joined) parent = (row - 1) * RS + run_start(mk, TK - 1);
        s_l[row * RS + q] = parent;
    }
    __syncthreads();
    // the other overlaps unite; one with the row behind adds nothing where the rows
    // above both of them touch it in one column
    const uint32_t both = mj && mi ? m & mj & mi & s_m[row - RI - KS] : 0u;
    for (uint32_t rest = m; rest;) {
        const int q = __ffs((int)rest) - 1;
        const uint32_t run = run_mask(rest, q);
        rest &= ~run;
        uint32_t o = run & mj;
        if (o) o &= ~run_mask(o, __ffs((int)o) - 1);
        for (; o;) {
            const int x = __ffs((int)o) - 1;
            o &= ~run_mask(o, x);
            unite(s_l, row * RS + q, (row - KS) * RS + run_start(mj, x), ok);
        }
        o = run & mi;
        if (o && !(run & mj)) o &= ~run_mask(o, __ffs((int)o) - 1);
        for (; o;) {
            const int x = __ffs((int)o) - 1;
            const uint32_t ov = run_mask(o, x);
            o &= ~ov;
            if (!(ov & both)) unite(s_l, row * RS + q, (row - RI) * RS + run_start(mi, x), ok);
        }
        if (q == 0 && joined && run & (mj | mi))
            unite(s_l, row * RS, (row - 1) * RS + run_start(mk, TK - 1), ok);
    }
    __syncthreads();
    for (uint32_t rest = m; rest;) {
        const int q = __ffs((int)rest) - 1;
        rest &= ~run_mask(rest, q);
        s_l[row * RS + q] = find_root(s_l, row * RS + q, ok);
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < 8; ++it) {
        const int row = row0 + it * RPW;
        int i, j, k;
        place(row, c, i, j, k);
        if (i >= n0 || j >= n1 || k >= n2) continue;
        int32_t l = -1;
        if (on[it]) {
            const int r = s_l[row * RS + run_start(s_m[row], c)];
            int ri, rj, rk;
            place(r / RS, r % RS, ri, rj, rk);
            l = (ri * n1 + rj) * n2 + rk;
        }
        L[(i * n1 + j) * n2 + k] = l;
    }
    if (!ok) atomicExch(&g_label_status, (int)TIPT_ERR_TIMEOUT);
}

struct FaceDivs {
    FastDiv per[3], in[3];   // by a face's sites, by the inner extent, of each direction
};

// Unions across the tile faces normal to blockIdx.y (0: i, 1: j, 2: k) and, on a
// periodic lattice, across its boundary.  Consecutive threads take neighbouring
// pairs, and a pair beside another masked pair of the same two tiles adds nothing.  Divisions by
// launch constants: 57.9 -> 53.2 us at 250x243x237.
template <int TI, int TJ, int TK>
__global__ void __launch_bounds__(256) label_faces_kernel(int32_t* L, int n0, int n1, int n2,
                                                          FaceDivs divs, int periodic) {
    static_assert(!(TI & (TI - 1)) && !(TJ & (TJ - 1)) && !(TK & (TK - 1)), "powers of two");
    const int d = blockIdx.y;
    const int n[3] = {n0, n1, n2}, t[3] = {TI, TJ, TK};
    const FastDiv dper = d == 0 ? divs.per[0] : d == 1 ? divs.per[1] : divs.per[2];
    const FastDiv din = d == 0 ? divs.in[0] : d == 1 ? divs.in[1] : divs.in[2];
    const int st[3] = {n1 * n2, n2, 1};
    // direction d, the outer and the inner (consecutive threads) of the other two
    const int in = d == 2 ? 1 : 2, ou = d == 0 ? 1 : 0;
    const unsigned inner = (unsigned)(n1 * n2), nf = (unsigned)((n[d] - 1) / t[d]);
    const unsigned faces = nf + (periodic && n[d] > 1 ? 1u : 0u);
    const unsigned per = d == 0 ? inner : (unsigned)n[ou] * (unsigned)n[in];
    // at most n[d] faces of N / n[d] sites: total <= N < 2^31, FastDiv's range
    const unsigned total = faces * per;
    const int lane = threadIdx.x & 31;
    bool ok = true;
    for (unsigned q0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); q0 < total;
         q0 += gridDim.x * blockDim.x) {
        const unsigned q = q0 + lane;
        bool pair = false;
        int32_t s = 0, o = 0;
        int a = 0, b = 0;
        if (q < total) {
            const unsigned face = dper.div(q), rem = q - face * per;
            b = (int)din.div(rem);
            a = (int)(rem - (unsigned)b * (unsigned)n[in]);
            const int x = face < nf ? (int)(face + 1) * t[d] : 0;
            s = x * st[d] + b * st[ou] + a * st[in];
            o = x > 0 ? s - st[d] : s + (n[d] - 1) * st[d];
            pair = L[s] >= 0 && L[o] >= 0;
        }
        const bool before = __shfl_up_sync(0xffffffffu, pair, 1);
        // the pair before it, in either direction along the face, joins the same runs
        if (pair && !(before && lane > 0 && (a & (t[in] - 1)) != 0) &&
            !((b & (t[ou] - 1)) != 0 && L[s - st[ou]] >= 0 && L[o - st[ou]] >= 0))
            unite(L, s, o, ok);
    }
    if (!ok) atomicExch(&g_label_status, (int)TIPT_ERR_TIMEOUT);
}

// Ranks of the roots (masked sites that are their own label) within their chunk
// of kChunk sites, in index order: R[root] = rank, and the chunk's number of
// roots.  A warp takes kChunk / 8 consecutive sites, 32 at a time; its lanes keep
// their flags in the bits of a word.
__global__ void __launch_bounds__(256) label_rank_kernel(const int32_t* L, int64_t N, int32_t* R,
                                                         int32_t* chunk_roots) {
    static_assert(kChunk == 8 * 32 * 32, "a flag word per lane");
    __shared__ int32_t s_warp[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t b0 = (int64_t)blockIdx.x * kChunk + warp * (kChunk / 8) + lane;
    uint32_t flags = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        int32_t l[16];  // sixteen loads in flight
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const int64_t s = b0 + (h * 16 + q) * 32;
            l[q] = s < N ? __ldg(L + s) : -1;
        }
#pragma unroll
        for (int q = 0; q < 16; ++q)
            flags |= (l[q] == (int32_t)(b0 + (h * 16 + q) * 32) ? 1u : 0u) << (h * 16 + q);
    }
    const int32_t cnt = (int32_t)__reduce_add_sync(0xffffffffu, __popc(flags));
    if (lane == 0) s_warp[warp] = cnt;
    __syncthreads();
    int32_t base = 0, total = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        if (w < warp) base += s_warp[w];
        total += s_warp[w];
    }
    if (threadIdx.x == 0) chunk_roots[blockIdx.x] = total;
    // the passes with a root in them
    uint32_t any = __reduce_or_sync(0xffffffffu, flags);
    while (any) {
        const int it = __ffs(any) - 1;
        any &= any - 1;
        const unsigned m = __ballot_sync(0xffffffffu, flags >> it & 1u);
        if (flags >> it & 1u) R[b0 + it * 32] = base + __popc(m & ((1u << lane) - 1u));
        base += __popc(m);
    }
}

// exclusive scan of the chunk counts (one block) and the total
__global__ void __launch_bounds__(1024) label_scan_kernel(int32_t* chunk_roots, int n_chunks,
                                                          int32_t* n_labels) {
    __shared__ int32_t s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = (n_chunks + blockDim.x - 1) / blockDim.x;
    const int b = threadIdx.x * per;
    int32_t sum = 0;
    for (int q = b; q < b + per && q < n_chunks; ++q) sum += chunk_roots[q];
    const auto warp_scan = [&](int32_t v) {   // inclusive
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        return v;
    };
    const int32_t inc = warp_scan(sum);
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) s_warp[lane] = warp_scan(s_warp[lane]);
    __syncthreads();
    int32_t run = inc - sum + (warp ? s_warp[warp - 1] : 0);
    if (threadIdx.x == blockDim.x - 1) *n_labels = run + sum;
    for (int q = b; q < b + per && q < n_chunks; ++q) {
        const int32_t v = chunk_roots[q];
        chunk_roots[q] = run;
        run += v;
    }
}

// label (1-based) of every site: its root's rank in the chunk plus the chunk's base
__global__ void __launch_bounds__(256) label_gather_kernel(const int32_t* L, const int32_t* R,
                                                           const int32_t* chunk_base, int32_t* out,
                                                           int64_t N) {
    bool ok = true;
    // four sites a thread, so that four chases are in flight
    for (int64_t s = (int64_t)blockIdx.x * 1024 + threadIdx.x; s < N; s += (int64_t)gridDim.x * 1024) {
        int32_t l[4], r[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) l[q] = s + 256 * q < N ? __ldg(L + s + 256 * q) : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q) r[q] = l[q] >= 0 ? __ldg(L + l[q]) : -1;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (r[q] != l[q]) r[q] = find_root(L, r[q], ok);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            l[q] = r[q] >= 0 ? __ldg(chunk_base + r[q] / kChunk) + __ldg(R + r[q]) + 1 : 0;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (s + 256 * q < N) out[s + 256 * q] = l[q];
    }
    if (!ok) atomicExch(&g_label_status, (int)TIPT_ERR_TIMEOUT);
}

// per-label statistics (index 0 = background, left at zero)
struct LabelStats {
    int64_t* count;     // [n+1]
    int64_t* sum_xyz;   // [n+1][3]
    int64_t* sum_sq;    // [n+1]  sum of x^2 + y^2 + z^2
    double* sum_val;    // [n+1]
    double* max_abs;    // [n+1]
};

__global__ void stats_zero_kernel(LabelStats st, int64_t n1) {
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n1;
         q += (int64_t)gridDim.x * blockDim.x) {
        st.count[q] = 0;
        st.sum_xyz[3 * q] = st.sum_xyz[3 * q + 1] = st.sum_xyz[3 * q + 2] = 0;
        st.sum_sq[q] = 0;
        st.sum_val[q] = 0.0;
        st.max_abs[q] = 0.0;
    }
}

template <int S>
__global__ void stats_kernel(const void* f, const int32_t* lab, int n0, int n1, int n2,
                             int32_t n_labels, LabelStats st) {
    const int64_t n12 = (int64_t)n1 * n2, N = (int64_t)n0 * n12;
    for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < N;
         s += (int64_t)gridDim.x * blockDim.x) {
        const int32_t l = lab[s];
        if (l <= 0 || l > n_labels) continue;
        const int64_t k = s % n2, r = s / n2, j = r % n1, i = r / n1;
        const double v = f ? field_val<S>(f, s, N) : 0.0;
        atomicAdd(reinterpret_cast<unsigned long long*>(&st.count[l]), 1ull);
        atomicAdd(reinterpret_cast<unsigned long long*>(&st.sum_xyz[3 * l]), (unsigned long long)i);
        atomicAdd(reinterpret_cast<unsigned long long*>(&st.sum_xyz[3 * l + 1]), (unsigned long long)j);
        atomicAdd(reinterpret_cast<unsigned long long*>(&st.sum_xyz[3 * l + 2]), (unsigned long long)k);
        atomicAdd(reinterpret_cast<unsigned long long*>(&st.sum_sq[l]),
                  (unsigned long long)(i * i + j * j + k * k));
        atomicAdd(&st.sum_val[l], v);
        // |v| >= 0: the IEEE bit patterns of non-negative doubles order like the values
        atomicMax(reinterpret_cast<unsigned long long*>(&st.max_abs[l]),
                  (unsigned long long)__double_as_longlong(fabs(v)));
    }
}

static int grid_for(int64_t N) {
    int64_t b = (N + 255) / 256;
    const int64_t cap = (int64_t)num_sms() * 16;
    return (int)(b < cap ? (b < 1 ? 1 : b) : cap);
}

// Tile labels, then the unions across tile faces.
template <int S, int TI, int TJ, int KS, int TK>
static void launch_tiles_as(const void* field, double thr, int32_t* L, int n0, int n1, int n2,
                            bool periodic, cudaStream_t st) {
    float thrf = (float)thr;
    if ((double)thrf > thr) thrf = nextafterf(thrf, -INFINITY);
    constexpr int TR = KS * TK;  // sites of a tile along the rows
    const int64_t tiles = (int64_t)((n0 + TI - 1) / TI) * ((n1 + TJ - 1) / TJ) * ((n2 + TR - 1) / TR);
    label_tile_kernel<S, TI, TJ, KS, TK><<<(unsigned)tiles, 256, 0, st>>>(field, thr, thrf, L, n0, n1, n2);
    // the direction with the most face pairs sets the grid
    const int64_t N = (int64_t)n0 * n1 * n2;
    const int64_t pi = ((n0 - 1) / TI + 1) * (N / n0), pj = ((n1 - 1) / TJ + 1) * (N / n1),
                  pk = ((n2 - 1) / TR + 1) * (N / n2);
    const int64_t most = pi > pj ? (pi > pk ? pi : pk) : (pj > pk ? pj : pk);
    const FaceDivs divs = {{FastDiv((uint32_t)(N / n0)), FastDiv((uint32_t)(N / n1)),
                            FastDiv((uint32_t)(N / n2))},
                           {FastDiv((uint32_t)n2), FastDiv((uint32_t)n2), FastDiv((uint32_t)n1)}};
    label_faces_kernel<TI, TJ, TR><<<dim3((unsigned)grid_for(most), 3), 256, 0, st>>>(
        L, n0, n1, n2, divs, periodic ? 1 : 0);
}

// The tiles of a lattice: 8 x 8 rows of 32 sites, 8 x 32 rows of 8 for short rows (fewer
// than 20 sites would leave lanes of the 32-site rows idle), 64 rows of 32 of a single
// plane.  A lattice that is thin in two directions, of which these would cover more than
// four times its sites with more tiles than are resident at once, takes the shape with
// the fewest tiles and pairs across their faces, 360 pairs to a tile.  (A resident tile
// costs nothing while it is empty: 2 x 2 x 5000 39 us in 157 tiles, 62 in ten; one that waits
// costs 2.3 ns.)  Float32 at a low threshold / above the field: 1 x 1 x 16e6 2836 / 1184 -> 298 /
// 69 us, 8e6 x 1 x 2 5115 / 2820 -> 804 / 143, 2 x 2 x 4e6 1917 / 370 -> 555 / 82, 1e6 x 4 x 4 1084 /
// 399 -> 322 / 101.
template <int S>
static void launch_tiles(const void* field, double thr, int32_t* L, int n0, int n1, int n2,
                         bool periodic, cudaStream_t st) {
    using Launch = void (*)(const void*, double, int32_t*, int, int, int, bool, cudaStream_t);
    struct Shape {
        int ti, tj, tr;
        Launch launch;
    };
    static const Shape longs[] = {{8, 8, 32, launch_tiles_as<S, 8, 8, 1, 32>},
                                  {1, 64, 32, launch_tiles_as<S, 1, 64, 1, 32>},
                                  {1, 1, 2048, launch_tiles_as<S, 1, 1, 64, 32>},
                                  {1, 8, 256, launch_tiles_as<S, 1, 8, 8, 32>},
                                  {8, 1, 256, launch_tiles_as<S, 8, 1, 8, 32>},
                                  {2, 2, 512, launch_tiles_as<S, 2, 2, 16, 32>},
                                  {64, 1, 32, launch_tiles_as<S, 64, 1, 1, 32>}};
    static const Shape shorts[] = {{8, 32, 8, launch_tiles_as<S, 8, 32, 1, 8>},
                                   {1, 256, 8, launch_tiles_as<S, 1, 256, 1, 8>},
                                   {256, 1, 8, launch_tiles_as<S, 256, 1, 1, 8>},
                                   {64, 4, 8, launch_tiles_as<S, 64, 4, 1, 8>},
                                   {4, 64, 8, launch_tiles_as<S, 4, 64, 1, 8>}};
    const bool single = n0 == 1, brief = !single && n2 < 20;
    const auto tiles = [&](const Shape& t) {
        return (int64_t)((n0 - 1) / t.ti + 1) * ((n1 - 1) / t.tj + 1) * ((n2 - 1) / t.tr + 1);
    };
    const Shape* pick = brief ? &shorts[0] : &longs[single ? 1 : 0];
    if (tiles(*pick) * 512 > (int64_t)n0 * n1 * n2 && tiles(*pick) > 8 * (int64_t)num_sms()) {
        const auto cost = [&](const Shape& t) {
            const int64_t pairs = (n0 - 1) / t.ti * ((int64_t)n1 * n2) +
                                  (n1 - 1) / t.tj * ((int64_t)n0 * n2) + (n2 - 1) / t.tr * ((int64_t)n0 * n1);
            return 360 * tiles(t) + pairs;
        };
        const auto least = [&](const auto& shapes) {
            for (const Shape& t : shapes)
                if (cost(t) < cost(*pick)) pick = &t;
        };
        least(longs);
        least(shorts);
    }
    pick->launch(field, thr, L, n0, n1, n2, periodic, st);
}

int64_t label_workspace_bytes(int64_t N) {
    const int64_t chunks = (N + kChunk - 1) / kChunk;
    return 4 * (2 * N + chunks + 64);
}

// Read (and optionally clear) the labeller's status word.
int label_status(int* status, int clear) {
    cudaError_t e = cudaMemcpyFromSymbol(status, g_label_status, sizeof(int));
    if (e == cudaSuccess && clear) {
        const int zero = 0;
        e = cudaMemcpyToSymbol(g_label_status, &zero, sizeof(int));
    }
    return e == cudaSuccess ? TIPT_OK : fail_cuda(e, "label status");
}

}  // namespace tipt

using namespace tipt;

extern "C" int64_t tipt_label_workspace_size(int64_t nx, int64_t ny, int64_t nz) {
    if (nx < 1 || ny < 1 || nz < 1) return 0;
    return label_workspace_bytes(nx * ny * nz);
}

extern "C" int tipt_label_components(int storage, const void* field, double threshold,
                                     int64_t nx, int64_t ny, int64_t nz, int periodic,
                                     int32_t* labels, int32_t* n_labels, void* workspace,
                                     int64_t workspace_bytes, void* stream) {
    int rc;
    if ((rc = check_storage(storage)) || (rc = check_dims(nx, ny, nz))) return rc;
    const int64_t N = nx * ny * nz;
    if (N >= (1ll << 31)) return fail(TIPT_ERR_UNSUPPORTED, "labelling takes < 2^31 sites");
    if ((rc = check_ptr(field, elem_align(storage), "field")) ||
        (rc = check_ptr(labels, 4, "labels")) || (rc = check_ptr(n_labels, 4, "n_labels")) ||
        (rc = check_ptr(workspace, 4, "workspace")))
        return rc;
    if (workspace_bytes < label_workspace_bytes(N))
        return fail(TIPT_ERR_ARG, "workspace of %lld bytes is smaller than the %lld needed",
                    (long long)workspace_bytes, (long long)label_workspace_bytes(N));
    const int64_t chunks = (N + kChunk - 1) / kChunk;
    int32_t* L = static_cast<int32_t*>(workspace);
    int32_t* R = L + N;
    int32_t* cr = R + N;
    cudaStream_t st = (cudaStream_t)stream;
    // (nx, ny, 1) has the components, indices and neighbours of (1, nx, ny), and
    // (nx, 1, 1) those of (1, 1, nx)
    int n0 = (int)nx, n1 = (int)ny, n2 = (int)nz;
    if (n2 == 1) {
        n2 = n1 > 1 ? n1 : n0;
        n1 = n1 > 1 ? n0 : 1;
        n0 = 1;
    }
    switch (storage) {
        case TIPT_F64: launch_tiles<TIPT_F64>(field, threshold, L, n0, n1, n2, periodic != 0, st); break;
        case TIPT_F32: launch_tiles<TIPT_F32>(field, threshold, L, n0, n1, n2, periodic != 0, st); break;
        default: launch_tiles<TIPT_F32C>(field, threshold, L, n0, n1, n2, periodic != 0, st); break;
    }
    label_rank_kernel<<<(unsigned)chunks, 256, 0, st>>>(L, N, R, cr);
    label_scan_kernel<<<1, 1024, 0, st>>>(cr, (int)chunks, n_labels);
    label_gather_kernel<<<grid_for((N + 3) / 4), 256, 0, st>>>(L, R, cr, labels, N);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TIPT_OK : fail_cuda(e, "labelling launch");
}

extern "C" int tipt_label_stats(int storage, const void* field, const int32_t* labels, int64_t nx,
                                int64_t ny, int64_t nz, int32_t n_labels, int64_t* count,
                                int64_t* sum_xyz, int64_t* sum_sq, double* sum_val,
                                double* max_abs, void* stream) {
    int rc;
    if ((rc = check_storage(storage)) || (rc = check_dims(nx, ny, nz))) return rc;
    if (field && (rc = check_ptr(field, elem_align(storage), "field"))) return rc;
    if ((rc = check_ptr(labels, 4, "labels")) || (rc = check_ptr(count, 8, "count")) ||
        (rc = check_ptr(sum_xyz, 8, "sum_xyz")) || (rc = check_ptr(sum_sq, 8, "sum_sq")) ||
        (rc = check_ptr(sum_val, 8, "sum_val")) || (rc = check_ptr(max_abs, 8, "max_abs")))
        return rc;
    if (n_labels < 0) return fail(TIPT_ERR_ARG, "n_labels < 0");
    const int64_t N = nx * ny * nz;
    LabelStats s{count, sum_xyz, sum_sq, sum_val, max_abs};
    cudaStream_t st = (cudaStream_t)stream;
    stats_zero_kernel<<<grid_for(n_labels + 1), 256, 0, st>>>(s, (int64_t)n_labels + 1);
    const int g = grid_for(N);
    switch (storage) {
        case TIPT_F64: stats_kernel<TIPT_F64><<<g, 256, 0, st>>>(field, labels, (int)nx, (int)ny, (int)nz, n_labels, s); break;
        case TIPT_F32: stats_kernel<TIPT_F32><<<g, 256, 0, st>>>(field, labels, (int)nx, (int)ny, (int)nz, n_labels, s); break;
        default: stats_kernel<TIPT_F32C><<<g, 256, 0, st>>>(field, labels, (int)nx, (int)ny, (int)nz, n_labels, s); break;
    }
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TIPT_OK : fail_cuda(e, "label statistics launch");
}
