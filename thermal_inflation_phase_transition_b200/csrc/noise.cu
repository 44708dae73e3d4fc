// Counter-based noise kernels: the hash pairs themselves (parity checks) and
// the noise-field fill that replaces the MT19937 generate_noise_field.
#include <type_traits>

#include "tipt_device.cuh"
#include "tipt_internal.h"

namespace tipt {

__global__ void hash_pairs_kernel(const uint64_t* __restrict__ keys, int64_t n, double* u1,
                                  double* u2, double* z) {
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n;
         q += (int64_t)gridDim.x * blockDim.x) {
        double a, b;
        hash_pair(keys[q], a, b);
        if (u1) u1[q] = a;
        if (u2) u2[q] = b;
        if (z) z[q] = gauss_cos(keys[q]);
    }
}

// Two sites a thread and pass: the transform's constants are loaded once for both
// (146 thread instructions a site instead of 166 with one site, 233 with CUDA's log,
// sqrt and cos).  256^3 float32: 142 us with those, 105 us with one site, 98 us here.
// PAIR off, for lattices that fit the resident threads: one site, a shorter chain (32^3 float32
// 2.1 -> 1.9 us, 48^3 2.4 -> 2.2 us, 64^3 3.1 -> 3.2 us).
template <typename OT, bool SIN, bool PAIR>
__global__ void __launch_bounds__(256) noise_fill_kernel(OT* __restrict__ out, int64_t N,
                                                         double scale, uint64_t step, uint64_t mul,
                                                         uint64_t seed) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t s0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if constexpr (!PAIR) {
        if (s0 >= N) return;
        const uint64_t key = noise_key((uint64_t)s0, step, mul, seed);
        out[s0] = (OT)__dmul_rn(scale, SIN ? gauss_sin(key) : gauss_cos(key));
        return;
    }
    for (int64_t s = s0; s < N; s += 2 * stride) {
        const uint64_t k0 = noise_key((uint64_t)s, step, mul, seed);
        const uint64_t k1 = noise_key((uint64_t)(s + stride), step, mul, seed);
        const double z0 = SIN ? gauss_sin(k0) : gauss_cos(k0);
        const double z1 = SIN ? gauss_sin(k1) : gauss_cos(k1);
        out[s] = (OT)__dmul_rn(scale, z0);
        if (s + stride < N) out[s + stride] = (OT)__dmul_rn(scale, z1);
    }
}

static unsigned grid_for(int64_t n, int threads) {
    int64_t b = (n + threads - 1) / threads;
    int64_t cap = (int64_t)num_sms() * 16;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (unsigned)b;
}

int launch_hash_pairs(const uint64_t* keys, int64_t n, double* u1, double* u2, double* z,
                      cudaStream_t st) {
    if (n == 0) return TIPT_OK;
    hash_pairs_kernel<<<grid_for(n, 256), 256, 0, st>>>(keys, n, u1, u2, z);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TIPT_OK : fail_cuda(e, "hash_pairs launch");
}

int launch_noise_fill(int storage, void* out, int64_t N, double scale, uint64_t step,
                      uint64_t mul, uint64_t seed, int component, cudaStream_t st) {
    if (N == 0) return TIPT_OK;
    const bool pair = N > 1024 * (int64_t)num_sms();
    const unsigned g = grid_for(pair ? (N + 1) / 2 : N, 256);
    const auto fill = [&](auto* o) {
        using OT = std::remove_pointer_t<decltype(o)>;
        auto kern = component ? (pair ? noise_fill_kernel<OT, true, true> : noise_fill_kernel<OT, true, false>)
                              : (pair ? noise_fill_kernel<OT, false, true> : noise_fill_kernel<OT, false, false>);
        kern<<<g, 256, 0, st>>>(o, N, scale, step, mul, seed);
    };
    if (storage == TIPT_F64) fill(static_cast<double*>(out));
    else fill(static_cast<float*>(out));
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TIPT_OK : fail_cuda(e, "noise_fill launch");
}

}  // namespace tipt
