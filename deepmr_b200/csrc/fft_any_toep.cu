// Toeplitz passes of run-time lengths (fftpass.cuh).
#include "fft_any.cuh"

namespace dmr {
namespace fftp {

template <int MX>
__global__ void __launch_bounds__(Gen<MX>::T, Gen<MX>::MINB) fft_toep_z_any_kernel(Fac f, int G0, int64_t gsize, ColArgs a,
                                                                     int64_t nk, const float2 *__restrict__ kern,
                                                                     float kscale, const float2 *__restrict__ tw,
                                                                     float2 *grid)
{
    extern __shared__ __align__(16) float2 fsm[];
    const int x = blockIdx.y * kFftLines + threadIdx.x % kFftLines;
    const int64_t bf = blockIdx.x, to = (int64_t)blockIdx.z * a.outer_stride + x;
    float2 *base = grid + bf * gsize + to;
    const float2 *kb = kern + (bf % nk) * gsize + to;
    with_radix<MX>(f.L1, [&](auto r) { cols_a<decltype(r)::value, false, false>(a, G0, x, fsm, f.L2, base, tw); });
    __syncthreads();
    with_radix<MX>(f.L2, [&](auto r) { toep_b<decltype(r)::value>(a, G0, x, fsm, f.L1, kb, kscale, tw); });
    __syncthreads();
    with_radix<MX>(f.L1, [&](auto r) { toep_c<decltype(r)::value>(a, G0, x, fsm, f.L2, base); });
}

int launch_toep_any(const Fac &f, const FftGeom &g, const ColArgs &a, int64_t nk, const float2 *kern, float kscale,
                    const float2 *tw, float2 *grid, cudaStream_t st)
{
    return by_size(f, [&](auto mx) {
        return launch_toep_k(fft_toep_z_any_kernel<decltype(mx)::value>, f.L, kFftLines * f.L2, g, a, nk, kern, kscale, tw,
                             grid, st, f);
    });
}

}  // namespace fftp
}  // namespace dmr
