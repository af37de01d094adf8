// Column passes of run-time lengths (fftpass.cuh).
#include "fft_any.cuh"

namespace dmr {
namespace fftp {

template <int MX, bool IN_ALL, bool OUT_ALL, bool INV>
__global__ void __launch_bounds__(Gen<MX>::T, Gen<MX>::MINB) fft_cols_any_kernel(Fac f, int G0, int64_t gsize, ColArgs a,
                                                                   const float2 *__restrict__ tw, float2 *grid)
{
    extern __shared__ __align__(16) float2 fsm[];
    const int x = blockIdx.x * kFftLines + threadIdx.x % kFftLines;
    float2 *base = grid + col_base(a, gsize);
    with_radix<MX>(f.L1, [&](auto r) { cols_a<decltype(r)::value, IN_ALL, INV>(a, G0, x, fsm, f.L2, base, tw); });
    __syncthreads();
    with_radix<MX>(f.L2, [&](auto r) { cols_b<decltype(r)::value, OUT_ALL, INV>(a, G0, x, fsm, f.L1, base); });
}

int launch_cols_any(const Fac &f, const FftGeom &g, const ColArgs &a, const float2 *tw, float2 *grid, cudaStream_t st)
{
    return by_size(f, [&](auto mx) {
        constexpr int MX = decltype(mx)::value;
        const int T = kFftLines * f.L2;
        return a.inv ? launch_cols_k(fft_cols_any_kernel<MX, true, false, true>, f.L, T, g, a, tw, grid, st, f)
                     : launch_cols_k(fft_cols_any_kernel<MX, false, true, false>, f.L, T, g, a, tw, grid, st, f);
    });
}

}  // namespace fftp
}  // namespace dmr
