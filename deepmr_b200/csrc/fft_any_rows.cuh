// Row passes of run-time lengths (fftpass.cuh), instantiated for padding and for
// cropping rows in files of their own.
#pragma once
#include "fft_any.cuh"

namespace dmr {
namespace fftp {

template <int MX, bool CROP, bool IL>
__global__ void __launch_bounds__(Gen<MX>::T, Gen<MX>::MINB) fft_rows_any_kernel(Fac f, RowArgs ra, const float2 *__restrict__ tw,
                                                                   const void *__restrict__ src, int src_real,
                                                                   float2 *__restrict__ dst)
{
    extern __shared__ __align__(16) float2 fsm[];
    with_radix<MX>(f.L1, [&](auto r) { rows_a<decltype(r)::value, CROP, IL>(ra, fsm, f.L, f.L2, tw, src, src_real); });
    __syncthreads();
    with_radix<MX>(f.L2, [&](auto r) { rows_b<decltype(r)::value, CROP, IL>(ra, fsm, f.L, f.L1, dst); });
}

template <bool CROP, bool IL>
int launch_rows_any(Fac f, const FftGeom &g, const float2 *tw, const void *src, int src_real, float2 *dst, cudaStream_t st)
{
    if (CROP) std::swap(f.L1, f.L2);
    return by_size(f, [&](auto mx) {
        return launch_rows_k<CROP, IL>(fft_rows_any_kernel<decltype(mx)::value, CROP, IL>, f.L1, f.L2, g, tw, src, src_real,
                                       dst, st, f);
    });
}

}  // namespace fftp
}  // namespace dmr
