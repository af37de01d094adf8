// Register transforms by run-time radix, for the passes of the lengths that have
// no kernel of their own.
#pragma once
#include "fftpass.cuh"

namespace dmr {
namespace fftp {

#define DMR_FFT_RADICES(X) \
    X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16) X(17) X(18) X(19) X(20) \
    X(21) X(22) X(23) X(24) X(25) X(26)
#define DMR_FFT_RADIX(R) \
    case R:              \
        if constexpr (R <= MX) fn(std::integral_constant<int, R>{}); \
        break;
template <int MX, class Fn>
__device__ __forceinline__ void with_radix(int r, Fn &&fn)
{
    switch (r) { DMR_FFT_RADICES(DMR_FFT_RADIX) }
}

// fn<MX> by the larger factor: small factors do not pay for the registers of large ones
template <class Fn>
int by_size(const Fac &f, Fn &&fn)
{
    const int m = std::max(f.L1, f.L2);
    if (m <= 13) return fn(std::integral_constant<int, 13>{});
    if (m <= 20) return fn(std::integral_constant<int, 20>{});
    return fn(std::integral_constant<int, kGenMax>{});
}

}  // namespace fftp
}  // namespace dmr
