// Cropping row passes of run-time lengths.
#include "fft_any_rows.cuh"

namespace dmr {
namespace fftp {

template int launch_rows_any<true, false>(Fac, const FftGeom &, const float2 *, const void *, int, float2 *, cudaStream_t);
template int launch_rows_any<true, true>(Fac, const FftGeom &, const float2 *, const void *, int, float2 *, cudaStream_t);

}  // namespace fftp
}  // namespace dmr
