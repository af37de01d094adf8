// 3D interpolation and gridding on a coil-interleaved grid (march.cu): plan
// structures and the calls of the pipelines.
//
// A batch of coils is cut into `n` chunks of `CS` coils (at most 32; the last
// chunk may hold fewer, its grid keeps the stride CS). The grid of a chunk is
// (frame, z, y, x, coil) in FFT order; rows are (sample in sorted order, coil)
// with the coil stride rounded up to even.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

struct dmr_plan;

namespace dmr {

struct ShortUnits;

struct MarchChunks {
    int64_t n;
    int CS;
};

// sorts the samples and builds the work lists (no-op, mp_W stays 0, where the
// kernels do not apply: not 3D, mixed widths or widths outside 2..6, or a grid
// huge for its samples). keys / keys_s / vals: total int32 each, vals = 0..total-1
// The lists' lengths are on their way to `totals` when it returns: march_lists
// takes them once the stream has been synchronised
struct MarchTotals {
    int n = 0;
    int32_t v[5] = {0};
};
int march_build(::dmr_plan *p, float *const rk[3], int32_t *keys, int32_t *keys_s, const int32_t *vals,
                MarchTotals &totals, cudaStream_t st);
void march_lists(::dmr_plan *p, const MarchTotals &totals);
int march_short_build(const ::dmr_plan *p, ShortUnits &out, cudaStream_t st);

// 2D: per-sample records in acquisition order, interpolation, and gridding by
// direct additions to the (zeroed) grid, for `nch` chunks of CS coils from coil
// b0 on, interleaved (direct2d.cu)
int d2_build(::dmr_plan *p, float *const rk[3], cudaStream_t st);
int d2_interp(const ::dmr_plan *p, const float2 *grid, float2 *ksp, int64_t b0, int64_t nch, int CS, int64_t batch,
              const float *weight, int wpb, cudaStream_t st);
int d2_grid(const ::dmr_plan *p, const void *ksp, int kreal, float2 *grid, int64_t b0, int64_t nch, int CS,
            int64_t batch, const float *weight, int wpb, cudaStream_t st);

// trajectory gradient from `nch` chunks of the interleaved forward grid, the
// first coil b0; calls with b0 > 0 add to the gradient of the coils before
int d2_grad(const ::dmr_plan *p, const float2 *grid, const float2 *v, int64_t b0, int64_t nch, int CS, int64_t batch,
            const float *weight, int wpb, float post, float *out, cudaStream_t st);

MarchChunks march_chunks(const ::dmr_plan *p, int64_t batch);
size_t march_rows_bytes(const ::dmr_plan *p, int CS);
size_t march_il_bytes(const ::dmr_plan *p, int CS);

// grid -> k-space, k-space -> grid for a batch. The grid is interleaved by
// chunks, or planar (coil, frame, z, y, x) with `il` the interleaved grid of one
// chunk; `rows`: the rows of one chunk. Deterministic gridding takes its
// scratch (every unit's plane of a chunk) from the library pool;
// DMR_ERR_UNSUPPORTED, before any launch, when that exceeds det_limit (> 0), the
// grid is too wide for its gather, or the pool has no memory.
int march_interp(const ::dmr_plan *p, const float2 *grid, bool planar, float2 *ksp, int64_t batch, const float *weight,
                 int wpb, float2 *rows, float2 *il, cudaStream_t st);
int march_grid(const ::dmr_plan *p, const void *ksp, int kreal, float2 *grid, bool planar, int64_t batch,
               const float *weight, int wpb, int det, int64_t det_limit, float2 *rows, float2 *il, cudaStream_t st);
// one chunk of a planar grid to interleaved
int march_interleave(const ::dmr_plan *p, const float2 *src, float2 *dst, int cact, int CS, cudaStream_t st);
// the same on planar grids with rows and il from the library pool
int march_interp_pool(const ::dmr_plan *p, const float2 *grid, float2 *ksp, int64_t batch, const float *weight,
                      int wpb, cudaStream_t st);
int march_grid_pool(const ::dmr_plan *p, const void *ksp, int kreal, float2 *grid, int64_t batch, const float *weight,
                    int wpb, int det, int64_t det_limit, cudaStream_t st);

}  // namespace dmr
