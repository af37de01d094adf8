// Device-resident NUFFT plan: geometry, bin structure and the sorted samples.
#pragma once

#include <cufft.h>

#include <atomic>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

#include "common.cuh"

namespace dmr {

// Geometry passed by value to every kernel. Axis index 0 = x (fastest),
// 1 = y, 2 = z; unused axes have G = N = W = T = nb = 1.
struct Geom {
    int ndim;
    int G[3];       // oversampled grid extent
    int N[3];       // image extent
    int W[3];       // kernel width (1: Cartesian axis, nearest node by truncation)
    int half[3];    // G // 2 (fftshift offset)
    int T[3];       // bin / tile extent
    int nb[3];      // bins per axis
    float beta[3];  // Kaiser-Bessel beta
    double inv_hw[3];  // 1 / (W / 2)
    int nbins;      // bins per frame
    int nframes;
    int64_t gsize;  // grid points per (batch, frame)
    int64_t isize;  // image points per (batch, frame)
    int64_t total;  // samples over all frames
    // register-tile gridding, set for its launches (PlanBins): block regions per
    // axis, and per frame
    int nr[3];
    int nregions;
};

// One block-level unit of interpolation / atomic-gridding work: a chunk of
// the samples of one bin (bin id includes the frame: f * nbins + local).
struct WorkItem {
    int bin;
    int begin;
    int end;
};

// Samples of a tensor-core gridding work item, at most: the MMA's fp32 sums in
// tensor memory lose accuracy over longer chains, and longer items would
// unbalance the blocks.
constexpr int kTgSegment = 2048;

// One block of register-tile gridding: part `begin` of `end` equal fractions
// of every window bin of block region `region` (frame included). slot < 0:
// the block writes the grid; otherwise it writes partial sums to scratch slot
// `slot`. A reduction item (region, first slot, end slot) sums the slots of a
// split region in order.
struct RtItem {
    int region;
    int begin;
    int end;
    int slot;
};

struct FftPlan {
    cufftHandle handle = 0;
    size_t work_bytes = 0;
    std::mutex mu;
};

// Process-wide cache of cuFFT plans keyed by (device, rank, dims, batch).
std::shared_ptr<FftPlan> get_fft_plan(int ndim, const int *dims_zyx, int64_t batch, int *err);

// stream-ordered plan memory: n elements of T from the plans' pool on `dev`
int plan_alloc_bytes(int dev, void **p, size_t bytes, cudaStream_t st);

template <typename T>
int plan_alloc(int dev, T **p, size_t n, cudaStream_t st)
{
    return plan_alloc_bytes(dev, (void **)p, n * sizeof(T), st);
}

// temporaries of plan building, freed (stream-ordered) at the end of the scope
struct PlanTemp {
    int dev;
    cudaStream_t st;
    std::vector<void *> ptrs;
    PlanTemp(int d, cudaStream_t s) : dev(d), st(s) {}
    ~PlanTemp()
    {
        for (void *q : ptrs) cudaFreeAsync(q, st);
    }
    template <typename T>
    int alloc(T **p, size_t n)
    {
        const int rc = plan_alloc(dev, p, n, st);
        if (rc == DMR_OK) ptrs.push_back(*p);
        return rc;
    }
};

// The bin kernels' structures of a plan: built aside by plan_bins and then
// published whole (dmr_plan::bins), so that a call sees all of them or none and
// nothing a call reads without them ever changes.
struct PlanBins {
    float *scoord[3] = {nullptr, nullptr, nullptr};  // sorted rescaled coordinates
    int32_t *sidx = nullptr;            // sorted position -> global sample index
    int32_t *bin_start = nullptr;       // (nframes * nbins + 1)
    WorkItem *work = nullptr;           // interpolation / atomic gridding items
    int nwork = 0;
    int32_t *work_order = nullptr;      // item order in 4x4x4-bin tiles (L2 reuse of halos and spokes)
    int32_t *tiles = nullptr;           // owner-gridding tile order (heavy first)
    int ntiles = 0;
    // deterministic gridding: whole non-empty bins grouped by colour; bins of
    // one colour have disjoint tile + halo regions
    WorkItem *det_work = nullptr;
    std::vector<int> det_color_start;   // host, ncolors + 1
    // register-tile gridding (3D): block regions per axis (0: not planned) and
    // frame, block items, reduction items for regions split over several blocks,
    // and the number of partial-sum slots
    int nr[3] = {0, 0, 0};
    int nregions = 0;
    RtItem *rt_items = nullptr;
    int nrt = 0;
    RtItem *rt_reduce = nullptr;
    int nrt_reduce = 0;
    int rt_slots = 0;
    // (the owner has synchronised, as ~dmr_plan's)
    ~PlanBins()
    {
        for (void *q : {(void *)scoord[0], (void *)scoord[1], (void *)scoord[2], (void *)sidx, (void *)bin_start,
                        (void *)work, (void *)work_order, (void *)tiles, (void *)det_work, (void *)rt_items,
                        (void *)rt_reduce})
            if (q) cudaFreeAsync(q, cudaStreamPerThread);
    }
};
// builds them on first use (plan.cu)
int plan_bins(const ::dmr_plan *p, cudaStream_t st);

// The bins of 3D tensor-core gridding (dmr_tc_min_coils), built and published the
// same way: bins of its own (tile T, x y z) whose region (tile + W - 1 per axis)
// is at most 7 x 6 x 6 = 252 points, one N = 256 MMA; the samples of a bin in
// acquisition order (consecutive samples of a spoke, which share 32-byte sectors
// of k-space, are read together); work items of at most kTgSegment samples,
// visited in 4 x 4 x 4-bin tiles.
struct TgBins {
    int T[3] = {0, 0, 0};
    int nb[3] = {1, 1, 1};
    int nbins = 0;
    int32_t *sidx = nullptr;
    // per sample (gridding order): the Kaiser-Bessel weights of its W taps on
    // each axis, [sample][axis][wp] (wp = 4), and the offsets of its first taps
    // inside its bin, x | y << 8 | z << 16
    float *w = nullptr;
    int32_t *l = nullptr;
    int wp = 0;
    WorkItem *work = nullptr;
    int nwork = 0;
    int32_t *order = nullptr;
    ~TgBins()
    {
        for (void *q : {(void *)sidx, (void *)w, (void *)l, (void *)work, (void *)order})
            if (q) cudaFreeAsync(q, cudaStreamPerThread);
    }
};
// whether a plan can have them (3D, one width of 2..4 on all axes), and the same for them
bool tg_geometry_ok(const ::dmr_plan *p);
int plan_tg(const ::dmr_plan *p, cudaStream_t st);
// Short gridding units of single planes (march.cu), the same way
struct ShortUnits {
    void *units = nullptr;
    int n = 0;
    ~ShortUnits()
    {
        if (units) cudaFreeAsync(units, cudaStreamPerThread);
    }
};
int plan_short(const ::dmr_plan *p, cudaStream_t st);
// Register-tile gridding: whether the geometry admits it (3D, grid at least
// a block region plus the kernel support on every axis); plan the block items after the bin sort (host
// bin offsets h_start, nframes * nbins + 1 entries); scratch bytes a call of
// `batch` coils needs (0 when the kernel does not apply).
bool rt_geometry_ok(const Geom &g);
int rt_build(const ::dmr_plan *p, PlanBins &b, const std::vector<int32_t> &h_start, cudaStream_t st);
size_t rt_scratch_bytes(const ::dmr_plan *p, int64_t batch);
// scratch bytes a gridding call of `batch` coils may need (either kernel)
size_t grid_scratch_bytes(const ::dmr_plan *p, int64_t batch);
// the plans' pool (nullptr where none exists and `create` is false)
cudaMemPool_t plan_pool(int dev, bool create);
// library-owned stream-ordered pool for the scratch of calls without a workspace
cudaMemPool_t scratch_pool(int dev);
// fused, pruned FFT passes of the NUFFT pipelines (fftpass.cu): whether they
// apply to the plan (2D or 3D, every grid extent at least the image's and a
// length they have; DMR_CUFFT=1 turns them off), the forward
// (apodise + pad + FFT into the grid) and the adjoint (inverse FFT of the grid,
// which it overwrites, + crop + 1/G + apodisation into the image)
bool fft3_applies(const ::dmr_plan *p);
// nframes: grids per batch element (the plan's frames, or the coefficients of a
// subspace transform)
int fft3_forward(const ::dmr_plan *p, const void *image, int image_real, int64_t batch, int64_t nframes, float2 *grid,
                 cudaStream_t st);
int fft3_adjoint(const ::dmr_plan *p, float2 *grid, int64_t batch, int64_t nframes, float2 *image, cudaStream_t st);
// the same with the coil-interleaved grid of march.cuh: nchunks chunks of CS
// coils, (chunk, frame, z, y, x, coil)
int fft3_forward_il(const ::dmr_plan *p, const void *image, int image_real, int64_t batch, int64_t nframes,
                    int64_t nchunks, int CS, float2 *grid, cudaStream_t st);
int fft3_adjoint_il(const ::dmr_plan *p, float2 *grid, int64_t batch, int64_t nframes, int64_t nchunks, int CS,
                    float2 *image, cudaStream_t st);
// the same passes for the 3D Toeplitz self-adjoint: whether they apply
// (kernel extents at least the image's and with a compiled transform), and
// pad + FFT + kernel multiply + inverse FFT + crop (data: batch kernel grids)
bool toep3_applies(int ndim, const int32_t *kshape, const int32_t *ishape);
// bytes after the `data_bytes` of kernel grids in a Toeplitz workspace: cuFFT's
// work area, or, where the passes apply, room for the batch's images (a quarter
// of the grids holds them whenever the grids are twice the images on two axes)
size_t toep_extra_bytes(int ndim, const int32_t *kshape, size_t data_bytes, size_t work_bytes);
int fft3_toeplitz(int ndim, const int32_t *kshape_zyx, const int32_t *ishape_zyx, const float2 *kernel, int64_t nk,
                  const void *image, int image_real, float2 *out, int64_t batch, float2 *data, cudaStream_t st);
// tensor-core gridding of 3D plans (tcgrid.cu: dispatch and health state,
// tmgrid.cu: the kernel); DMR_ERR_UNSUPPORTED when the plan has no gridding bins
int grid_tc_dispatch(const ::dmr_plan *p, const void *ksp, int kreal, float2 *grid, int64_t batch,
                     const float *weight, int wpb, cudaStream_t st);
// smallest batch of atomic tensor-core gridding (dmr_tc_min_coils), DMR_NO_TC,
// and the deterministic scratch limit (dmr_det_scratch_limit)
int tc_min_coils();
bool tc_disabled();
int64_t det_scratch_limit();
// whether gridding of `batch` coils runs on the plane kernel (march.cuh)
bool grid_march_applies(const ::dmr_plan *p, int64_t batch, int det);
// atomic tensor-core gridding with the plan's gridding bins (tmgrid.cu);
// `timeouts` is the device address of the process-wide counter of blocks that
// stopped on a bounded wait
int grid_tm_dispatch(const ::dmr_plan *p, const void *ksp, int kreal, float2 *grid, int64_t batch,
                     const float *weight, int wpb, int *timeouts, int stall, cudaStream_t st);

}  // namespace dmr

struct dmr_plan {
    dmr::Geom g;
    int device;
    double scale;                       // kernel-sum normalisation
    std::vector<int64_t> frame_offsets;  // host CSR
    float os[3];
    // device buffers: apodisation tables and frame offsets, rescaled coordinates
    // in acquisition order
    char *tables = nullptr;
    float *rk[3] = {nullptr, nullptr, nullptr};
    // bin structures: null until plan_bins has published them
    mutable std::mutex bins_mu;
    mutable std::atomic<const dmr::PlanBins *> bins_ptr{nullptr};
    const dmr::PlanBins &bins() const { return *bins_ptr.load(std::memory_order_acquire); }
    mutable std::atomic<const dmr::TgBins *> tg_ptr{nullptr};
    mutable std::atomic<const dmr::ShortUnits *> short_ptr{nullptr};
    float *apod[3] = {nullptr, nullptr, nullptr};  // per-axis apodisation (image index)
    int64_t *foff_dev = nullptr;        // frame offsets on the device (nframes + 1)
    // march order (march.cu; mp_W == 0: not planned; 3D, and 2D plans dense enough
    // for tiles, which have gridding units only): tiles along x and y,
    // CSR offsets per cell, sorted position -> sample and back, per sorted
    // sample the tap weights and z cell, gridding units for 1, 2, 4 and 8
    // planes per warp (int4), the first unit of each (frame tile, plane), and
    // interpolation items (int4)
    int mp_W = 0;
    int mp_nt[2] = {0, 0};
    int32_t *mp_cstart = nullptr;
    int32_t *mp_sidx = nullptr;
    int32_t *mp_inv = nullptr;
    int32_t *mp_zc = nullptr;
    float *mp_rec = nullptr;
    void *mp_units[4] = {nullptr, nullptr, nullptr, nullptr};
    int mp_nunits[4] = {0, 0, 0, 0};
    int32_t *mp_ustart = nullptr;
    void *mp_items = nullptr;
    int mp_nitems = 0;
    // 2D, acquisition order (direct2d.cu; d2_W == 0: not planned): tap weights
    // and (first tap position, frame) per sample (int2)
    int d2_W = 0;
    float *d2_rec = nullptr;
    void *d2_base = nullptr;
    // whether forward transforms run on the interleaved grid
    bool il_forward() const { return (g.ndim == 3 && mp_W) || d2_W; }
    // device status word: blocks of this plan's calls whose bounded wait ran out
    // (dmr_plan_status; 0 while every result is valid)
    int32_t *status = nullptr;

    // (the owner has synchronised the device, or the stream that a plan was being
    // built on: nothing uses the buffers any more)
    ~dmr_plan()
    {
        auto drop = [](void *q) {
            if (q) cudaFreeAsync(q, cudaStreamPerThread);
        };
        drop(tables);
        delete bins_ptr.load();
        delete tg_ptr.load();
        delete short_ptr.load();
        for (int a = 0; a < 3; a++) drop(rk[a]);
        drop(status);
        drop(mp_cstart);
        drop(mp_sidx);
        drop(mp_inv);
        drop(mp_zc);
        drop(mp_rec);
        for (void *u : mp_units) drop(u);
        drop(mp_ustart);
        drop(mp_items);
        drop(d2_rec);
        drop(d2_base);
    }
};
