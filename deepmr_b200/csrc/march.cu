// 3D interpolation and gridding on a coil-interleaved grid.
//
// Reference: apply_interpolation / apply_gridding and their 3D kernels
// (src/deepmr/fft/_interp/interp.py:14-120, 189-227 and
//  src/deepmr/fft/_interp/grid.py:14-125, 253-284):
//   y[p]          = sum_taps w_z w_y w_x grid[taps]      (then / scale)
//   grid[taps(p)] += w_z w_y w_x y[p]                    (then / scale)
//
// Layouts. The grid of a chunk of CS coils is stored (frame, z, y, x, coil),
// FFT order on every axis: the coils of a grid point are contiguous, so a warp
// whose lanes are coils reads and updates whole 256-byte rows. Samples pass
// through a buffer of rows [sample in sorted order][coil] for the same reason;
// rows_in_kernel / rows_out_kernel transpose between it and the caller's
// (coil, sample) k-space, applying density weight and scale on the way.
//
// Order. Samples are sorted by (frame, tile of T x T cells in (x, y), cell of
// the tile, z cell), a cell being the grid cell of the first tap, with a CSR
// offset per cell: the samples that touch a grid plane z of a tile are, per
// cell column, one contiguous range (two when the range wraps around z = 0).
//
// Every tap weight comes from the plan (mp_rec: the x, y and z weights, padded
// to 16 bytes). The kernels read records with warp-wide broadcasts, which cost
// their bytes per lane in shared-memory bandwidth: storing weights twice, as
// operand pairs of the packed FP32 instructions, made both kernels slower (7.6
// vs 6.5 ms gridding, 9.5 vs 8.7 ms interpolation, 192^3 kooshball, 32 coils).
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <type_traits>

#include "kb.cuh"
#include "march.cuh"
#include "plan.cuh"

namespace dmr {

namespace {

// tile extent by kernel width: the tile plus its halo is at most 8 x 8 points,
// which a lane of the gridding kernel holds in registers
__host__ __device__ constexpr int march_tile(int W) { return W <= 4 ? 4 : 3; }
__host__ __device__ constexpr int march_rec(int W, int ndim = 3) { return (ndim * W + 3) / 4 * 4; }

// visits of a gridding unit / samples of an interpolation item, at most: heavier
// ones (the centre of k-space) are split so that no warp runs far behind. A
// unit's sums are a chain in float32 and the units of a plane are another (a
// quarter as long where a block's warps add theirs first), so that errors grow
// with a unit's length and with its inverse: 64 visits is where they are least
// (adjoint of 48^3, 12 coils, W 6, os 1.25, against 64 bits: 7.4e-6 of the result
// at 8 visits, 4.4 at 64, 3.7 with blocks adding first, 5.9 at 512; 64^3, 8 coils,
// W 4: 8.1e-7 at 64, 10.2 at 512), and several planes to a warp cost no more in
// short units (512 and 64: 772 and 790 us; 64^3, 8 coils: 265 and 240). With a
// plane per warp a unit's flush weighs more (192^3, 32 coils: 12.2 ms at 512, 13.7
// at 64), so these are long, and short where a call needs it: see short_planes. At
// width 6 all are short (144^3, 32 coils: 5.1 and 5.4 ms)
constexpr int kShortUnit = 64, kLongUnit = 512;
// unit lists of a plan: planes per warp
constexpr int kUnitLists = 4;
constexpr int kUnitPlanes[kUnitLists] = {1, 2, 4, 8};
constexpr int unit_visits(int ndim, int W, int list) { return ndim == 3 && W <= 5 && list == 0 ? kLongUnit : kShortUnit; }
constexpr int kItemSamples = 144;
constexpr int kItemZ = 8;  // z cells of an interpolation item
// rows of cell columns of an interpolation item (a tile has T / march_rows items per z block)
__host__ __device__ constexpr int march_rows(int W) { return W <= 4 ? 2 : 3; }

struct MarchGeom {
    int G[3], half[3];
    int T, nt0, nt1;  // tile extent, tiles along x and y
    int CS;           // coils of the chunk = coil stride of the grid
    int RS;           // coil stride of the rows (CS rounded up to even)
    bool join;        // gridding: a block's warps add their pieces of a plane first
    int64_t plane;    // G[0] * G[1]
    int64_t gsize;
};

__device__ __forceinline__ float2 dup(float v) { return make_float2(v, v); }

__device__ __forceinline__ void cp16(uint32_t dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void cp8(uint32_t dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void cp4(uint32_t dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---------------------------------------------------------------------------
// plan
// ---------------------------------------------------------------------------
// cell key of every sample: (frame, tile y, tile x, y in tile, x in tile, z)
__global__ void march_key_kernel(Geom g, int T, int nt0, int nt1, const int64_t *__restrict__ foff,
                                 const float *__restrict__ rk0, const float *__restrict__ rk1,
                                 const float *__restrict__ rk2, int32_t *__restrict__ keys,
                                 int32_t *__restrict__ counts)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < g.total;
         i += (int64_t)gridDim.x * blockDim.x) {
        int lo = 0, hi = g.nframes;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (foff[mid] <= i) lo = mid; else hi = mid;
        }
        const int x = pmod(first_tap_dev(rk0[i], g.W[0]), g.G[0]);
        const int y = pmod(first_tap_dev(rk1[i], g.W[1]), g.G[1]);
        const int z = g.ndim == 3 ? pmod(first_tap_dev(rk2[i], g.W[2]), g.G[2]) : 0;
        const int tx = x / T, ty = y / T;
        const int col = ((lo * nt1 + ty) * nt0 + tx) * (T * T) + (y - ty * T) * T + (x - tx * T);
        const int key = col * g.G[2] + z;
        keys[i] = key;
        atomicAdd(&counts[key], 1);
    }
}

// per sorted sample: tap weights, z cell, and the inverse permutation
__global__ void march_rec_kernel(Geom g, const int32_t *__restrict__ sidx, const float *__restrict__ rk0,
                                 const float *__restrict__ rk1, const float *__restrict__ rk2,
                                 float *__restrict__ rec, int32_t *__restrict__ zc, int32_t *__restrict__ inv)
{
    const int W = g.W[0], R = march_rec(W, g.ndim);
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < g.total;
         j += (int64_t)gridDim.x * blockDim.x) {
        const int32_t i = sidx[j];
        inv[i] = (int32_t)j;
        const float k[3] = {rk0[i], rk1[i], g.ndim == 3 ? rk2[i] : 0.0f};
        float *r = rec + j * R;
        for (int a = 0; a < g.ndim; a++) {
            const int x0 = first_tap_dev(k[a], W);
            for (int t = 0; t < W; t++) {
                const float w = tap_weight(x0, t, k[a], W, g.inv_hw[a], g.beta[a]);
                r[a * W + t] = w;
            }
            if (a == 2) zc[j] = pmod(x0, g.G[2]);
        }
    }
}

// z-cell ranges of the samples that touch planes [z0, z1] (z1 < G): the main
// one [a, b) and the one that wraps around the end of the axis [wa, G)
__device__ __forceinline__ void plane_cells(int z0, int z1, int W, int G, int &a, int &b, int &wa)
{
    a = max(0, z0 - (W - 1));
    b = z1 + 1;
    wa = z0 < W - 1 ? max(G + z0 - (W - 1), 0) : G;
}

// gridding units of np planes: number of pieces of each (frame tile, plane group)
__global__ void march_unit_count_kernel(const int32_t *__restrict__ cstart, int64_t nft, int TT, int G2, int W, int np,
                                        int nzu, int most, int32_t *__restrict__ counts)
{
    const int64_t n = nft * nzu;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= n; i += (int64_t)gridDim.x * blockDim.x) {
        if (i == n) {
            counts[n] = 0;
            continue;
        }
        const int64_t ft = i / nzu;
        const int zu = (int)(i - ft * nzu);
        const int z0 = zu * np, z1 = min(z0 + np, G2) - 1;
        int a, b, wa;
        plane_cells(z0, z1, W, G2, a, b, wa);
        int visits = 0;
        for (int c = 0; c < TT; c++) {
            const int32_t *cs = cstart + (ft * TT + c) * G2;
            visits += cs[b] - cs[a] + (cs[G2] - cs[wa]);
        }
        counts[i] = (visits + most - 1) / most;
    }
}

// (frame tile, plane group, first visit, end visit) of every unit
__global__ void march_unit_fill_kernel(const int32_t *__restrict__ start, int64_t nft, int nzu, int most,
                                       int4 *__restrict__ units)
{
    const int64_t n = nft * nzu;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int s = start[i], e = start[i + 1];
        const int ft = (int)(i / nzu), zu = (int)(i - (int64_t)ft * nzu);
        for (int u = s; u < e; u++)
            units[u] = make_int4(ft, zu, (u - s) * most, u + 1 == e ? 0x7fffffff : (u - s + 1) * most);
    }
}

// interpolation items (frame tile, z block, row part): pieces of at most kItemSamples samples
__global__ void march_item_count_kernel(const int32_t *__restrict__ cstart, int64_t nft, int TT, int cols, int G2, int nzb,
                                        int32_t *__restrict__ counts)
{
    const int nh = TT / cols;
    const int64_t n = nft * nzb * nh;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i <= n; i += (int64_t)gridDim.x * blockDim.x) {
        if (i == n) {
            counts[n] = 0;
            continue;
        }
        const int64_t ft = i / (nzb * nh);
        const int r = (int)(i - ft * (nzb * nh));
        const int z0 = r / nh * kItemZ, z1 = min(z0 + kItemZ, G2), h = r % nh;
        int cnt = 0;
        for (int c = h * cols; c < (h + 1) * cols; c++) {
            const int32_t *cs = cstart + (ft * TT + c) * G2;
            cnt += cs[z1] - cs[z0];
        }
        counts[i] = (cnt + kItemSamples - 1) / kItemSamples;
    }
}

// (frame tile, z block and row part, part, parts)
__global__ void march_item_fill_kernel(const int32_t *__restrict__ start, int64_t nft, int nzbh, int4 *__restrict__ items)
{
    const int64_t n = nft * nzbh;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int s = start[i], e = start[i + 1];
        const int ft = (int)(i / nzbh), zb = (int)(i - (int64_t)ft * nzbh);
        for (int u = s; u < e; u++) items[u] = make_int4(ft, zb, u - s, e - s);
    }
}

// ---------------------------------------------------------------------------
// rows <-> k-space
// ---------------------------------------------------------------------------
// samples (grid points) per block of the transposing kernels: 2048 values
__host__ __device__ constexpr int row_tile(int CC) { return 2048 / CC; }

// rows[inv[i]][c] = ksp[b0 + c][i] * weight * scale: reads run along the
// samples, writes are whole rows, CC lanes (a power of two >= RS) per row.
// DRAM-bound: 8 B in and out per value, 1.6 ms for 32 x 19.2 M samples (6.2 TB/s).
template <int CC>
__global__ void __launch_bounds__(256) rows_in_kernel(const void *__restrict__ ksp, int kreal, int64_t total, int64_t b0,
                                                      int cact, int RS, const float *__restrict__ weight, int wpb,
                                                      float scale, const int32_t *__restrict__ inv,
                                                      float2 *__restrict__ rows)
{
    constexpr int NT = row_tile(CC);
    __shared__ float2 s[NT][CC + 1];
    __shared__ int32_t sj[NT];
    const int64_t i0 = blockIdx.x * (int64_t)NT;
    const int n = (int)min((int64_t)NT, total - i0);
    for (int t = threadIdx.x; t < n; t += 256) sj[t] = inv[i0 + t];
    float2 v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int e = threadIdx.x + 256 * k, c = e / NT, t = e % NT;
        v[k] = make_float2(0.0f, 0.0f);
        if (c < cact && t < n) {
            const int64_t o = (b0 + c) * total + i0 + t;
            if (kreal) v[k].x = reinterpret_cast<const float *>(ksp)[o];
            else v[k] = reinterpret_cast<const float2 *>(ksp)[o];
        }
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int e = threadIdx.x + 256 * k, c = e / NT, t = e % NT;
        float w = 1.0f;
        if (weight && c < cact && t < n) w = weight[wpb ? (b0 + c) * total + i0 + t : i0 + t];
        s[t][c] = make_float2(v[k].x * w * scale, v[k].y * w * scale);
    }
    __syncthreads();
    const int c = threadIdx.x % CC;
    if (c < RS)
#pragma unroll 4
        for (int r = threadIdx.x / CC; r < n; r += 256 / CC) rows[(int64_t)sj[r] * RS + c] = s[r][c];
}

// ksp[b0 + c][i] = rows[inv[i]][c] * scale * weight
template <int CC>
__global__ void __launch_bounds__(256) rows_out_kernel(const float2 *__restrict__ rows, int64_t total, int64_t b0,
                                                       int cact, int RS, const float *__restrict__ weight, int wpb,
                                                       float scale, const int32_t *__restrict__ inv,
                                                       float2 *__restrict__ ksp)
{
    constexpr int NT = row_tile(CC);
    __shared__ float2 s[NT][CC + 1];
    const int64_t i0 = blockIdx.x * (int64_t)NT;
    const int n = (int)min((int64_t)NT, total - i0);
    const int c = threadIdx.x % CC;
    float2 v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int r = threadIdx.x / CC + k * (256 / CC);
        v[k] = make_float2(0.0f, 0.0f);
        if (r < n && c < RS) v[k] = __ldcs(rows + (int64_t)__ldg(inv + i0 + r) * RS + c);
    }
#pragma unroll
    for (int k = 0; k < 8; k++) s[threadIdx.x / CC + k * (256 / CC)][c] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int e = threadIdx.x + 256 * k, cc = e / NT, t = e % NT;
        if (cc >= cact || t >= n) continue;
        const int64_t o = (b0 + cc) * total + i0 + t;
        float w = scale;
        if (weight) w *= weight[wpb ? o : i0 + t];
        const float2 x = s[t][cc];
        ksp[o] = make_float2(x.x * w, x.y * w);
    }
}

// planar (coil, point) <-> interleaved (point, coil) grids of one chunk
template <int CC, bool PLANAR>
__global__ void __launch_bounds__(256) transpose_kernel(const float2 *__restrict__ src, float2 *__restrict__ dst,
                                                        int64_t npts, int cact, int CS)
{
    constexpr int NT = row_tile(CC);
    __shared__ float2 s[NT][CC + 1];
    const int64_t p0 = blockIdx.x * (int64_t)NT;
    const int n = (int)min((int64_t)NT, npts - p0);
    float2 v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int e = threadIdx.x + 256 * k;
        v[k] = make_float2(0.0f, 0.0f);
        if (PLANAR) {
            if (e < n * CS) v[k] = __ldcs(src + p0 * CS + e);
        } else {
            const int c = e / NT, t = e % NT;
            if (c < cact && t < n) v[k] = __ldcs(src + (int64_t)c * npts + p0 + t);
        }
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int e = threadIdx.x + 256 * k;
        if (PLANAR) {
            const int t = e / CS;
            if (t < NT) s[t][e - t * CS] = v[k];
        } else {
            s[e % NT][e / NT] = v[k];
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int e = threadIdx.x + 256 * k;
        if (PLANAR) {
            const int c = e / NT, t = e % NT;
            if (c < cact && t < n) dst[(int64_t)c * npts + p0 + t] = s[t][c];
        } else if (e < n * CS) {
            const int t = e / CS;
            dst[p0 * CS + e] = s[t][e - t * CS];
        }
    }
}

// ---------------------------------------------------------------------------
// Gridding. A warp owns one plane z of a tile's region (R x R points, R = T +
// W - 1) in registers, lane = coil (32 / NP coils, and NP consecutive planes
// side by side in the warp), and visits every sample that touches the plane:
// per column of cells (compile-time tap positions, one case of a switch) the
// samples of its W z-cells. The plane is then added to the grid once, 8 B per
// lane and point, coils contiguous (pieces of a heavy plane that a block's warps
// hold are added first). The only atomics are the R^2 additions per unit, 10.8 GB
// for the 192^3, 32-coil
// kooshball against 24.8 GB of per-bin regions. Rows and weight records of 16
// visits at a time come through a double-buffered shared-memory ring of the
// warp (cp.async).
// With `scratch` (deterministic mode) a unit stores its plane to its own slot
// instead, and grid_planes_gather_kernel adds the slots per grid point in a
// fixed order.
// ---------------------------------------------------------------------------
constexpr int kGridWarps = 4;
constexpr int kVisitBatch = 16;

template <int W, int NP, int ND>
struct PlaneShape {
    static constexpr int T = march_tile(W), R = T + W - 1, REC = march_rec(W, ND);
    static constexpr int CC = 32 / NP;     // coil lanes
    static constexpr int ROWB = CC * 8;    // bytes of a staged row
    static constexpr int RECS = kVisitBatch * ROWB, ZCS = RECS + kVisitBatch * REC * 4;
    static constexpr int BUF = ZCS + kVisitBatch * 4;  // one buffer of the ring: rows, records, z cells
    // shared memory of a pair of warps: their rings, then one of their planes
    static constexpr int PLANE = R * R * 32 * 8, PAIR = 4 * BUF > PLANE ? 4 * BUF : PLANE;
    static constexpr int SMEM = kGridWarps / 2 * PAIR;
};

template <int W, int NP, int ND>
__global__ void __launch_bounds__(32 * kGridWarps, W <= 4 ? 4 : 3)
    grid_planes_kernel(MarchGeom g, const int4 *__restrict__ units, int nunits, const int32_t *__restrict__ cstart,
                       const float *__restrict__ rec, const int32_t *__restrict__ zc, const float2 *__restrict__ rows,
                       float2 *__restrict__ grid, float2 *__restrict__ scratch)
{
    using S = PlaneShape<W, NP, ND>;
    constexpr int T = S::T, R = S::R, REC = S::REC, CC = S::CC, TT = T * T;
    extern __shared__ __align__(16) unsigned char msm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int u = blockIdx.x * kGridWarps + warp;
    if (u >= nunits) return;  // warp-uniform; barriers join warps of one tile and plane only
    const int ring = (warp >> 1) * S::PAIR + (warp & 1) * 2 * S::BUF;
    const int4 un = units[u];
    const int ft = un.x, z0 = un.y * NP, z1 = min(z0 + NP, g.G[2]) - 1;
    const int c = lane % CC, z = z0 + lane / CC;

    // ranges of the columns: lane = (wrapped, column)
    int beg = 0, cnt = 0;
    {
        const int col = lane & 15, wrapped = lane >> 4;
        if (col < TT) {
            int a, b, wa;
            plane_cells(z0, z1, ND == 3 ? W : 1, g.G[2], a, b, wa);
            const int32_t *cs = cstart + ((int64_t)ft * TT + col) * g.G[2];
            beg = cs[wrapped ? wa : a];
            cnt = cs[wrapped ? g.G[2] : b] - beg;
        }
    }
    auto scan = [&](int v) {
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, v, d);
            if (lane >= d) v += o;
        }
        return v;
    };
    {
        // the unit's part of the visits
        const int incl = scan(cnt), excl = incl - cnt;
        const int lo = max(excl, un.z), hi = min(incl, un.w);
        beg += max(lo - excl, 0);
        cnt = max(hi - lo, 0);
    }
    const int incl = scan(cnt);
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    const int first = beg - (incl - cnt);  // sample of visit v in this lane's range: first + v

    // visits [v0, v0 + kVisitBatch) into buffer b of the ring
    auto fetch = [&](int v0, int b) {
        const int v = min(v0 + (lane & (kVisitBatch - 1)), total - 1);
        int s = 0;  // range of visit v: the first lane whose inclusive count exceeds it
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            const int t = __shfl_sync(0xffffffffu, incl, s + d - 1);
            if (t <= v) s += d;
        }
        const int j = __shfl_sync(0xffffffffu, first, s) + v;
        const uint32_t dst = smem_addr(msm + ring + b * S::BUF);
        constexpr int LPR = CC / 2;  // lanes per row, 16 bytes each
#pragma unroll
        for (int k = 0; k < kVisitBatch * LPR / 32; k++) {
            const int r = k * (32 / LPR) + lane / LPR, piece = lane % LPR;
            const int jr = __shfl_sync(0xffffffffu, j, r);
            if (2 * piece < g.RS) cp16(dst + r * S::ROWB + piece * 16, rows + (int64_t)jr * g.RS + 2 * piece);
        }
#pragma unroll
        for (int k = 0; k < (kVisitBatch * REC / 4 + 31) / 32; k++) {
            const int p = k * 32 + lane, r = p / (REC / 4), piece = p - r * (REC / 4);
            const int jr = __shfl_sync(0xffffffffu, j, r & (kVisitBatch - 1));
            if (r < kVisitBatch) cp16(dst + S::RECS + p * 16, rec + (int64_t)jr * REC + 4 * piece);
        }
        if (ND == 3 && lane < kVisitBatch) cp4(dst + S::ZCS + lane * 4, zc + j);
    };

    float2 acc[R][R];
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
        for (int k = 0; k < R; k++) acc[i][k] = make_float2(0.0f, 0.0f);

    // one visit: sample i of the current buffer, column K of the tile
    auto visit = [&](auto kc, int buf, int i, int zoff) {
        constexpr int K = decltype(kc)::value, ky = K / T, kx = K % T;
        const float2 v = *reinterpret_cast<const float2 *>(msm + buf + i * S::ROWB + c * 8);
        const float *wp = reinterpret_cast<const float *>(msm + buf + S::RECS) + i * REC;
        float w[REC];
#pragma unroll
        for (int q = 0; q < (2 * W + 3) / 4; q++)
            *reinterpret_cast<float4 *>(w + 4 * q) = *reinterpret_cast<const float4 *>(wp + 4 * q);
        float2 t = v;
        if constexpr (ND == 3) {
            const int iz = zoff - *reinterpret_cast<const int *>(msm + buf + S::ZCS + i * 4);  // this lane's plane is tap iz
            t = make_float2(0.0f, 0.0f);
            // (a select, not a zero weight: values that are not finite stay in their W planes)
            if (NP == 1 || (unsigned)iz < (unsigned)W) t = __fmul2_rn(dup(wp[2 * W + iz]), v);
        }
#pragma unroll
        for (int jy = 0; jy < W; jy++) {
            const float2 ty = __fmul2_rn(dup(w[W + jy]), t);
#pragma unroll
            for (int jx = 0; jx < W; jx++)
                acc[ky + jy][kx + jx] = __ffma2_rn(dup(w[jx]), ty, acc[ky + jy][kx + jx]);
        }
    };

    unsigned ranges = __ballot_sync(0xffffffffu, cnt > 0);
    fetch(0, 0);
    cp_commit();
    if (total > kVisitBatch) fetch(kVisitBatch, 1);
    cp_commit();
    cp_wait<1>();
    __syncwarp();
    int base = 0;  // first visit of the current buffer
    int pos = 0, left = 0, col = 0, zoff = 0, buf = ring;
    while (ranges || left) {
        if (!left) {
            const int s = __ffs(ranges) - 1;
            ranges &= ranges - 1;
            left = __shfl_sync(0xffffffffu, cnt, s);
            col = s & 15;
            zoff = s >> 4 ? z + g.G[2] : z;
        }
        if (pos == kVisitBatch) {
            // the other buffer next; this one takes the batch after it
            __syncwarp();
            base += kVisitBatch;
            if (base + kVisitBatch < total) fetch(base + kVisitBatch, (base / kVisitBatch + 1) & 1);
            cp_commit();
            cp_wait<1>();
            __syncwarp();
            buf = ring + ((base / kVisitBatch) & 1) * S::BUF;
            pos = 0;
        }
        const int n = min(left, kVisitBatch - pos);
        const int end = pos + n;
        left -= n;
        switch (col) {
#define DMR_COL(K)                                                                                       \
    case K:                                                                                              \
        if constexpr (K < TT) {                                                                          \
            for (; pos < end; pos++) visit(std::integral_constant<int, K>{}, buf, pos, zoff);            \
        }                                                                                                \
        break;
            DMR_COL(0) DMR_COL(1) DMR_COL(2) DMR_COL(3) DMR_COL(4) DMR_COL(5) DMR_COL(6) DMR_COL(7)
            DMR_COL(8) DMR_COL(9) DMR_COL(10) DMR_COL(11) DMR_COL(12) DMR_COL(13) DMR_COL(14) DMR_COL(15)
#undef DMR_COL
        }
    }
    cp_wait<0>();

    if (scratch) {
        float2 *d = scratch + (int64_t)u * (R * R) * g.CS + c;
        if (c < g.CS && z <= z1) {
#pragma unroll
            for (int i = 0; i < R; i++)
#pragma unroll
                for (int k = 0; k < R; k++) __stcs(d + (int64_t)(i * R + k) * g.CS, acc[i][k]);
        }
        return;
    }
    // pieces of one tile's plane that neighbouring warps hold are added before they
    // go to the grid: warps 1 and 3 to 0 and 2, then 2 to 0 (through the pair's
    // shared memory, `give` to `take`, whose barriers both sides reach). A heavy
    // plane's sum is then a tree over units of a block and a chain over blocks, a
    // quarter as long: it is the chain in the grid that rounds most (64^3, 8 coils:
    // 8.4e-7 of the result without, see unit_visits). Long units gain nothing from it
    // (192^3, 32 coils: 1.2e-6 either way, 0.06 of 11.5 ms)
    static_assert(kGridWarps == 4, "pairs of warps");
    auto same = [&](int v) {  // unit v is a piece of the same plane
        if (v < 0 || v >= nunits) return false;
        const int4 o = units[v];
        return o.x == un.x && o.y == un.y;
    };
    auto join = [](int id) {
        __syncwarp();
        asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
    };
    auto give = [&](int at) {
        float2 *d = reinterpret_cast<float2 *>(msm + at) + lane;
#pragma unroll
        for (int i = 0; i < R; i++)
#pragma unroll
            for (int k = 0; k < R; k++) d[(i * R + k) * 32] = acc[i][k];
    };
    auto take = [&](int at) {
        const float2 *d = reinterpret_cast<const float2 *>(msm + at) + lane;
#pragma unroll
        for (int i = 0; i < R; i++)
#pragma unroll
            for (int k = 0; k < R; k++) acc[i][k] = __fadd2_rn(acc[i][k], d[(i * R + k) * 32]);
    };
    const int pair = (warp >> 1) * S::PAIR;
    if (g.join && same(warp & 1 ? u - 1 : u + 1)) {
        join(1 + (warp >> 1));  // both are done with their rings
        if (warp & 1) give(pair);
        join(1 + (warp >> 1));
        if (warp & 1) return;
        take(pair);
    }
    if (g.join && !(warp & 1) && same(warp ? u - 2 : u + 2)) {  // (the unit between is one of the plane's, too)
        join(3);  // warp 0 has taken what lay in its pair's memory
        if (warp) give(0);
        join(3);
        if (warp) return;
        take(0);
    }
    if (c >= g.CS || z > z1) return;
    const int ntile = g.nt0 * g.nt1;
    const int f = ft / ntile, t2 = ft - f * ntile, ty = t2 / g.nt0, tx = t2 - ty * g.nt0;
    int pz = z - g.half[2], px = tx * T - g.half[0], py = ty * T - g.half[1];
    if (pz < 0) pz += g.G[2];
    if (px < 0) px += g.G[0];
    if (py < 0) py += g.G[1];
    float2 *gz = grid + (f * g.gsize + pz * g.plane) * g.CS + c;
    int xo[R];
#pragma unroll
    for (int k = 0; k < R; k++) {
        xo[k] = px * g.CS;
        px = px + 1 == g.G[0] ? 0 : px + 1;
    }
#pragma unroll
    for (int i = 0; i < R; i++) {
        float2 *row = gz + (int64_t)py * g.G[0] * g.CS;
        py = py + 1 == g.G[1] ? 0 : py + 1;
#pragma unroll
        for (int k = 0; k < R; k++) atomicAdd(row + xo[k], acc[i][k]);
    }
}

// The tiles (extent T, region R <= 8) that cover centred position t of an axis,
// as 16-bit entries (tile << 3 | offset) + 1 in increasing offset, 0 after the
// last (tile origins b T < G; offsets past the end of the axis wrap)
template <int T, int R>
__device__ __forceinline__ uint4 tile_cover(int t, int G)
{
    uint32_t e[4] = {0, 0, 0, 0};
    int n = 0;
    for (int u = 0; u < R; u++) {
        int o = t - u;
        while (o < 0) o += G;
        if (o % T == 0) {
            e[n >> 1] |= ((uint32_t)(o / T << 3 | u) + 1u) << (16 * (n & 1));
            n++;
        }
    }
    return make_uint4(e[0], e[1], e[2], e[3]);
}

__device__ __forceinline__ int cover_at(const uint4 &c, int k)
{
    const uint32_t w = k < 4 ? (k < 2 ? c.x : c.y) : (k < 6 ? c.z : c.w);
    return (int)((w >> (16 * (k & 1))) & 0xffff) - 1;
}

// Deterministic mode: a grid point adds the slots of the units whose tile
// regions cover it (tiles by y, then x offset, then a unit's pieces in visit
// order). Blocks loop over grid rows (frame, z, y): the row's y tiles and the
// unit ranges of all their x tiles come into shared memory once, threads run
// along (x, coil), the slots of up to four tiles are loaded together. Every
// point is written.
template <int W>
__global__ void __launch_bounds__(256) grid_planes_gather_kernel(MarchGeom g, int nframes,
                                                                 const int32_t *__restrict__ ustart,
                                                                 const float2 *__restrict__ scratch,
                                                                 float2 *__restrict__ grid)
{
    constexpr int T = march_tile(W), R = T + W - 1;
    extern __shared__ __align__(16) unsigned char msm[];
    uint4 *xcov = reinterpret_cast<uint4 *>(msm);             // G[0]
    int2 *su = reinterpret_cast<int2 *>(xcov + g.G[0]);       // R x nt0 unit ranges
    for (int x = threadIdx.x; x < g.G[0]; x += blockDim.x) {
        int t = x + g.half[0];
        xcov[x] = tile_cover<T, R>(t >= g.G[0] ? t - g.G[0] : t, g.G[0]);
    }
    const int64_t nrows = (int64_t)nframes * g.G[2] * g.G[1];
    for (int64_t row = blockIdx.x; row < nrows; row += gridDim.x) {
        const int64_t r2 = row / g.G[1];
        const int y = (int)(row - r2 * g.G[1]), f = (int)(r2 / g.G[2]), z = (int)(r2 - (int64_t)f * g.G[2]);
        int lz = z + g.half[2], ly = y + g.half[1];  // centred positions
        if (lz >= g.G[2]) lz -= g.G[2];
        if (ly >= g.G[1]) ly -= g.G[1];
        const uint4 ycov = tile_cover<T, R>(ly, g.G[1]);
        int ny = 0;
        while (ny < 8 && cover_at(ycov, ny) >= 0) ny++;
        __syncthreads();  // the previous row's ranges are consumed
        for (int e = threadIdx.x; e < ny * g.nt0; e += blockDim.x) {
            const int k = e / g.nt0, tx = e - k * g.nt0;
            const int64_t ft = ((int64_t)f * g.nt1 + (cover_at(ycov, k) >> 3)) * g.nt0 + tx;
            const int s0 = __ldg(ustart + ft * g.G[2] + lz);
            su[e] = make_int2(s0, __ldg(ustart + ft * g.G[2] + lz + 1) - s0);
        }
        __syncthreads();
        for (int e = threadIdx.x; e < g.G[0] * g.CS; e += blockDim.x) {
            const int x = e / g.CS, c = e - x * g.CS;
            const uint4 xc = xcov[x];
            float2 acc = make_float2(0.0f, 0.0f);
            const int x0 = cover_at(xc, 0), x1 = cover_at(xc, 1);
            auto slot = [&](int s, int ky, int vx) {
                const int dy = cover_at(ycov, ky) & 7;
                return scratch + ((int64_t)s * (R * R) + dy * R + (vx & 7)) * g.CS + c;
            };
            // a split unit's further pieces; short ones (width 6) eight at a time, the
            // chain of a heavy plane's pieces rounds most (long ones that way: 1.11e-6
            // of the result both ways, 64^3, W 4, and 2 % of the call's time)
            auto rest = [&](int2 u, int ky, int vx) {
                if constexpr (W < 6) {
                    for (int s = 1; s < u.y; s++) acc = __fadd2_rn(acc, __ldcs(slot(u.x + s, ky, vx)));
                } else {
                    for (int s = 1; s < u.y;) {
                        float2 sum = __ldcs(slot(u.x + s, ky, vx));
                        for (const int e = min(s + 8, u.y); ++s < e;) sum = __fadd2_rn(sum, __ldcs(slot(u.x + s, ky, vx)));
                        acc = __fadd2_rn(acc, sum);
                    }
                }
            };
            if (ny <= 2 && cover_at(xc, 2) < 0) {
                int2 u[4];
                float2 v[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int ky = q >> 1, vx = q & 1 ? x1 : x0;
                    u[q] = ky < ny && vx >= 0 ? su[ky * g.nt0 + (vx >> 3)] : make_int2(0, 0);
                    if (u[q].y > 0) v[q] = __ldcs(slot(u[q].x, ky, vx));
                }
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (u[q].y > 0) {
                        acc = __fadd2_rn(acc, v[q]);
                        rest(u[q], q >> 1, q & 1 ? x1 : x0);
                    }
            } else {
                for (int ky = 0; ky < ny; ky++)
                    for (int k = 0; k < 8; k++) {
                        const int vx = cover_at(xc, k);
                        if (vx < 0) break;
                        const int2 u = su[ky * g.nt0 + (vx >> 3)];
                        if (u.y > 0) {
                            acc = __fadd2_rn(acc, __ldcs(slot(u.x, ky, vx)));
                            rest(u, ky, vx);
                        }
                    }
            }
            grid[row * g.G[0] * g.CS + e] = acc;
        }
    }
}

// ---------------------------------------------------------------------------
// Interpolation. A block stages the region of an item (march_rows(W) rows of a
// tile's columns over kItemZ z cells, plus the halo, CC coils) and the
// weight records of its samples (at most kItemSamples) in shared memory. The
// samples, in (column, z) order, are cut evenly among the warps. Lane = (plane
// group, row group, coil): the W^3 taps of the current cell sit in registers,
// plane z in slot z mod P of its lane group, and moving to the next z cell of
// a column loads only the planes that enter (W^2 taps instead of W^3). The
// groups' partial sums are added with shuffles and the sample's row stored
// (coils contiguous). 192^3 kooshball, 32 coils: 8.7 ms and 1.6 ms for the
// rows (cell-cube kernel on planar grids: 15.6 ms); the FMAs alone are 2.8 ms,
// the rest is latency at 3 warps per scheduler (168 registers: the cube).
// ---------------------------------------------------------------------------
constexpr int kItemCap = kItemSamples + 8;   // a part of an item rounds up per column

template <int W, int NZ, int NY>
struct InterpShape {
    static constexpr int T = march_tile(W), REC = march_rec(W);
    static constexpr int SPL = (W + NZ - 1) / NZ, P = NZ * SPL;  // plane slots per lane, in all
    static constexpr int RY = (W + NY - 1) / NY;                 // tap rows per lane
    static_assert(SPL <= 4, "slots per lane");
    static constexpr int NG = NZ * NY, CC = 32 / NG;             // lane groups, coils per group
    static constexpr int NW = NZ == 1 ? 6 : 4;                   // warps
    static constexpr int H = march_rows(W), COLS = T * H;        // rows of columns, columns
    static constexpr int RX = T + W - 1, RYE = H + W - 1, RZ = kItemZ + W - 1, PTS = RX * RYE * RZ;
    static constexpr int TILE = (PTS * CC * 8 + 15) / 16 * 16;
    static constexpr int SMEM = TILE + kItemCap * (REC * 4 + 4);
    static constexpr int MINB = NZ == 1 || SPL * RY * W > 64 ? 2 : 4;
};

template <int W, int NZ, int NY>
__global__ void __launch_bounds__(32 * InterpShape<W, NZ, NY>::NW, InterpShape<W, NZ, NY>::MINB)
    interp_march_kernel(MarchGeom g, const int4 *__restrict__ items, const int32_t *__restrict__ cstart,
                        const float *__restrict__ rec, const int32_t *__restrict__ zc, const float2 *__restrict__ grid,
                        float2 *__restrict__ rows)
{
    using S = InterpShape<W, NZ, NY>;
    constexpr int T = S::T, TT = T * T, REC = S::REC, SPL = S::SPL, P = S::P, RY = S::RY, CC = S::CC, RX = S::RX,
                  RYE = S::RYE, COLS = S::COLS, NW = S::NW, NH = TT / COLS;
    extern __shared__ __align__(16) unsigned char msm[];
    __shared__ int s_beg[COLS], s_pre[COLS + 1];
    __shared__ int s_x[RX];
    __shared__ int64_t s_y[RYE], s_z[S::RZ];
    float2 *tile = reinterpret_cast<float2 *>(msm);
    float *srec = reinterpret_cast<float *>(msm + S::TILE);
    int *szc = reinterpret_cast<int *>(msm + S::TILE + kItemCap * REC * 4);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int4 it = items[blockIdx.x];
    const int ft = it.x, h = it.y % NH, z0 = it.y / NH * kItemZ, z1 = min(z0 + kItemZ, g.G[2]);
    const int c0 = blockIdx.y * CC;
    const int ntile = g.nt0 * g.nt1;
    const int f = ft / ntile, t2 = ft - f * ntile, ty = t2 / g.nt0, tx = t2 - ty * g.nt0;
    if (warp == 0) {
        // the columns' sample ranges (this part of them) and their offsets in the item
        int beg = 0, cnt = 0;
        if (lane < COLS) {
            const int32_t *cs = cstart + ((int64_t)ft * TT + h * COLS + lane) * g.G[2];
            const int b = cs[z0], n = cs[z1] - b;
            const int lo = (int)((int64_t)n * it.z / it.w), hi = (int)((int64_t)n * (it.z + 1) / it.w);
            beg = b + lo;
            cnt = hi - lo;
        }
        int incl = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += o;
        }
        if (lane < COLS) {
            s_beg[lane] = beg;
            s_pre[lane + 1] = incl;
        }
        if (lane == 0) s_pre[0] = 0;
    } else {
        // grid offsets of the region's positions on each axis
        const int e = tid - 32;
        if (e < RX) s_x[e] = (tx * T + e + g.G[0] - g.half[0]) % g.G[0] * g.CS;
        else if (e < RX + RYE)
            s_y[e - RX] = (int64_t)((ty * T + h * S::H + e - RX + g.G[1] - g.half[1]) % g.G[1]) * g.G[0] * g.CS;
        else if (e < RX + RYE + S::RZ)
            s_z[e - RX - RYE] = (int64_t)((z0 + e - RX - RYE + g.G[2] - g.half[2]) % g.G[2]) * g.plane * g.CS;
    }
    __syncthreads();
    // region rows: RX points of CC coils each
    {
        const float2 *gf = grid + f * g.gsize * g.CS + c0;
        const bool pair = (CC & 1) == 0 && (g.CS & 1) == 0;
        for (int row = warp; row < RYE * S::RZ; row += NW) {
            const int rz = row / RYE;
            const float2 *src = gf + s_z[rz] + s_y[row - rz * RYE];
            const uint32_t dst = smem_addr(tile + row * (RX * CC));
            if (pair) {
                constexpr int LPR = CC > 1 ? CC / 2 : 1;
#pragma unroll
                for (int q = lane; q < RX * LPR; q += 32) {
                    const int pt = q / LPR, e = 2 * (q - pt * LPR);
                    if (c0 + e < g.CS) cp16(dst + q * 16, src + s_x[pt] + e);
                }
            } else {
#pragma unroll
                for (int q = lane; q < RX * CC; q += 32) {
                    const int pt = q / CC, e = q - pt * CC;
                    if (c0 + e < g.CS) cp8(dst + q * 8, src + s_x[pt] + e);
                }
            }
        }
    }
    const int n = s_pre[COLS];
    // weight records and z cells, item order
    for (int s = warp; s < COLS; s += NW) {
        const int pre = s_pre[s], m = s_pre[s + 1] - pre, beg = s_beg[s];
        const uint32_t d = smem_addr(srec + pre * REC), dz = smem_addr(szc + pre);
        for (int q = lane; q < m * (REC / 4); q += 32) cp16(d + q * 16, rec + (int64_t)beg * REC + 4 * q);
        for (int q = lane; q < m; q += 32) cp4(dz + q * 4, zc + beg + q);
    }
    cp_commit();
    cp_wait<0>();
    __syncthreads();

    // (lanes past the last group idle as a copy of it; nothing of theirs is used)
    const int lg = min(lane / CC, S::NG - 1), c = lane % CC, gz = lg % NZ, gy = lg / NZ;
    const bool store = lane < CC && c0 + c < g.CS;
    const int f1 = n * (warp + 1) / NW;
    int q = n * warp / NW;
    int s = 0;
    float2 cube[SPL][RY][W];
    // taps of plane rz of the column into slot kc of the lane
    auto load = [&](auto kc, int off) {
        constexpr int k = decltype(kc)::value;
        const float2 *tp = reinterpret_cast<const float2 *>(msm + off);
        if constexpr (k < SPL) {
            // (a marker per slot: merged branches would index the registers)
            asm volatile("// slot %0" ::"n"(k));
#pragma unroll
            for (int i = 0; i < RY; i++)
                if (NY == 1 || gy * RY + i < W) {
#pragma unroll
                    for (int j = 0; j < W; j++) cube[k][i][j] = tp[(i * RX + j) * CC];
                }
        }
    };
    // sum over the x taps, then y, of slot k
    auto plane_sum = [&](int k, const float *w, const float *wy) {
        float2 r[RY], t = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int j = 0; j < W; j++)
#pragma unroll
            for (int i = 0; i < RY; i++) {
                const float2 wx = dup(w[j]);
                r[i] = j == 0 ? __fmul2_rn(wx, cube[k][i][j]) : __ffma2_rn(wx, cube[k][i][j], r[i]);
            }
#pragma unroll
        for (int i = 0; i < RY; i++) {
            if (NY > 1 && gy * RY + i >= W) continue;
            t.x = i == 0 ? wy[i] * r[i].x : fmaf(wy[i], r[i].x, t.x);
            t.y = i == 0 ? wy[i] * r[i].y : fmaf(wy[i], r[i].y, t.y);
        }
        return t;
    };
    while (q < f1) {
        while (s_pre[s + 1] <= q) s++;
        const int qe = min(f1, s_pre[s + 1]);
        const int tcol = (((s / T + gy * RY) * RX + s % T) * CC + c) * 8;
        float2 *orow = rows + (int64_t)(s_beg[s] - s_pre[s] + q) * g.RS + c0 + c;
        int wo = S::TILE + q * (REC * 4);  // the sample's record (offset in shared memory)
        int have = 0;  // planes below `have` are loaded
        while (q < qe) {
            // runs of samples of one z cell, found for 32 samples at a time
            const int m = min(32, qe - q);
            const int zl = szc[q + min(lane, m - 1)] - z0;
            const int zp = __shfl_up_sync(0xffffffffu, zl, 1);
            unsigned heads = __ballot_sync(0xffffffffu, lane < m && (lane == 0 || zl != zp));
            q += m;
            while (heads) {
                const int h0 = __ffs(heads) - 1;
                heads &= heads - 1;
                int cnt = (heads ? __ffs(heads) - 1 : m) - h0;
                const int zz = __shfl_sync(0xffffffffu, zl, h0);
                // tap of each slot's plane; the planes that entered since the
                // column's last run (local z >= have) are loaded
                int wi[SPL];
                const int zm = zz % P;
#pragma unroll
                for (int k = 0; k < SPL; k++) {
                    wi[k] = gz + NZ * k - zm;
                    if (wi[k] < 0) wi[k] += P;
                }
                auto enter = [&](auto kc) {
                    constexpr int k = decltype(kc)::value;
                    if constexpr (k < SPL)
                        if (wi[k] < W && zz + wi[k] >= have) load(kc, tcol + (zz + wi[k]) * (RX * RYE * CC * 8));
                };
                enter(std::integral_constant<int, 0>{});
                enter(std::integral_constant<int, 1>{});
                enter(std::integral_constant<int, 2>{});
                enter(std::integral_constant<int, 3>{});
                have = zz + W;
                for (; cnt > 0; cnt--, wo += REC * 4) {
                    const float *wp = reinterpret_cast<const float *>(msm + wo);
                    float w[REC];
#pragma unroll
                    for (int e = 0; e < ((NY == 1 ? 2 * W : W) + 3) / 4; e++)
                        *reinterpret_cast<float4 *>(w + 4 * e) = *reinterpret_cast<const float4 *>(wp + 4 * e);
                    float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
                    for (int k = 0; k < SPL; k++) {
                        const float2 t = plane_sum(k, w, NY == 1 ? w + W : wp + W + gy * RY);
                        if (P == W || wi[k] < W) {
                            const float wz = wp[2 * W + wi[k]];
                            acc.x = fmaf(wz, t.x, acc.x);
                            acc.y = fmaf(wz, t.y, acc.y);
                        }
                    }
                    // groups 0 .. NG - 1 added into group 0
#pragma unroll
                    for (int m = S::NG; m > 1; m = (m + 1) / 2) {
                        const int h = (m + 1) / 2;
                        const float ox = __shfl_down_sync(0xffffffffu, acc.x, h * CC);
                        const float oy = __shfl_down_sync(0xffffffffu, acc.y, h * CC);
                        if (lg + h < m) {
                            acc.x += ox;
                            acc.y += oy;
                        }
                    }
                    if (store) *orow = acc;
                    orow += g.RS;
                }
            }
        }
    }
}

// Few coils: the same items and regions, a thread per sample. Lanes as (plane
// group, coil) leave most of a warp idle then, and a region staged for more coils
// than there are keeps blocks off the SM.
constexpr int kFewThreads = 128;

template <int W, int CC>
__global__ void __launch_bounds__(kFewThreads)
    interp_few_kernel(MarchGeom g, const int4 *__restrict__ items, const int32_t *__restrict__ cstart,
                      const float *__restrict__ rec, const int32_t *__restrict__ zc, const float2 *__restrict__ grid,
                      float2 *__restrict__ rows)
{
    using S = InterpShape<W, W, 1>;
    constexpr int T = S::T, TT = T * T, REC = S::REC, RX = S::RX, RYE = S::RYE, COLS = S::COLS, NH = TT / COLS;
    __shared__ __align__(16) float2 tile[S::PTS * CC];
    __shared__ int s_beg[COLS], s_pre[COLS + 1];
    const int tid = threadIdx.x, lane = tid & 31;
    const int4 it = items[blockIdx.x];
    const int ft = it.x, h = it.y % NH, z0 = it.y / NH * kItemZ, z1 = min(z0 + kItemZ, g.G[2]);
    const int ntile = g.nt0 * g.nt1;
    const int f = ft / ntile, t2 = ft - f * ntile, ty = t2 / g.nt0, tx = t2 - ty * g.nt0;
    // region points, CC coils each
    const float2 *gf = grid + f * g.gsize * g.CS;
    for (int e = tid; e < S::PTS * CC; e += kFewThreads) {
        const int pt = e / CC, c = e - pt * CC;
        const int x = pt % RX, r = pt / RX, y = r % RYE, z = r / RYE;
        const int gx = (tx * T + x + g.G[0] - g.half[0]) % g.G[0], gy = (ty * T + h * S::H + y + g.G[1] - g.half[1]) % g.G[1],
                  gz = (z0 + z + g.G[2] - g.half[2]) % g.G[2];
        if (c < g.CS) cp8(smem_addr(tile + e), gf + (gz * g.plane + (int64_t)gy * g.G[0] + gx) * g.CS + c);
    }
    cp_commit();
    if (tid < 32) {
        // the columns' sample ranges (this part of them) and their offsets in the item
        int beg = 0, cnt = 0;
        if (lane < COLS) {
            const int32_t *cs = cstart + ((int64_t)ft * TT + h * COLS + lane) * g.G[2];
            const int b = cs[z0], n = cs[z1] - b;
            const int lo = (int)((int64_t)n * it.z / it.w), hi = (int)((int64_t)n * (it.z + 1) / it.w);
            beg = b + lo;
            cnt = hi - lo;
        }
        int incl = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += o;
        }
        if (lane < COLS) {
            s_beg[lane] = beg;
            s_pre[lane + 1] = incl;
        }
        if (lane == 0) s_pre[0] = 0;
    }
    cp_wait<0>();
    __syncthreads();
    const int n = s_pre[COLS];
    for (int q = tid; q < n; q += kFewThreads) {
        int s = 0;
        while (s_pre[s + 1] <= q) s++;
        const int64_t j = s_beg[s] + q - s_pre[s];
        float w[REC];
#pragma unroll
        for (int e = 0; e < REC / 4; e++)
            *reinterpret_cast<float4 *>(w + 4 * e) = __ldg(reinterpret_cast<const float4 *>(rec + j * REC) + e);
        const float2 *tp = tile + ((((zc[j] - z0) * RYE + s / T) * RX) + s % T) * CC;
        float2 acc[CC];
#pragma unroll
        for (int c = 0; c < CC; c++) acc[c] = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int k = 0; k < W; k++) {
            float2 t[CC];
#pragma unroll
            for (int i = 0; i < W; i++) {
                float2 r[CC];
#pragma unroll
                for (int x = 0; x < W; x++)
#pragma unroll
                    for (int c = 0; c < CC; c++) {
                        const float2 v = tp[((k * RYE + i) * RX + x) * CC + c];
                        r[c] = x == 0 ? __fmul2_rn(dup(w[x]), v) : __ffma2_rn(dup(w[x]), v, r[c]);
                    }
#pragma unroll
                for (int c = 0; c < CC; c++)
                    t[c] = i == 0 ? __fmul2_rn(dup(w[W + i]), r[c]) : __ffma2_rn(dup(w[W + i]), r[c], t[c]);
            }
#pragma unroll
            for (int c = 0; c < CC; c++) acc[c] = __ffma2_rn(dup(w[2 * W + k]), t[c], acc[c]);
        }
#pragma unroll
        for (int c = 0; c < CC; c++)
            if (c < g.CS) rows[j * g.RS + c] = acc[c];
    }
}

int march_blocks(int64_t n)
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, 256), (int64_t)sms * 16));
}

MarchGeom march_geom(const dmr_plan *p, int CS)
{
    const Geom &g = p->g;
    MarchGeom m;
    for (int a = 0; a < 3; a++) {
        m.G[a] = g.G[a];
        m.half[a] = g.half[a];
    }
    m.T = march_tile(g.W[0]);
    m.nt0 = p->mp_nt[0];
    m.nt1 = p->mp_nt[1];
    m.CS = CS;
    m.RS = (CS + 1) & ~1;
    m.join = true;
    m.plane = (int64_t)g.G[0] * g.G[1];
    m.gsize = g.gsize;
    return m;
}

template <int W, int NP, int ND>
int launch_planes_np(const dmr_plan *p, const MarchGeom &m, const void *units, int n, const float2 *rows, float2 *grid,
                     float2 *scratch, cudaStream_t st)
{
    using S = PlaneShape<W, NP, ND>;
    if (n == 0) return DMR_OK;
    auto kern = grid_planes_kernel<W, NP, ND>;
    DMR_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM));
    kern<<<(unsigned)ceil_div(n, kGridWarps), 32 * kGridWarps, S::SMEM, st>>>(m, (const int4 *)units, n,
                                                                             p->mp_cstart, p->mp_rec, p->mp_zc, rows,
                                                                             grid, scratch);
    DMR_LAUNCHED("grid_planes_kernel");
    return DMR_OK;
}

// Single planes come in long units from 20 coils on, where these took the place of
// tensor-core sums (64^3, W 4: 3.7e-6 of the result, now 1.1e-6); 17 to 19 coils
// had the sums of the cell-cube kernel (8.0e-7) and get short ones (8.2e-7), built
// by a plan's first such call
bool short_planes(const dmr_plan *p, int CS) { return p->g.ndim == 3 && p->mp_W <= 5 && CS > 16 && CS < 20; }

// planes per warp by the coils of the chunk: lanes = coils x planes (96^3, 8
// coils: 385 us with 4 planes, 760 us with the cell-cube kernel; 1 coil: 227 and
// 411 us)
template <int W>
int launch_planes(const dmr_plan *p, const MarchGeom &m, const float2 *rows, float2 *grid, float2 *scratch,
                  cudaStream_t st)
{
    const auto units = p->mp_units;
    const int *n = p->mp_nunits;
    if (p->g.ndim == 2) return launch_planes_np<W, 1, 2>(p, m, units[0], n[0], rows, grid, scratch, st);
    // deterministic units are always single planes of one list, so that a coil's
    // sums do not depend on how many coils it is gridded with
    if (!scratch && short_planes(p, m.CS)) {
        const ShortUnits &s = *p->short_ptr.load(std::memory_order_acquire);
        return launch_planes_np<W, 1, 3>(p, m, s.units, s.n, rows, grid, scratch, st);
    }
    if (scratch || m.CS > 16) {
        MarchGeom long_units = m;
        long_units.join = W == 6;
        return launch_planes_np<W, 1, 3>(p, long_units, units[0], n[0], rows, grid, scratch, st);
    }
    if (m.CS > 8) return launch_planes_np<W, 2, 3>(p, m, units[1], n[1], rows, grid, scratch, st);
    if (m.CS > 4) return launch_planes_np<W, 4, 3>(p, m, units[2], n[2], rows, grid, scratch, st);
    return launch_planes_np<W, 8, 3>(p, m, units[3], n[3], rows, grid, scratch, st);
}

// dynamic shared memory of a gather block: cover lists of the x positions, unit
// ranges of up to 8 rows of tiles
size_t gather_smem(const MarchGeom &m) { return (size_t)m.G[0] * sizeof(uint4) + (size_t)8 * m.nt0 * sizeof(int2); }

template <int W>
int launch_gather(const dmr_plan *p, const MarchGeom &m, const float2 *scratch, float2 *grid, cudaStream_t st)
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t smem = gather_smem(m);
    auto kern = grid_planes_gather_kernel<W>;
    DMR_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int64_t nrows = (int64_t)p->g.nframes * m.G[2] * m.G[1];
    kern<<<(unsigned)std::min<int64_t>(nrows, (int64_t)sms * 8), 256, smem, st>>>(m, p->g.nframes, p->mp_ustart, scratch,
                                                                               grid);
    DMR_LAUNCHED("grid_planes_gather_kernel");
    return DMR_OK;
}

template <int W, int NZ, int NY>
int launch_interp_n(const dmr_plan *p, const MarchGeom &m, const float2 *grid, float2 *rows, cudaStream_t st)
{
    using S = InterpShape<W, NZ, NY>;
    auto kern = interp_march_kernel<W, NZ, NY>;
    DMR_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM));
    kern<<<dim3(p->mp_nitems, (unsigned)ceil_div(m.CS, S::CC)), 32 * S::NW, S::SMEM, st>>>(
        m, (const int4 *)p->mp_items, p->mp_cstart, p->mp_rec, p->mp_zc, grid, rows);
    DMR_LAUNCHED("interp_march_kernel");
    return DMR_OK;
}

template <int W, int CC>
int launch_interp_few(const dmr_plan *p, const MarchGeom &m, const float2 *grid, float2 *rows, cudaStream_t st)
{
    interp_few_kernel<W, CC><<<p->mp_nitems, kFewThreads, 0, st>>>(m, (const int4 *)p->mp_items, p->mp_cstart, p->mp_rec,
                                                                  p->mp_zc, grid, rows);
    DMR_LAUNCHED("interp_few_kernel");
    return DMR_OK;
}

template <int W>
int launch_interp(const dmr_plan *p, const MarchGeom &m, const float2 *grid, float2 *rows, cudaStream_t st)
{
    // a thread per sample for 1 coil (96^3, 1.8 M samples: W 3, os 1.25, 247 us with
    // lane groups and 105 with this; W 6, os 2, 1,477 and 535), for 2 at the widths
    // whose groups take 3 coils or more at a time (W 2 and 3: 0.95 to 1.8 times the
    // groups' speed, W 6 1.1 to 2.1, W 4 and 5 0.86 to 1.5), and for 3 and 4 at widths
    // 2 and 3 where items have 16 samples or more (4 coils at 65: 1.2 to 1.4 times, at
    // 16: 1.0 to 1.1, at 2: 0.9 to 1.0; W 4 0.6 to 1.0)
    if (m.CS == 1) return launch_interp_few<W, 1>(p, m, grid, rows, st);
    if constexpr (W <= 3 || W == 6)
        if (m.CS == 2) return launch_interp_few<W, 2>(p, m, grid, rows, st);
    if constexpr (W <= 3)
        if (m.CS <= 4 && p->g.total >= 16 * (int64_t)p->mp_nitems) return launch_interp_few<W, 4>(p, m, grid, rows, st);
    // width 6: 10 coils at a time take 1.7 times as long as 5
    if constexpr (W == 6)
        if (5 * ceil_div(m.CS, 10) < 3 * ceil_div(m.CS, 5)) return launch_interp_n<6, 3, 1>(p, m, grid, rows, st);
    // lane groups by the coils of the chunk: as few as leave the lanes filled
    // (each group adds a share of a plane's work and a round of shuffles); a
    // lane holds at most 64 taps
    if constexpr (W <= 4) {
        if (m.CS > 16) return launch_interp_n<W, 1, 1>(p, m, grid, rows, st);
        if (m.CS > 32 / W) return launch_interp_n<W, 2, 1>(p, m, grid, rows, st);
    }
    if (m.CS > (W == 3 ? 3 : 16 / W) || W == 6) return launch_interp_n<W, W, 1>(p, m, grid, rows, st);
    if constexpr (W <= 5) {
        if constexpr (W >= 4)
            if (m.CS > 32 / (W * W)) return launch_interp_n<W, W, 2>(p, m, grid, rows, st);
        return launch_interp_n<W, W, W>(p, m, grid, rows, st);
    }
    return DMR_ERR_UNSUPPORTED;
}

}  // namespace

// ---------------------------------------------------------------------------
// plan building and entry points (march.cuh)
// ---------------------------------------------------------------------------
int march_build(dmr_plan *p, float *const rk[3], int32_t *keys, int32_t *keys_s, const int32_t *vals,
                MarchTotals &totals, cudaStream_t st)
{
    const Geom &g = p->g;
    const int W = g.W[0], dev = p->device;
    if (g.ndim < 2 || g.total == 0 || W < 2 || W > 6 || g.W[1] != W || (g.ndim == 3 && g.W[2] != W)) return DMR_OK;
    const int T = march_tile(W), TT = T * T;
    const int nt0 = (int)ceil_div(g.G[0], T), nt1 = (int)ceil_div(g.G[1], T);
    const int64_t nft = (int64_t)g.nframes * nt0 * nt1, ncells = nft * TT * g.G[2];
    // the CSR offsets take 4 bytes per cell: not for grids that are huge for
    // their samples (their plans keep the bin kernels)
    if (ncells >= INT32_MAX || ncells > 16 * g.total + (1 << 24)) return DMR_OK;
    // 2D tiles pay from a few samples per tile on (below, a tile's flush costs
    // more than its samples' own additions: direct2d.cu), and go with the
    // interleaved grids of direct2d.cu, which has built its records before
    if (g.ndim == 2 && (p->d2_W == 0 || g.total < 4 * nft)) return DMR_OK;
    const bool d3 = g.ndim == 3;
    // lists: gridding units (2D: the first), interpolation items (3D)
    const int nl = d3 ? kUnitLists + 1 : 1;
    const auto np = kUnitPlanes;
    const int nzb = (int)ceil_div(g.G[2], kItemZ), cols = T * march_rows(W), nzbh = nzb * (TT / cols);
    int per[kUnitLists + 1];  // entries per frame tile before splitting
    int64_t off[kUnitLists + 2] = {0};
    for (int l = 0; l < nl; l++) {
        per[l] = l < kUnitLists ? (int)ceil_div(g.G[2], np[l]) : nzbh;
        off[l + 1] = off[l] + nft * per[l] + 1;
    }
    PlanTemp tmp(dev, st);
    int32_t *counts = nullptr, *starts = nullptr;
    DMR_TRY(tmp.alloc(&counts, ncells + 1));
    DMR_TRY(tmp.alloc(&starts, off[nl]));
    DMR_TRY(plan_alloc(dev, &p->mp_cstart, ncells + 1, st));
    DMR_TRY(plan_alloc(dev, &p->mp_sidx, g.total, st));
    DMR_TRY(plan_alloc(dev, &p->mp_inv, g.total, st));
    DMR_TRY(plan_alloc(dev, &p->mp_zc, d3 ? g.total : 1, st));
    DMR_TRY(plan_alloc(dev, &p->mp_rec, (size_t)g.total * march_rec(W, g.ndim), st));
    DMR_TRY(plan_alloc(dev, &p->mp_ustart, off[1], st));
    DMR_CUDA(cudaMemsetAsync(counts, 0, (ncells + 1) * sizeof(int32_t), st));
    march_key_kernel<<<march_blocks(g.total), 256, 0, st>>>(g, T, nt0, nt1, p->foff_dev, rk[0], rk[1], rk[2], keys,
                                                            counts);
    DMR_LAUNCHED("march_key_kernel");
    int bits = 1;
    while ((1ll << bits) < ncells) bits++;
    size_t tb = 0, t1 = 0;
    DMR_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, keys, keys_s, vals, p->mp_sidx, (int)g.total, 0, bits, st));
    DMR_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, t1, counts, p->mp_cstart, (int)(ncells + 1), st));
    tb = std::max(tb, t1);
    char *temp = nullptr;
    DMR_TRY(tmp.alloc(&temp, tb));
    DMR_CUDA(cub::DeviceRadixSort::SortPairs(temp, tb, keys, keys_s, vals, p->mp_sidx, (int)g.total, 0, bits, st));
    DMR_CUDA(cub::DeviceScan::ExclusiveSum(temp, tb, counts, p->mp_cstart, (int)(ncells + 1), st));
    g_launches.fetch_add(2);
    march_rec_kernel<<<march_blocks(g.total), 256, 0, st>>>(g, p->mp_sidx, rk[0], rk[1], rk[2], p->mp_rec, p->mp_zc,
                                                           p->mp_inv);
    DMR_LAUNCHED("march_rec_kernel");
    // counts -> offsets -> lists (`counts` has room: every list has at most one
    // entry per (frame tile, z) plus one). A list holds at most one entry per
    // non-empty group and one per `most` samples or visits, so it is allocated
    // before its length is known
    for (int l = 0; l < nl; l++) {
        const int64_t n = off[l + 1] - off[l];
        const int most = l < kUnitLists ? unit_visits(g.ndim, W, l) : kItemSamples;
        int4 *list = nullptr;
        if (l < kUnitLists) {
            const int64_t visits = g.total * (d3 ? ceil_div(np[l] + W - 1, np[l]) + 1 : 1);
            DMR_TRY(plan_alloc(dev, &list, std::min(n, visits) + visits / most + 1, st));
            march_unit_count_kernel<<<march_blocks(n), 256, 0, st>>>(p->mp_cstart, nft, TT, g.G[2], d3 ? W : 1, np[l],
                                                                    per[l], most, counts);
        } else {
            DMR_TRY(plan_alloc(dev, &list, std::min(n, g.total) + g.total / most + 1, st));
            march_item_count_kernel<<<march_blocks(n), 256, 0, st>>>(p->mp_cstart, nft, TT, cols, g.G[2], nzb, counts);
        }
        (l < kUnitLists ? p->mp_units[l] : p->mp_items) = list;
        DMR_LAUNCHED("march_count_kernel");
        DMR_CUDA(cub::DeviceScan::ExclusiveSum(temp, tb, counts, starts + off[l], (int)n, st));
        g_launches.fetch_add(1);
        if (l < kUnitLists)
            march_unit_fill_kernel<<<march_blocks(n), 256, 0, st>>>(starts + off[l], nft, per[l], most, list);
        else
            march_item_fill_kernel<<<march_blocks(n), 256, 0, st>>>(starts + off[l], nft, per[l], list);
        DMR_LAUNCHED("march_fill_kernel");
        DMR_CUDA(cudaMemcpyAsync(&totals.v[l], starts + off[l + 1] - 1, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    }
    // the gather finds the units of a (frame tile, plane) by their offsets
    DMR_CUDA(cudaMemcpyAsync(p->mp_ustart, starts, off[1] * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
    totals.n = nl;
    p->mp_nt[0] = nt0;
    p->mp_nt[1] = nt1;
    p->mp_W = W;
    return DMR_OK;
}

// the short units of single planes (short_planes), from the plan's cell offsets
int march_short_build(const dmr_plan *p, ShortUnits &out, cudaStream_t st)
{
    const Geom &g = p->g;
    const int W = p->mp_W, T = march_tile(W), TT = T * T;
    const int64_t nft = (int64_t)g.nframes * p->mp_nt[0] * p->mp_nt[1], n = nft * g.G[2] + 1;
    PlanTemp tmp(p->device, st);
    int32_t *counts = nullptr, *starts = nullptr;
    char *temp = nullptr;
    size_t tb = 0;
    DMR_TRY(tmp.alloc(&counts, n));
    DMR_TRY(tmp.alloc(&starts, n));
    DMR_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, counts, starts, (int)n, st));
    DMR_TRY(tmp.alloc(&temp, tb));
    march_unit_count_kernel<<<march_blocks(n), 256, 0, st>>>(p->mp_cstart, nft, TT, g.G[2], W, 1, g.G[2], kShortUnit,
                                                            counts);
    DMR_LAUNCHED("march_unit_count_kernel");
    DMR_CUDA(cub::DeviceScan::ExclusiveSum(temp, tb, counts, starts, (int)n, st));
    g_launches.fetch_add(1);
    DMR_CUDA(cudaMemcpyAsync(&out.n, starts + n - 1, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    DMR_CUDA(cudaStreamSynchronize(st));
    int4 *list = nullptr;
    DMR_TRY(plan_alloc(p->device, &list, out.n, st));
    out.units = list;
    march_unit_fill_kernel<<<march_blocks(n), 256, 0, st>>>(starts, nft, g.G[2], kShortUnit, list);
    DMR_LAUNCHED("march_unit_fill_kernel");
    DMR_CUDA(cudaStreamSynchronize(st));
    return DMR_OK;
}

void march_lists(dmr_plan *p, const MarchTotals &totals)
{
    for (int l = 0; l < totals.n; l++) (l < kUnitLists ? p->mp_nunits[l] : p->mp_nitems) = totals.v[l];
}

MarchChunks march_chunks(const dmr_plan *p, int64_t batch)
{
    // up to 32 coils at a time, fewer when the rows would take over 8 GB
    int64_t most = 32;
    if (p->mp_W) while (most > 4 && p->g.total * most * (int64_t)sizeof(float2) > (8ll << 30)) most /= 2;
    MarchChunks c;
    c.n = ceil_div(batch, most);
    c.CS = (int)ceil_div(batch, c.n);
    return c;
}

size_t march_rows_bytes(const dmr_plan *p, int CS)
{
    if (!p->mp_W) return 0;  // 2D without tiles: no rows
    return align_up((size_t)p->g.total * ((CS + 1) & ~1) * sizeof(float2), 256);
}

size_t march_il_bytes(const dmr_plan *p, int CS)
{
    return align_up((size_t)p->g.nframes * p->g.gsize * CS * sizeof(float2), 256);
}

#define DMR_MARCH_W(F, ...)                 \
    switch (p->mp_W) {                      \
    case 2: return F<2>(__VA_ARGS__);       \
    case 3: return F<3>(__VA_ARGS__);       \
    case 4: return F<4>(__VA_ARGS__);       \
    case 5: return F<5>(__VA_ARGS__);       \
    case 6: return F<6>(__VA_ARGS__);       \
    default: return DMR_ERR_UNSUPPORTED;    \
    }

static int interp_chunk(const dmr_plan *p, const MarchGeom &m, const float2 *grid, float2 *rows, cudaStream_t st)
{
    DMR_MARCH_W(launch_interp, p, m, grid, rows, st)
}

static int grid_chunk(const dmr_plan *p, const MarchGeom &m, const float2 *rows, float2 *grid, float2 *scratch,
                      cudaStream_t st)
{
    DMR_MARCH_W(launch_planes, p, m, rows, grid, scratch, st)
}

static int gather_chunk(const dmr_plan *p, const MarchGeom &m, const float2 *scratch, float2 *grid, cudaStream_t st)
{
    DMR_MARCH_W(launch_gather, p, m, scratch, grid, st)
}

// coil lanes of the transposing kernels
static int row_lanes(int n) { return n > 16 ? 32 : (n > 8 ? 16 : (n > 4 ? 8 : 4)); }

static int rows_in(const dmr_plan *p, const MarchGeom &m, const void *ksp, int kreal, int64_t b0, int cact,
                   const float *weight, int wpb, float2 *rows, cudaStream_t st)
{
    const int CC = row_lanes(m.RS);
    const auto kern = CC == 32 ? rows_in_kernel<32>
                               : (CC == 16 ? rows_in_kernel<16> : (CC == 8 ? rows_in_kernel<8> : rows_in_kernel<4>));
    kern<<<(unsigned)ceil_div(p->g.total, row_tile(CC)), 256, 0, st>>>(ksp, kreal, p->g.total, b0, cact, m.RS, weight,
                                                                      wpb, (float)(1.0 / p->scale), p->mp_inv, rows);
    DMR_LAUNCHED("rows_in_kernel");
    return DMR_OK;
}

static int rows_out(const dmr_plan *p, const MarchGeom &m, const float2 *rows, int64_t b0, int cact,
                    const float *weight, int wpb, float2 *ksp, cudaStream_t st)
{
    const int CC = row_lanes(m.RS);
    const auto kern = CC == 32 ? rows_out_kernel<32>
                               : (CC == 16 ? rows_out_kernel<16> : (CC == 8 ? rows_out_kernel<8> : rows_out_kernel<4>));
    kern<<<(unsigned)ceil_div(p->g.total, row_tile(CC)), 256, 0, st>>>(rows, p->g.total, b0, cact, m.RS, weight, wpb,
                                                                      (float)(1.0 / p->scale), p->mp_inv, ksp);
    DMR_LAUNCHED("rows_out_kernel");
    return DMR_OK;
}

template <bool PLANAR>
static int transpose(const float2 *src, float2 *dst, int64_t npts, int cact, int CS, cudaStream_t st)
{
    const int CC = row_lanes(CS);
    const auto kern = CC == 32 ? transpose_kernel<32, PLANAR>
                               : (CC == 16 ? transpose_kernel<16, PLANAR>
                                           : (CC == 8 ? transpose_kernel<8, PLANAR> : transpose_kernel<4, PLANAR>));
    kern<<<(unsigned)ceil_div(npts, row_tile(CC)), 256, 0, st>>>(src, dst, npts, cact, CS);
    DMR_LAUNCHED("transpose_kernel");
    return DMR_OK;
}

int march_interleave(const dmr_plan *p, const float2 *src, float2 *dst, int cact, int CS, cudaStream_t st)
{
    return transpose<false>(src, dst, (int64_t)p->g.nframes * p->g.gsize, cact, CS, st);
}

int march_interp(const dmr_plan *p, const float2 *grid, bool planar, float2 *ksp, int64_t batch, const float *weight,
                 int wpb, float2 *rows, float2 *il, cudaStream_t st)
{
    const MarchChunks ch = march_chunks(p, batch);
    const MarchGeom m = march_geom(p, ch.CS);
    const int64_t npts = (int64_t)p->g.nframes * p->g.gsize;
    DMR_CHECK(ch.n < 65536, DMR_ERR_UNSUPPORTED, "batch too large");
    if (p->d2_W && !planar) return d2_interp(p, grid, ksp, 0, ch.n, ch.CS, batch, weight, wpb, st);
    for (int64_t k = 0; k < ch.n; k++) {
        const int64_t b0 = k * ch.CS;
        const int cact = (int)std::min<int64_t>(ch.CS, batch - b0);
        const float2 *src = grid + b0 * npts;
        if (planar && ch.CS > 1) {
            DMR_TRY(transpose<false>(src, il, npts, cact, ch.CS, st));
            src = il;
        }
        if (p->d2_W) {
            DMR_TRY(d2_interp(p, src, ksp, b0, 1, ch.CS, batch, weight, wpb, st));
            continue;
        }
        DMR_TRY(interp_chunk(p, m, src, rows, st));
        DMR_TRY(rows_out(p, m, rows, b0, cact, weight, wpb, ksp, st));
    }
    return DMR_OK;
}

// scratch of deterministic gridding: every unit's plane of one chunk of coils.
// DMR_ERR_UNSUPPORTED (another deterministic kernel takes the call) where that
// is over the caller's limit, and on grids too wide for the gather: its lists
// must fit in shared memory (7,264 x positions at widths 2..4, 6,225 at 5 and 6)
// and its entries hold a tile in 13 bits
static int det_scratch(const dmr_plan *p, const MarchGeom &m, int64_t det_limit, size_t *need)
{
    const int R = m.T + p->mp_W - 1;
    *need = std::max<size_t>((size_t)p->mp_nunits[0] * R * R * m.CS * sizeof(float2), 256);
    if (det_limit > 0 && *need > (size_t)det_limit) return DMR_ERR_UNSUPPORTED;
    int dev = 0, limit = 0;
    DMR_CUDA(cudaGetDevice(&dev));
    DMR_CUDA(cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    return gather_smem(m) > (size_t)limit || std::max(m.nt0, m.nt1) > 8191 ? DMR_ERR_UNSUPPORTED : DMR_OK;
}

int march_grid(const dmr_plan *p, const void *ksp, int kreal, float2 *grid, bool planar, int64_t batch,
               const float *weight, int wpb, int det, int64_t det_limit, float2 *rows, float2 *il, cudaStream_t st)
{
    const MarchChunks ch = march_chunks(p, batch);
    const MarchGeom m = march_geom(p, ch.CS);
    const int64_t npts = (int64_t)p->g.nframes * p->g.gsize;
    const size_t chunk_bytes = (size_t)npts * ch.CS * sizeof(float2);
    float2 *scratch = nullptr;
    DMR_CHECK(ch.n < 65536, DMR_ERR_UNSUPPORTED, "batch too large");
    if (!det && short_planes(p, ch.CS)) DMR_TRY(plan_short(p, st));
    if (!p->mp_W) {
        // 2D, too sparse for tiles
        if (det) return DMR_ERR_UNSUPPORTED;
        if (!planar || ch.CS == 1) {
            DMR_CUDA(cudaMemsetAsync(grid, 0, chunk_bytes * ch.n, st));
            return d2_grid(p, ksp, kreal, grid, 0, ch.n, ch.CS, batch, weight, wpb, st);
        }
        for (int64_t k = 0; k < ch.n; k++) {
            const int64_t b0 = k * ch.CS;
            DMR_CUDA(cudaMemsetAsync(il, 0, chunk_bytes, st));
            DMR_TRY(d2_grid(p, ksp, kreal, il, b0, 1, ch.CS, batch, weight, wpb, st));
            DMR_TRY(transpose<true>(il, grid + b0 * npts, npts, (int)std::min<int64_t>(ch.CS, batch - b0), ch.CS, st));
        }
        return DMR_OK;
    }
    if (det) {
        size_t need = 0;
        DMR_TRY(det_scratch(p, m, det_limit, &need));
        cudaMemPool_t pool = scratch_pool(p->device);
        if (pool == nullptr) return DMR_ERR_UNSUPPORTED;
        void *owned = nullptr;
        const cudaError_t e = cudaMallocFromPoolAsync(&owned, need, pool, st);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            return DMR_ERR_UNSUPPORTED;
        }
        if (e != cudaSuccess) return cuda_fail(e, "cudaMallocFromPoolAsync", __FILE__, __LINE__);
        scratch = (float2 *)owned;
    }
    auto run = [&]() -> int {
        for (int64_t k = 0; k < ch.n; k++) {
            const int64_t b0 = k * ch.CS;
            const int cact = (int)std::min<int64_t>(ch.CS, batch - b0);
            float2 *dst = planar && ch.CS > 1 ? il : grid + b0 * npts;
            DMR_TRY(rows_in(p, m, ksp, kreal, b0, cact, weight, wpb, rows, st));
            if (!det) DMR_CUDA(cudaMemsetAsync(dst, 0, chunk_bytes, st));
            DMR_TRY(grid_chunk(p, m, rows, dst, scratch, st));
            if (det) DMR_TRY(gather_chunk(p, m, scratch, dst, st));
            if (planar && ch.CS > 1) DMR_TRY(transpose<true>(il, grid + b0 * npts, npts, cact, ch.CS, st));
        }
        return DMR_OK;
    };
    const int rc = run();
    if (scratch) cudaFreeAsync(scratch, st);
    return rc;
}

// rows and interleaved grid of a call without a workspace, from the library pool
struct MarchPool {
    float2 *rows = nullptr, *il = nullptr;
    cudaStream_t st;
    void *owned = nullptr;
    MarchPool(const dmr_plan *p, int64_t batch, cudaStream_t s) : st(s)
    {
        const int CS = march_chunks(p, batch).CS;
        const size_t a = march_rows_bytes(p, CS), b = march_il_bytes(p, CS);
        cudaMemPool_t pool = scratch_pool(p->device);
        if (pool && cudaMallocFromPoolAsync(&owned, a + b, pool, st) == cudaSuccess) {
            rows = (float2 *)owned;
            il = (float2 *)((char *)owned + a);
        } else {
            owned = nullptr;
            cudaGetLastError();
        }
    }
    ~MarchPool()
    {
        if (owned) cudaFreeAsync(owned, st);
    }
};

int march_interp_pool(const dmr_plan *p, const float2 *grid, float2 *ksp, int64_t batch, const float *weight, int wpb,
                      cudaStream_t st)
{
    MarchPool b(p, batch, st);
    if (!b.owned) return DMR_ERR_UNSUPPORTED;
    return march_interp(p, grid, true, ksp, batch, weight, wpb, b.rows, b.il, st);
}

int march_grid_pool(const dmr_plan *p, const void *ksp, int kreal, float2 *grid, int64_t batch, const float *weight,
                    int wpb, int det, int64_t det_limit, cudaStream_t st)
{
    if (det && p->mp_W) {  // (before the buffers are allocated)
        size_t need = 0;
        DMR_TRY(det_scratch(p, march_geom(p, march_chunks(p, batch).CS), det_limit, &need));
    }
    MarchPool b(p, batch, st);
    if (!b.owned) return DMR_ERR_UNSUPPORTED;
    return march_grid(p, ksp, kreal, grid, true, batch, weight, wpb, det, det_limit, b.rows, b.il, st);
}

}  // namespace dmr
