// 2D interpolation and sparse gridding, straight between the coil-interleaved
// grid (march.cuh) and the caller's k-space, in acquisition order.
//
// Reference: the 2D kernels of apply_interpolation / apply_gridding
// (src/deepmr/fft/_interp/interp.py:14-120, 150-186 and
//  src/deepmr/fft/_interp/grid.py:14-125, 205-250).
//
// A 2D sample has W^2 <= 36 taps, few enough that no tile pays: consecutive
// samples of a readout share their grid rows in L1, every tap is one coalesced
// access of the coils, and neither a sort nor a transposed copy of the k-space
// is needed. Lane = (sample, coil); a block's samples pass through shared
// memory so that the k-space side runs along the samples. Weights and the
// first tap's grid position come from the plan (d2_rec, d2_base).
#include <algorithm>
#include <cmath>

#include "kb.cuh"
#include "march.cuh"
#include "plan.cuh"

namespace dmr {

namespace {

__host__ __device__ constexpr int d2_rec(int W) { return (2 * W + 3) / 4 * 4; }
// samples per block
__host__ __device__ constexpr int d2_tile(int CC) { return CC <= 4 ? 256 : 1024 / CC; }

struct D2Geom {
    int G0, G1, CS;
    int64_t gsize, npts, total;  // points per frame, per chunk grid; samples
};

// per sample, acquisition order: x and y tap weights, FFT-order position of the
// first tap (x | y << 16) and frame
__global__ void d2_rec_kernel(Geom g, const int64_t *__restrict__ foff, const float *__restrict__ rk0,
                              const float *__restrict__ rk1, float *__restrict__ rec, int2 *__restrict__ base)
{
    const int W = g.W[0], R = d2_rec(W);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < g.total;
         i += (int64_t)gridDim.x * blockDim.x) {
        int lo = 0, hi = g.nframes;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (foff[mid] <= i) lo = mid; else hi = mid;
        }
        const float k[2] = {rk0[i], rk1[i]};
        int pos[2];
        for (int a = 0; a < 2; a++) {
            const int x0 = first_tap_dev(k[a], W);
            pos[a] = pmod(x0 - g.half[a], g.G[a]);
            for (int t = 0; t < W; t++)
                rec[i * R + a * W + t] = tap_weight(x0, t, k[a], W, g.inv_hw[a], g.beta[a]);
        }
        base[i] = make_int2(pos[0] | pos[1] << 16, lo);
    }
}

// grid offsets (in coils) of the taps of a sample: rows and columns
template <int W>
struct Taps {
    float w[d2_rec(W)];
    int xo[W];
    int64_t yo[W];
    __device__ __forceinline__ Taps(const D2Geom &g, const float *__restrict__ rec, int2 b)
    {
#pragma unroll
        for (int q = 0; q < d2_rec(W) / 4; q++)
            *reinterpret_cast<float4 *>(w + 4 * q) = __ldg(reinterpret_cast<const float4 *>(rec) + q);
        int x = b.x & 0xffff, y = b.x >> 16;
        const int64_t f = (int64_t)b.y * g.gsize;
#pragma unroll
        for (int t = 0; t < W; t++) {
            xo[t] = x * g.CS;
            yo[t] = (f + (int64_t)y * g.G0) * g.CS;
            x = x + 1 == g.G0 ? 0 : x + 1;
            y = y + 1 == g.G1 ? 0 : y + 1;
        }
    }
};

template <int W, int CC>
__global__ void __launch_bounds__(256) interp2_kernel(D2Geom g, const float *__restrict__ rec,
                                                      const int2 *__restrict__ base, const float2 *__restrict__ grid,
                                                      float2 *__restrict__ ksp, int64_t b00, int64_t batch,
                                                      const float *__restrict__ weight, int wpb, float scale)
{
    constexpr int NS = d2_tile(CC);
    __shared__ float2 s[CC == 1 ? 1 : NS][CC + 1];
    const int64_t i0 = blockIdx.x * (int64_t)NS, b0 = b00 + (int64_t)blockIdx.y * g.CS;
    const int n = (int)min((int64_t)NS, g.total - i0), cact = (int)min((int64_t)g.CS, batch - b0);
    const int c = threadIdx.x % CC;
    const float2 *gc = grid + blockIdx.y * g.npts * g.CS + c;
    float2 acc = make_float2(0.0f, 0.0f);
    for (int r = threadIdx.x / CC; r < n; r += 256 / CC) {
        if (c >= cact) continue;
        const int64_t i = i0 + r;
        const Taps<W> t(g, rec + i * d2_rec(W), __ldg(base + i));
        float2 v[W][W];
#pragma unroll
        for (int jy = 0; jy < W; jy++)
#pragma unroll
            for (int jx = 0; jx < W; jx++) v[jy][jx] = __ldg(gc + t.yo[jy] + t.xo[jx]);
        acc = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int jy = 0; jy < W; jy++) {
            float2 q = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int jx = 0; jx < W; jx++) {
                q.x = fmaf(t.w[jx], v[jy][jx].x, q.x);
                q.y = fmaf(t.w[jx], v[jy][jx].y, q.y);
            }
            acc.x = fmaf(t.w[W + jy], q.x, acc.x);
            acc.y = fmaf(t.w[W + jy], q.y, acc.y);
        }
        if (CC > 1) s[r][c] = acc;
    }
    if (CC > 1) __syncthreads();
    for (int e = threadIdx.x; e < NS * CC; e += 256) {
        const int cc = e / NS, t = e % NS;
        if (cc >= cact || t >= n) continue;
        const int64_t o = (b0 + cc) * g.total + i0 + t;
        float w = scale;
        if (weight) w *= weight[wpb ? o : i0 + t];
        const float2 x = CC == 1 ? acc : s[t][cc];
        ksp[o] = make_float2(x.x * w, x.y * w);
    }
}

// sparse gridding: every tap of every sample added to the (zeroed) grid, 8 B
// per lane, coils contiguous
template <int W, int CC>
__global__ void __launch_bounds__(256) grid2_kernel(D2Geom g, const float *__restrict__ rec,
                                                    const int2 *__restrict__ base, const void *__restrict__ ksp,
                                                    int kreal, float2 *__restrict__ grid, int64_t b00, int64_t batch,
                                                    const float *__restrict__ weight, int wpb, float scale)
{
    constexpr int NS = d2_tile(CC);
    __shared__ float2 s[NS][CC + 1];
    const int64_t i0 = blockIdx.x * (int64_t)NS, b0 = b00 + (int64_t)blockIdx.y * g.CS;
    const int n = (int)min((int64_t)NS, g.total - i0), cact = (int)min((int64_t)g.CS, batch - b0);
    for (int e = threadIdx.x; e < NS * CC; e += 256) {
        const int cc = e / NS, t = e % NS;
        if (cc >= cact || t >= n) continue;
        const int64_t o = (b0 + cc) * g.total + i0 + t;
        float2 v = make_float2(0.0f, 0.0f);
        if (kreal) v.x = reinterpret_cast<const float *>(ksp)[o];
        else v = reinterpret_cast<const float2 *>(ksp)[o];
        const float w = weight ? weight[wpb ? o : i0 + t] : 1.0f;
        s[t][cc] = make_float2(v.x * w * scale, v.y * w * scale);
    }
    __syncthreads();
    const int c = threadIdx.x % CC;
    if (c >= cact) return;
    float2 *gc = grid + blockIdx.y * g.npts * g.CS + c;
    for (int r = threadIdx.x / CC; r < n; r += 256 / CC) {
        const int64_t i = i0 + r;
        const Taps<W> t(g, rec + i * d2_rec(W), __ldg(base + i));
        const float2 v = s[r][c];
#pragma unroll
        for (int jy = 0; jy < W; jy++) {
            const float2 u = make_float2(t.w[W + jy] * v.x, t.w[W + jy] * v.y);
#pragma unroll
            for (int jx = 0; jx < W; jx++)
                atomicAdd(gc + t.yo[jy] + t.xo[jx], make_float2(t.w[jx] * u.x, t.w[jx] * u.y));
        }
    }
}

// Trajectory gradient (gradient.cu): out[i, a] = post * sum_b Re(conj(v_b[i])
// dy_b[i] / dcoord[i, a]) over coils b0 .. of `nch` interleaved chunks.
// The block evaluates its samples' tap weights and their derivatives once; lane
// = (sample, coil) sums its coil's taps, coils are added with shuffles.
struct D2Grad {
    float beta[2], inv_hw[2], rs[2];
};

template <int W, int CC>
__global__ void __launch_bounds__(256) grad2_kernel(D2Geom g, D2Grad gr, const float *__restrict__ rk0,
                                                    const float *__restrict__ rk1, const float *__restrict__ rec,
                                                    const int2 *__restrict__ base, const float2 *__restrict__ grid,
                                                    const float2 *__restrict__ v, int64_t batch, int64_t nch,
                                                    const float *__restrict__ weight, int wpb, float scale, float post,
                                                    int64_t b00, float *__restrict__ out)
{
    constexpr int NS = d2_tile(CC), GS = CC;  // samples per block, lanes per sample
    __shared__ float2 s[NS][CC + 1];
    __shared__ float dw[NS][2 * W + 1];
    const int64_t i0 = blockIdx.x * (int64_t)NS;
    const int n = (int)min((int64_t)NS, g.total - i0);
    for (int e = threadIdx.x; e < 2 * W * NS; e += 256) {
        const int t = e / (2 * W), q = e - t * (2 * W), a = q / W, k = q - a * W;
        if (t >= n) continue;
        const float c = a ? rk1[i0 + t] : rk0[i0 + t];
        const int x0 = first_tap_dev(c, W);
        const float u = (float)(((double)(x0 + k) - (double)c) * (2.0 / W));
        float d;
        kb_and_derivative(u, gr.beta[a], &d);
        dw[t][q] = d * -gr.inv_hw[a] * gr.rs[a];
    }
    const int c = threadIdx.x % CC;
    constexpr int K = (NS * CC + 255) / 256;  // samples of this lane
    float acc[K][2];
#pragma unroll
    for (int k = 0; k < K; k++) acc[k][0] = acc[k][1] = 0.0f;
    for (int64_t ch = 0; ch < nch; ch++) {
        const int64_t b0 = b00 + ch * g.CS;
        const int cact = (int)min((int64_t)g.CS, batch - b0);
        __syncthreads();
        for (int e = threadIdx.x; e < NS * CC; e += 256) {
            const int cc = e / NS, t = e % NS;
            if (cc >= cact || t >= n) continue;
            const int64_t o = (b0 + cc) * g.total + i0 + t;
            const float2 x = v[o];
            float w = scale;
            if (weight) w *= weight[wpb ? o : i0 + t];
            s[t][cc] = make_float2(x.x * w, x.y * w);
        }
        __syncthreads();
        const float2 *gc = grid + ch * g.npts * g.CS + c;
#pragma unroll
        for (int k = 0; k < K; k++) {
            const int r = threadIdx.x / CC + k * (256 / CC);
            if (r >= n || c >= cact) continue;
            const Taps<W> t(g, rec + (i0 + r) * d2_rec(W), __ldg(base + i0 + r));
            float2 dx = make_float2(0.0f, 0.0f), dy = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int jy = 0; jy < W; jy++) {
                float2 q = make_float2(0.0f, 0.0f), qd = make_float2(0.0f, 0.0f);
#pragma unroll
                for (int jx = 0; jx < W; jx++) {
                    const float2 x = __ldg(gc + t.yo[jy] + t.xo[jx]);
                    q.x = fmaf(t.w[jx], x.x, q.x);
                    q.y = fmaf(t.w[jx], x.y, q.y);
                    qd.x = fmaf(dw[r][jx], x.x, qd.x);
                    qd.y = fmaf(dw[r][jx], x.y, qd.y);
                }
                dx.x = fmaf(t.w[W + jy], qd.x, dx.x);
                dx.y = fmaf(t.w[W + jy], qd.y, dx.y);
                dy.x = fmaf(dw[r][W + jy], q.x, dy.x);
                dy.y = fmaf(dw[r][W + jy], q.y, dy.y);
            }
            const float2 vb = s[r][c];
            acc[k][0] += vb.x * dx.x + vb.y * dx.y;  // Re(conj(v) D)
            acc[k][1] += vb.x * dy.x + vb.y * dy.y;
        }
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
        const int r = threadIdx.x / CC + k * (256 / CC);
#pragma unroll
        for (int d = 1; d < GS; d <<= 1) {
            acc[k][0] += __shfl_xor_sync(0xffffffffu, acc[k][0], d);
            acc[k][1] += __shfl_xor_sync(0xffffffffu, acc[k][1], d);
        }
        if (r < n && c == 0) {
            // (chunks given one call at a time add to the first one's)
            float *o = out + (i0 + r) * 2;
            o[0] = (b00 ? o[0] : 0.0f) + acc[k][0] * post;
            o[1] = (b00 ? o[1] : 0.0f) + acc[k][1] * post;
        }
    }
}

D2Geom d2_geom(const dmr_plan *p, int CS)
{
    D2Geom g;
    g.G0 = p->g.G[0];
    g.G1 = p->g.G[1];
    g.CS = CS;
    g.gsize = p->g.gsize;
    g.npts = (int64_t)p->g.nframes * p->g.gsize;
    g.total = p->g.total;
    return g;
}

template <int W, int CC>
int launch_interp2(const dmr_plan *p, const D2Geom &g, const float2 *grid, float2 *ksp, int64_t b0, int64_t nch,
                   int64_t batch, const float *weight, int wpb, cudaStream_t st)
{
    interp2_kernel<W, CC><<<dim3((unsigned)ceil_div(g.total, d2_tile(CC)), (unsigned)nch), 256, 0, st>>>(
        g, p->d2_rec, (const int2 *)p->d2_base, grid, ksp, b0, batch, weight, wpb, (float)(1.0 / p->scale));
    DMR_LAUNCHED("interp2_kernel");
    return DMR_OK;
}

template <int W, int CC>
int launch_grid2(const dmr_plan *p, const D2Geom &g, const void *ksp, int kreal, float2 *grid, int64_t b0, int64_t nch,
                 int64_t batch, const float *weight, int wpb, cudaStream_t st)
{
    grid2_kernel<W, CC><<<dim3((unsigned)ceil_div(g.total, d2_tile(CC)), (unsigned)nch), 256, 0, st>>>(
        g, p->d2_rec, (const int2 *)p->d2_base, ksp, kreal, grid, b0, batch, weight, wpb, (float)(1.0 / p->scale));
    DMR_LAUNCHED("grid2_kernel");
    return DMR_OK;
}

template <int W, int CC>
int launch_grad2(const dmr_plan *p, const D2Geom &g, const float2 *grid, const float2 *v, int64_t b0, int64_t nch,
                 int64_t batch,
                 const float *weight, int wpb, float post, float *out, cudaStream_t st)
{
    D2Grad gr;
    for (int a = 0; a < 2; a++) {
        gr.beta[a] = p->g.beta[a];
        gr.inv_hw[a] = (float)p->g.inv_hw[a];
        gr.rs[a] = std::ceil(p->os[a] * (float)p->g.N[a]) / (float)p->g.N[a];
    }
    grad2_kernel<W, CC><<<(unsigned)ceil_div(g.total, d2_tile(CC)), 256, 0, st>>>(
        g, gr, p->rk[0], p->rk[1], p->d2_rec, (const int2 *)p->d2_base, grid, v, batch, nch, weight, wpb,
        (float)(1.0 / p->scale), post, b0, out);
    DMR_LAUNCHED("grad2_kernel");
    return DMR_OK;
}

// coil lanes: the smallest power of two that covers the chunk
#define DMR_D2_CC(F, W, CS, ...)                                                   \
    return CS > 16  ? F<W, 32>(__VA_ARGS__)                                        \
           : CS > 8 ? F<W, 16>(__VA_ARGS__)                                        \
           : CS > 4 ? F<W, 8>(__VA_ARGS__)                                         \
           : CS > 2 ? F<W, 4>(__VA_ARGS__) : CS > 1 ? F<W, 2>(__VA_ARGS__) : F<W, 1>(__VA_ARGS__)
#define DMR_D2(F, CS, ...)                                   \
    switch (p->d2_W) {                                       \
    case 2: DMR_D2_CC(F, 2, CS, __VA_ARGS__);                \
    case 3: DMR_D2_CC(F, 3, CS, __VA_ARGS__);                \
    case 4: DMR_D2_CC(F, 4, CS, __VA_ARGS__);                \
    case 5: DMR_D2_CC(F, 5, CS, __VA_ARGS__);                \
    case 6: DMR_D2_CC(F, 6, CS, __VA_ARGS__);                \
    default: return DMR_ERR_UNSUPPORTED;                     \
    }

}  // namespace

int d2_build(dmr_plan *p, float *const rk[3], cudaStream_t st)
{
    const Geom &g = p->g;
    const int W = g.W[0];
    if (g.ndim != 2 || g.total == 0 || W < 2 || W > 6 || g.W[1] != W) return DMR_OK;
    // a record holds its first tap as x | y << 16, y in the upper half of a
    // signed int: longer grids keep the bin kernels
    if (g.G[0] > 65536 || g.G[1] > 32768) return DMR_OK;
    DMR_TRY(plan_alloc(p->device, &p->d2_rec, (size_t)g.total * d2_rec(W), st));
    int2 *base = nullptr;
    DMR_TRY(plan_alloc(p->device, &base, g.total, st));
    p->d2_base = base;
    const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(g.total, 256), 148 * 16);
    d2_rec_kernel<<<blocks, 256, 0, st>>>(g, p->foff_dev, rk[0], rk[1], p->d2_rec, base);
    DMR_LAUNCHED("d2_rec_kernel");
    p->d2_W = W;
    return DMR_OK;
}

int d2_interp(const dmr_plan *p, const float2 *grid, float2 *ksp, int64_t b0, int64_t nch, int CS, int64_t batch,
              const float *weight, int wpb, cudaStream_t st)
{
    const D2Geom g = d2_geom(p, CS);
    DMR_D2(launch_interp2, CS, p, g, grid, ksp, b0, nch, batch, weight, wpb, st)
}

int d2_grid(const dmr_plan *p, const void *ksp, int kreal, float2 *grid, int64_t b0, int64_t nch, int CS,
            int64_t batch, const float *weight, int wpb, cudaStream_t st)
{
    const D2Geom g = d2_geom(p, CS);
    DMR_D2(launch_grid2, CS, p, g, ksp, kreal, grid, b0, nch, batch, weight, wpb, st)
}

int d2_grad(const dmr_plan *p, const float2 *grid, const float2 *v, int64_t b0, int64_t nch, int CS, int64_t batch,
            const float *weight, int wpb, float post, float *out, cudaStream_t st)
{
    const D2Geom g = d2_geom(p, CS);
    DMR_D2(launch_grad2, CS, p, g, grid, v, b0, nch, batch, weight, wpb, post, out, st)
}

}  // namespace dmr
