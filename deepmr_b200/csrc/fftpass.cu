// Host side of the FFT passes (fftpass.cuh): the compiled lengths, twiddle tables,
// launches, and the transforms of the NUFFT and Toeplitz pipelines.
#include <cmath>
#include <map>
#include <mutex>
#include <vector>

#include "fftpass.cuh"

namespace dmr {

using namespace fftp;

namespace {

// the lengths with a compiled transform (grid extents of common matrix sizes
// at oversampling 1.25 and 2), as (L, L1, L2); other lengths run with
// their factors at run time (any_factors) or through cuFFT. The
// smaller factor first: more threads wait for fewer loads each in step A, and no
// warp is idle there (rows forward, 280 = 14 x 20, 500 x 16 images of 224^2:
// 1.98 ms with 20 first, 1.53 with 14; columns 1.73 and 1.60). The cropping row
// pass is the other way round (1.40 ms, 1.56; its stores are the scattered side)
#define DMR_FFT_LENGTHS(X)                                                                            \
    X(32, 4, 8) X(40, 5, 8) X(48, 3, 16) X(56, 7, 8) X(64, 8, 8) X(80, 5, 16) X(96, 6, 16)              \
    X(112, 7, 16) X(120, 10, 12) X(128, 8, 16) X(140, 7, 20) X(144, 12, 12) X(160, 10, 16)               \
    X(168, 12, 14) X(192, 12, 16) X(200, 10, 20) X(224, 14, 16) X(240, 15, 16) X(256, 16, 16)            \
    X(280, 14, 20) X(288, 16, 18) X(320, 16, 20) X(336, 14, 24) X(384, 16, 24) X(400, 20, 20)            \
    X(480, 20, 24) X(512, 16, 32) X(640, 20, 32)

// the factors of a length, smaller first, as near to each other as they can be;
// L == 0: none (a prime factor above 23, no two factors up to 26, or below 32
// points, where a block of 16 lines has a warp or two)
Fac any_factors(int L)
{
    Fac f;
    if (L < 32) return f;
    for (int a = 2; a * a <= L; a++)
        if (L % a == 0 && L / a <= kGenMax) f = Fac{L, a, L / a};
    return f;
}

bool has_len(int L)
{
    switch (L) {
#define DMR_FFT_CASE(L, L1, L2) case L: return true;
        DMR_FFT_LENGTHS(DMR_FFT_CASE)
#undef DMR_FFT_CASE
    default: return any_factors(L).L != 0;
    }
}

// per-device twiddle tables of a length: entry k1 L2 + n2 is
// exp(-2 pi i n2 k1 / L), from double precision; then the same with the factors
// exchanged, for the cropping row pass (`crop`). Both are uploaded at once, on a
// stream of their own, so that a call can be captured whatever ran before it
std::mutex g_tw_mu;
std::map<std::pair<int, int>, float2 *> g_tw;

int second_factor(int L, bool crop)
{
    switch (L) {
#define DMR_FFT_CASE(L, L1, L2) case L: return crop ? L1 : L2;
        DMR_FFT_LENGTHS(DMR_FFT_CASE)
#undef DMR_FFT_CASE
    default: return crop ? any_factors(L).L1 : any_factors(L).L2;
    }
}

int twiddles(int L, bool crop, const float2 **out)
{
    int dev = 0;
    DMR_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_tw_mu);
    float2 *&d = g_tw[{dev, L}];
    if (!d) {
        std::vector<float2> h(2 * L);
        const double two_pi = 6.283185307179586476925286766559;
        for (int t = 0; t < 2 * L; t++) {
            const int L2 = second_factor(L, t >= L), e = t % L;
            const double ang = two_pi * (double)((e / L2) * (e % L2)) / (double)L;
            h[t] = make_float2((float)std::cos(ang), (float)-std::sin(ang));
        }
        const Uncaptured mode;
        cudaStream_t st = nullptr;
        float2 *p = nullptr;
        DMR_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        cudaError_t e = cudaMalloc(&p, h.size() * sizeof(float2));
        if (e == cudaSuccess) e = cudaMemcpyAsync(p, h.data(), h.size() * sizeof(float2), cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        cudaStreamDestroy(st);
        if (e != cudaSuccess) {
            if (p) cudaFree(p);
            return cuda_fail(e, "twiddle table", __FILE__, __LINE__);
        }
        d = p;
    }
    *out = d + (crop ? L : 0);
    return DMR_OK;
}

int fft_disabled()
{
    static const int v = [] {
        const char *e = getenv("DMR_CUFFT");
        return e && atoi(e) ? 1 : 0;
    }();
    return v;
}

// the forward passes read part of each line and write all of it, the
// adjoint passes the other way round
int launch_cols(int L, const FftGeom &g, const ColArgs &a, const float2 *tw, float2 *grid, cudaStream_t st)
{
    switch (L) {
#define DMR_FFT_CASE(L, L1, L2)                                                                                        \
    case L: {                                                                                                          \
        using F = Len<L, L1, L2>;                                                                                      \
        return a.inv ? launch_cols_k(fft_cols_kernel<F, true, false, true>, L, F::T, g, a, tw, grid, st)               \
                     : launch_cols_k(fft_cols_kernel<F, false, true, false>, L, F::T, g, a, tw, grid, st);             \
    }
        DMR_FFT_LENGTHS(DMR_FFT_CASE)
#undef DMR_FFT_CASE
    default: break;
    }
    const Fac f = any_factors(L);
    return f.L ? launch_cols_any(f, g, a, tw, grid, st) : DMR_ERR_UNSUPPORTED;
}

template <bool CROP, bool IL>
int launch_rows_c(int L, const FftGeom &g, const float2 *tw, const void *src, int src_real, float2 *dst, cudaStream_t st)
{
    switch (L) {
#define DMR_FFT_CASE(L, L1, L2)                                                                                          \
    case L: {                                                                                                            \
        constexpr int A = CROP ? L2 : L1, B = CROP ? L1 : L2;                                                            \
        return launch_rows_k<CROP, IL>(fft_rows_kernel<Len<L, A, B>, CROP, IL>, A, B, g, tw, src, src_real, dst, st);     \
    }
        DMR_FFT_LENGTHS(DMR_FFT_CASE)
#undef DMR_FFT_CASE
    default: break;
    }
    const Fac f = any_factors(L);
    return f.L ? launch_rows_any<CROP, IL>(f, g, tw, src, src_real, dst, st) : DMR_ERR_UNSUPPORTED;
}

template <bool IL = false>
int launch_rows(int L, bool crop, const FftGeom &g, const float2 *tw, const void *src, int src_real, float2 *dst,
                cudaStream_t st)
{
    return crop ? launch_rows_c<true, IL>(L, g, tw, src, src_real, dst, st)
                : launch_rows_c<false, IL>(L, g, tw, src, src_real, dst, st);
}

int launch_toep_z(int L, const FftGeom &g, const ColArgs &a, int64_t nk, const float2 *kern, float kscale,
                  const float2 *tw, float2 *grid, cudaStream_t st)
{
    switch (L) {
#define DMR_FFT_CASE(L, L1, L2)                                                                                          \
    case L: return launch_toep_k(fft_toep_z_kernel<Len<L, L1, L2>>, L, Len<L, L1, L2>::T, g, a, nk, kern, kscale, tw, grid, st);
        DMR_FFT_LENGTHS(DMR_FFT_CASE)
#undef DMR_FFT_CASE
    default: break;
    }
    const Fac f = any_factors(L);
    return f.L ? launch_toep_any(f, g, a, nk, kern, kscale, tw, grid, st) : DMR_ERR_UNSUPPORTED;
}

FftGeom make_geom(const dmr_plan *p, int64_t batch, int64_t nframes, float scale)
{
    const Geom &gg = p->g;
    FftGeom g;
    for (int a = 0; a < 3; a++) {
        g.N[a] = gg.N[a];
        g.G[a] = gg.G[a];
        g.apod[a] = gg.W[a] != 1 ? p->apod[a] : nullptr;
        g.off[a] = -(gg.N[a] / 2);  // FFT order: centred index N/2 at 0
    }
    g.nbf = batch * nframes;
    g.gsize = gg.gsize;
    g.isize = gg.isize;
    g.scale = scale;
    return g;
}

void set_ranges(ColArgs &a, int L)
{
    a.in = range(a.in_q0, a.in_n, L);
    a.out = range(a.out_q0, a.out_n, L);
}

ColArgs y_pass(const FftGeom &g, bool inv)
{
    // y columns of the N2 planes that hold data; the forward reads the N1
    // valid y only, the adjoint writes the N1 kept y only
    ColArgs a;
    a.S = g.G[0];
    a.outer_stride = (int64_t)g.G[0] * g.G[1];
    a.nouter = g.N[2];
    a.outer_q0 = wrapi(g.off[2], g.G[2]);
    a.outer_G = g.G[2];
    const int q0 = wrapi(g.off[1], g.G[1]);
    a.in_q0 = inv ? 0 : q0;
    a.in_n = inv ? g.G[1] : g.N[1];
    a.out_q0 = inv ? q0 : 0;
    a.out_n = inv ? g.N[1] : g.G[1];
    a.inv = inv;
    set_ranges(a, g.G[1]);
    return a;
}

ColArgs z_pass(const FftGeom &g, bool inv)
{
    // z columns of every (y, x); the forward reads the N2 valid z only, the
    // adjoint writes the N2 kept z only
    ColArgs a;
    a.S = (int64_t)g.G[0] * g.G[1];
    a.outer_stride = g.G[0];
    a.nouter = g.G[1];
    a.outer_q0 = 0;
    a.outer_G = g.G[1];
    const int q0 = wrapi(g.off[2], g.G[2]);
    a.in_q0 = inv ? 0 : q0;
    a.in_n = inv ? g.G[2] : g.N[2];
    a.out_q0 = inv ? q0 : 0;
    a.out_n = inv ? g.N[2] : g.G[2];
    a.inv = inv;
    set_ranges(a, g.G[2]);
    return a;
}

}  // namespace

bool fft3_applies(const dmr_plan *p)
{
    const Geom &g = p->g;
    if (fft_disabled() || (g.ndim != 2 && g.ndim != 3)) return false;
    for (int a = 0; a < g.ndim; a++)
        if (g.G[a] < g.N[a] || !has_len(g.G[a])) return false;
    return true;
}

// apodise + zero-pad + forward 3D FFT of `image` into `grid` (FFT order)
int fft3_forward(const dmr_plan *p, const void *image, int image_real, int64_t batch, int64_t nframes, float2 *grid,
                 cudaStream_t st)
{
    const FftGeom g = make_geom(p, batch, nframes, 1.0f);
    const float2 *tw[3] = {nullptr, nullptr, nullptr};
    for (int a = 0; a < p->g.ndim; a++) DMR_TRY(twiddles(g.G[a], false, &tw[a]));
    if (g.nbf == 0) return DMR_OK;
    DMR_TRY(launch_rows(g.G[0], false, g, tw[0], image, image_real, grid, st));
    DMR_TRY(launch_cols(g.G[1], g, y_pass(g, false), tw[1], grid, st));
    if (g.G[2] == 1) return DMR_OK;  // 2D
    return launch_cols(g.G[2], g, z_pass(g, false), tw[2], grid, st);
}

// inverse 3D FFT of `grid` (FFT order, overwritten) + crop + 1/G + apodisation into `image`
int fft3_adjoint(const dmr_plan *p, float2 *grid, int64_t batch, int64_t nframes, float2 *image, cudaStream_t st)
{
    const FftGeom g = make_geom(p, batch, nframes, (float)(1.0 / (double)p->g.gsize));
    const float2 *tw[3] = {nullptr, nullptr, nullptr};
    for (int a = 0; a < p->g.ndim; a++) DMR_TRY(twiddles(g.G[a], a == 0, &tw[a]));
    if (g.nbf == 0) return DMR_OK;
    if (g.G[2] > 1) DMR_TRY(launch_cols(g.G[2], g, z_pass(g, true), tw[2], grid, st));
    DMR_TRY(launch_cols(g.G[1], g, y_pass(g, true), tw[1], grid, st));
    return launch_rows(g.G[0], true, g, tw[0], grid, 0, image, st);
}

namespace {

// geometry of the column passes on an interleaved grid: x and coil are one
// contiguous axis
FftGeom il_cols(const FftGeom &g)
{
    FftGeom c = g;
    c.G[0] *= g.CS;
    c.gsize *= g.CS;
    return c;
}

FftGeom il_geom(const dmr_plan *p, int64_t batch, int64_t nframes, int64_t nchunks, int CS, float scale)
{
    FftGeom g = make_geom(p, nchunks, nframes, scale);  // nbf: (chunk, frame) sets
    g.CS = CS;
    g.nframes = (int)nframes;
    g.batch = batch;
    return g;
}

}  // namespace

int fft3_forward_il(const dmr_plan *p, const void *image, int image_real, int64_t batch, int64_t nframes,
                    int64_t nchunks, int CS, float2 *grid, cudaStream_t st)
{
    if (CS == 1) return fft3_forward(p, image, image_real, batch, nframes, grid, st);  // the same layout
    const FftGeom g = il_geom(p, batch, nframes, nchunks, CS, 1.0f), c = il_cols(g);
    const float2 *tw[3] = {nullptr, nullptr, nullptr};
    for (int a = 0; a < p->g.ndim; a++) DMR_TRY(twiddles(g.G[a], false, &tw[a]));
    DMR_TRY(launch_rows<true>(g.G[0], false, g, tw[0], image, image_real, grid, st));
    DMR_TRY(launch_cols(g.G[1], c, y_pass(c, false), tw[1], grid, st));
    if (g.G[2] == 1) return DMR_OK;  // 2D
    return launch_cols(g.G[2], c, z_pass(c, false), tw[2], grid, st);
}

int fft3_adjoint_il(const dmr_plan *p, float2 *grid, int64_t batch, int64_t nframes, int64_t nchunks, int CS,
                    float2 *image, cudaStream_t st)
{
    if (CS == 1) return fft3_adjoint(p, grid, batch, nframes, image, st);
    const FftGeom g = il_geom(p, batch, nframes, nchunks, CS, (float)(1.0 / (double)p->g.gsize)), c = il_cols(g);
    const float2 *tw[3] = {nullptr, nullptr, nullptr};
    for (int a = 0; a < p->g.ndim; a++) DMR_TRY(twiddles(g.G[a], a == 0, &tw[a]));
    if (g.G[2] > 1) DMR_TRY(launch_cols(g.G[2], c, z_pass(c, true), tw[2], grid, st));
    DMR_TRY(launch_cols(g.G[1], c, y_pass(c, true), tw[1], grid, st));
    return launch_rows<true>(g.G[0], true, g, tw[0], grid, 0, image, st);
}

bool toep3_applies(int ndim, const int32_t *kshape, const int32_t *ishape)
{
    if (fft_disabled() || (ndim != 2 && ndim != 3) || !kshape || !ishape) return false;
    for (int a = 0; a < ndim; a++)
        if (kshape[a] < ishape[a] || !has_len(kshape[a])) return false;
    return true;
}

size_t toep_extra_bytes(int ndim, const int32_t *kshape, size_t data_bytes, size_t work_bytes)
{
    size_t b = align_up(work_bytes, 256);
    if (toep3_applies(ndim, kshape, kshape)) b = std::max(b, align_up(data_bytes / 4, 256));
    return b;
}

// Toeplitz self-adjoint of a 3D image batch (src/deepmr/fft/nufft.py:609-669,
// _interp/toeplitz.py:84-87): zero-pad to the kernel grid (resize offsets
// K/2 - N/2, no shift), FFT, times kernel[b mod nk] / K (the two orthonormal
// 1/sqrt(K)), inverse FFT, crop; `data` is a workspace of batch kernel grids.
int fft3_toeplitz(int ndim, const int32_t *kshape_zyx, const int32_t *ishape_zyx, const float2 *kernel, int64_t nk,
                  const void *image, int image_real, float2 *out, int64_t batch, float2 *data, cudaStream_t st)
{
    FftGeom g;
    g.gsize = g.isize = 1;
    for (int a = 0; a < 3; a++) {
        g.G[a] = a < ndim ? kshape_zyx[ndim - 1 - a] : 1;
        g.N[a] = a < ndim ? ishape_zyx[ndim - 1 - a] : 1;
        g.off[a] = g.G[a] / 2 - g.N[a] / 2;
        g.apod[a] = nullptr;
        g.gsize *= g.G[a];
        g.isize *= g.N[a];
    }
    g.nbf = batch;
    g.scale = 1.0f;
    const float2 *tw[3] = {nullptr, nullptr, nullptr}, *twc = nullptr;
    for (int a = 0; a < ndim; a++) DMR_TRY(twiddles(g.G[a], false, &tw[a]));
    DMR_TRY(twiddles(g.G[0], true, &twc));
    if (batch == 0) return DMR_OK;
    const float kscale = (float)(1.0 / (double)g.gsize);
    DMR_TRY(launch_rows(g.G[0], false, g, tw[0], image, image_real, data, st));
    if (ndim == 2) {
        // the y pass is the fused one: its lines with data in, kept lines out
        ColArgs y = y_pass(g, false);
        y.out_q0 = y.in_q0;
        y.out_n = y.in_n;
        set_ranges(y, g.G[1]);
        DMR_TRY(launch_toep_z(g.G[1], g, y, nk, kernel, kscale, tw[1], data, st));
    } else {
        DMR_TRY(launch_cols(g.G[1], g, y_pass(g, false), tw[1], data, st));
        ColArgs z = z_pass(g, false);
        z.out_q0 = z.in_q0;
        z.out_n = z.in_n;  // only the kept z leave the fused transform
        set_ranges(z, g.G[2]);
        DMR_TRY(launch_toep_z(g.G[2], g, z, nk, kernel, kscale, tw[2], data, st));
        DMR_TRY(launch_cols(g.G[1], g, y_pass(g, true), tw[1], data, st));
    }
    return launch_rows(g.G[0], true, g, twc, data, 0, out, st);
}

}  // namespace dmr

extern "C" int dmr_fft3_fused(dmr_plan *plan) { return plan && dmr::fft3_applies(plan) ? 1 : 0; }
