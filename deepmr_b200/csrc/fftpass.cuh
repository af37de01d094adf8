// 3D FFT passes of the NUFFT pipelines, fused with the zero-padding /
// cropping and the apodisation, and pruned to the lines that hold data.
//
// The forward NUFFT (src/deepmr/fft/nufft.py:450-528) apodises the image,
// zero-pads it to the oversampled grid (src/deepmr/_signal/resize.py:11-102),
// and takes a centred FFT (src/deepmr/fft/fft.py:9-87); the adjoint
// (nufft.py:531-606) takes a centred inverse FFT (norm "backward", 1/G), crops
// and apodises. The grid lives in FFT order (centred index c at
// (c - G//2) mod G), so image index i of an axis sits at grid index
// (i - N//2) mod G, and only N of the G positions of an axis hold image data.
// A 3D transform is three passes of 1D transforms, and each pass touches only
// the lines that matter:
//   forward: x rows of the N1*N2 image rows (reading the image, apodising and
//   padding on the fly), y columns of the N2 planes with data (reading only
//   the N1 valid y), z columns everywhere (reading only the N2 valid z);
//   adjoint: z columns everywhere (writing only the N2 kept z), y columns of
//   the N2 kept planes (writing only the N1 kept y), x rows of the N1*N2 kept
//   rows (writing the cropped, scaled, apodised image directly).
// With G = 1.25 N that is 15.5 GB of DRAM traffic per 240^3 x 32 transform
// against 26.6 GB for a full-grid pad kernel plus three full passes.
//
// Each block transforms 16 lines in two steps (the four-step form of the
// Cooley-Tukey algorithm, L = L1 L2): a thread takes L1 points of a line
// straight from global memory into registers, transforms and twiddles them,
// one exchange through shared memory, and L2 points per thread go from
// registers to global memory. Nothing is staged in shared memory before or
// after: with 16 lines of 8 bytes next to each other (columns, interleaved
// rows) a half-warp reads and writes 128 contiguous bytes, along image rows
// neighbouring threads take neighbouring points.
// What bounds these passes is DRAM, once there are few instructions and enough
// warps: 500 x 16 images of 224^2 to 280^2 and back take 1.53 + 1.60 ms and
// 1.55 + 1.40 ms, 4.7 to 5.6 TB/s; 192^3 x 32 coils 0.80 + 2.25 and 2.22 + 0.76.
// Tiles staged by asynchronous copies, roots of unity read from shared memory and
// a run-time direction took 93 instructions per point (now about 55) at 18 warps
// per SM: 2.44 + 2.08, 2.11 + 2.12, and 1.23 + 2.56, 2.52 + 1.07. So constants are
// immediates, co-prime factors of a register transform need no twiddles (Good, "The interaction
// algorithm and practical Fourier analysis", 1958), the direction is a template
// argument, and the twiddles between the steps are stored in the order in which
// they are used, in double precision rounded once.
#pragma once
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "plan.cuh"

namespace dmr {
namespace fftp {


// lines per block: 8 are as fast on small grids, but their 64-byte pieces cost a
// quarter on large ones (192^3, 32 coils, columns: 2.27 ms with 16, 2.96 with 8)
constexpr int kFftLines = 16;

__device__ __forceinline__ float2 cmulf(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// complex add / subtract as packed FP32 (one instruction each)
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
// a + s b and s b for a real constant s
__device__ __forceinline__ float2 axpy(float s, float2 b, float2 a)
{
    return make_float2(fmaf(s, b.x, a.x), fmaf(s, b.y, a.y));
}
__device__ __forceinline__ float2 scl(float s, float2 b) { return make_float2(s * b.x, s * b.y); }

// cos and sin of 2 pi t / n at compile time: the angle is brought to [0, pi/4]
// exactly (in eighths of a turn), then the power series in double precision
constexpr double series(double x, bool odd)
{
    double term = odd ? x : 1.0, sum = term;
    for (int k = odd ? 3 : 2; k < 26; k += 2) {
        term *= -x * x / ((double)k * (k - 1));
        sum += term;
    }
    return sum;
}
constexpr double cos_turn(int t, int n)  // 0 <= t < n
{
    if (2 * t > n) t = n - t;                              // cos(2 pi - a)
    if (4 * t > n) return -cos_turn(n - 2 * t, 2 * n);     // -cos(pi - a)
    const double x = 6.283185307179586476925286766559 / n;
    // above an eighth of a turn: sin(pi/2 - a), the complement as an exact fraction
    return 8 * t > n ? series((n - 4 * t) * (x / 4), true) : series(t * x, false);
}
constexpr double sin_turn(int t, int n)
{
    // sin a = cos(a - quarter turn), in quarters of 1/n
    int q = (4 * t - n) % (4 * n);
    if (q < 0) q += 4 * n;
    return cos_turn(q, 4 * n);
}
// exp(-+2 pi i t / n): forward (INV false) and inverse
template <int T, int N, bool INV>
struct Root {
    static constexpr float re = (float)cos_turn(T % N, N);
    static constexpr float im = (float)(INV ? sin_turn(T % N, N) : -sin_turn(T % N, N));
};
// v times exp(-+2 pi i T / N), without arithmetic for quarter turns
template <int T, int N, bool INV>
__device__ __forceinline__ float2 rot(float2 v)
{
    if constexpr (T % N == 0) {
        return v;
    } else if constexpr (4 * (T % N) == N) {
        return INV ? make_float2(-v.y, v.x) : make_float2(v.y, -v.x);
    } else if constexpr (2 * (T % N) == N) {
        return make_float2(-v.x, -v.y);
    } else if constexpr (4 * (T % N) == 3 * N) {
        return INV ? make_float2(v.y, -v.x) : make_float2(-v.y, v.x);
    } else {
        constexpr float c = Root<T, N, INV>::re, s = Root<T, N, INV>::im;
        return make_float2(v.x * c - v.y * s, v.x * s + v.y * c);
    }
}

template <int... I, class Fn>
__device__ __forceinline__ void unroll_seq(std::integer_sequence<int, I...>, Fn &&fn)
{
    (fn(std::integral_constant<int, I>{}), ...);
}
template <int N, class Fn>
__device__ __forceinline__ void unroll(Fn &&fn)
{
    unroll_seq(std::make_integer_sequence<int, N>{}, fn);
}

// factors of a register transform: co-prime where there are any
template <int M>
struct Split {
    static constexpr int pow2 = M % 32 == 0 ? 32 : (M % 16 == 0 ? 16 : (M % 8 == 0 ? 8 : (M % 4 == 0 ? 4 : (M % 2 == 0 ? 2 : 1))));
    static constexpr int odd = M / pow2;
    static constexpr int A = odd > 1 && pow2 > 1 ? pow2 : (odd == 1 ? (M == 8 ? 2 : 4) : (M % 3 == 0 ? 3 : 5));
    static constexpr int B = M / A;
    static constexpr bool coprime = A % 2 != B % 2 && !(A % 3 == 0 && B % 3 == 0) && !(A % 5 == 0 && B % 5 == 0) ||
                                    (A == 3 && B % 3 != 0) || (A == 5 && B % 5 != 0);
};

// M-point DFT of registers v, natural order in and out. Odd prime lengths R:
// with a_k = v_k + v_(R-k), b_k = v_k - v_(R-k),
//   V_m, V_(R-m) = v0 + sum_k cos(k m) a_k -+ i sum_k sin(k m) b_k.
// M = A B co-prime: n = B n1 + A n2 and k = (k mod A, k mod B) separate the two
// (no twiddles); otherwise n = B n1 + n2, k = k1 + A k2 with twiddles w_M^(n2 k1).
// Every index is a compile-time constant once unrolled.
template <int M, bool INV>
__device__ __forceinline__ void reg_dft(float2 *v)
{
    if constexpr (M == 2) {
        const float2 a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if constexpr (M == 4) {
        const float2 s02 = cadd(v[0], v[2]), d02 = csub(v[0], v[2]);
        const float2 s13 = cadd(v[1], v[3]), jd = rot<1, 4, INV>(csub(v[1], v[3]));
        v[0] = cadd(s02, s13);
        v[1] = cadd(d02, jd);
        v[2] = csub(s02, s13);
        v[3] = csub(d02, jd);
    } else if constexpr (M == 3 || M == 5 || M == 7 || M == 11 || M == 13 || M == 17 || M == 19 || M == 23) {
        constexpr int H = M / 2;
        float2 a[H + 1], b[H + 1];
        const float2 v0 = v[0];
#pragma unroll
        for (int k = 1; k <= H; k++) {
            a[k] = cadd(v[k], v[M - k]);
            b[k] = csub(v[k], v[M - k]);
            v[0] = cadd(v[0], a[k]);
        }
        unroll<H>([&](auto mi) {
            constexpr int m = decltype(mi)::value + 1;
            float2 re = axpy(Root<m, M, INV>::re, a[1], v0), im = scl(Root<m, M, INV>::im, b[1]);
            // sums of five and more: two chains, added last (rounding)
            constexpr int SPLIT = M > 7 ? H / 2 : H;
            float2 re2 = make_float2(0.0f, 0.0f), im2 = re2;
            unroll<H - 1>([&](auto ki) {
                constexpr int k = decltype(ki)::value + 2;
                constexpr float c = Root<k * m, M, INV>::re, s = Root<k * m, M, INV>::im;
                if constexpr (k <= SPLIT) {
                    re = axpy(c, a[k], re);
                    im = axpy(s, b[k], im);
                } else if constexpr (k == SPLIT + 1) {
                    re2 = scl(c, a[k]);
                    im2 = scl(s, b[k]);
                } else {
                    re2 = axpy(c, a[k], re2);
                    im2 = axpy(s, b[k], im2);
                }
            });
            if constexpr (SPLIT < H) {
                re = cadd(re, re2);
                im = cadd(im, im2);
            }
            v[m] = make_float2(re.x - im.y, re.y + im.x);  // + i im
            v[M - m] = make_float2(re.x + im.y, re.y - im.x);
        });
    } else {
        constexpr int A = Split<M>::A, B = Split<M>::B;
        static_assert(A > 1 && B > 1 && A * B == M, "factors");
        float2 y[M];
        unroll<B>([&](auto bi) {
            constexpr int n2 = decltype(bi)::value;
            float2 a[A];
#pragma unroll
            for (int n1 = 0; n1 < A; n1++) a[n1] = v[Split<M>::coprime ? (B * n1 + A * n2) % M : B * n1 + n2];
            reg_dft<A, INV>(a);
            unroll<A>([&](auto ai) {
                constexpr int k1 = decltype(ai)::value;
                y[n2 * A + k1] = Split<M>::coprime ? a[k1] : rot<n2 * k1, M, INV>(a[k1]);
            });
        });
        unroll<A>([&](auto ai) {
            constexpr int k1 = decltype(ai)::value;
            float2 b[B];
#pragma unroll
            for (int n2 = 0; n2 < B; n2++) b[n2] = y[n2 * A + k1];
            reg_dft<B, INV>(b);
            if constexpr (!Split<M>::coprime) {
#pragma unroll
                for (int k2 = 0; k2 < B; k2++) v[k1 + A * k2] = b[k2];
            } else {
#pragma unroll
                for (int k = 0; k < M; k++)
                    if (k % A == k1) v[k] = b[k % B];
            }
        });
    }
}

// A transform length L = L1 L2 (both at most 32).
// Step A, one thread per (line, n2): the L1 points L2 n1 + n2, times w_L^(n2 k1)
// after the transform. Step B, one thread per (line, k1): the L2 values n2,
// which become the transform at k1 + L1 k2.
template <int L_, int L1_, int L2_>
struct Len {
    static constexpr int L = L_, L1 = L1_, L2 = L2_;
    static constexpr int MX = L1 > L2 ? L1 : L2;
    static constexpr int T = kFftLines * MX;
    // resident blocks that the registers are planned for, from registers a thread
    // would like; more warps beat a few spilled words (280 points, 500 x 16 images
    // forward: 3.13 ms at 64 registers, 3 blocks; 3.95 at 96, 2 blocks) up to 24
    // points a thread. The Toeplitz pass holds two transforms' values (288 points:
    // 0.73 ms at 3 blocks, 0.91 at 4)
    static constexpr int blocks(int regs) { return 65536 / (T * regs) > 0 ? 65536 / (T * regs) : 1; }
    static constexpr int MINB = blocks(MX > 24 ? 128 : 56), TOEP_MINB = blocks(MX > 24 ? 128 : 64);
    static_assert(L1 * L2 == L, "factors");
};

// v times the twiddle between the steps, conjugated for the inverse
template <bool INV>
__device__ __forceinline__ float2 twiddle(float2 v, float2 w)
{
    return INV ? make_float2(v.x * w.x + v.y * w.y, v.y * w.x - v.x * w.y)
               : make_float2(v.x * w.x - v.y * w.y, v.x * w.y + v.y * w.x);
}

// step A from registers (a[n1]) into the exchange buffer, rows k1 of pitch S1;
// `sm` points at (n2, line), tw at table entry n2
template <int L1, bool INV>
__device__ __forceinline__ void step_a(float2 *a, float2 *sm, int S1, const float2 *__restrict__ tw, int L2)
{
    reg_dft<L1, INV>(a);
    sm[0] = a[0];
#pragma unroll
    for (int k1 = 1; k1 < L1; k1++) sm[k1 * S1] = twiddle<INV>(a[k1], __ldg(tw + k1 * L2));
}

// step B from the exchange buffer (`sm` at row k1, line; positions of pitch S2) into registers
template <int L2, bool INV>
__device__ __forceinline__ void step_b(const float2 *sm, int S2, float2 *b)
{
#pragma unroll
    for (int n2 = 0; n2 < L2; n2++) b[n2] = sm[n2 * S2];
    reg_dft<L2, INV>(b);
}

// positions of a line that hold data: l < e1 or s2 <= l < e2 (a cyclic range)
struct Range {
    int e1, s2, e2;
    __device__ __forceinline__ bool has(int l) const { return l < e1 || (l >= s2 && l < e2); }
};

struct FftGeom {
    int N[3], G[3];       // image / grid extents (x, y, z)
    int off[3];           // image index i sits at grid position (i + off) mod G
    int64_t nbf;          // batch * frames
    int64_t gsize, isize; // points per grid / image
    const float *apod[3]; // per-axis apodisation by image index (nullptr: 1)
    float scale;
    // coil-interleaved grids (row passes with IL): the line set of a (chunk,
    // frame) is (z, y, coil), element stride CS; images stay (batch, frame, z, y, x)
    int CS = 1;
    int nframes = 1;
    int64_t batch = 0;
};

__host__ __device__ __forceinline__ int wrapi(int v, int n)
{
    v %= n;
    return v < 0 ? v + n : v;
}

// the cyclic range [q0, q0 + n) of a length-L line
inline Range range(int q0, int n, int L)
{
    return q0 + n > L ? Range{q0 + n - L, q0, L} : Range{0, q0, q0 + n};
}

// division of 0 <= v < 2^31 by a run-time constant
struct FastDiv {
    unsigned d, m, s;
    explicit FastDiv(unsigned d_ = 1) : d(d_), s(31)
    {
        while ((1ull << (s - 31)) < d) s++;
        m = (unsigned)(((1ull << s) + d - 1) / d);
    }
    __device__ __forceinline__ unsigned div(unsigned v) const { return (unsigned)(((unsigned long long)v * m) >> s); }
};

// Lines of a row pass: line `row` of set bf (a (batch, frame) grid; with IL a
// (chunk, frame) and line row % CS of image row row / CS).
struct RowArgs {
    FftGeom g;
    FastDiv cs, n1, nf;
    int nrows;   // lines of a set
    int64_t bf0; // first set of the launch
};

// image offset (-1: a coil past the batch), grid offset and, times the scale,
// the apodisation of a line
struct RowLine {
    int64_t img, grid;
    float s;
};

template <bool IL>
__device__ __forceinline__ RowLine row_line(const RowArgs &ra, int row)
{
    const FftGeom &g = ra.g;
    const int64_t bf = ra.bf0 + blockIdx.y;
    int coil = 0, rr = row;
    if (IL) {
        rr = ra.cs.div(row);
        coil = row - rr * g.CS;
    }
    const int z = ra.n1.div(rr), y = rr - z * g.N[1];
    int qy = y + g.off[1], qz = z + g.off[2];
    if (qy < 0) qy += g.G[1];
    if (qz < 0) qz += g.G[2];
    RowLine ln;
    ln.img = bf * g.isize + (int64_t)rr * g.N[0];
    ln.grid = bf * g.gsize + ((int64_t)qz * g.G[1] + qy) * g.G[0];
    if (IL) {
        const int64_t chunk = ra.nf.div((unsigned)bf), f = bf - chunk * g.nframes, b = chunk * g.CS + coil;
        ln.img = b < g.batch ? (b * g.nframes + f) * g.isize + (int64_t)rr * g.N[0] : -1;
        ln.grid = ln.grid * g.CS + coil;
    }
    ln.s = g.scale;
    if (g.apod[1]) ln.s *= g.apod[1][y];
    if (g.apod[2]) ln.s *= g.apod[2][z];
    return ln;
}

// Row passes (x), a block per 16 rows.
//   forward (CROP false): image rows (real or complex) are placed at their
//   FFT-order positions (zero elsewhere), apodised, transformed and written
//   as full grid rows;
//   adjoint (CROP true): grid rows are inverse-transformed and the kept x,
//   scaled and apodised, written to the image.
// With IL the lines are 16 neighbouring (row, coil) pairs and the grid is
// interleaved, so its accesses run along the lines; the image's along x.
//
// The two steps take the transform length and the other factor as arguments:
// constants in the kernels of compiled lengths, run-time numbers in the others.
template <bool CROP, bool IL>
struct RowShape {
    // lanes of step A / B along the points of a line (else across the lines)
    static constexpr bool XA = !(IL && CROP), XB = !(IL && !CROP);
    // pitches of the exchange buffer (row k1, position n2, line): the lanes of a
    // half-warp are neighbours when they write and an odd pitch apart when they
    // read across, so that they hit distinct banks
    int S1, S2, SC;
    __host__ __device__ constexpr explicit RowShape(int L2)
        : S1(XA ? kFftLines * (L2 | 1) : L2 * kFftLines), S2(XA ? 1 : kFftLines), SC(XA ? L2 | 1 : 1)
    {
        if (XB) S1 |= 1;
    }
};

template <int L1, bool CROP, bool IL>
__device__ __forceinline__ void rows_a(const RowArgs &ra, float2 *fsm, int L, int L2, const float2 *__restrict__ tw,
                                       const void *__restrict__ src, int src_real)
{
    constexpr bool XA = RowShape<CROP, IL>::XA;
    const RowShape<CROP, IL> S(L2);
    const FftGeom &g = ra.g;
    const int w = threadIdx.x, row0 = blockIdx.x * kFftLines;
    // grid position q holds image index (q + h0) mod L (when below N0)
    const int N0 = g.N[0], h0 = g.off[0] > 0 ? L - g.off[0] : -g.off[0];
    if (w >= kFftLines * L2) return;
    const int c = XA ? w / L2 : w % kFftLines, n2 = XA ? w - c * L2 : w / kFftLines;
    float2 a[L1];
#pragma unroll
    for (int n1 = 0; n1 < L1; n1++) a[n1] = make_float2(0.0f, 0.0f);
    if (row0 + c < ra.nrows) {
        const RowLine ln = row_line<IL>(ra, row0 + c);
        if (CROP) {
            const float2 *sp = reinterpret_cast<const float2 *>(src) + ln.grid + (int64_t)n2 * (IL ? g.CS : 1);
            const int step = IL ? L2 * g.CS : L2;
#pragma unroll
            for (int n1 = 0; n1 < L1; n1++) a[n1] = IL ? __ldcg(sp + (int64_t)step * n1) : sp[step * n1];
        } else if (ln.img >= 0) {
            const float *ap = g.apod[0];
            // image index of position L2 n1 + n2: i0 + L2 n1, less L after the wrap
            const int i0 = n2 + h0;
            if (src_real) {
                const float *sp = reinterpret_cast<const float *>(src) + ln.img;
#pragma unroll
                for (int n1 = 0; n1 < L1; n1++) {
                    const int i = i0 + L2 * n1 - (i0 + L2 * n1 >= L ? L : 0);
                    if (i < N0) a[n1].x = sp[i] * (ap ? ln.s * __ldg(ap + i) : ln.s);
                }
            } else {
                const float2 *sp = reinterpret_cast<const float2 *>(src) + ln.img;
#pragma unroll
                for (int n1 = 0; n1 < L1; n1++) {
                    const int i = i0 + L2 * n1 - (i0 + L2 * n1 >= L ? L : 0);
                    if (i < N0) a[n1] = sp[i];
                }
#pragma unroll
                for (int n1 = 0; n1 < L1; n1++) {
                    const int i = i0 + L2 * n1 - (i0 + L2 * n1 >= L ? L : 0);
                    if (i < N0) a[n1] = scl(ap ? ln.s * __ldg(ap + i) : ln.s, a[n1]);
                }
            }
        }
    }
    step_a<L1, CROP>(a, fsm + n2 * S.S2 + c * S.SC, S.S1, tw + n2, L2);
}

template <int L2, bool CROP, bool IL>
__device__ __forceinline__ void rows_b(const RowArgs &ra, const float2 *fsm, int L, int L1, float2 *__restrict__ dst)
{
    constexpr bool XB = RowShape<CROP, IL>::XB;
    const RowShape<CROP, IL> S(L2);
    const FftGeom &g = ra.g;
    const int w = threadIdx.x, row0 = blockIdx.x * kFftLines;
    const int N0 = g.N[0], h0 = g.off[0] > 0 ? L - g.off[0] : -g.off[0];
    if (w >= kFftLines * L1) return;
    const int c = XB ? w / L1 : w % kFftLines, k1 = XB ? w - c * L1 : w / kFftLines;
    float2 b[L2];
    step_b<L2, CROP>(fsm + k1 * S.S1 + c * S.SC, S.S2, b);
    if (row0 + c >= ra.nrows) return;
    const RowLine ln = row_line<IL>(ra, row0 + c);
    if (!CROP) {
        float2 *d = dst + ln.grid + (int64_t)k1 * (IL ? g.CS : 1);
        const int step = IL ? L1 * g.CS : L1;
#pragma unroll
        for (int k2 = 0; k2 < L2; k2++) d[(int64_t)step * k2] = b[k2];
    } else if (ln.img >= 0) {
        const float *ap = g.apod[0];
        const int i0 = k1 + h0;
        float2 *d = dst + ln.img;
#pragma unroll
        for (int k2 = 0; k2 < L2; k2++) {
            const int i = i0 + L1 * k2 - (i0 + L1 * k2 >= L ? L : 0);
            if (i < N0) d[i] = scl(ap ? ln.s * __ldg(ap + i) : ln.s, b[k2]);
        }
    }
}

template <class F, bool CROP, bool IL>
__global__ void __launch_bounds__(F::T, F::MINB) fft_rows_kernel(RowArgs ra, const float2 *__restrict__ tw,
                                                        const void *__restrict__ src, int src_real,
                                                        float2 *__restrict__ dst)
{
    extern __shared__ __align__(16) float2 fsm[];
    rows_a<F::L1, CROP, IL>(ra, fsm, F::L, F::L2, tw, src, src_real);
    __syncthreads();
    rows_b<F::L2, CROP, IL>(ra, fsm, F::L, F::L1, dst);
}

// Column pass along y or z, in place on the grid: a block per 16 consecutive x
// (x, coil) of one line set (set, outer index), the line running along the axis
// with element stride S. Input positions outside `in` are zero and not read;
// outputs outside `out` are not written. Outer index k selects plane / row
// (outer_q0 + k) mod outer_G with stride outer_stride.
struct ColArgs {
    int64_t S, outer_stride;
    int nouter, outer_q0, outer_G;
    int in_q0, in_n, out_q0, out_n;
    int inv;
    Range in, out;
};

// column of the block's thread w: grid position x, first element at line position 0
__device__ __forceinline__ int64_t col_base(const ColArgs &a, int64_t gsize)
{
    int qo = a.outer_q0 + blockIdx.y;
    if (qo >= a.outer_G) qo -= a.outer_G;
    return blockIdx.z * gsize + (int64_t)qo * a.outer_stride + blockIdx.x * kFftLines + threadIdx.x % kFftLines;
}

template <int L1, bool IN_ALL, bool INV>
__device__ __forceinline__ void cols_a(const ColArgs &a, int G0, int x, float2 *fsm, int L2, const float2 *base,
                                       const float2 *__restrict__ tw)
{
    const int w = threadIdx.x, r = w / kFftLines, step = (int)(L2 * a.S);
    if (r >= L2) return;
    float2 v[L1];
    base += r * a.S;
#pragma unroll
    for (int n1 = 0; n1 < L1; n1++) {
        v[n1] = make_float2(0.0f, 0.0f);
        if (x < G0 && (IN_ALL || a.in.has(r + L2 * n1))) v[n1] = __ldcg(base + (int64_t)step * n1);
    }
    step_a<L1, INV>(v, fsm + w, L2 * kFftLines, tw + r, L2);
}

template <int L2, bool OUT_ALL, bool INV>
__device__ __forceinline__ void cols_b(const ColArgs &a, int G0, int x, const float2 *fsm, int L1, float2 *base)
{
    const int w = threadIdx.x, r = w / kFftLines, step = (int)(L1 * a.S);
    if (r >= L1 || x >= G0) return;
    float2 b[L2];
    step_b<L2, INV>(fsm + r * L2 * kFftLines + w % kFftLines, kFftLines, b);
    base += r * a.S;
#pragma unroll
    for (int k2 = 0; k2 < L2; k2++)
        if (OUT_ALL || a.out.has(r + L1 * k2)) base[(int64_t)step * k2] = b[k2];
}

template <class F, bool IN_ALL, bool OUT_ALL, bool INV>
__global__ void __launch_bounds__(F::T, F::MINB) fft_cols_kernel(int G0, int64_t gsize, ColArgs a,
                                                        const float2 *__restrict__ tw, float2 *grid)
{
    extern __shared__ __align__(16) float2 fsm[];
    const int x = blockIdx.x * kFftLines + threadIdx.x % kFftLines;
    float2 *base = grid + col_base(a, gsize);
    cols_a<F::L1, IN_ALL, INV>(a, G0, x, fsm, F::L2, base, tw);
    __syncthreads();
    cols_b<F::L2, OUT_ALL, INV>(a, G0, x, fsm, F::L1, base);
}

// Toeplitz z pass: per 16 x of one (batch, y), the z columns (reading the N2 z
// with data only), forward FFT, times kernel[b mod nk][z][y][x] * kscale,
// inverse FFT, and the N2 kept z written back. After step B a thread holds the
// transform at k1 + L1 k2, all k2: the inverse runs the two steps backwards from
// there (L2 points over k2, twiddles, the same row of the exchange buffer, L1
// points over k1), so two barriers serve both transforms. Blocks run
// batch-fastest: those that read one kernel tile run together and share it in L2.
template <int L2>
__device__ __forceinline__ void toep_b(const ColArgs &a, int G0, int x, float2 *fsm, int L1, const float2 *kb, float kscale,
                                       const float2 *__restrict__ tw)
{
    const int w = threadIdx.x, r = w / kFftLines, step = (int)(L1 * a.S);
    if (r >= L1) return;
    float2 b[L2];
    float2 *row = fsm + r * L2 * kFftLines + w % kFftLines;
    step_b<L2, false>(row, kFftLines, b);
    // kernel values six loads at a time (left to itself the compiler takes one load,
    // one use: 288 points, 8 coils of 144^3, 1.31 ms against 0.75, and 512 points 48
    // us a call against 24; all at once spills: 28 us)
    constexpr int GRP = 6;
    const bool on = x < G0;
    kb += r * a.S;
#pragma unroll
    for (int k0 = 0; k0 < L2; k0 += GRP) {
        float2 kv[GRP];
#pragma unroll
        for (int j = 0; j < GRP; j++)
            kv[j] = on && k0 + j < L2 ? __ldg(kb + (int64_t)step * (k0 + j)) : make_float2(0.0f, 0.0f);
#pragma unroll
        for (int j = 0; j < GRP; j++)
            if (k0 + j < L2) b[k0 + j] = scl(kscale, cmulf(kv[j], b[k0 + j]));
    }
    reg_dft<L2, true>(b);
#pragma unroll
    for (int n2 = 0; n2 < L2; n2++) row[n2 * kFftLines] = twiddle<true>(b[n2], __ldg(tw + r * L2 + n2));
}

template <int L1>
__device__ __forceinline__ void toep_c(const ColArgs &a, int G0, int x, const float2 *fsm, int L2, float2 *base)
{
    const int w = threadIdx.x, r = w / kFftLines, step = (int)(L2 * a.S);
    if (r >= L2 || x >= G0) return;
    float2 v[L1];
#pragma unroll
    for (int k1 = 0; k1 < L1; k1++) v[k1] = fsm[k1 * L2 * kFftLines + w];
    reg_dft<L1, true>(v);
    base += r * a.S;
#pragma unroll
    for (int n1 = 0; n1 < L1; n1++)
        if (a.out.has(r + L2 * n1)) base[(int64_t)step * n1] = v[n1];
}

template <class F>
__global__ void __launch_bounds__(F::T, F::TOEP_MINB) fft_toep_z_kernel(int G0, int64_t gsize, ColArgs a, int64_t nk,
                                                          const float2 *__restrict__ kern, float kscale,
                                                          const float2 *__restrict__ tw, float2 *grid)
{
    extern __shared__ __align__(16) float2 fsm[];
    const int x = blockIdx.y * kFftLines + threadIdx.x % kFftLines;
    const int64_t bf = blockIdx.x, to = (int64_t)blockIdx.z * a.outer_stride + x;
    float2 *base = grid + bf * gsize + to;
    cols_a<F::L1, false, false>(a, G0, x, fsm, F::L2, base, tw);
    __syncthreads();
    toep_b<F::L2>(a, G0, x, fsm, F::L1, kern + (bf % nk) * gsize + to, kscale, tw);
    __syncthreads();
    toep_c<F::L1>(a, G0, x, fsm, F::L2, base);
}

// Other lengths L = L1 L2, both at most MX: the same steps with the factors at
// run time, a switch over the register transforms. Three sizes of kernel (13, 20
// and 26), so that small factors do not pay for the registers of large ones.
struct Fac {
    int L = 0, L1 = 0, L2 = 0;
};
constexpr int kGenMax = 26;
template <int MX>
struct Gen {
    static constexpr int T = kFftLines * MX, MINB = 65536 / (T * (MX > 20 ? 72 : 64));
};
// the run-time lengths' passes (fft_any_rows.cuh, fft_any_cols.cu, fft_any_toep.cu)
template <bool CROP, bool IL>
int launch_rows_any(Fac f, const FftGeom &g, const float2 *tw, const void *src, int src_real, float2 *dst, cudaStream_t st);
int launch_cols_any(const Fac &f, const FftGeom &g, const ColArgs &a, const float2 *tw, float2 *grid, cudaStream_t st);
int launch_toep_any(const Fac &f, const FftGeom &g, const ColArgs &a, int64_t nk, const float2 *kern, float kscale,
                    const float2 *tw, float2 *grid, cudaStream_t st);

// sets (batch, frame) per launch: the grid's y and z extents are 16 bits
constexpr int64_t kMaxSets = 65535;

template <class K>
inline int opt_in(K kern, size_t smem)
{
    if (smem > 48 * 1024) DMR_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return DMR_OK;
}

// a column pass with any kernel that takes (G0, gsize, a, tw, grid)
template <class K, class... A>
inline int launch_cols_k(K kern, int L, int T, const FftGeom &g, const ColArgs &a, const float2 *tw, float2 *grid, cudaStream_t st,
                  A... head)
{
    const size_t smem = (size_t)L * kFftLines * sizeof(float2);
    DMR_TRY(opt_in(kern, smem));
    for (int64_t b = 0; b < g.nbf; b += kMaxSets) {
        const dim3 blocks((unsigned)ceil_div(g.G[0], kFftLines), (unsigned)a.nouter,
                          (unsigned)std::min<int64_t>(g.nbf - b, kMaxSets));
        kern<<<blocks, T, smem, st>>>(head..., g.G[0], g.gsize, a, tw, grid + b * g.gsize);
        DMR_LAUNCHED("fft_cols_kernel");
    }
    return DMR_OK;
}

template <bool CROP, bool IL, class K, class... A>
inline int launch_rows_k(K kern, int L1, int L2, const FftGeom &g, const float2 *tw, const void *src, int src_real, float2 *dst,
                  cudaStream_t st, A... head)
{
    const size_t smem = (size_t)L1 * RowShape<CROP, IL>(L2).S1 * sizeof(float2);
    DMR_TRY(opt_in(kern, smem));
    const int64_t nrows = (int64_t)g.N[2] * g.N[1] * (IL ? g.CS : 1);
    DMR_CHECK(nrows < INT32_MAX - kFftLines && g.nbf <= INT32_MAX, DMR_ERR_UNSUPPORTED, "too many image rows");
    RowArgs ra{g, FastDiv(IL ? g.CS : 1), FastDiv(g.N[1]), FastDiv(g.nframes), (int)nrows, 0};
    for (; ra.bf0 < g.nbf; ra.bf0 += kMaxSets) {
        const dim3 blocks((unsigned)ceil_div(nrows, kFftLines), (unsigned)std::min<int64_t>(g.nbf - ra.bf0, kMaxSets));
        kern<<<blocks, kFftLines * std::max(L1, L2), smem, st>>>(head..., ra, tw, src, src_real, dst);
        DMR_LAUNCHED(CROP ? "fft_crop_rows_kernel" : "fft_pad_rows_kernel");
    }
    return DMR_OK;
}

template <class K, class... A>
inline int launch_toep_k(K kern, int L, int T, const FftGeom &g, const ColArgs &a, int64_t nk, const float2 *kernel, float kscale,
                  const float2 *tw, float2 *grid, cudaStream_t st, A... head)
{
    const size_t smem = (size_t)L * kFftLines * sizeof(float2);
    DMR_TRY(opt_in(kern, smem));
    const dim3 blocks((unsigned)g.nbf, (unsigned)ceil_div(g.G[0], kFftLines), (unsigned)a.nouter);
    kern<<<blocks, T, smem, st>>>(head..., g.G[0], g.gsize, a, nk, kernel, kscale, tw, grid);
    DMR_LAUNCHED("fft_toep_z_kernel");
    return DMR_OK;
}

}  // namespace fftp
}  // namespace dmr
