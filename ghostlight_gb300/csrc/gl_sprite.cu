// gl_sprite.cu — the SPRITE starburst engine: one FFT of the stop pupil,
// baked over wavelength into an RGB sprite, splatted at every source.
//
// Restates the reference's default engine (render_starburst's sprite path,
// ghostlight/src/starburst_render.cu:969-1073, kernels :194-389):
//   |FFT(A)|^2 with DC at the grid centre -> normalised to unit sum -> the
//   sprite texel (i, j) = sum_l cmf_l * PSF(c + (i, j - c) lambda_ref /
//   lambda_l) (lambda_ref / lambda_l)^2 (Fourier scaling theorem, bilinear,
//   zero outside) -> box-summed by ds toward the output pitch -> each output
//   pixel integrates the sprite over its own footprint (area-weighted box
//   resample), times the source colour and the gain.
//
// GB300 layout (one GPU, everything resident in the plan):
//   * 2-D FFT of the real pupil as two shared-memory passes (gl_fft.cuh): (1)
//     column transforms, two real columns per complex transform, split into
//     their half spectra ky <= N / 2; a CTA whose columns the pupil leaves dark
//     only says so (the pupil fills a centred disc of `fill` of the grid, so
//     most are); (2) two rows ky per CTA over the lit columns, whose last stage
//     writes |X|^2 straight to its fftshifted place and, the pupil being real,
//     to the mirrored one, and adds the CTA's energy to one FP64 sum;
//   * the wavelength bake and the ds x ds box sum fused in one kernel, so the
//     N x N x 3 fine sprite (805 MB at N = 8192) never exists in HBM; the
//     1 / energy normalisation is read on the device (no host round trip);
//   * the splat: one thread per (source, output pixel in the footprint),
//     float atomics into the caller's planes (sources overlap), as the
//     reference does.
#include "gl_internal.h"
#include "gl_fft.cuh"
#include "gl_launch.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

namespace gl {
namespace {

constexpr int kSpriteThreads = 256;
constexpr int kMaxSpriteGrid = 8192;   // a complex row pair fits the 227 KB of shared memory

struct StarSource { float px, py, r, g, b; };

// ---- 2-D transform of a real grid ------------------------------------------------
// N = 2048 with a pupil of 0.3 of it: rows then columns of the full complex
// spectrum took 28 + 110 us (139 KB of shared memory and 8 warps per CTA, one
// CTA per SM, 16-byte pieces of each row), the half spectrum's two passes
// 19 + 20 us.
constexpr int kShortGrid = 1024;    // ping-pong stages up to here, in place above (gl_fft.cuh)

// Half spectrum of the first pass: column x, row ky <= N / 2 at
// ((ky / 2) N + x) 2 + ky % 2, so a pair of rows is one contiguous block.
__device__ __forceinline__ size_t half_index(int N, int pair, int x) { return ((size_t)pair * N + x) * 2; }

// Pass 1: columns 4 blockIdx.x .. + 3, two real ones per complex sequence; rows
// ky < 2 pairs kept.  lit[blockIdx.x]
// = 0 where all are zero (nothing is written then).  The grid may be a caller's
// that starts at an odd float: pairs of columns are read as such only from 8-byte
// boundaries (N is even, so the base decides for all rows).
template <bool PP>
__global__ void __launch_bounds__(1024) grid_cols(const float* __restrict__ in, int N, int pairs,
                                                  const __grid_constant__ FftDims d, const float2* __restrict__ tw,
                                                  float2* __restrict__ half, unsigned char* __restrict__ lit)
{
    after_previous();
    extern __shared__ float2 sm[];
    float2* x = sm;
    float2* y = PP ? sm + padded((size_t)N * 2) : sm;
    const int c0 = blockIdx.x * 4;
    const bool pairwise = (reinterpret_cast<uintptr_t>(in) & 7) == 0;
    int any = 0;
    for (int i = threadIdx.x; i < 2 * N; i += blockDim.x)
    {
        const float* q = in + (size_t)(i >> 1) * N + c0 + 2 * (i & 1);
        float2 v;
        if (pairwise) v = *reinterpret_cast<const float2*>(q);
        else
        {
            v.x = q[0];
            v.y = q[1];
        }
        any |= (v.x != 0.0f) | (v.y != 0.0f);
        x[fft_slot<2, true>(i >> 1, i & 1, N)] = v;
    }
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) lit[blockIdx.x] = any ? 1 : 0;
    if (!any) return;
    for (int st = 0; st < d.nrad; ++st) fft_any<2, true, false, PP, false, false, true>(x, y, d, st, tw, FftNone{}, FftNone{});
    // Z = FFT(a + i b): FFT(a)[k] = (Z[k] + conj Z[N - k]) / 2, FFT(b)[k] = (Z[k] - conj Z[N - k]) / 2i;
    // per pair of rows: 2 x 2 columns x 2 rows, one 64-byte piece
    for (int t = threadIdx.x; t < pairs * 2; t += blockDim.x)
    {
        const int pr = t >> 1, s = t & 1;
        float2 a[2], b[2];
        #pragma unroll
        for (int c = 0; c < 2; ++c)
        {
            const int k = 2 * pr + c;
            a[c] = b[c] = make_float2(0.0f, 0.0f);
            if (k <= N / 2)
            {
                const float2 z = x[fft_slot<2, true>(k, s, N)], w = x[fft_slot<2, true>((N - k) & (N - 1), s, N)];
                a[c] = make_float2(0.5f * (z.x + w.x), 0.5f * (z.y - w.y));
                b[c] = make_float2(0.5f * (z.y + w.y), 0.5f * (w.x - z.x));
            }
        }
        float4* o = reinterpret_cast<float4*>(half + half_index(N, pr, c0 + 2 * s));
        o[0] = make_float4(a[0].x, a[0].y, a[1].x, a[1].y);
        o[1] = make_float4(b[0].x, b[0].y, b[1].x, b[1].y);
    }
}

// Rows ky = 2 pair + s of the half spectrum; dark columns are zero.
struct HalfRows {
    const float2* half;            // the pair's block
    const unsigned char* lit;      // shared memory
    __device__ __forceinline__ float2 operator()(int s, int x) const
    {
        return lit[x >> 2] ? half[2 * x + s] : make_float2(0.0f, 0.0f);
    }
};

// |X|^2 at its fftshifted place and at the mirrored one.
struct PsfStore {
    float* psf;
    float* sum;                    // this thread's energy
    int N, pair;
    __device__ __forceinline__ void operator()(int s, int kx, float2 z) const
    {
        const int ky = 2 * pair + s, h = N / 2, m = N - 1;
        if (ky > h) return;
        const float p = z.x * z.x + z.y * z.y;
        psf[(size_t)((ky + h) & m) * N + ((kx + h) & m)] = p;
        const bool own = ky == 0 || ky == h;             // these rows hold their own mirror
        *sum += own ? p : 2.0f * p;
        if (own) return;
        psf[(size_t)((h - ky) & m) * N + ((h - kx) & m)] = p;
    }
};

// The matrix-DFT engine's compact autocorrelation (mdft_render.cu:88-99,
// 247-262), from the transform of the fftshifted PSF: lags within +-mc,
// C[a][b] (a = y lag + mc, b = x lag + mc) = (-1)^(lx + ly) Re X[ly][lx] /
// (energy N^2).  The sign undoes the fftshift of the PSF (a shift by N/2
// multiplies the transform by (-1)^l); energy = sum |FFT A|^2 = G[0][0].  A real
// pupil has a real, point-symmetric autocorrelation: the imaginary part is
// rounding, and C[-ly][-lx] is C[ly][lx].
struct LagStore {
    float* C;
    int N, pair, mc, ldc;
    float scale, scale_lo;         // the scale in two floats: one rounding would be in every lag
    __device__ __forceinline__ void operator()(int s, int kx, float2 z) const
    {
        const int ly = 2 * pair + s, lx = kx <= N / 2 ? kx : kx - N;
        if (ly > mc || lx < -mc || lx > mc) return;
        const float x = ((lx + ly) & 1) ? -z.x : z.x, v = fmaf(x, scale, x * scale_lo);
        C[(size_t)(mc + ly) * ldc + (mc + lx)] = v;
        if (ly > 0) C[(size_t)(mc - ly) * ldc + (mc - lx)] = v;
    }
};

// Pass 2: rows ky of pair blockIdx.x.  LAGS: the autocorrelation's lags, else
// the PSF and its energy.
template <bool PP, bool LAGS>
__global__ void __launch_bounds__(1024) grid_rows(const float2* __restrict__ half, const unsigned char* __restrict__ lit,
                                                  int N, const __grid_constant__ FftDims d, const float2* __restrict__ tw,
                                                  float* __restrict__ out, double* __restrict__ energy, int mc, int ldc)
{
    after_previous();
    extern __shared__ float2 sm[];
    __shared__ double red[32];
    float2* x = sm;
    float2* y = PP ? sm + padded((size_t)N * 2) : sm;
    unsigned char* flags = reinterpret_cast<unsigned char*>(sm + (PP ? 2 : 1) * padded((size_t)N * 2));
    const int pair = blockIdx.x;
    for (int i = threadIdx.x; i < N / 4; i += blockDim.x) flags[i] = lit[i];
    __syncthreads();
    const HalfRows load{half + half_index(N, pair, 0), flags};
    fft_any<2, true, false, PP, true, false, true>(x, y, d, 0, tw, load, FftNone{});
    for (int st = 1; st + 1 < d.nrad; ++st) fft_any<2, true, false, PP, false, false, true>(x, y, d, st, tw, FftNone{}, FftNone{});
    if (LAGS)
    {
        const double e = *energy;
        const double k = e > 0.0 ? 1.0 / (e * (double)N * (double)N) : 0.0;
        const float scale = (float)k, scale_lo = (float)(k - (double)scale);
        fft_any<2, true, false, PP, false, true, true>(x, y, d, d.nrad - 1, tw, FftNone{}, LagStore{out, N, pair, mc, ldc, scale, scale_lo});
        return;
    }
    float own = 0.0f;
    fft_any<2, true, false, PP, false, true, true>(x, y, d, d.nrad - 1, tw, FftNone{}, PsfStore{out, &own, N, pair});
    double part = (double)own;        // (from here on in FP64: the sum's rounding is in every lag)
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = part;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        atomicAdd(energy, t);
    }
}

// Bake over wavelength + box sum of d x d fine texels (d a power of two up to
// 32): coarse texel (a, b) of M x M.
//
// A lane owns one fine column and T fine rows of it; a CTA's eight warps stack
// to 32 columns x 8 T rows.  The rows' source positions are tabled per
// wavelength in shared memory, the column's is formed once per wavelength.
// Neighbouring fine rows sample source rows 0.8 to 1.4 apart, so the
// horizontal blend of the lower source row of one is mostly the upper one of
// the next: about 2.5 loads per texel and wavelength where separate samples
// take 4, and all loads of a thread's rows are in flight at once (carrying the
// blend from row to row behind a branch left each row waiting for its own
// load).
// The box sum goes over the thread's rows, then lanes, then (d > T) warps, in
// a fixed order.  Every fine texel is a thread's, so a strongly minified sprite
// (few coarse texels) still fills the chip.  Bound by load latency and issue in
// equal parts (issue slots 56% busy, L1 49%); eight rows per thread, or more
// CTAs per SM at fewer registers, are slower.
// N = 2048, 31 wavelengths, d = 2: 221 -> 157 us; N = 1024, 16 wavelengths,
// d = 16 (one thread per coarse texel: 16 CTAs): 1404 -> 28 us.
constexpr int kBakeSpec = 32;      // wavelengths staged at a time

// A fine row's source rows at one wavelength: byte offset of the lower one, its
// lowest bit set where the upper one is the lower one of the fine row before
// (offsets are multiples of 4 N), and the blend of the two (zero outside).
struct __align__(16) RowAt { uint32_t lower; float up, lo, pad; };

// A float of the grid by its byte offset (a grid has at most 2^28 bytes).
__device__ __forceinline__ float grid_at(const float* g, uint32_t byte)
{
    return __ldg(reinterpret_cast<const float*>(reinterpret_cast<const char*>(g) + byte));
}

template <int T>
__global__ void __launch_bounds__(kSpriteThreads) sprite_bake(const float* __restrict__ psf, int N,
                                                              const float4* __restrict__ spec, int n_spec,
                                                              float lambda_ref, int d, int M,
                                                              const double* __restrict__ energy,
                                                              float* __restrict__ sprite)
{
    after_previous();
    constexpr int kRows = kSpriteThreads / 32 * T;       // fine rows of the CTA
    __shared__ float4 lam[kBakeSpec];                    // lambda_ref / lambda, colour weights
    __shared__ RowAt row_at[kBakeSpec][kRows];
    __shared__ float part[kSpriteThreads / 32][32][3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane, j0 = blockIdx.y * kRows + warp * T;
    const double e = *energy;
    const float scale = (e > 0.0) ? (float)(1.0 / e) : 0.0f;
    const float half = (float)(N / 2), top = (float)(N - 1);
    const float dx = (float)(i - N / 2);
    float acc[T][3] = {};
    for (int l0 = 0; l0 < n_spec; l0 += kBakeSpec)
    {
        const int nl = min(kBakeSpec, n_spec - l0);
        __syncthreads();
        for (int q = threadIdx.x; q < nl * kRows; q += kSpriteThreads)
        {
            const int l = q / kRows, r = q - l * kRows;
            const float4 s = spec[l0 + l];
            const float k = lambda_ref / s.x;
            const float dy = (float)((int)blockIdx.y * kRows + r - N / 2);
            const float fy = half + dy * k;
            const bool in = fy >= 0.0f && fy < top;
            const int y0 = in ? (int)floorf(fy) : 0;
            // the row before, of the same thread
            const float fz = half + (dy - 1.0f) * k;
            const bool carried = r % T != 0 && in && fz >= 0.0f && y0 == (int)floorf(fz) + 1;
            RowAt at;
            at.lower = (uint32_t)(y0 + 1) * (uint32_t)N * 4u | (carried ? 1u : 0u);
            at.lo = in ? fy - (float)y0 : 0.0f;
            at.up = in ? 1.0f - at.lo : 0.0f;
            at.pad = 0.0f;
            row_at[l][r] = at;
            if (r == 0) lam[l] = make_float4(k, s.y * (k * k * scale), s.z * (k * k * scale), s.w * (k * k * scale));
        }
        __syncthreads();
        #pragma unroll 2
        for (int l = 0; l < nl; ++l)
        {
            const float4 s = lam[l];
            const float fx = half + dx * s.x;
            const bool in = fx >= 0.0f && fx < top;
            if (!__any_sync(0xffffffffu, in)) continue;
            const int x0 = in ? (int)floorf(fx) : 0;
            const float tx = fx - (float)x0;
            // a column outside blends to zero
            const float b0 = in ? 1.0f - tx : 0.0f, b1 = in ? tx : 0.0f;
            const uint32_t x4 = 4u * (uint32_t)x0, n4 = 4u * (uint32_t)N;
            // lower source row of each fine row; the upper one where it is not
            // the row before's (the same for the whole warp)
            float lo[T], up[T];
            #pragma unroll
            for (int r = 0; r < T; ++r)
            {
                const uint32_t o = (row_at[l][warp * T + r].lower & ~1u) + x4;
                lo[r] = grid_at(psf, o) * b0 + grid_at(psf, o + 4) * b1;
            }
            #pragma unroll
            for (int r = 0; r < T; ++r)
            {
                const uint32_t f = row_at[l][warp * T + r].lower;
                up[r] = lo[max(r - 1, 0)];
                if (!(f & 1u))
                {
                    const uint32_t o = f + x4 - n4;
                    up[r] = grid_at(psf, o) * b0 + grid_at(psf, o + 4) * b1;
                }
            }
            #pragma unroll
            for (int r = 0; r < T; ++r)
            {
                const RowAt& at = row_at[l][warp * T + r];
                const float v = up[r] * at.up + lo[r] * at.lo;
                acc[r][0] += s.y * v;
                acc[r][1] += s.z * v;
                acc[r][2] += s.w * v;
            }
        }
    }
    // rows of the thread, then lanes
    const int g = min(d, T);                             // rows per sum
    #pragma unroll
    for (int r = 0; r < T; ++r)
        #pragma unroll
        for (int c = 0; c < 3; ++c)
        {
            float v = acc[r][c];
            #pragma unroll
            for (int q = 1; q < T; ++q)
                if (r + q < T && q < g && r % g == 0) v += acc[r + q][c];
            for (int o = 1; o < d; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (r % g == 0 && (lane & (d - 1)) == 0)
            {
                if (d <= T) sprite[3 * ((size_t)((j0 + r) / d) * M + i / d) + c] = v;
                else part[warp][lane][c] = v;
            }
        }
    if (d <= T) return;                                  // uniform over the grid
    // d > T: each coarse texel is d / T warps of this CTA
    __syncthreads();
    const int wpt = d / T, cols = 32 / d, rows = (kSpriteThreads / 32) / wpt;
    for (int t = threadIdx.x; t < rows * cols * 3; t += kSpriteThreads)
    {
        const int c = t % 3, a = (t / 3) % cols, b = t / (3 * cols);
        float v = 0.0f;
        for (int w = 0; w < wpt; ++w) v += part[b * wpt + w][a * d][c];
        sprite[3 * ((size_t)(blockIdx.y * rows + b) * M + blockIdx.x * cols + a) + c] = v;
    }
}

// The rest of a box sum above 32: f x f sums of the 32-texel sums.
__global__ void __launch_bounds__(kSpriteThreads) sprite_box(const float* __restrict__ fine, int f, int M,
                                                             float* __restrict__ sprite)
{
    after_previous();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 3 * M * M) return;
    const int c = t % 3, a = (t / 3) % M, b = t / (3 * M);
    float v = 0.0f;
    for (int y = 0; y < f; ++y)
        for (int x = 0; x < f; ++x) v += fine[3 * ((size_t)(b * f + y) * M * f + a * f + x) + c];
    sprite[t] = v;
}

// One output pixel of one source's footprint (offset t in its
// (2 rx + 1) x (2 ry + 1) box): the sprite integrated over the pixel's sensor
// footprint (texel overlap areas), tinted, added.
__device__ __forceinline__ void splat_pixel(const float* __restrict__ sprite, int M, float sx_ds, float sy_ds,
                                            float px_mm_x, float px_mm_y, int rx, int ry, const StarSource& s,
                                            long long t, float gain, float* __restrict__ out_r,
                                            float* __restrict__ out_g, float* __restrict__ out_b, int width,
                                            int height)
{
    const long long span_x = 2LL * rx + 1;
    const int oy = (int)(t / span_x) - ry, ox = (int)(t % span_x) - rx;
    const int ix = (int)floorf(s.px) + ox, iy = (int)floorf(s.py) + oy;
    if (ix < 0 || ix >= width || iy < 0 || iy >= height) return;
    // the pixel [ix, ix+1) x [iy, iy+1) in texel-cell coordinates (texel a
    // covers [a, a+1), its centre at sensor offset (a - M/2 + 0.5) pitch)
    const float xlo = ((ix - s.px) * px_mm_x) / sx_ds + 0.5f * M - 0.5f + 0.5f;
    const float xhi = ((ix + 1.0f - s.px) * px_mm_x) / sx_ds + 0.5f * M - 0.5f + 0.5f;
    const float ylo = ((iy - s.py) * px_mm_y) / sy_ds + 0.5f * M - 0.5f + 0.5f;
    const float yhi = ((iy + 1.0f - s.py) * px_mm_y) / sy_ds + 0.5f * M - 0.5f + 0.5f;
    int i0 = (int)floorf(xlo), i1 = (int)floorf(xhi - 1e-6f);
    int j0 = (int)floorf(ylo), j1 = (int)floorf(yhi - 1e-6f);
    i0 = max(i0, 0);
    i1 = min(i1, M - 1);
    j0 = max(j0, 0);
    j1 = min(j1, M - 1);
    if (i1 < i0 || j1 < j0) return;
    i1 = min(i1, i0 + 64);   // bounded box for a pathologically minified sprite
    j1 = min(j1, j0 + 64);
    float ar = 0.0f, ag = 0.0f, ab = 0.0f;
    for (int j = j0; j <= j1; ++j)
    {
        const float yov = fminf(yhi, (float)(j + 1)) - fmaxf(ylo, (float)j);
        if (yov <= 0.0f) continue;
        const float* row = sprite + 3 * ((size_t)j * M);
        for (int i = i0; i <= i1; ++i)
        {
            const float xov = fminf(xhi, (float)(i + 1)) - fmaxf(xlo, (float)i);
            if (xov <= 0.0f) continue;
            const float w = xov * yov;
            const float* p = row + 3 * i;
            ar += p[0] * w;
            ag += p[1] * w;
            ab += p[2] * w;
        }
    }
    const float vr = ar * s.r * gain, vg = ag * s.g * gain, vb = ab * s.b * gain;
    const size_t pix = (size_t)iy * width + ix;
    if (fabsf(vr) > 1e-20f) atomicAdd(&out_r[pix], vr);
    if (fabsf(vg) > 1e-20f) atomicAdd(&out_g[pix], vg);
    if (fabsf(vb) > 1e-20f) atomicAdd(&out_b[pix], vb);
}

__global__ void __launch_bounds__(kSpriteThreads) sprite_splat(const float* __restrict__ sprite, int M, float sx_ds,
                                                               float sy_ds, float px_mm_x, float px_mm_y, int rx,
                                                               int ry, const StarSource* __restrict__ src,
                                                               int n_src, float gain, float* __restrict__ out_r,
                                                               float* __restrict__ out_g, float* __restrict__ out_b,
                                                               int width, int height)
{
    const long long per_src = (2LL * rx + 1) * (2LL * ry + 1);
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= (long long)n_src * per_src) return;
    const int si = (int)(tid / per_src);
    splat_pixel(sprite, M, sx_ds, sy_ds, px_mm_x, px_mm_y, rx, ry, src[si], tid % per_src, gain, out_r, out_g,
                out_b, width, height);
}

// One source passed by value: no staging buffer, so splats of one resident
// sprite on many streams run side by side.
__global__ void __launch_bounds__(kSpriteThreads) sprite_splat_one(const float* __restrict__ sprite, int M,
                                                                   float sx_ds, float sy_ds, float px_mm_x,
                                                                   float px_mm_y, int rx, int ry, StarSource s,
                                                                   float gain, float* __restrict__ out_r,
                                                                   float* __restrict__ out_g,
                                                                   float* __restrict__ out_b, int width, int height)
{
    const long long per_src = (2LL * rx + 1) * (2LL * ry + 1);
    const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= per_src) return;
    splat_pixel(sprite, M, sx_ds, sy_ds, px_mm_x, px_mm_y, rx, ry, s, tid, gain, out_r, out_g, out_b, width, height);
}

}  // namespace

struct SpritePlan {
    int N = 0, n_spec = 0, M = 0, device = 0;
    float lambda_ref = 550.0f;
    FftDims dims{};
    float2* tw = nullptr;        // stage twiddles
    float2* half = nullptr;      // half spectrum, N / 4 + 1 row pairs x N columns
    unsigned char* lit = nullptr;   // per four columns: anything lit
    float* psf = nullptr;
    float* sprite = nullptr;
    size_t sprite_cap = 0;       // floats; grown by the bake to 3 M^2 (and the scratch of a large box sum)
    float4* spec = nullptr;
    double* energy = nullptr;
    StarSource* src = nullptr;
    int src_cap = 0;
    bool pp = false;
    int threads = 0;
    size_t smem = 0;
};

}  // namespace gl

struct gl_sprite_plan { gl::SpritePlan* p; };

using namespace gl;

static void sprite_free(SpritePlan* p)
{
    cudaFree(p->tw);
    cudaFree(p->half);
    cudaFree(p->lit);
    cudaFree(p->psf);
    cudaFree(p->sprite);
    cudaFree(p->spec);
    cudaFree(p->energy);
    cudaFree(p->src);
    delete p;
}

extern "C" int gl_sprite_plan_create(int N, const gl_spectral_sample* spec, int n_spec, float lambda_ref,
                                     gl_sprite_plan** out)
{
    if (!out || !spec || n_spec < 1) return fail(GL_ERR_INVALID, "sprite_plan_create: bad arguments");
    if (N < 256 || N > kMaxSpriteGrid || (N & (N - 1)) != 0)
        return fail(GL_ERR_INVALID, "sprite_plan_create: grid must be a power of two in [256, 8192]");
    if (!(lambda_ref > 0.0f)) return fail(GL_ERR_INVALID, "sprite_plan_create: lambda_ref must be positive");
    for (int l = 0; l < n_spec; ++l)
        if (!(spec[l].lambda > 0.0f)) return fail(GL_ERR_INVALID, "sprite_plan_create: wavelengths must be positive");
    SpritePlan* p = new SpritePlan();
    p->N = N;
    p->n_spec = n_spec;
    p->lambda_ref = lambda_ref;
    p->dims = make_dims(N);
    cudaGetDevice(&p->device);
    const size_t NN = (size_t)N * N;
    p->pp = N <= kShortGrid;
    p->threads = fft_threads(N, 2, p->pp);
    p->smem = (p->pp ? 2 : 1) * padded((size_t)N * 2) * sizeof(float2) + N / 4;
    cudaError_t e = cudaSuccess;
    auto chk = [&](cudaError_t x) { if (e == cudaSuccess) e = x; };
    const std::vector<float2> tw = stage_twiddles(p->dims);
    chk(cudaMalloc(&p->tw, sizeof(float2) * tw.size()));
    chk(cudaMalloc(&p->half, sizeof(float2) * 2 * (size_t)N * (N / 4 + 1)));
    chk(cudaMalloc(&p->lit, N / 4));
    chk(cudaMalloc(&p->psf, sizeof(float) * NN));
    chk(cudaMalloc(&p->spec, sizeof(float4) * n_spec));
    chk(cudaMalloc(&p->energy, sizeof(double)));
    if (e == cudaSuccess)
    {
        std::vector<float4> sp((size_t)n_spec);
        for (int l = 0; l < n_spec; ++l) sp[l] = make_float4(spec[l].lambda, spec[l].cmf_r, spec[l].cmf_g, spec[l].cmf_b);
        chk(cudaMemcpy(p->tw, tw.data(), sizeof(float2) * tw.size(), cudaMemcpyHostToDevice));
        chk(cudaMemcpy(p->spec, sp.data(), sizeof(float4) * n_spec, cudaMemcpyHostToDevice));
        if (p->pp)
        {
            chk((cudaError_t)raise_smem_limit((const void*)grid_cols<true>, p->smem));
            chk((cudaError_t)raise_smem_limit((const void*)grid_rows<true, false>, p->smem));
            chk((cudaError_t)raise_smem_limit((const void*)grid_rows<true, true>, p->smem));
        }
        else
        {
            chk((cudaError_t)raise_smem_limit((const void*)grid_cols<false>, p->smem));
            chk((cudaError_t)raise_smem_limit((const void*)grid_rows<false, false>, p->smem));
            chk((cudaError_t)raise_smem_limit((const void*)grid_rows<false, true>, p->smem));
        }
    }
    if (e != cudaSuccess)
    {
        sprite_free(p);
        return fail(e == cudaErrorMemoryAllocation ? GL_ERR_OOM : GL_ERR_CUDA,
                    std::string("sprite_plan_create: ") + cudaGetErrorString(e));
    }
    *out = new gl_sprite_plan{p};
    return GL_OK;
}

// The transforms and the bake follow each other through launches that are set up
// while the one before drains (gl_launch.cuh): a 512^2 bake at 3 wavelengths 26.6 ->
// 20.9 us, its autocorrelation 38 -> 30.  `after`: the stream's last kernel is one of
// this plan's.
static cudaError_t sprite_cols(const SpritePlan* p, const float* d_grid, int pairs, bool after, cudaStream_t st)
{
    auto kernel = p->pp ? grid_cols<true> : grid_cols<false>;
    if (after) return launch_after(kernel, dim3(p->N / 4), p->threads, p->smem, st, d_grid, p->N, pairs, p->dims, p->tw, p->half, p->lit);
    kernel<<<p->N / 4, p->threads, p->smem, st>>>(d_grid, p->N, pairs, p->dims, p->tw, p->half, p->lit);
    return cudaGetLastError();
}

template <bool LAGS>
static cudaError_t sprite_rows(const SpritePlan* p, int pairs, float* d_out, int mc, int ldc, cudaStream_t st)
{
    return launch_after(p->pp ? grid_rows<true, LAGS> : grid_rows<false, LAGS>, dim3(pairs), p->threads, p->smem, st, p->half,
                        p->lit, p->N, p->dims, p->tw, d_out, p->energy, mc, ldc);
}

// The fftshifted |FFT(grid)|^2 into p->psf, its sum added to p->energy.
static cudaError_t sprite_psf(const SpritePlan* p, const float* d_grid, cudaStream_t st)
{
    const cudaError_t e = sprite_cols(p, d_grid, p->N / 4 + 1, false, st);
    return e != cudaSuccess ? e : sprite_rows<false>(p, p->N / 4 + 1, p->psf, 0, 0, st);
}

extern "C" int gl_sprite_plan_bake(gl_sprite_plan* plan, const float* d_pupil, int ds, void* stream)
{
    if (!plan || !d_pupil) return fail(GL_ERR_INVALID, "sprite_bake: bad arguments");
    SpritePlan* p = plan->p;
    const int N = p->N;
    if (ds < 1 || (ds & (ds - 1)) != 0 || ds > N / 8)
        return fail(GL_ERR_INVALID, "sprite_bake: ds must be a power of two in [1, N/8]");
    cudaStream_t st = (cudaStream_t)stream;
    // a box sum above 32 goes through the 32-texel sums, kept behind the sprite
    const size_t need = 3 * (size_t)(N / ds) * (N / ds) + (ds > 32 ? 3 * (size_t)(N / 32) * (N / 32) : 0);
    if (need > p->sprite_cap)
    {
        // an earlier splat on this stream may still read the old sprite
        GL_CUDA_TRY(cudaStreamSynchronize(st));
        cudaFree(p->sprite);
        p->sprite = nullptr;
        p->sprite_cap = 0;
        GL_CUDA_TRY(cudaMalloc(&p->sprite, sizeof(float) * need));
        p->sprite_cap = need;
    }
    p->M = N / ds;
    GL_CUDA_TRY(cudaMemsetAsync(p->energy, 0, sizeof(double), st));
    GL_CUDA_TRY(sprite_psf(p, d_pupil, st));
    // rows per thread: four and two wavelengths in flight measured best at 1024
    // and 2048; the smallest grid takes one, for enough warps (256 CTAs)
    const int d = std::min(ds, 32), m1 = N / d;
    float* fine = ds > 32 ? p->sprite + 3 * (size_t)p->M * p->M : p->sprite;
    const int T = N >= 512 || d > 8 ? 4 : 1;                 // a CTA's 8 T rows hold whole box sums
    GL_CUDA_TRY(launch_after(T == 4 ? sprite_bake<4> : sprite_bake<1>, dim3(N / 32, N / (8 * T)), kSpriteThreads, 0, st, p->psf, N,
                             p->spec, p->n_spec, p->lambda_ref, d, m1, p->energy, fine));
    if (ds > 32)
        GL_CUDA_TRY(launch_after(sprite_box, dim3((3 * p->M * p->M + kSpriteThreads - 1) / kSpriteThreads), kSpriteThreads, 0, st,
                                 fine, ds / 32, p->M, p->sprite));
    GL_CUDA_TRY(cudaGetLastError());
    g_last_launches = ds > 32 ? 4 : 3;
    return GL_OK;
}

extern "C" int gl_sprite_plan_splat(gl_sprite_plan* plan, const float* sources, int n_src, float sx_ds, float sy_ds,
                                    float px_mm_x, float px_mm_y, int rx, int ry, float gain, float* d_out_r,
                                    float* d_out_g, float* d_out_b, int width, int height, void* stream)
{
    if (!plan || n_src < 0 || (n_src > 0 && !sources) || !d_out_r || !d_out_g || !d_out_b || width < 1 || height < 1)
        return fail(GL_ERR_INVALID, "sprite_splat: bad arguments");
    SpritePlan* p = plan->p;
    if (p->M == 0) return fail(GL_ERR_INVALID, "sprite_splat: bake the sprite first");
    if (!(sx_ds > 0.0f) || !(sy_ds > 0.0f) || !(px_mm_x > 0.0f) || !(px_mm_y > 0.0f) || rx < 0 || ry < 0)
        return fail(GL_ERR_INVALID, "sprite_splat: pitches must be positive");
    if (n_src == 0) return GL_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (n_src > p->src_cap)
    {
        // the previous buffer may still be read by an earlier splat on this stream
        GL_CUDA_TRY(cudaStreamSynchronize(st));
        cudaFree(p->src);
        p->src = nullptr;
        p->src_cap = 0;
        GL_CUDA_TRY(cudaMalloc(&p->src, sizeof(StarSource) * n_src));
        p->src_cap = n_src;
    }
    GL_CUDA_TRY(cudaMemcpyAsync(p->src, sources, sizeof(StarSource) * n_src, cudaMemcpyHostToDevice, st));
    const long long total = (long long)n_src * (2LL * rx + 1) * (2LL * ry + 1);
    if (total > (1LL << 40)) return fail(GL_ERR_INVALID, "sprite_splat: footprint too large");
    const long long blocks = (total + kSpriteThreads - 1) / kSpriteThreads;
    if (blocks > 0x7fffffffLL) return fail(GL_ERR_INVALID, "sprite_splat: footprint too large");
    sprite_splat<<<(unsigned)blocks, kSpriteThreads, 0, st>>>(p->sprite, p->M, sx_ds, sy_ds, px_mm_x, px_mm_y, rx, ry,
                                                              p->src, n_src, gain, d_out_r, d_out_g, d_out_b, width,
                                                              height);
    GL_CUDA_TRY(cudaGetLastError());
    // the host sources are staged through pageable memory: the copy is done
    // when the call returns, so the caller may reuse them
    g_last_launches = 1;
    return GL_OK;
}

extern "C" int gl_sprite_splat_source(const float* d_sprite, int M, float px, float py, float r, float g, float b,
                                      float sx_ds, float sy_ds, float px_mm_x, float px_mm_y, int rx, int ry,
                                      float gain, float* d_out_r, float* d_out_g, float* d_out_b, int width,
                                      int height, void* stream)
{
    if (!d_sprite || M < 1 || !d_out_r || !d_out_g || !d_out_b || width < 1 || height < 1)
        return fail(GL_ERR_INVALID, "sprite_splat_source: bad arguments");
    if (!(sx_ds > 0.0f) || !(sy_ds > 0.0f) || !(px_mm_x > 0.0f) || !(px_mm_y > 0.0f) || rx < 0 || ry < 0)
        return fail(GL_ERR_INVALID, "sprite_splat_source: pitches must be positive");
    const long long total = (2LL * rx + 1) * (2LL * ry + 1);
    const long long blocks = (total + kSpriteThreads - 1) / kSpriteThreads;
    if (blocks > 0x7fffffffLL) return fail(GL_ERR_INVALID, "sprite_splat_source: footprint too large");
    const StarSource s{px, py, r, g, b};
    sprite_splat_one<<<(unsigned)blocks, kSpriteThreads, 0, (cudaStream_t)stream>>>(
        d_sprite, M, sx_ds, sy_ds, px_mm_x, px_mm_y, rx, ry, s, gain, d_out_r, d_out_g, d_out_b, width, height);
    GL_CUDA_TRY(cudaGetLastError());
    g_last_launches = 1;
    return GL_OK;
}

extern "C" int gl_sprite_plan_autocorr(gl_sprite_plan* plan, const float* d_pupil, int mc, float* d_C, int ldc,
                                       int rows, void* stream)
{
    if (!plan || !d_pupil || !d_C) return fail(GL_ERR_INVALID, "autocorr: bad arguments");
    SpritePlan* p = plan->p;
    const int N = p->N;
    if (mc < 0 || mc > N / 2 - 1) return fail(GL_ERR_INVALID, "autocorr: lag radius must lie in [0, N/2 - 1]");
    if (ldc < 2 * mc + 1 || rows < 2 * mc + 1)
        return fail(GL_ERR_INVALID, "autocorr: the output must hold (2 mc + 1)^2 lags");
    cudaStream_t st = (cudaStream_t)stream;
    GL_CUDA_TRY(cudaMemsetAsync(d_C, 0, sizeof(float) * (size_t)ldc * rows, st));
    GL_CUDA_TRY(cudaMemsetAsync(p->energy, 0, sizeof(double), st));
    // |FFT A|^2 (fftshifted) and its sum, as the sprite bake computes them
    GL_CUDA_TRY(sprite_psf(p, d_pupil, st));
    // the second transform, kept only at lags within +-mc
    const int pairs = mc / 2 + 1;
    GL_CUDA_TRY(sprite_cols(p, p->psf, pairs, true, st));
    GL_CUDA_TRY(sprite_rows<true>(p, pairs, d_C, mc, ldc, st));
    GL_CUDA_TRY(cudaGetLastError());
    // the bake's sprite no longer matches the PSF buffer's contents
    p->M = 0;
    g_last_launches = 4;
    return GL_OK;
}

extern "C" int gl_sprite_plan_read(gl_sprite_plan* plan, float* d_psf, float* d_sprite, double* energy, int* M,
                                   void* stream)
{
    if (!plan) return fail(GL_ERR_INVALID, "sprite_read: bad arguments");
    SpritePlan* p = plan->p;
    cudaStream_t st = (cudaStream_t)stream;
    const size_t NN = (size_t)p->N * p->N;
    if (d_psf) GL_CUDA_TRY(cudaMemcpyAsync(d_psf, p->psf, sizeof(float) * NN, cudaMemcpyDeviceToDevice, st));
    if (d_sprite && p->M)
        GL_CUDA_TRY(cudaMemcpyAsync(d_sprite, p->sprite, sizeof(float) * 3 * (size_t)p->M * p->M,
                                    cudaMemcpyDeviceToDevice, st));
    if (energy)
    {
        GL_CUDA_TRY(cudaMemcpyAsync(energy, p->energy, sizeof(double), cudaMemcpyDeviceToHost, st));
        GL_CUDA_TRY(cudaStreamSynchronize(st));
    }
    if (M) *M = p->M;
    return GL_OK;
}

extern "C" int gl_sprite_plan_destroy(gl_sprite_plan* plan)
{
    if (!plan) return GL_OK;
    cudaDeviceSynchronize();
    sprite_free(plan->p);
    delete plan;
    return GL_OK;
}
