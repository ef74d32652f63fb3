// gl_conv.cu — PSF / veil convolution of the flare image with a large FP32
// kernel, by FFT.
//
// The reference has no image convolution on this path (its veil is an
// analytic glare-spread sprite splatted per source, veil_render.cu:94-243);
// the flare path adds one: out_c = in_c (*) k, 'same' size, k centred.
//
// GB300 route:
//   * linear convolution by zero-padded circular convolution of size P x Q,
//     P, Q = the smallest 2^a 3^b >= image + kernel - 1 (2048 + 257 - 1 = 2304
//     = 16 * 16 * 9: no power-of-two padding waste);
//   * image and kernel are real: two rows of a plane make one complex row
//     transform, whose Hermitian parts are the two rows' spectra, so only
//     Q / 2 + 1 columns exist;
//   * Stockham FFTs with large radices held in registers (16, 8, 4, 2 and 9,
//     3), 16 elements per thread and one shared-memory buffer per transform
//     (gl_fft.cuh);
//   * three passes: (1) forward row FFTs of two row pairs per CTA, split into
//     the rows' half spectra; (2) per two columns: forward FFT, times the
//     kernel spectrum, inverse FFT.  The inverse takes the radices in the
//     opposite order, so the product stays in the registers that the last
//     forward butterfly left it in; (3) the row pairs' spectra rebuilt, inverse
//     row FFTs, the cropped W x H planes written from registers.
// The kernel spectrum (normalisation 1/(PQ) folded in) is built once per plan
// and stays resident.
// 2048^2 x 3 (*) 257^2: 0.325 -> 0.157 ms (two planes packed in one complex
// transform, the third alone, ping-pong buffers, 18 warps per SM before); the
// passes take 46, 73 and 43 us cold, issue slots half busy: bound by instruction
// issue and fetch (each CTA runs a long straight line of code once), not by HBM
// (15%) or shared memory (40%).  Passes 2 and 3 are launched while the pass before
// them drains (gl_launch.cuh): 100^2 (*) 7^2, calls back to back, 20.5 -> 16 us (18.5
// with the passes' form before half spectra), one alone 36 -> 31; 2048^2 (*) 257^2
// 163 -> 157.
#include "gl_internal.h"
#include "gl_fft.cuh"
#include "gl_launch.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

namespace gl {
namespace {

// HBM layout of the intermediate: column pairs.  Half spectrum (row r, column
// q <= Q / 2) of plane p at ((p G + q / 2) rows + r) 2 + q % 2, G = pairs of
// columns, rows even.  A column pair is one contiguous block for the column
// pass; a row pair's piece of it is one 32-byte sector for the row passes, and
// the pieces of a CTA's row pairs are neighbours.
__device__ __forceinline__ size_t pair_index(int plane, int G, int rows, int g, int r)
{
    return (((size_t)plane * G + g) * rows + r) * 2;
}

constexpr int kPairs = 2;          // row pairs per CTA in the row passes
constexpr int kColsPerCta = 2;     // one column pair per CTA in the column pass
constexpr int kConvThreads = 384;  // 3072 points, two transforms of them, 16 elements per thread
// Ping-pong stages (gl_fft.cuh) up to this length, in place above.  Three
// planes, calls back to back, ping-pong against in place: 162 x 486 points 18.4 /
// 34.9 us, 512 x 512 22.6 / 28.8, 512 x 729 27.0 / 31.1, 768 x 768 37.0 / 30.8, 972 x
// 972 52 / 45.
constexpr int kShort = 740;

struct ConvPlanes {
    const float* in[3];
    const float* add[3];           // a second layer summed in on load, or null
    float* out[3];
};

// Input of pass 1: rows row0 + 2 s and the next as one complex row.
struct RowLoad {
    const float* in;
    const float* add;
    int W, H, row0;
    __device__ __forceinline__ float2 operator()(int s, int i) const
    {
        const int r = row0 + 2 * s;
        float2 z = make_float2(0.0f, 0.0f);
        if (i < W)
        {
            const size_t o = (size_t)r * W + i;
            if (r < H) z.x = in[o];
            if (r + 1 < H) z.y = in[o + W];
            if (add)
            {
                if (r < H) z.x += add[o];
                if (r + 1 < H) z.y += add[o + W];
            }
        }
        return z;
    }
};

// Output of pass 3: real part -> row row0 + 2 s, imaginary part -> the next.
struct RowStore {
    float* out;
    int W, H, row0;
    __device__ __forceinline__ void operator()(int s, int i, float2 v) const
    {
        if (i >= W) return;
        const int r = row0 + 2 * s;
        const size_t o = (size_t)r * W + i;
        if (r < H) out[o] = v.x;
        if (r + 1 < H) out[o + W] = v.y;
    }
};

// A column pair: rows at and past `rows` are zero, and not written.
struct ColLoad {
    const float2* base;
    int rows;
    __device__ __forceinline__ float2 operator()(int s, int r) const
    {
        return r < rows ? base[2 * (size_t)r + s] : make_float2(0.0f, 0.0f);
    }
};
struct ColStore {
    float2* base;
    int rows;
    __device__ __forceinline__ void operator()(int s, int r, float2 v) const
    {
        if (r < rows) base[2 * (size_t)r + s] = v;
    }
};
struct ColMul {
    const float2* k;
    __device__ __forceinline__ float2 operator()(int s, int r, float2 v) const { return cmul(v, __ldg(k + 2 * (size_t)r + s)); }
};

// Pass 1: plane blockIdx.y, row pairs blockIdx.x kPairs + s.  Rows of width W,
// zero-padded to Q.
template <bool PP>
__global__ void __launch_bounds__(PP ? 512 : kConvThreads, PP ? 2 : 3) conv_rows_fwd(const __grid_constant__ ConvPlanes A, int W, int H, int rows, int G,
                                                                float2* __restrict__ buf, const __grid_constant__ FftDims d,
                                                                const float2* __restrict__ tw)
{
    extern __shared__ float2 sm[];
    float2* x = sm;
    float2* y = PP ? sm + kPairs * padded((size_t)d.n) : sm;
    const int Q = d.n, row0 = blockIdx.x * 2 * kPairs;
    const RowLoad load{A.in[blockIdx.y], A.add[blockIdx.y], W, H, row0};
    if (d.nrad == 0)
    {
        if (threadIdx.x < kPairs) x[fft_slot<kPairs, false>(0, threadIdx.x, Q)] = load(threadIdx.x, 0);
        __syncthreads();
    }
    else
        fft_any<kPairs, false, false, PP, true, false, PP>(x, y, d, 0, tw, load, FftNone{});
    for (int st = 1; st < d.nrad; ++st) fft_any<kPairs, false, false, PP, false, false, PP>(x, y, d, st, tw, FftNone{}, FftNone{});
    // Z = FFT(a + i b): FFT(a)[q] = (Z[q] + conj Z[Q - q]) / 2, FFT(b)[q] = (Z[q] - conj Z[Q - q]) / 2i;
    // the pairs of one column pair are neighbouring sectors, so they go to neighbouring threads
    for (int t = threadIdx.x; t < G * kPairs; t += blockDim.x)
    {
        const int g = t / kPairs, s = t % kPairs, r = row0 + 2 * s;
        if (r >= rows) continue;
        float2 a[2], b[2];
        #pragma unroll
        for (int c = 0; c < 2; ++c)
        {
            const int q = 2 * g + c;
            a[c] = b[c] = make_float2(0.0f, 0.0f);
            if (q <= Q / 2)
            {
                const float2 z = x[fft_slot<kPairs, false>(q, s, Q)], w = x[fft_slot<kPairs, false>(q == 0 ? 0 : Q - q, s, Q)];
                a[c] = make_float2(0.5f * (z.x + w.x), 0.5f * (z.y - w.y));
                b[c] = make_float2(0.5f * (z.y + w.y), 0.5f * (w.x - z.x));
            }
        }
        float4* o = reinterpret_cast<float4*>(buf + pair_index(blockIdx.y, G, rows, g, r));
        o[0] = make_float4(a[0].x, a[0].y, a[1].x, a[1].y);
        o[1] = make_float4(b[0].x, b[0].y, b[1].x, b[1].y);
    }
}

// The middle of a column: last forward stage, times the kernel spectrum, first
// inverse stage, all on the same registers (that stage's outputs j + p m are
// the inputs of the inverse's first stage of the same radix).
template <int R, bool FINE, class MUL>
__device__ __forceinline__ void conv_turn(float2 (&v)[R], int it, const FftStage& d, const MUL& mul)
{
    const int m = d.n / R, s = it % kColsPerCta, j = it / kColsPerCta;
    #pragma unroll
    for (int p = 0; p < R; ++p) v[p] = mul(s, j + p * m, v[p]);
    dft<R, FINE>(v, 1.0f);
}

template <int R, bool PP, bool FIRST, bool LAST, class LD, class MUL, class ST>
__device__ __forceinline__ void conv_middle(const float2* x, float2* y, const FftStage& d, const LD& ld, const MUL& mul,
                                            const ST& st)
{
    constexpr int NB = kColsPerCta;
    const int items = d.n / R * NB;
    FftStage back = d;
    back.Ls = 1;                       // the first stage of the way back
    if (PP)
    {
        for (int it = threadIdx.x; it < items; it += blockDim.x)
        {
            float2 v[R];
            fft_take<R, NB, true, false, FIRST, PP>(v, x, it, d, ld);
            conv_turn<R, PP>(v, it, d, mul);
            fft_put<R, NB, true, LAST>(v, y, it, back, st);
        }
    }
    else
    {
        constexpr int I = (16 + R - 1) / R;
        float2 v[I][R] = {};
        #pragma unroll
        for (int u = 0; u < I; ++u)
        {
            const int it = threadIdx.x + u * blockDim.x;
            if (it >= items) continue;
            fft_take<R, NB, true, false, FIRST, PP>(v[u], x, it, d, ld);
            conv_turn<R, PP>(v[u], it, d, mul);
        }
        if (!FIRST) __syncthreads();
        #pragma unroll
        for (int u = 0; u < I; ++u)
        {
            const int it = threadIdx.x + u * blockDim.x;
            if (it < items) fft_put<R, NB, true, LAST>(v[u], y, it, back, st);
        }
    }
    if (!LAST) __syncthreads();
}

template <bool PP, bool FIRST, bool LAST, class LD, class MUL, class ST>
__device__ __forceinline__ void conv_middle_any(float2*& x, float2*& y, const FftDims& d, const float2* __restrict__ tws,
                                                const LD& ld, const MUL& mul, const ST& st)
{
    const FftStage f = fft_stage_of(d, d.nrad - 1, tws);
    switch (d.rad[d.nrad - 1])
    {
    case 16: conv_middle<16, PP, FIRST, LAST>(x, y, f, ld, mul, st); break;
    case 9: conv_middle<9, PP, FIRST, LAST>(x, y, f, ld, mul, st); break;
    case 8: conv_middle<8, PP, FIRST, LAST>(x, y, f, ld, mul, st); break;
    case 4: conv_middle<4, PP, FIRST, LAST>(x, y, f, ld, mul, st); break;
    case 3: conv_middle<3, PP, FIRST, LAST>(x, y, f, ld, mul, st); break;
    default: conv_middle<2, PP, FIRST, LAST>(x, y, f, ld, mul, st); break;
    }
    float2* t = x;
    x = y;
    y = t;
}

// Pass 2: column pair blockIdx.x of plane blockIdx.y: forward FFT over P rows
// (rows >= rows_in are zero), times the kernel spectrum, inverse FFT; rows
// [0, rows_in) back in place.
template <bool PP>
__global__ void __launch_bounds__(PP ? 512 : kConvThreads, PP ? 2 : 3) conv_cols(float2* __restrict__ buf, const float2* __restrict__ khat,
                                                            int rows_in, int rows, int k_rows, int G, const __grid_constant__ FftDims d,
                                                            const __grid_constant__ FftDims di,
                                                            const float2* __restrict__ tw, const float2* __restrict__ twi)
{
    after_previous();
    extern __shared__ float2 sm[];
    float2* x = sm;
    float2* y = PP ? sm + padded((size_t)d.n * kColsPerCta) : sm;
    const int g = blockIdx.x;
    float2* base = buf + pair_index(blockIdx.y, G, rows, g, 0);
    const ColLoad load{base, rows_in};
    const ColStore store{base, rows_in};
    const ColMul mul{khat + pair_index(0, G, k_rows, g, 0)};
    if (d.nrad < 2)
    {
        if (d.nrad == 1) conv_middle_any<PP, true, true>(x, y, d, tw, load, mul, store);
        else if (threadIdx.x < 2) store(threadIdx.x, 0, mul(threadIdx.x, 0, load(threadIdx.x, 0)));
        return;
    }
    fft_any<2, true, false, PP, true, false, PP>(x, y, d, 0, tw, load, FftNone{});
    for (int st = 1; st + 1 < d.nrad; ++st) fft_any<2, true, false, PP, false, false, PP>(x, y, d, st, tw, FftNone{}, FftNone{});
    conv_middle_any<PP, false, false>(x, y, d, tw, FftNone{}, mul, FftNone{});
    for (int st = 1; st + 1 < d.nrad; ++st) fft_any<2, true, true, PP, false, false, PP>(x, y, di, st, twi, FftNone{}, FftNone{});
    fft_any<2, true, true, PP, false, true, PP>(x, y, di, d.nrad - 1, twi, FftNone{}, store);
}

// Pass 3: the row pairs' transforms Z = FFT(a) + i FFT(b) from the half
// spectra, inverse FFT, real part -> row r, imaginary part -> row r + 1.
template <bool PP>
__global__ void __launch_bounds__(PP ? 512 : kConvThreads, PP ? 2 : 3) conv_rows_inv(const float2* __restrict__ buf, const __grid_constant__ ConvPlanes A, int W,
                                                                int H, int rows, int G, const __grid_constant__ FftDims d,
                                                                const float2* __restrict__ tw)
{
    after_previous();
    extern __shared__ float2 sm[];
    float2* x = sm;
    float2* y = PP ? sm + kPairs * padded((size_t)d.n) : sm;
    const int Q = d.n, row0 = blockIdx.x * 2 * kPairs;
    float* out = A.out[blockIdx.y];
    for (int t = threadIdx.x; t < G * kPairs; t += blockDim.x)
    {
        const int g = t / kPairs, s = t % kPairs, r = row0 + 2 * s;
        float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a;
        if (r < rows)
        {
            const float4* p = reinterpret_cast<const float4*>(buf + pair_index(blockIdx.y, G, rows, g, r));
            a = __ldg(p);
            b = __ldg(p + 1);
        }
        #pragma unroll
        for (int c = 0; c < 2; ++c)
        {
            const int q = 2 * g + c;
            if (q > Q / 2) continue;
            const float2 u = c ? make_float2(a.z, a.w) : make_float2(a.x, a.y);
            const float2 w = c ? make_float2(b.z, b.w) : make_float2(b.x, b.y);
            x[fft_slot<kPairs, false>(q, s, Q)] = make_float2(u.x - w.y, u.y + w.x);
            // conj U + i conj W at Q - q; the middle of an even Q is its own mirror
            if (q > 0 && 2 * q != Q) x[fft_slot<kPairs, false>(Q - q, s, Q)] = make_float2(u.x + w.y, w.x - u.y);
        }
    }
    __syncthreads();
    const RowStore store{out, W, H, row0};
    if (d.nrad == 0)
    {
        if (threadIdx.x < kPairs) store(threadIdx.x, 0, x[fft_slot<kPairs, false>(0, threadIdx.x, Q)]);
        return;
    }
    for (int st = 0; st + 1 < d.nrad; ++st) fft_any<kPairs, false, true, PP, false, false, PP>(x, y, d, st, tw, FftNone{}, FftNone{});
    fft_any<kPairs, false, true, PP, false, true, PP>(x, y, d, d.nrad - 1, tw, FftNone{}, store);
}

// ---- kernel spectrum, once per plan ----------------------------------------------
// In FP64 and rounded once: a third of the rounding of forward transform, product
// and inverse was the kernel's own float transform, the same in every call (noise, 2048^2
// (*) 257^2: 3.7e-7 off 64 bits with it, 2.8e-7 without).  One CTA a row of the
// kernel, then one a column: Stockham stages of radix 4, 3, 2 between two arrays
// in shared memory.  A plan for 2304^2 points takes the time it took with the float
// transform (3.2 ms, most of it the tables).
constexpr int kSpecThreads = 256;

// exp(-2 pi i t / n), t < n
__global__ void spec_circle(int n, double2* __restrict__ tw)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    double s, c;
    sincospi(2.0 * (double)t / (double)n, &s, &c);
    tw[t] = make_double2(c, -s);
}

template <int R>
__device__ __forceinline__ void spec_stage(const double2* x, double2* y, int n, int Ls, const double2* __restrict__ tw)
{
    const int m = n / R;
    for (int j = threadIdx.x; j < m; j += kSpecThreads)
    {
        const int g = j / Ls, k = j - g * Ls;
        double2 v[R];
        #pragma unroll
        for (int q = 0; q < R; ++q)
        {
            const double2 a = x[j + q * m], w = tw[q * k * (m / Ls)];
            v[q] = make_double2(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
        }
        #pragma unroll
        for (int p = 0; p < R; ++p)
        {
            double2 o = v[0];
            #pragma unroll
            for (int q = 1; q < R; ++q)
            {
                const double2 w = tw[p * q % R * m];
                o.x += v[q].x * w.x - v[q].y * w.y;
                o.y += v[q].x * w.y + v[q].y * w.x;
            }
            y[g * Ls * R + k + p * Ls] = o;
        }
    }
    __syncthreads();
}

// The transform of x; returns the array that holds it (x or y).
__device__ const double2* spec_fft(double2* x, double2* y, int n, const double2* __restrict__ tw)
{
    __syncthreads();
    for (int Ls = 1; Ls < n;)
    {
        const int left = n / Ls, R = left % 4 == 0 ? 4 : (left % 2 == 0 ? 2 : 3);
        if (R == 4) spec_stage<4>(x, y, n, Ls, tw);
        else if (R == 3) spec_stage<3>(x, y, n, Ls, tw);
        else spec_stage<2>(x, y, n, Ls, tw);
        double2* t = x;
        x = y;
        y = t;
        Ls *= R;
    }
    return x;
}

// Row blockIdx.x of the kernel, its centre at column 0, wrapped: its half spectrum
// (cols of them, zero past Q / 2).
__global__ void __launch_bounds__(kSpecThreads) spec_rows(const float* __restrict__ k, int kw, int Q, int cols, double norm,
                                                          const double2* __restrict__ tw, double2* __restrict__ a)
{
    extern __shared__ double2 arrays[];
    const float* row = k + (size_t)blockIdx.x * kw;
    for (int c = threadIdx.x; c < Q; c += kSpecThreads)
    {
        const int v = (c + kw / 2) % Q;
        arrays[c] = make_double2(v < kw ? (double)row[v] * norm : 0.0, 0.0);
    }
    const double2* r = spec_fft(arrays, arrays + Q, Q, tw);
    for (int q = threadIdx.x; q < cols; q += kSpecThreads)
        a[(size_t)blockIdx.x * cols + q] = q <= Q / 2 ? r[q] : make_double2(0.0, 0.0);
}

// Column blockIdx.x of the rows' spectra, the centre row at row 0, wrapped: its
// transform to the column pairs of the intermediate (pair_index).
__global__ void __launch_bounds__(kSpecThreads) spec_cols(const double2* __restrict__ a, int kh, int P, int cols, int k_rows,
                                                          const double2* __restrict__ tw, float2* __restrict__ khat)
{
    extern __shared__ double2 arrays[];
    const int q = blockIdx.x;
    for (int y = threadIdx.x; y < P; y += kSpecThreads)
    {
        const int u = (y + kh / 2) % P;
        arrays[y] = u < kh ? a[(size_t)u * cols + q] : make_double2(0.0, 0.0);
    }
    const double2* r = spec_fft(arrays, arrays + P, P, tw);
    for (int y = threadIdx.x; y < P; y += kSpecThreads)
        khat[((size_t)(q >> 1) * k_rows + y) * 2 + (q & 1)] = make_float2((float)r[y].x, (float)r[y].y);
}

int good_size(int need)
{
    int best = 1 << 30;
    for (long long p2 = 1; p2 < (1LL << 31); p2 *= 2)
        for (long long v = p2; v < (1LL << 31); v *= 3)
        {
            if (v >= need && v < best) best = (int)v;
            if (v >= need) break;
        }
    return best;
}

}  // namespace

struct ConvPlan {
    int W = 0, H = 0, KW = 0, KH = 0, P = 0, Q = 0;
    int G = 0, rows = 0, k_rows = 0;  // column pairs, rows of the intermediate and of the kernel spectrum (even)
    float2* khat = nullptr;   // column pairs, k_rows rows
    float2* buf = nullptr;    // column pairs, 3 planes x rows
    float2* tw_q = nullptr;   // stage twiddles: rows, columns, columns in the opposite order
    float2* tw_p = nullptr;
    float2* tw_pi = nullptr;
    FftDims dq{}, dp{}, dpi{};
    size_t smem_row = 0, smem_col = 0;
    int thr_row = 0, thr_col = 0;
    bool pp_row = false, pp_col = false;      // ping-pong stages
};

}  // namespace gl

struct gl_conv_plan { gl::ConvPlan* p; };

using namespace gl;

static void conv_free(ConvPlan* p)
{
    cudaFree(p->khat);
    cudaFree(p->buf);
    cudaFree(p->tw_q);
    cudaFree(p->tw_p);
    cudaFree(p->tw_pi);
    delete p;
}

// The kernel's spectrum (centre at the origin, so the circular convolution lands
// 'same'-aligned; 1 / (P Q) folded in) into p->khat.
static cudaError_t conv_spectrum(const ConvPlan* p, const float* h_kernel, cudaStream_t st)
{
    const size_t nk = (size_t)p->KH * p->KW, cols = 2 * (size_t)p->G, cells = p->KH * cols;
    const size_t k_at = sizeof(double2) * (cells + (size_t)p->Q + p->P);
    const size_t smem_q = 2 * sizeof(double2) * p->Q, smem_p = 2 * sizeof(double2) * p->P;
    char* block = nullptr;         // the rows' spectra, the circles of both axes, the kernel
    cudaError_t e = cudaMalloc(&block, k_at + sizeof(float) * nk);
    auto chk = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
    double2 *a = reinterpret_cast<double2*>(block), *twq = a + cells, *twp = twq + p->Q;
    float* k = reinterpret_cast<float*>(block + k_at);
    if (e == cudaSuccess) chk((cudaError_t)raise_smem_limit((const void*)spec_rows, smem_q));
    if (e == cudaSuccess) chk((cudaError_t)raise_smem_limit((const void*)spec_cols, smem_p));
    if (e == cudaSuccess) chk(cudaMemcpyAsync(k, h_kernel, sizeof(float) * nk, cudaMemcpyHostToDevice, st));
    if (e == cudaSuccess)
    {
        const double norm = 1.0 / ((double)p->P * (double)p->Q);
        spec_circle<<<(p->Q + 255) / 256, 256, 0, st>>>(p->Q, twq);
        spec_circle<<<(p->P + 255) / 256, 256, 0, st>>>(p->P, twp);
        spec_rows<<<p->KH, kSpecThreads, smem_q, st>>>(k, p->KW, p->Q, (int)cols, norm, twq, a);
        spec_cols<<<(unsigned)cols, kSpecThreads, smem_p, st>>>(a, p->KH, p->P, (int)cols, p->k_rows, twp, p->khat);
        chk(cudaGetLastError());
    }
    chk(cudaStreamSynchronize(st));
    cudaFree(block);
    return e;
}

extern "C" int gl_conv2d_plan_create(int width, int height, const float* h_kernel, int kw, int kh, void* stream,
                                     gl_conv_plan** out)
{
    if (!out || !h_kernel) return fail(GL_ERR_INVALID, "conv2d_plan_create: null argument");
    if (width <= 0 || height <= 0 || kw <= 0 || kh <= 0 || (kw % 2) == 0 || (kh % 2) == 0)
        return fail(GL_ERR_INVALID, "conv2d_plan_create: positive sizes and an odd (centred) kernel required");
    ConvPlan* p = new ConvPlan();
    p->W = width; p->H = height; p->KW = kw; p->KH = kh;
    p->Q = good_size(width + kw - 1);
    p->P = good_size(height + kh - 1);
    if (p->P > 3072 || p->Q > 3072)
    {
        delete p;
        return fail(GL_ERR_INVALID, "conv2d_plan_create: padded transform above 3072 points per axis");
    }
    p->G = (p->Q / 2 + 1 + 1) / 2;
    p->rows = (p->H + 1) / 2 * 2;
    p->k_rows = (p->P + 1) / 2 * 2;
    p->dq = make_dims(p->Q);
    p->dp = make_dims(p->P);
    p->dpi = reversed(p->dp);
    p->pp_row = p->Q <= kShort;
    p->pp_col = p->P <= kShort;
    p->smem_row = (p->pp_row ? 2 : 1) * kPairs * padded((size_t)p->Q) * sizeof(float2);
    p->smem_col = (p->pp_col ? 2 : 1) * padded((size_t)p->P * kColsPerCta) * sizeof(float2);
    p->thr_row = fft_threads(p->Q, kPairs, p->pp_row);
    p->thr_col = fft_threads(p->P, kColsPerCta, p->pp_col);
    cudaStream_t st = (cudaStream_t)stream;
    const std::vector<float2> twq = stage_twiddles(p->dq), twp = stage_twiddles(p->dp), twi = stage_twiddles(p->dpi);
    cudaError_t e = cudaSuccess;
    auto chk = [&](cudaError_t x) { if (e == cudaSuccess) e = x; };
    chk(cudaMalloc(&p->khat, sizeof(float2) * 2 * (size_t)p->G * p->k_rows));
    chk(cudaMalloc(&p->buf, sizeof(float2) * 3 * 2 * (size_t)p->G * p->rows));
    chk(cudaMalloc(&p->tw_q, sizeof(float2) * twq.size()));
    chk(cudaMalloc(&p->tw_p, sizeof(float2) * twp.size()));
    chk(cudaMalloc(&p->tw_pi, sizeof(float2) * twi.size()));
    chk((cudaError_t)raise_smem_limit(p->pp_col ? (const void*)conv_cols<true> : (const void*)conv_cols<false>, p->smem_col));
    chk((cudaError_t)raise_smem_limit(p->pp_row ? (const void*)conv_rows_fwd<true> : (const void*)conv_rows_fwd<false>, p->smem_row));
    chk((cudaError_t)raise_smem_limit(p->pp_row ? (const void*)conv_rows_inv<true> : (const void*)conv_rows_inv<false>, p->smem_row));
    if (e == cudaSuccess)
    {
        chk(cudaMemcpyAsync(p->tw_q, twq.data(), sizeof(float2) * twq.size(), cudaMemcpyHostToDevice, st));
        chk(cudaMemcpyAsync(p->tw_p, twp.data(), sizeof(float2) * twp.size(), cudaMemcpyHostToDevice, st));
        chk(cudaMemcpyAsync(p->tw_pi, twi.data(), sizeof(float2) * twi.size(), cudaMemcpyHostToDevice, st));
    }
    // (waits for the tables' copies too)
    if (e == cudaSuccess) chk(conv_spectrum(p, h_kernel, st));
    if (e != cudaSuccess)
    {
        conv_free(p);
        return fail(e == cudaErrorMemoryAllocation ? GL_ERR_OOM : GL_ERR_CUDA, std::string("conv2d_plan_create: ") + cudaGetErrorString(e));
    }
    *out = new gl_conv_plan{p};
    return GL_OK;
}

extern "C" int gl_conv2d_plan_execute2(gl_conv_plan* plan, const float* d_in_r, const float* d_in_g,
                                       const float* d_in_b, const float* d_add_r, const float* d_add_g,
                                       const float* d_add_b, float* d_out_r, float* d_out_g, float* d_out_b,
                                       void* stream)
{
    if (!plan || !d_in_r || !d_in_g || !d_in_b || !d_out_r || !d_out_g || !d_out_b)
        return fail(GL_ERR_INVALID, "conv2d_plan_execute: null argument");
    if ((d_add_r == nullptr) != (d_add_g == nullptr) || (d_add_r == nullptr) != (d_add_b == nullptr))
        return fail(GL_ERR_INVALID, "conv2d_plan_execute: the added layer needs all three planes or none");
    ConvPlan* p = plan->p;
    cudaStream_t st = (cudaStream_t)stream;
    const ConvPlanes A{{d_in_r, d_in_g, d_in_b}, {d_add_r, d_add_g, d_add_b}, {d_out_r, d_out_g, d_out_b}};
    const dim3 rb((unsigned)((p->rows + 2 * kPairs - 1) / (2 * kPairs)), 3);
    const dim3 cb(p->G, 3);
    if (p->pp_row) conv_rows_fwd<true><<<rb, p->thr_row, p->smem_row, st>>>(A, p->W, p->H, p->rows, p->G, p->buf, p->dq, p->tw_q);
    else conv_rows_fwd<false><<<rb, p->thr_row, p->smem_row, st>>>(A, p->W, p->H, p->rows, p->G, p->buf, p->dq, p->tw_q);
    GL_CUDA_TRY(launch_after(p->pp_col ? conv_cols<true> : conv_cols<false>, cb, p->thr_col, p->smem_col, st, p->buf, p->khat,
                             p->H, p->rows, p->k_rows, p->G, p->dp, p->dpi, p->tw_p, p->tw_pi));
    GL_CUDA_TRY(launch_after(p->pp_row ? conv_rows_inv<true> : conv_rows_inv<false>, rb, p->thr_row, p->smem_row, st, p->buf, A,
                             p->W, p->H, p->rows, p->G, p->dq, p->tw_q));
    GL_CUDA_TRY(cudaGetLastError());
    g_last_launches = 3;
    return GL_OK;
}

extern "C" int gl_conv2d_plan_execute(gl_conv_plan* plan, const float* d_in_r, const float* d_in_g, const float* d_in_b,
                                      float* d_out_r, float* d_out_g, float* d_out_b, void* stream)
{
    return gl_conv2d_plan_execute2(plan, d_in_r, d_in_g, d_in_b, nullptr, nullptr, nullptr, d_out_r, d_out_g, d_out_b,
                                   stream);
}

extern "C" int gl_conv2d_plan_info(const gl_conv_plan* plan, int* P, int* Q)
{
    if (!plan) return fail(GL_ERR_INVALID, "conv2d_plan_info: null plan");
    if (P) *P = plan->p->P;
    if (Q) *Q = plan->p->Q;
    return GL_OK;
}

extern "C" int gl_conv2d_plan_destroy(gl_conv_plan* plan)
{
    if (!plan) return GL_OK;
    conv_free(plan->p);
    delete plan;
    return GL_OK;
}
