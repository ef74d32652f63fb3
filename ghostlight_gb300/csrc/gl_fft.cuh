// gl_fft.cuh — shared-memory Stockham FFT building blocks (complex float):
// radix 16 / 9 / 8 / 4 / 3 / 2 butterflies held in registers, one stage per
// pass over shared memory, twiddles from a table computed in FP64.  Used by
// the image convolution (gl_conv.cu) and the starburst sprite (gl_sprite.cu).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

namespace gl {

// Radix plan of one transform length n = 2^a 3^b: per stage its radix r, the
// span Ls of the sub-transforms done before it, ceil(2^32 / Ls) and
// ceil(2^32 / (n / r)) for exact divisions by multiply-high (indices < 2^16),
// and the stage's place in the stage tables (stage_twiddles).
struct FftDims {
    int n, nrad;                       // at most five radices below 2^14
    int rad[6];
    int ls[6];
    uint32_t lmag[6], mmag[6];
    int twoff[7];
};

__device__ __forceinline__ float2 cmul(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// (sign i) * a
__device__ __forceinline__ float2 cis(float2 a, float sign) { return make_float2(-sign * a.y, sign * a.x); }

// a times the constant c + sign i s.  FINE: the constant in two floats each; one
// rounded to one float is off by up to 3e-8 in every product with it, the same way
// every time.  Error of a transform of 1024^2 noise against 64 bits 2.0e-7, FINE
// 1.65e-7.  The sprite's transforms take it (1 to 2 us each, code to fetch) and the
// convolution's short ones; its long ones would be 4 % slower (161 -> 168 us).
template <bool FINE>
__device__ __forceinline__ float2 cmul_const(float2 a, double c, double s, float sign)
{
    const float ch = (float)c, sh = sign * (float)s;
    if (!FINE) return cmul(a, make_float2(ch, sh));
    const float cl = (float)(c - (double)(float)c), sl = sign * (float)(s - (double)(float)s);
    return make_float2(fmaf(a.x, ch, fmaf(-a.y, sh, fmaf(a.x, cl, -a.y * sl))),
                       fmaf(a.x, sh, fmaf(a.y, ch, fmaf(a.x, sl, a.y * cl))));
}

// Padded shared-memory index: one spare word per 16 elements, so a warp
// writing 16-element runs at a stride of 16 hits 16 different banks.
__device__ __forceinline__ int pad(int i) { return i + (i >> 4); }
__host__ __device__ inline size_t padded(size_t n) { return n + (n >> 4) + 1; }

// ---- small DFTs in registers: X[p] = sum_q v[q] w^(pq), w = exp(sign 2 pi i / R) ----
__device__ __forceinline__ void dft2(float2& a, float2& b)
{
    const float2 t = a;
    a = cadd(t, b);
    b = csub(t, b);
}

__device__ __forceinline__ void dft4(float2& v0, float2& v1, float2& v2, float2& v3, float sign)
{
    const float2 t0 = cadd(v0, v2), t1 = csub(v0, v2), t2 = cadd(v1, v3), t3 = cis(csub(v1, v3), sign);
    v0 = cadd(t0, t2);
    v2 = csub(t0, t2);
    v1 = cadd(t1, t3);
    v3 = csub(t1, t3);
}

template <bool FINE>
__device__ __forceinline__ void dft3(float2& v0, float2& v1, float2& v2, float sign)
{
    constexpr double c = 0.86602540378443864676;   // sqrt(3)/2
    constexpr float ch = (float)c, cl = FINE ? (float)(c - (double)ch) : 0.0f;
    const float2 t1 = cadd(v1, v2);
    const float2 t2 = csub(v1, v2);
    const float2 base = make_float2(v0.x - 0.5f * t1.x, v0.y - 0.5f * t1.y);
    const float2 rot = cis(FINE ? make_float2(fmaf(ch, t2.x, cl * t2.x), fmaf(ch, t2.y, cl * t2.y)) : make_float2(ch * t2.x, ch * t2.y), sign);
    v0 = cadd(v0, t1);
    v1 = cadd(base, rot);
    v2 = csub(base, rot);
}

// 8 = 2 x 4: q = q1 + 2 q2; inner DFT4 over q2, twiddle w8^(q1 p1), outer DFT2.
template <bool FINE>
__device__ __forceinline__ void dft8(float2 (&v)[8], float sign)
{
    constexpr double h = 0.70710678118654752440;
    dft4(v[0], v[2], v[4], v[6], sign);   // q1 = 0 -> A0[p1] at v[0], v[2], v[4], v[6]
    dft4(v[1], v[3], v[5], v[7], sign);   // q1 = 1 -> A1[p1]
    v[3] = cmul_const<FINE>(v[3], h, h, sign);
    v[5] = cis(v[5], sign);
    v[7] = cmul_const<FINE>(v[7], -h, h, sign);
    float2 x[8];
    #pragma unroll
    for (int p1 = 0; p1 < 4; ++p1)
    {
        x[p1] = cadd(v[2 * p1], v[2 * p1 + 1]);
        x[p1 + 4] = csub(v[2 * p1], v[2 * p1 + 1]);
    }
    #pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = x[i];
}

// 16 = 4 x 4: q = q1 + 4 q2; inner DFT4 over q2, twiddle w16^(q1 p1), outer DFT4 over q1.
template <bool FINE>
__device__ __forceinline__ void dft16(float2 (&v)[16], float sign)
{
    constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173, h = 0.70710678118654752440;
    #pragma unroll
    for (int q1 = 0; q1 < 4; ++q1) dft4(v[q1], v[q1 + 4], v[q1 + 8], v[q1 + 12], sign);
    // v[q1 + 4 p1] = A[q1][p1]; multiply by w16^(q1 p1)
    v[5] = cmul_const<FINE>(v[5], c1, s1, sign);     // q1 1, p1 1: k 1
    v[9] = cmul_const<FINE>(v[9], h, h, sign);       // 1,2: k 2
    v[13] = cmul_const<FINE>(v[13], s1, c1, sign);   // 1,3: k 3
    v[6] = cmul_const<FINE>(v[6], h, h, sign);       // 2,1: k 2
    v[10] = cis(v[10], sign);                // 2,2: k 4
    v[14] = cmul_const<FINE>(v[14], -h, h, sign);    // 2,3: k 6
    v[7] = cmul_const<FINE>(v[7], s1, c1, sign);     // 3,1: k 3
    v[11] = cmul_const<FINE>(v[11], -h, h, sign);    // 3,2: k 6
    v[15] = cmul_const<FINE>(v[15], -c1, -s1, sign); // 3,3: k 9
    #pragma unroll
    for (int p1 = 0; p1 < 4; ++p1) dft4(v[4 * p1], v[4 * p1 + 1], v[4 * p1 + 2], v[4 * p1 + 3], sign);
    // now v[4 p1 + p2] = X[p1 + 4 p2]: transpose the 4 x 4 index
    float2 x[16];
    #pragma unroll
    for (int p1 = 0; p1 < 4; ++p1)
        #pragma unroll
        for (int p2 = 0; p2 < 4; ++p2) x[p1 + 4 * p2] = v[4 * p1 + p2];
    #pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = x[i];
}

// 9 = 3 x 3: q = q1 + 3 q2; inner DFT3 over q2, twiddle w9^(q1 p1), outer DFT3 over q1.
template <bool FINE>
__device__ __forceinline__ void dft9(float2 (&v)[9], float sign)
{
    constexpr double c1 = 0.76604444311897803520, s1 = 0.64278760968653932632;   // 2 pi / 9
    constexpr double c2 = 0.17364817766693034885, s2 = 0.98480775301220805936;   // 4 pi / 9
    constexpr double c4 = -0.93969262078590838405, s4 = 0.34202014332566873304; // 8 pi / 9
    #pragma unroll
    for (int q1 = 0; q1 < 3; ++q1) dft3<FINE>(v[q1], v[q1 + 3], v[q1 + 6], sign);
    v[4] = cmul_const<FINE>(v[4], c1, s1, sign);   // q1 1, p1 1: k 1
    v[7] = cmul_const<FINE>(v[7], c2, s2, sign);   // 1,2: k 2
    v[5] = cmul_const<FINE>(v[5], c2, s2, sign);   // 2,1: k 2
    v[8] = cmul_const<FINE>(v[8], c4, s4, sign);   // 2,2: k 4
    #pragma unroll
    for (int p1 = 0; p1 < 3; ++p1) dft3<FINE>(v[3 * p1], v[3 * p1 + 1], v[3 * p1 + 2], sign);
    float2 x[9];
    #pragma unroll
    for (int p1 = 0; p1 < 3; ++p1)
        #pragma unroll
        for (int p2 = 0; p2 < 3; ++p2) x[p1 + 3 * p2] = v[3 * p1 + p2];
    #pragma unroll
    for (int i = 0; i < 9; ++i) v[i] = x[i];
}

template <int R, bool FINE>
__device__ __forceinline__ void dft(float2 (&v)[R], float sign)
{
    if constexpr (R == 2) dft2(v[0], v[1]);
    else if constexpr (R == 3) dft3<FINE>(v[0], v[1], v[2], sign);
    else if constexpr (R == 4) dft4(v[0], v[1], v[2], v[3], sign);
    else if constexpr (R == 8) dft8<FINE>(v, sign);
    else if constexpr (R == 9) dft9<FINE>(v, sign);
    else dft16<FINE>(v, sign);
}

// ---- stages between registers and shared memory ---------------------------------
// Two forms.  In place (PP = false): every thread holds 16 elements (one
// radix-16 butterfly, two of radix 8 or 9, ...), reads a stage's inputs, waits,
// and writes the outputs to the same shared buffer: one buffer per transform
// where ping-pong needs two, so twice the CTAs fit an SM; blockDim >= n NB / 16.
// Ping-pong (PP = true): a loop over butterflies from one buffer to the other,
// a fraction of the code, for short transforms, whose time is latency and
// instruction fetch.  The first stage can read its inputs straight from global
// memory, the last write its outputs there (both are in natural order across
// threads).  Twiddles come from per-stage tables in the order the threads read
// them (a whole-circle table is read with strides that take a line per lane).
// NB sequences; INTER: element i of sequence s at pad(i NB + s), else at
// s padded(n) + pad(i).
template <int NB, bool INTER>
__device__ __forceinline__ int fft_slot(int i, int s, int n)
{
    return INTER ? pad(i * NB + s) : s * (int)padded((size_t)n) + pad(i);
}

struct FftNone {
    __device__ float2 operator()(int, int) const { return make_float2(0.0f, 0.0f); }
    __device__ void operator()(int, int, float2) const {}
};

// What one stage needs of the dims.
struct FftStage {
    int n, Ls;
    uint32_t lmag, mmag;
    const float2* tw;
};

__device__ __forceinline__ FftStage fft_stage_of(const FftDims& d, int stage, const float2* tws)
{
    return {d.n, d.ls[stage], d.lmag[stage], d.mmag[stage], tws + d.twoff[stage]};
}

// The item `it` of a stage with m = n / R butterflies per sequence: its
// sequence and butterfly.
template <int NB, bool INTER>
__device__ __forceinline__ void fft_item(int it, int m, uint32_t mmag, int& s, int& j)
{
    if (INTER) { s = it % NB; j = it / NB; }
    else if (NB == 1) { s = 0; j = it; }
    else
    {
        s = m > 1 ? (int)__umulhi((uint32_t)it, mmag) : it;
        j = it - s * m;
    }
}

// v[q] *= w^q, w = exp(-+2 pi i k / (Ls R)), every power from the table (a
// product of two entries carries twice the error of one), two of them in each
// 16-byte read.
template <int R>
__device__ __forceinline__ void fft_twiddle(float2 (&v)[R], int k, int Ls, const float2* __restrict__ tw, bool inv)
{
    const float4* t = reinterpret_cast<const float4*>(tw) + k;
    #pragma unroll
    for (int p = 0; p < R / 2; ++p)
    {
        const float4 w = __ldg(t + p * Ls);
        const int q = 2 * p + 1;
        v[q] = cmul(v[q], make_float2(w.x, inv ? -w.y : w.y));
        if (q + 1 < R) v[q + 1] = cmul(v[q + 1], make_float2(w.z, inv ? -w.w : w.w));
    }
}

// The butterfly of item `it`: inputs from ld (FIRST) or shared memory, twiddled, transformed.
template <int R, int NB, bool INTER, bool INV, bool FIRST, bool FINE, class LD>
__device__ __forceinline__ void fft_take(float2 (&v)[R], const float2* x, int it, const FftStage& d, const LD& ld)
{
    const int n = d.n, m = n / R;
    int s, j;
    fft_item<NB, INTER>(it, m, d.mmag, s, j);
    #pragma unroll
    for (int q = 0; q < R; ++q) v[q] = FIRST ? ld(s, j + q * m) : x[fft_slot<NB, INTER>(j + q * m, s, n)];
    if (d.Ls > 1) fft_twiddle<R>(v, j - (int)__umulhi((uint32_t)j, d.lmag) * d.Ls, d.Ls, d.tw, INV);
    dft<R, FINE>(v, INV ? 1.0f : -1.0f);
}

// Its outputs, to st (LAST) or shared memory.
template <int R, int NB, bool INTER, bool LAST, class ST>
__device__ __forceinline__ void fft_put(const float2 (&v)[R], float2* y, int it, const FftStage& d, const ST& st)
{
    const int n = d.n, m = n / R;
    int s, j;
    fft_item<NB, INTER>(it, m, d.mmag, s, j);
    const int g = d.Ls > 1 ? (int)__umulhi((uint32_t)j, d.lmag) : j;
    const int ob = g * d.Ls * R + (j - g * d.Ls);
    #pragma unroll
    for (int p = 0; p < R; ++p)
    {
        if (LAST) st(s, ob + p * d.Ls, v[p]);
        else y[fft_slot<NB, INTER>(ob + p * d.Ls, s, n)] = v[p];
    }
}

// One stage, x -> y (in place: the same buffer).  FIRST: inputs from ld(s, i);
// LAST: outputs to st(s, i, value).  Ends on a barrier unless LAST.  In place,
// the elements start as zeros: set under a condition only, they count as live
// from the kernel's start and every radix's stage adds to the spills.
template <int R, int NB, bool INTER, bool INV, bool PP, bool FIRST, bool LAST, bool FINE, class LD, class ST>
__device__ __forceinline__ void fft_stage(const float2* x, float2* y, const FftStage& d, const LD& ld, const ST& st)
{
    const int items = d.n / R * NB;
    if (PP)
    {
        for (int it = threadIdx.x; it < items; it += blockDim.x)
        {
            float2 v[R];
            fft_take<R, NB, INTER, INV, FIRST, FINE>(v, x, it, d, ld);
            fft_put<R, NB, INTER, LAST>(v, y, it, d, st);
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
            if (it < items) fft_take<R, NB, INTER, INV, FIRST, FINE>(v[u], x, it, d, ld);
        }
        if (!FIRST) __syncthreads();
        #pragma unroll
        for (int u = 0; u < I; ++u)
        {
            const int it = threadIdx.x + u * blockDim.x;
            if (it < items) fft_put<R, NB, INTER, LAST>(v[u], y, it, d, st);
        }
    }
    if (!LAST) __syncthreads();
}

// The stage of whatever radix; leaves the result's buffer in x (in place: y == x).
template <int NB, bool INTER, bool INV, bool PP, bool FIRST, bool LAST, bool FINE, class LD, class ST>
__device__ __forceinline__ void fft_any(float2*& x, float2*& y, const FftDims& d, int stage,
                                        const float2* __restrict__ tws, const LD& ld, const ST& st)
{
    const FftStage f = fft_stage_of(d, stage, tws);
    switch (d.rad[stage])
    {
    case 16: fft_stage<16, NB, INTER, INV, PP, FIRST, LAST, FINE>(x, y, f, ld, st); break;
    case 9: fft_stage<9, NB, INTER, INV, PP, FIRST, LAST, FINE>(x, y, f, ld, st); break;
    case 8: fft_stage<8, NB, INTER, INV, PP, FIRST, LAST, FINE>(x, y, f, ld, st); break;
    case 4: fft_stage<4, NB, INTER, INV, PP, FIRST, LAST, FINE>(x, y, f, ld, st); break;
    case 3: fft_stage<3, NB, INTER, INV, PP, FIRST, LAST, FINE>(x, y, f, ld, st); break;
    default: fft_stage<2, NB, INTER, INV, PP, FIRST, LAST, FINE>(x, y, f, ld, st); break;
    }
    float2* t = x;
    x = y;
    y = t;
}

// Threads of a CTA that holds NB transforms of n points.
inline int fft_threads(int n, int nb, bool pp)
{
    return std::min(pp ? 512 : 1024, std::max(pp ? 64 : 32, pp ? (n * nb / 4 + 31) / 32 * 32 : (n * nb + 511) / 512 * 32));
}

// Spans, division constants and table places of the radices in d.
inline void set_spans(FftDims& d)
{
    int Ls = 1, off = 0;
    for (int s = 0; s < d.nrad; ++s)
    {
        const int m = d.n / d.rad[s];
        d.ls[s] = Ls;
        d.lmag[s] = Ls > 1 ? (uint32_t)((((uint64_t)1 << 32) + Ls - 1) / Ls) : 0u;
        d.mmag[s] = m > 1 ? (uint32_t)((((uint64_t)1 << 32) + m - 1) / m) : 0u;
        d.twoff[s] = off;
        if (Ls > 1) off += d.rad[s] / 2 * 2 * Ls;
        Ls *= d.rad[s];
    }
    d.twoff[d.nrad] = off;
}

inline FftDims make_dims(int n)
{
    FftDims d{};
    d.n = n;
    int m = n;
    while (m % 16 == 0) { d.rad[d.nrad++] = 16; m /= 16; }
    if (m % 8 == 0) { d.rad[d.nrad++] = 8; m /= 8; }
    if (m % 4 == 0) { d.rad[d.nrad++] = 4; m /= 4; }
    if (m % 2 == 0) { d.rad[d.nrad++] = 2; m /= 2; }
    while (m % 9 == 0) { d.rad[d.nrad++] = 9; m /= 9; }
    if (m % 3 == 0) { d.rad[d.nrad++] = 3; m /= 3; }
    set_spans(d);
    return d;
}

// The same stages in the opposite order.
inline FftDims reversed(FftDims d)
{
    std::reverse(d.rad, d.rad + d.nrad);
    set_spans(d);
    return d;
}

// Per-stage twiddles exp(-2 pi i q k / (Ls r)), entry ((q - 1) / 2 Ls + k) 2 +
// (q - 1) % 2 of the stage's table at twoff, in double then rounded (at least
// one entry; an even radix leaves the last power's neighbour unused).
inline std::vector<float2> stage_twiddles(const FftDims& d)
{
    std::vector<float2> t((size_t)std::max(1, d.twoff[d.nrad]));
    const double pi = 3.14159265358979323846;
    for (int s = 0; s < d.nrad; ++s)
    {
        if (d.ls[s] == 1) continue;
        for (int q = 1; q < d.rad[s]; ++q)
            for (int k = 0; k < d.ls[s]; ++k)
            {
                const double a = 2.0 * pi * (double)(q * k) / (double)(d.ls[s] * d.rad[s]);
                t[(size_t)d.twoff[s] + ((size_t)((q - 1) / 2) * d.ls[s] + k) * 2 + (q - 1) % 2] = make_float2((float)std::cos(a), (float)-std::sin(a));
            }
    }
    return t;
}

}  // namespace gl
