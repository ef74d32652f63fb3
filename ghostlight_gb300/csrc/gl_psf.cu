// gl_psf.cu — PSF grid renderer: per source, the lens's primary-ray spot
// (every pupil sample at every wavelength) splatted into its own tile of a
// composite atlas (psf_kernel, psf_render.cu:30-232).
//
// GB300 layout: the packed lens records and the per-wavelength IOR slices are
// staged in shared memory once per CTA; one thread per (source, pupil sample)
// walks the wavelengths with the reference-formulation primary trace; the
// splat is bilinear, or a normalised Gaussian of the configured physical
// width, clipped to the source's tile.  A wide Gaussian takes the dense kernel
// below: the tile as a sum of outer products in registers.
#include "gl_internal.h"
#include "gl_render.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

namespace gl {
namespace {

constexpr int kPsfThreads = 256;
constexpr float kTapMin = 1e-6f;        // taps of less of their splat are left out
constexpr float kDepositMin = 1e-14f;   // colour times weight up to which a plane takes nothing of a ray

struct PsfArgs {
    const SurfRec* recs;
    const float* ior_at;         // [spec][surf]
    const float4* spec;          // lambda, cmf r g b
    const gl_psf_source* src;
    const float2* grid;
    int n_surf, n_spec, n_src, n_grid;
    float front_R, start_z, mm_per_pixel, ray_weight;
    int tile_w, tile_h, comp_w, comp_h, mono;
    float sigma_px;
    int radius_px;
    float* out_r;
    float* out_g;
    float* out_b;
    int tile_smem;       // 1: the CTA's source tile is accumulated in shared memory
    // dense path: landings [source][wavelength][sample] as (x, y, weight, 1), the
    // last 0 where there is none near the tile, of n_land wavelengths from l_base
    // on; samples per CTA in steps of the CTA's threads
    float4* land;
    int l_base, n_land, s_base, rounds;
};

// Adds a ray-wavelength's weighted colour to one composite pixel: into the
// CTA's shared-memory copy of its source's tile (planes of tile_w x tile_h),
// or straight into the composite with global atomics.
__device__ __forceinline__ void deposit(const PsfArgs& A, float* tile, int tx, int ty, int pix, float lum,
                                       float cr, float cg, float cb, float wt)
{
    if (tile != nullptr)
    {
        const int t = ty * A.tile_w + tx, plane = A.tile_w * A.tile_h;
        if (A.mono)
        {
            if (fabsf(lum) > kDepositMin) atomicAdd(tile + t, lum * wt);
        }
        else
        {
            if (fabsf(cr) > kDepositMin) atomicAdd(tile + t, cr * wt);
            if (fabsf(cg) > kDepositMin) atomicAdd(tile + plane + t, cg * wt);
            if (fabsf(cb) > kDepositMin) atomicAdd(tile + 2 * plane + t, cb * wt);
        }
        return;
    }
    if (A.mono)
    {
        if (fabsf(lum) > kDepositMin) atomicAdd(A.out_r + pix, lum * wt);
    }
    else
    {
        if (fabsf(cr) > kDepositMin) atomicAdd(A.out_r + pix, cr * wt);
        if (fabsf(cg) > kDepositMin) atomicAdd(A.out_g + pix, cg * wt);
        if (fabsf(cb) > kDepositMin) atomicAdd(A.out_b + pix, cb * wt);
    }
}

template <bool LAND>
__device__ __forceinline__ void psf_trace_one(const PsfArgs& A, const SurfRec* lens, const float* at, float* tile,
                                              int si, int gi);

// LAND: the landings go to A.land instead of the tiles (the dense path), the
// wavelengths split over grid.z.
template <bool LAND>
__global__ void __launch_bounds__(kPsfThreads) psf_kernel(PsfArgs A)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SurfRec* lens = reinterpret_cast<SurfRec*>(smem_raw);
    float* at = reinterpret_cast<float*>(lens + A.n_surf);
    {
        const int words = A.n_surf * (int)(sizeof(SurfRec) / 4);
        const int* s = reinterpret_cast<const int*>(A.recs);
        int* d = reinterpret_cast<int*>(lens);
        for (int i = threadIdx.x; i < words; i += blockDim.x) d[i] = s[i];
        for (int i = threadIdx.x; i < A.n_spec * A.n_surf; i += blockDim.x) at[i] = A.ior_at[i];
    }
    // every ray of this CTA belongs to source blockIdx.x and deposits only in
    // its tile: accumulate the tile in shared memory, add it to the composite once
    float* tile = nullptr;
    const int planes = A.mono ? 1 : 3, tile_px = A.tile_w * A.tile_h;
    if (A.tile_smem)
    {
        tile = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(at + A.n_spec * A.n_surf) +
                                        ((16 - (((uintptr_t)(at + A.n_spec * A.n_surf)) & 15)) & 15));
        for (int i = threadIdx.x; i < planes * tile_px; i += blockDim.x) tile[i] = 0.0f;
    }
    __syncthreads();
    const int si = LAND ? A.s_base + blockIdx.x : blockIdx.x;
    const int gi = blockIdx.y * kPsfThreads + threadIdx.x;
    if (si < A.n_src && gi < A.n_grid) psf_trace_one<LAND>(A, lens, at, tile, si, gi);
    if (LAND || !A.tile_smem || si >= A.n_src) return;
    __syncthreads();
    const gl_psf_source S = A.src[si];
    float* outs[3] = {A.out_r, A.out_g, A.out_b};
    for (int i = threadIdx.x; i < planes * tile_px; i += blockDim.x)
    {
        const float v = tile[i];
        if (v == 0.0f) continue;
        const int pl = i / tile_px, t = i - pl * tile_px;
        const int xi = S.tile_x0 + t % A.tile_w, yi = S.tile_y0 + t / A.tile_w;
        if (xi < 0 || xi >= A.comp_w || yi < 0 || yi >= A.comp_h) continue;
        atomicAdd(outs[pl] + (size_t)yi * A.comp_w + xi, v);
    }
}

// One pupil sample of one source through every wavelength, splatted into the
// source's tile (tile != nullptr: the CTA's shared-memory copy of it).  LAND:
// landings (px, py, weight) of the wavelengths in hand instead of the splat.
template <bool LAND>
__device__ __forceinline__ void psf_trace_one(const PsfArgs& A, const SurfRec* lens, const float* at, float* tile,
                                              int si, int gi)
{
    const gl_psf_source S = A.src[si];
    const float2 uv = A.grid[gi];
    const float bx = tanf(S.angle_x), by = tanf(S.angle_y);
    const V3 dir = normalized(v3(bx, by, 1.0f));
    const V3 org = v3(uv.x * A.front_R - kSpawnOffset * bx, uv.y * A.front_R - kSpawnOffset * by, A.start_z);
    const int tx_min = S.tile_x0, ty_min = S.tile_y0, tx_max = S.tile_x0 + A.tile_w, ty_max = S.tile_y0 + A.tile_h;
    const int per = LAND ? (A.n_land + (int)gridDim.z - 1) / (int)gridDim.z : A.n_spec;
    const int l0 = LAND ? A.l_base + (int)blockIdx.z * per : 0;
    const int l1 = LAND ? min(A.l_base + A.n_land, l0 + per) : A.n_spec;
    for (int l = l0; l < l1; ++l)
    {
        float4* land = nullptr;
        if (LAND)
        {
            land = A.land + ((size_t)(si - A.s_base) * A.n_land + (l - A.l_base)) * A.n_grid + gi;
            land->w = 0.0f;
        }
        const float4 sp = A.spec[l];
        const TraceOut r = trace_primary(lens, A.n_surf, at + l * A.n_surf, org, dir, sp.x);
        if (r.status != GL_TRACE_OK || !isfinite(r.x) || !isfinite(r.y)) continue;
        const float tx = (r.x - S.chief_x_mm) / A.mm_per_pixel + (float)A.tile_w * 0.5f;
        const float ty = (r.y - S.chief_y_mm) / A.mm_per_pixel + (float)A.tile_h * 0.5f;
        const float margin = (float)(A.radius_px > 0 ? A.radius_px + 1 : 1);
        if (tx < -margin || tx > (float)A.tile_w + margin || ty < -margin || ty > (float)A.tile_h + margin) continue;
        const float px = tx + (float)S.tile_x0, py = ty + (float)S.tile_y0;
        const float w = r.w * A.ray_weight;
        if (LAND)
        {
            // (an attenuator's weight may have either sign; one that is not a number
            // is left out, as the taps leave it out)
            if (w == w) *land = make_float4(px, py, w, 1.0f);
            continue;
        }
        const float lum = (S.r + S.g + S.b) * (1.0f / 3.0f) * sp.z * w;
        const float cr = S.r * sp.y * w, cg = S.g * sp.z * w, cb = S.b * sp.w * w;
        if (A.sigma_px <= 0.0f)
        {
            const int x0 = (int)floorf(px - 0.5f), y0 = (int)floorf(py - 0.5f);
            const float fx = (px - 0.5f) - (float)x0, fy = (py - 0.5f) - (float)y0;
            const float bw[4] = {(1.0f - fx) * (1.0f - fy), fx * (1.0f - fy), (1.0f - fx) * fy, fx * fy};
            #pragma unroll
            for (int k = 0; k < 4; ++k)
            {
                const int xi = x0 + (k & 1), yi = y0 + (k >> 1);
                if (xi < tx_min || xi >= tx_max || yi < ty_min || yi >= ty_max || xi < 0 || xi >= A.comp_w ||
                    yi < 0 || yi >= A.comp_h)
                    continue;
                deposit(A, tile, xi - S.tile_x0, yi - S.tile_y0, yi * A.comp_w + xi, lum, cr, cg, cb, bw[k]);
            }
        }
        else
        {
            const float inv2 = 1.0f / (2.0f * A.sigma_px * A.sigma_px);
            const int cx = (int)floorf(px), cy = (int)floorf(py);
            const float ox = px - ((float)cx + 0.5f), oy = py - ((float)cy + 0.5f);
            const int R = A.radius_px;
            float wsum = 0.0f;
            for (int dy = -R; dy <= R; ++dy)
            {
                const float dyr = (float)dy - oy;
                for (int dx = -R; dx <= R; ++dx)
                {
                    const float dxr = (float)dx - ox;
                    wsum += expf(-(dxr * dxr + dyr * dyr) * inv2);
                }
            }
            const float inv_wsum = wsum > 1e-20f ? 1.0f / wsum : 0.0f;
            for (int dy = -R; dy <= R; ++dy)
            {
                const int yi = cy + dy;
                if (yi < ty_min || yi >= ty_max || yi < 0 || yi >= A.comp_h) continue;
                const float dyr = (float)dy - oy;
                for (int dx = -R; dx <= R; ++dx)
                {
                    const int xi = cx + dx;
                    if (xi < tx_min || xi >= tx_max || xi < 0 || xi >= A.comp_w) continue;
                    const float dxr = (float)dx - ox;
                    const float wt = expf(-(dxr * dxr + dyr * dyr) * inv2) * inv_wsum;
                    if (wt < kTapMin) continue;
                    deposit(A, tile, xi - S.tile_x0, yi - S.tile_y0, yi * A.comp_w + xi, lum, cr, cg, cb, wt);
                }
            }
        }
    }
}

// ---- dense Gaussian tiles ---------------------------------------------------
// The Gaussian of a landing is an outer product gx(x) gy(y), so a source's
// tile at one wavelength is the matrix product Gy^T diag(w) Gx over the rays
// that land near it: no exponentials per tap (2 (2R + 1) per ray instead of
// 2 (2R + 1)^2) and no shared-memory atomics (3 per tap).  One CTA holds the
// tile of one (source, wavelength, range of pupil samples) in registers, 8 x 8
// pixels per thread; it
//   1. packs the landings near the tile, as psf_kernel<true> left them, into a
//      list;
//   2. for 32 landings at a time writes the rows gx and gy (zero outside the
//      window, gy times weight / sum of the window) to shared memory, one warp
//      per landing, and adds their outer products, each group of threads that
//      covers the tile taking every G-th landing;
//   3. sums the groups through shared memory and adds the tile, times the
//      wavelength's colour weights, to the composite.
// Bound by the FP32 pipes in step 2 (64 FMA per 4 shared 16-byte loads); the
// trace before it is most of the time left.  8 x 8 tiles of 64^2, 16
// wavelengths, radius 13 (the default settings): 3.96 -> 0.35 ms for both
// kernels.  Taps and rays that are too faint are left out as psf_kernel<false>
// leaves them out.  The trace stays a kernel of its own (landings through a scratch
// that fits L2): inlined here it rounded some landings differently.
constexpr int kDenseChunk = 32;       // landings per outer-product step
constexpr size_t kDenseLandings = (size_t)4 << 20;   // 64 MB: stays in L2 between the two kernels
constexpr long long kLandingBytes = (long long)(kDenseLandings * sizeof(float4));
constexpr int kDenseRoundsMax = 16;   // pupil samples per thread and CTA, at most

struct DenseGeom {
    int tx, ty, groups;               // 8 x 8 blocks across and down the tile, thread groups that cover it
};

__host__ __device__ inline DenseGeom dense_geom(int tile_w, int tile_h)
{
    DenseGeom g;
    g.tx = (tile_w + 7) / 8;
    g.ty = (tile_h + 7) / 8;
    g.groups = g.tx * g.ty <= kPsfThreads ? kPsfThreads / (g.tx * g.ty) : 0;
    return g;
}

// floats: the landing list, then the gx / gy rows, which the group sum reuses
// as one plane
inline size_t dense_smem_floats(const DenseGeom& g, int rounds)
{
    const size_t rows = (size_t)kDenseChunk * 8 * (g.tx + g.ty), plane = (size_t)64 * g.tx * g.ty;
    return 4 * (size_t)rounds * kPsfThreads + std::max(rows, plane);
}

// CUT: taps below kTapMin of their splat are left out one by one, as the tap kernel
// leaves them out (a window much wider than 2.5 sigma has such taps): three
// instructions per pixel and landing in place of one.
template <bool CUT>
__global__ void __launch_bounds__(kPsfThreads, 2) psf_dense_kernel(PsfArgs A)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int n_list;
    const DenseGeom G = dense_geom(A.tile_w, A.tile_h);
    const int W8 = 8 * G.tx, H8 = 8 * G.ty;
    float4* list = reinterpret_cast<float4*>(smem_raw);              // local px, py, weight
    float* gx = reinterpret_cast<float*>(list + A.rounds * kPsfThreads);         // [landing][W8]
    float* gy = gx + kDenseChunk * W8;                               // [landing][H8]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int si = A.s_base + blockIdx.x, l = A.l_base + blockIdx.y;
    if (tid == 0) n_list = 0;
    __syncthreads();
    const gl_psf_source S = A.src[si];
    const float4 sp = A.spec[l];
    const int R = A.radius_px;
    const int planes = A.mono ? 1 : 3;
    const float lum = (S.r + S.g + S.b) * (1.0f / 3.0f) * sp.z;
    const float c[3] = {A.mono ? lum : S.r * sp.y, A.mono ? 0.0f : S.g * sp.z, A.mono ? 0.0f : S.b * sp.w};
    const float4* land = A.land + ((size_t)blockIdx.x * A.n_land + blockIdx.y) * A.n_grid;
    // a plane takes nothing of a ray that is too faint in it; where that differs
    // between planes (a dim source, the end of the spectrum) each has its own pass
    int mixed = 0;
    for (int q = 0; q < A.rounds; ++q)
    {
        const int gi = (blockIdx.z * A.rounds + q) * kPsfThreads + tid;
        float4 e = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (gi < A.n_grid) e = land[gi];
        int seen = 0, faint = 0;
        #pragma unroll
        for (int k = 0; k < 3; ++k)
        {
            const bool takes = fabsf(c[k] * e.z) > kDepositMin;
            seen |= takes;
            faint |= fabsf(c[k]) > 0.0f && !takes;
        }
        const bool in = e.w != 0.0f && seen;
        mixed |= in && faint;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        int base = 0;
        if (lane == 0 && m) base = atomicAdd(&n_list, __popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (in) list[base + __popc(m & ((1u << lane) - 1u))] = e;
    }
    mixed = __syncthreads_or(mixed);
    const int n = n_list;
    if (n == 0) return;
    const float inv2 = 1.0f / (2.0f * A.sigma_px * A.sigma_px);
    const int per = G.tx * G.ty, grp = tid / per, cell = tid - grp * per;
    const int mx = (cell % G.tx) * 8, my = (cell / G.tx) * 8;
    #pragma unroll 1
    for (int p0 = 0; p0 < (mixed ? planes : 1); ++p0)
    {
        const float cp = p0 == 0 ? c[0] : (p0 == 1 ? c[1] : c[2]);
        float acc[8][8] = {};
        for (int c0 = 0; c0 < n; c0 += kDenseChunk)
        {
            const int cnt = min(kDenseChunk, n - c0);
            for (int r = warp; r < cnt; r += kPsfThreads / 32)
            {
                const float4 e = list[c0 + r];
                const int cx = (int)floorf(e.x), cy = (int)floorf(e.y);
                const float ox = e.x - ((float)cx + 0.5f), oy = e.y - ((float)cy + 0.5f);
                // window offset of this lane: R <= 16, at most 33 entries per axis
                float wx = 0.0f, wy = 0.0f;
                for (int d = lane - R; d <= R; d += 32)
                {
                    const float dx = (float)d - ox, dy = (float)d - oy;
                    wx += expf(-(dx * dx) * inv2);
                    wy += expf(-(dy * dy) * inv2);
                }
                #pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                {
                    wx += __shfl_xor_sync(0xffffffffu, wx, o);
                    wy += __shfl_xor_sync(0xffffffffu, wy, o);
                }
                const float ws = wx * wy;
                const bool seen = ws > 1e-20f && (!mixed || fabsf(cp * e.z) > kDepositMin);
                const float amp = !seen ? 0.0f : (CUT ? 1.0f / ws : e.z / ws);
                const int lx = cx - S.tile_x0, ly = cy - S.tile_y0;
                for (int i = lane; i < W8; i += 32)
                {
                    const float dx = (float)(i - lx) - ox;
                    gx[r * W8 + i] = (i < A.tile_w && abs(i - lx) <= R) ? expf(-(dx * dx) * inv2) : 0.0f;
                }
                for (int i = lane; i < H8; i += 32)
                {
                    const float dy = (float)(i - ly) - oy;
                    gy[r * H8 + i] = (i < A.tile_h && abs(i - ly) <= R) ? expf(-(dy * dy) * inv2) * amp : 0.0f;
                }
            }
            __syncthreads();
            if (grp < G.groups)
            {
                for (int r = grp; r < cnt; r += G.groups)
                {
                    const float4* px = reinterpret_cast<const float4*>(gx + r * W8 + mx);
                    const float4* py = reinterpret_cast<const float4*>(gy + r * H8 + my);
                    const float4 x0 = px[0], x1 = px[1], y0 = py[0], y1 = py[1];
                    const float vx[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
                    const float vy[8] = {y0.x, y0.y, y0.z, y0.w, y1.x, y1.y, y1.z, y1.w};
                    const float w = CUT ? list[c0 + r].z : 0.0f;
                    #pragma unroll
                    for (int j = 0; j < 8; ++j)
                        #pragma unroll
                        for (int i = 0; i < 8; ++i)
                        {
                            if (!CUT) acc[j][i] = fmaf(vy[j], vx[i], acc[j][i]);
                            else
                            {
                                const float t = vy[j] * vx[i];
                                if (t >= kTapMin) acc[j][i] = fmaf(t, w, acc[j][i]);
                            }
                        }
                }
            }
            __syncthreads();
        }
        // sum of the groups, in order, in the rows' place (the loop ended on a barrier)
        float* sum = gx;
        for (int g = 0; g < G.groups; ++g)
        {
            if (grp == g)
            {
                #pragma unroll
                for (int j = 0; j < 8; ++j)
                    #pragma unroll
                    for (int i = 0; i < 8; ++i)
                    {
                        float* q = sum + (my + j) * W8 + mx + i;
                        *q = g == 0 ? acc[j][i] : *q + acc[j][i];
                    }
            }
            __syncthreads();
        }
        float* const outs[3] = {A.out_r, A.out_g, A.out_b};
        for (int t = tid; t < A.tile_w * A.tile_h; t += kPsfThreads)
        {
            const int y = t / A.tile_w, x = t - y * A.tile_w;
            const int xi = S.tile_x0 + x, yi = S.tile_y0 + y;
            if (xi < 0 || xi >= A.comp_w || yi < 0 || yi >= A.comp_h) continue;
            const float v = sum[y * W8 + x];
            if (v == 0.0f) continue;
            #pragma unroll
            for (int pl = 0; pl < 3; ++pl)
                if ((!mixed || pl == p0) && fabsf(c[pl]) > 0.0f) atomicAdd(outs[pl] + (size_t)yi * A.comp_w + xi, c[pl] * v);
        }
        __syncthreads();
    }
}

// Whether a landing's window may hold taps below kTapMin: its corner, seen from
// the far end of the centre pixel.
inline bool faint_taps(float sigma_px, int radius_px)
{
    const double inv2 = 0.5 / ((double)sigma_px * sigma_px), far = radius_px + 0.5;
    double wx = 0.0;
    for (int d = -radius_px; d <= radius_px; ++d) wx += std::exp(-(d + 0.5) * (d + 0.5) * inv2);
    return !(std::exp(-2.0 * far * far * inv2) >= 1.01 * (double)kTapMin * wx * wx);
}

// The dense kernel pays for the whole tile per landing, the sparse one for the
// (2R + 1)^2 taps.  Atlas of 64 sources, 16 wavelengths, 64^2 grid, sparse
// against dense: 64^2 tiles, R = 2 0.40 / 0.43 ms, R = 3 0.52 / 0.43, R = 13
// 3.96 / 0.44; 32^2 tiles, R = 2 0.41 / 0.42, R = 3 0.55 / 0.42; 128^2 tiles,
// R = 3 0.43 / 0.48, R = 4 0.54 / 0.48 (the trace is 0.35 of each).
inline bool dense_tile(int tile_w, int tile_h, float sigma_px, int radius_px)
{
    const DenseGeom g = dense_geom(tile_w, tile_h);
    return sigma_px > 0.0f && g.groups >= 1 && radius_px >= (64 * g.tx * g.ty <= 8192 ? 3 : 4);
}

// Landings kept at a time: of as many wavelengths and sources as fit the scratch
// (0 sources: not one wavelength of one source does).
struct Landings { int l, s; };

inline Landings landings(int n_sources, int n_grid, int n_spec, long long bytes)
{
    const size_t most = std::min<size_t>(kDenseLandings, (size_t)std::max(0LL, bytes) / sizeof(float4));
    Landings k{0, 0};
    if (most < (size_t)n_grid) return k;
    k.l = (int)std::min<size_t>(std::min(n_spec, 65535), most / n_grid);
    k.s = (int)std::min<size_t>(n_sources, most / ((size_t)n_grid * k.l));
    return k;
}

}  // namespace
}  // namespace gl

using namespace gl;

// The render of both entries: the scratch (lens records, index table,
// spectrum, sources, pupil grid: one block, one copy) comes from the device's
// stream-ordered pool and is freed in stream order; the plain entry then waits
// for the stream, `ordered` does not.
static int psf_render_impl(const gl_surface* surfaces, int n_surfaces, const gl_psf_source* sources, int n_sources,
                           const gl_pupil_sample* grid, int n_grid, const gl_spectral_sample* spec, int n_spec,
                           int tile_w, int tile_h, int composite_w, int composite_h, float mm_per_pixel,
                           int monochromatic, float splat_sigma_px, int splat_radius_px, float* d_out_r,
                           float* d_out_g, float* d_out_b, long long landing_bytes, void* stream, bool ordered)
{
    if (!surfaces || n_surfaces <= 0) return fail(GL_ERR_INVALID, "psf_render: lens has no surfaces");
    if (n_sources < 0 || n_grid < 0 || n_spec < 1 || (n_sources > 0 && !sources) || (n_grid > 0 && !grid) || !spec)
        return fail(GL_ERR_INVALID, "psf_render: bad arguments");
    if (tile_w <= 0 || tile_h <= 0 || composite_w <= 0 || composite_h <= 0 || !(mm_per_pixel > 0.0f))
        return fail(GL_ERR_INVALID, "psf_render: grid and tile dimensions must be positive");
    if ((long long)composite_w * composite_h > (1LL << 31)) return fail(GL_ERR_INVALID, "psf_render: too many pixels");
    if (!d_out_r || (!monochromatic && (!d_out_g || !d_out_b))) return fail(GL_ERR_INVALID, "psf_render: null output");
    if (splat_radius_px < 0 || splat_radius_px > 16) return fail(GL_ERR_INVALID, "psf_render: splat radius must be 0..16");
    if (n_sources == 0 || n_grid == 0) return GL_OK;
    int dev = 0;
    GL_CUDA_TRY(cudaGetDevice(&dev));
    std::vector<SurfRec> recs((size_t)n_surfaces);
    int rc = pack_lens(surfaces, n_surfaces, recs.data(), dev);
    if (rc) return rc;
    std::vector<float> lams((size_t)n_spec), at((size_t)n_spec * n_surfaces), bf((size_t)n_spec * n_surfaces);
    std::vector<float4> sp((size_t)n_spec);
    for (int i = 0; i < n_spec; ++i)
    {
        lams[i] = spec[i].lambda;
        sp[i] = make_float4(spec[i].lambda, spec[i].cmf_r, spec[i].cmf_g, spec[i].cmf_b);
    }
    build_ior_tables(surfaces, n_surfaces, lams.data(), n_spec, at.data(), bf.data());
    cudaStream_t st = (cudaStream_t)stream;
    // one scratch block, each part 256-byte aligned, filled by one copy
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t o_recs = 0, o_at = o_recs + up(recs.size() * sizeof(SurfRec)), o_spec = o_at + up(at.size() * sizeof(float)),
                 o_src = o_spec + up(sp.size() * sizeof(float4)), o_grid = o_src + up((size_t)n_sources * sizeof(gl_psf_source)),
                 total = o_grid + up((size_t)n_grid * sizeof(float2));
    std::vector<char> host(total, 0);
    std::memcpy(host.data() + o_recs, recs.data(), recs.size() * sizeof(SurfRec));
    std::memcpy(host.data() + o_at, at.data(), at.size() * sizeof(float));
    std::memcpy(host.data() + o_spec, sp.data(), sp.size() * sizeof(float4));
    std::memcpy(host.data() + o_src, sources, (size_t)n_sources * sizeof(gl_psf_source));
    std::memcpy(host.data() + o_grid, grid, (size_t)n_grid * sizeof(float2));
    char* block = nullptr;
    cudaMemPool_t pool;
    cudaError_t e = shared_device_pool(dev, &pool);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(reinterpret_cast<void**>(&block), total, pool, st);
    if (e != cudaSuccess)
        return fail(e == cudaErrorMemoryAllocation ? GL_ERR_OOM : GL_ERR_CUDA, std::string("psf_render: ") + cudaGetErrorString(e));
    SurfRec* d_recs = reinterpret_cast<SurfRec*>(block + o_recs);
    float* d_at = reinterpret_cast<float*>(block + o_at);
    float4* d_spec = reinterpret_cast<float4*>(block + o_spec);
    gl_psf_source* d_src = reinterpret_cast<gl_psf_source*>(block + o_src);
    float2* d_grid = reinterpret_cast<float2*>(block + o_grid);
    e = cudaMemcpyAsync(block, host.data(), total, cudaMemcpyHostToDevice, st);
    // the CTA's source tile in shared memory when it fits (96 KB of tile)
    const size_t tile_bytes = (size_t)(monochromatic ? 1 : 3) * tile_w * tile_h * sizeof(float);
    const bool tile_smem = tile_bytes <= 96 * 1024;
    const DenseGeom dg = dense_geom(tile_w, tile_h);
    // samples per CTA: as many as keep about four CTAs per resident slot (two
    // per SM), so that few CTAs add the same tile to the composite
    int rounds = kDenseRoundsMax, n_sm = 0;
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
    auto dense_z = [&](int r) { return ((long long)n_grid + r * kPsfThreads - 1) / (r * kPsfThreads); };
    while (rounds > 1 && dense_z(rounds) * n_sources * n_spec < 8LL * n_sm) rounds /= 2;
    const size_t dense_smem = dense_smem_floats(dg, rounds) * sizeof(float);
    const Landings k = landings(n_sources, n_grid, n_spec, landing_bytes);
    const int land_l = k.l, land_s = k.s;
    bool dense = dense_tile(tile_w, tile_h, splat_sigma_px, splat_radius_px) && dense_smem <= 220 * 1024 && land_s > 0;
    float4* d_land = nullptr;
    if (e == cudaSuccess && dense)
    {
        e = cudaMallocFromPoolAsync(reinterpret_cast<void**>(&d_land), sizeof(float4) * (size_t)land_s * land_l * n_grid, pool, st);
        if (e == cudaErrorMemoryAllocation)
        {
            // no room for them: the taps need none
            cudaGetLastError();
            d_land = nullptr;
            dense = false;
            e = cudaSuccess;
        }
    }
    const size_t smem = recs.size() * sizeof(SurfRec) + at.size() * sizeof(float) + (tile_smem && !dense ? tile_bytes + 16 : 0);
    if (e == cudaSuccess && smem > 48 * 1024)
        e = (cudaError_t)raise_smem_limit(dense ? (const void*)psf_kernel<true> : (const void*)psf_kernel<false>, smem);
    auto dense_kernel = faint_taps(splat_sigma_px, splat_radius_px) ? psf_dense_kernel<true> : psf_dense_kernel<false>;
    if (e == cudaSuccess && dense && dense_smem > 47 * 1024)   // the kernel has a static word besides
        e = (cudaError_t)raise_smem_limit((const void*)dense_kernel, dense_smem);
    int launches = dense ? 0 : 1;
    if (e == cudaSuccess)
    {
        PsfArgs A;
        A.recs = d_recs; A.ior_at = d_at; A.spec = d_spec; A.src = d_src; A.grid = d_grid;
        A.n_surf = n_surfaces; A.n_spec = n_spec; A.n_src = n_sources; A.n_grid = n_grid;
        A.front_R = surfaces[0].semi_aperture; A.start_z = surfaces[0].z - kSpawnOffset;
        A.mm_per_pixel = mm_per_pixel; A.ray_weight = 1.0f / (float)n_grid;
        A.tile_w = tile_w; A.tile_h = tile_h; A.comp_w = composite_w; A.comp_h = composite_h;
        A.mono = monochromatic ? 1 : 0;
        A.sigma_px = splat_sigma_px; A.radius_px = splat_radius_px;
        A.out_r = d_out_r; A.out_g = d_out_g; A.out_b = d_out_b;
        A.tile_smem = tile_smem && !dense ? 1 : 0;
        A.land = d_land;
        A.l_base = 0; A.n_land = 0; A.s_base = 0;
        A.rounds = rounds;
        const unsigned blocks = (unsigned)((n_grid + kPsfThreads - 1) / kPsfThreads);
        if (!dense) psf_kernel<false><<<dim3((unsigned)n_sources, blocks), kPsfThreads, smem, st>>>(A);
        for (int s0 = 0; dense && s0 < n_sources; s0 += land_s)
            for (int l0 = 0; l0 < n_spec; l0 += land_l)
            {
                const unsigned ns = (unsigned)std::min(land_s, n_sources - s0);
                A.s_base = s0; A.l_base = l0;
                A.n_land = std::min(land_l, n_spec - l0);
                // wavelengths over grid.z until there are about eight CTAs per
                // resident slot (four of 58 registers x 256 per SM): 64 cells of
                // 2816 samples are 704 CTAs, a second wave of 96 with all 16
                // wavelengths in each: landings 330 -> 256 us in eight parts
                // (0.96 -> 0.88 ms a call; in two 0.92, four 0.89, sixteen 0.89)
                const long long ctas = (long long)ns * blocks, want = 32LL * n_sm;
                const int parts = (int)std::min<long long>(A.n_land, std::max(1LL, (want + ctas - 1) / ctas));
                const int per = (A.n_land + parts - 1) / parts;
                psf_kernel<true><<<dim3(ns, blocks, (unsigned)((A.n_land + per - 1) / per)), kPsfThreads, smem, st>>>(A);
                dense_kernel<<<dim3(ns, (unsigned)A.n_land, (unsigned)dense_z(rounds)), kPsfThreads, dense_smem, st>>>(A);
                launches += 2;
            }
        e = cudaGetLastError();
    }
    if (d_land)
    {
        const cudaError_t f = cudaFreeAsync(d_land, st);
        if (e == cudaSuccess) e = f;
    }
    const cudaError_t f = cudaFreeAsync(block, st);
    if (e == cudaSuccess) e = f;
    if (!ordered)
    {
        const cudaError_t w = cudaStreamSynchronize(st);
        if (e == cudaSuccess) e = w;
    }
    if (e != cudaSuccess)
        return fail(e == cudaErrorMemoryAllocation ? GL_ERR_OOM : GL_ERR_CUDA, std::string("psf_render: ") + cudaGetErrorString(e));
    g_last_launches = launches;
    return GL_OK;
}

extern "C" long long gl_psf_scratch_bytes(int n_sources, int n_grid, int n_spec, int tile_w, int tile_h, float splat_sigma_px,
                                          int splat_radius_px)
{
    if (n_sources <= 0 || n_grid <= 0 || n_spec <= 0 || tile_w <= 0 || tile_h <= 0) return 0;
    // lens records, index table, spectrum, sources and pupil grid, each rounded up
    const long long tables = (long long)kMaxSurfaces * (sizeof(SurfRec) + sizeof(float) * n_spec) + sizeof(float4) * n_spec +
                             sizeof(gl_psf_source) * (long long)n_sources + sizeof(float2) * (long long)n_grid + 5 * 256;
    if (!dense_tile(tile_w, tile_h, splat_sigma_px, splat_radius_px)) return tables;
    const Landings k = landings(n_sources, n_grid, n_spec, kLandingBytes);
    return tables + (long long)sizeof(float4) * k.s * k.l * n_grid;
}

extern "C" int gl_psf_render(const gl_surface* surfaces, int n_surfaces, const gl_psf_source* sources, int n_sources,
                             const gl_pupil_sample* grid, int n_grid, const gl_spectral_sample* spec, int n_spec,
                             int tile_w, int tile_h, int composite_w, int composite_h, float mm_per_pixel,
                             int monochromatic, float splat_sigma_px, int splat_radius_px, float* d_out_r,
                             float* d_out_g, float* d_out_b, void* stream)
{
    return psf_render_impl(surfaces, n_surfaces, sources, n_sources, grid, n_grid, spec, n_spec, tile_w, tile_h,
                           composite_w, composite_h, mm_per_pixel, monochromatic, splat_sigma_px, splat_radius_px,
                           d_out_r, d_out_g, d_out_b, kLandingBytes, stream, false);
}

extern "C" int gl_psf_render_async(const gl_surface* surfaces, int n_surfaces, const gl_psf_source* sources,
                                   int n_sources, const gl_pupil_sample* grid, int n_grid,
                                   const gl_spectral_sample* spec, int n_spec, int tile_w, int tile_h,
                                   int composite_w, int composite_h, float mm_per_pixel, int monochromatic,
                                   float splat_sigma_px, int splat_radius_px, float* d_out_r, float* d_out_g,
                                   float* d_out_b, void* stream)
{
    return psf_render_impl(surfaces, n_surfaces, sources, n_sources, grid, n_grid, spec, n_spec, tile_w, tile_h,
                           composite_w, composite_h, mm_per_pixel, monochromatic, splat_sigma_px, splat_radius_px,
                           d_out_r, d_out_g, d_out_b, kLandingBytes, stream, true);
}

extern "C" int gl_psf_render_async2(const gl_surface* surfaces, int n_surfaces, const gl_psf_source* sources,
                                    int n_sources, const gl_pupil_sample* grid, int n_grid,
                                    const gl_spectral_sample* spec, int n_spec, int tile_w, int tile_h,
                                    int composite_w, int composite_h, float mm_per_pixel, int monochromatic,
                                    float splat_sigma_px, int splat_radius_px, float* d_out_r, float* d_out_g,
                                    float* d_out_b, long long landing_bytes, void* stream)
{
    return psf_render_impl(surfaces, n_surfaces, sources, n_sources, grid, n_grid, spec, n_spec, tile_w, tile_h,
                           composite_w, composite_h, mm_per_pixel, monochromatic, splat_sigma_px, splat_radius_px,
                           d_out_r, d_out_g, d_out_b, landing_bytes, stream, true);
}
