// gl_survive.cu — which part of the pupil an off-axis beam gets through: the
// centroid of its surviving launches (solve_survivor_center,
// starburst_render.cu:503-583) and the cat's-eye envelope over the pupil
// (build_survivor_envelope, :393-491).
//
// Both classify a grid of launches (does the ray reach the sensor?), then take
// the cells on the border between classes apart into ss x ss launches of their
// own.  Here both passes make their launches where they trace them: one thread a
// cell for the classes, one warp a cell for the borders (its lanes take the
// sub-launches), and nothing but the result comes back.  With the launches built
// and the classes compared on the host, three batches of rays went there and back
// and every step in between was a pass over host arrays: centre and envelope of a
// 12-surface lens, 81^2 and 192^2 cells, 2.1 ms; so 0.33.
// Bound by latency: 30,000 launches in two waves of some 10 us each.
#include "gl_disp.cuh"
#include "gl_render.h"

#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <vector>

namespace gl {
namespace {

constexpr int kThreads = 128;
constexpr unsigned kAll = 0xffffffffu;
constexpr unsigned char kOutside = 2;            // the cell's centre is outside the stop: not traced

struct SurviveArgs {
    const SurfRec* recs;
    const DispRec* disp;
    const float* cu;             // cell centres along x: launch positions (centre) or pupil coordinates (envelope)
    const float* cv;             // along y
    const float* ou;             // ss offsets of a cell's sub-launches along x
    const float* ov;
    unsigned char* cls;          // m x m: 0 dies, 1 survives, kOutside
    int n_surf, m, ss;
    float lam, z, dx, dy, dz;
    float cx, cy, ep_x, ep_y;    // envelope: launch = centre + pupil coordinate * ep
};

struct Lens {
    SurfRec recs[kMaxSurfaces];
    float at[kMaxSurfaces];
};

__device__ __forceinline__ void load_lens(const SurviveArgs& A, Lens& L)
{
    const int words = A.n_surf * (int)(sizeof(SurfRec) / 4);
    for (int i = threadIdx.x; i < words; i += kThreads)
        reinterpret_cast<int*>(L.recs)[i] = reinterpret_cast<const int*>(A.recs)[i];
    for (int i = threadIdx.x; i < A.n_surf; i += kThreads) L.at[i] = disp_ior(A.disp[i], A.lam);
    __syncthreads();
}

__device__ __forceinline__ bool survives(const SurviveArgs& A, const Lens& L, float x, float y)
{
    const TraceOut t = trace_primary(L.recs, A.n_surf, L.at, v3(x, y, A.z), v3(A.dx, A.dy, A.dz), A.lam);
    return t.status == GL_TRACE_OK && isfinite(t.x) && isfinite(t.y);
}

// PupilMask::contains (pupil_contains) on the device.
__device__ __forceinline__ bool inside_stop(const PupilMask& m, float u, float v)
{
    const float ux = __fdiv_rn(u, m.aspect);
    const float r2 = __fadd_rn(__fmul_rn(ux, ux), __fmul_rn(v, v));
    if (r2 > 1.0f) return false;
    if (m.n_blades < 3) return true;
    const float r = __fsqrt_rn(r2);
    if (m.blade.deformed) return r <= blade_radius_at(m.blade, atan2f(v, ux));
    if (r <= m.apothem) return true;
    float sector = fmodf(atan2f(v, ux) - m.rot_rad, m.sector);
    if (sector < 0.0f) sector += m.sector;
    return !(r * cosf(sector - m.sector * 0.5f) > m.apothem);
}

// The launch of a sub-sample: centre, the position itself; envelope, on the spawn
// plane through the pupil coordinate.
template <bool ENV>
__device__ __forceinline__ bool survives_at(const SurviveArgs& A, const Lens& L, float u, float v)
{
    if (!ENV) return survives(A, L, u, v);
    return survives(A, L, __fadd_rn(A.cx, __fmul_rn(u, A.ep_x)), __fadd_rn(A.cy, __fmul_rn(v, A.ep_y)));
}

template <bool ENV>
__global__ void __launch_bounds__(kThreads) classify_kernel(const SurviveArgs A, const PupilMask mask)
{
    __shared__ Lens L;
    load_lens(A, L);
    const int k = blockIdx.x * kThreads + threadIdx.x;
    if (k >= A.m * A.m) return;
    const float u = A.cu[k % A.m], v = A.cv[k / A.m];
    A.cls[k] = (ENV && !inside_stop(mask, u, v)) ? kOutside : (unsigned char)survives_at<ENV>(A, L, u, v);
}

// A cell's value.  Centre: {sum of x, sum of y, weight} of its survivors, a border
// cell's sub-launches weighted 1 / ss^2.  Envelope: the surviving fraction of a
// border cell's sub-launches inside the stop, else the class (-1 outside).
template <bool ENV>
__global__ void __launch_bounds__(kThreads) border_kernel(const SurviveArgs A, const PupilMask mask, double* __restrict__ sums,
                                                          float* __restrict__ env)
{
    __shared__ Lens L;
    const int lane = threadIdx.x & 31;
    const int k = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5), cells = A.m * A.m;
    const int i = k % A.m, j = k / A.m;
    bool border = false;
    int own = kOutside;
    if (k < cells)
    {
        own = A.cls[k];
        // lanes 0 .. 8: the 3 x 3 around the cell
        bool differs = false;
        const int ni = i + lane % 3 - 1, nj = j + lane / 3 - 1;
        if (lane < 9 && own != kOutside && ni >= 0 && ni < A.m && nj >= 0 && nj < A.m)
        {
            const int c = A.cls[nj * A.m + ni];
            differs = c != kOutside && c != own;
        }
        border = __any_sync(kAll, differs);
    }
    if (__syncthreads_or(border)) load_lens(A, L);
    if (k >= cells) return;
    const float u0 = A.cu[i], v0 = A.cv[j];
    double sx = 0.0, sy = 0.0;
    int n_in = 0, n_ok = 0;
    if (border)
    {
        for (int q = lane; q < A.ss * A.ss; q += 32)
        {
            const float u = __fadd_rn(u0, A.ou[q % A.ss]), v = __fadd_rn(v0, A.ov[q / A.ss]);
            if (ENV && !inside_stop(mask, u, v)) continue;
            ++n_in;
            if (!survives_at<ENV>(A, L, u, v)) continue;
            ++n_ok;
            sx += (double)u;
            sy += (double)v;
        }
        __syncwarp();
        for (int s = 16; s > 0; s >>= 1)
        {
            n_in += __shfl_xor_sync(kAll, n_in, s);
            n_ok += __shfl_xor_sync(kAll, n_ok, s);
            if (!ENV)
            {
                sx += __shfl_xor_sync(kAll, sx, s);
                sy += __shfl_xor_sync(kAll, sy, s);
            }
        }
    }
    if (lane != 0) return;
    if (ENV)
    {
        float e = own == kOutside ? -1.0f : (float)own;
        if (border && n_in > 0) e = __fdiv_rn((float)n_ok, (float)n_in);
        env[k] = e;
        return;
    }
    const double part = border ? 1.0 / (double)(A.ss * A.ss) : (double)own;
    sums[3 * (size_t)k] = (border ? sx : (double)u0) * part;
    sums[3 * (size_t)k + 1] = (border ? sy : (double)v0) * part;
    sums[3 * (size_t)k + 2] = (border ? (double)n_ok : 1.0) * part;
}

// The cells' sums added up by one block (always in the same order).
__global__ void __launch_bounds__(512) total_kernel(const double* __restrict__ sums, int cells, double* __restrict__ out)
{
    __shared__ double part[3][16];
    double v[3] = {0.0, 0.0, 0.0};
    for (int k = threadIdx.x; k < cells; k += 512)
        for (int c = 0; c < 3; ++c) v[c] += sums[3 * (size_t)k + c];
    for (int c = 0; c < 3; ++c)
    {
        for (int s = 16; s > 0; s >>= 1) v[c] += __shfl_xor_sync(kAll, v[c], s);
        if ((threadIdx.x & 31) == 0) part[c][threadIdx.x >> 5] = v[c];
    }
    __syncthreads();
    if (threadIdx.x < 3)
    {
        double t = 0.0;
        for (int w = 0; w < 16; ++w) t += part[threadIdx.x][w];
        out[threadIdx.x] = t;
    }
}

// Cells outside the stop take the largest value within two cells (0 where that is
// none).
__global__ void __launch_bounds__(256) dilate_kernel(const float* __restrict__ env, int m, float* __restrict__ out)
{
    const int k = blockIdx.x * 256 + threadIdx.x;
    if (k >= m * m) return;
    float e = env[k];
    if (e < 0.0f)
    {
        const int i = k % m, j = k / m;
        e = 0.0f;
        for (int y = max(j - 2, 0); y <= min(j + 2, m - 1); ++y)
            for (int x = max(i - 2, 0); x <= min(i + 2, m - 1); ++x) e = fmaxf(e, env[(size_t)y * m + x]);
    }
    out[k] = e;
}

// One block of device memory: the staged records and tables, then the scratch.
struct Staged {
    std::vector<char> host;
    size_t add(const void* p, size_t bytes)
    {
        const size_t at = (host.size() + 255) & ~(size_t)255;
        host.resize(at + bytes);
        std::memcpy(host.data() + at, p, bytes);
        return at;
    }
};

template <bool ENV>
int run(const gl_surface* surfaces, int n, SurviveArgs A, const std::vector<float> t[4], double* sums, float* d_env, cudaStream_t st)
{
    int dev = 0;
    GL_CUDA_TRY(cudaGetDevice(&dev));
    std::vector<SurfRec> recs((size_t)n);
    const int rc = pack_lens(surfaces, n, recs.data(), dev);
    if (rc) return rc;
    const std::vector<DispRec> disp = disp_records(surfaces, n);
    PupilMask mask = resolve_pupil_mask(surfaces, n, 0, 0.0f);
    mask.aspect = 1.0f;
    Staged in;
    const size_t o_recs = in.add(recs.data(), sizeof(SurfRec) * n), o_disp = in.add(disp.data(), sizeof(DispRec) * n);
    size_t o_t[4];
    for (int k = 0; k < 4; ++k) o_t[k] = in.add(t[k].data(), sizeof(float) * t[k].size());
    const int cells = A.m * A.m;
    const size_t o_cls = (in.host.size() + 255) & ~(size_t)255, o_val = (o_cls + (size_t)cells + 255) & ~(size_t)255;
    const size_t o_out = o_val + (ENV ? sizeof(float) : 3 * sizeof(double)) * (size_t)cells, bytes = o_out + 3 * sizeof(double);
    cudaMemPool_t pool;
    char* block = nullptr;
    GL_CUDA_TRY(shared_device_pool(dev, &pool));
    GL_CUDA_TRY(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&block), bytes, pool, st));
    cudaError_t e = cudaMemcpyAsync(block, in.host.data(), in.host.size(), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
    {
        A.recs = reinterpret_cast<SurfRec*>(block + o_recs);
        A.disp = reinterpret_cast<DispRec*>(block + o_disp);
        A.n_surf = n;
        A.cu = reinterpret_cast<float*>(block + o_t[0]);
        A.cv = reinterpret_cast<float*>(block + o_t[1]);
        A.ou = reinterpret_cast<float*>(block + o_t[2]);
        A.ov = reinterpret_cast<float*>(block + o_t[3]);
        A.cls = reinterpret_cast<unsigned char*>(block + o_cls);
        double* val = reinterpret_cast<double*>(block + o_val);
        double* out = reinterpret_cast<double*>(block + o_out);
        const int warps = kThreads / 32;
        classify_kernel<ENV><<<(cells + kThreads - 1) / kThreads, kThreads, 0, st>>>(A, mask);
        border_kernel<ENV><<<(cells + warps - 1) / warps, kThreads, 0, st>>>(A, mask, val, reinterpret_cast<float*>(val));
        if (ENV) dilate_kernel<<<(cells + 255) / 256, 256, 0, st>>>(reinterpret_cast<float*>(val), A.m, d_env);
        else total_kernel<<<1, 512, 0, st>>>(val, cells, out);
        e = cudaGetLastError();
        if (!ENV && e == cudaSuccess) e = cudaMemcpyAsync(sums, out, 3 * sizeof(double), cudaMemcpyDeviceToHost, st);
    }
    const cudaError_t f = cudaFreeAsync(block, st);
    // the staged block and the sums are host memory of this call
    const cudaError_t w = cudaStreamSynchronize(st);
    GL_CUDA_TRY(e);
    GL_CUDA_TRY(f);
    GL_CUDA_TRY(w);
    g_last_launches = 3;
    return GL_OK;
}

}  // namespace
}  // namespace gl

using namespace gl;

extern "C" {

int gl_survivor_center(const gl_surface* surfaces, int n, float lambda, const float* dir, float launch_z, float span_x,
                       float span_y, int scan, int ss, double* out, void* stream)
{
    if (!surfaces || n <= 0 || !dir || !out || scan < 2 || scan > 4096 || ss < 1 || ss > 64)
        return fail(GL_ERR_INVALID, "survivor_center: bad arguments");
    SurviveArgs A{};
    A.m = scan; A.ss = ss;
    A.lam = lambda; A.z = launch_z; A.dx = dir[0]; A.dy = dir[1]; A.dz = dir[2];
    std::vector<float> t[4];
    const float hx = span_x / (float)(scan - 1), hy = span_y / (float)(scan - 1);
    for (int k = 0; k < scan; ++k)
    {
        const float g = 2.0f * (float)k / (float)(scan - 1) - 1.0f;
        t[0].push_back(span_x * g);
        t[1].push_back(span_y * g);
    }
    for (int k = 0; k < ss; ++k)
    {
        const float o = 2.0f * ((float)k + 0.5f) / (float)ss - 1.0f;
        t[2].push_back(hx * o);
        t[3].push_back(hy * o);
    }
    return run<false>(surfaces, n, A, t, out, nullptr, (cudaStream_t)stream);
}

int gl_survivor_envelope(const gl_surface* surfaces, int n, float lambda, const float* dir, float launch_z, float cx, float cy,
                         float ep_x, float ep_y, int me, int ss, float* d_env, void* stream)
{
    if (!surfaces || n <= 0 || !dir || !d_env || me < 1 || me > 32768 || ss < 1 || ss > 64)
        return fail(GL_ERR_INVALID, "survivor_envelope: bad arguments");
    SurviveArgs A{};
    A.m = me; A.ss = ss;
    A.lam = lambda; A.z = launch_z; A.dx = dir[0]; A.dy = dir[1]; A.dz = dir[2];
    A.cx = cx; A.cy = cy; A.ep_x = ep_x; A.ep_y = ep_y;
    std::vector<float> t[4];
    const float du = 2.0f / (float)me;
    for (int k = 0; k < me; ++k) t[0].push_back(((float)k + 0.5f) / (float)me * 2.0f - 1.0f);
    for (int k = 0; k < ss; ++k) t[2].push_back(du * (((float)k + 0.5f) / (float)ss - 0.5f));
    t[1] = t[0];
    t[3] = t[2];
    return run<true>(surfaces, n, A, t, nullptr, d_env, (cudaStream_t)stream);
}

}  // extern "C"
