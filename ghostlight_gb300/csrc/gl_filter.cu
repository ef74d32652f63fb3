// gl_filter.cu — ghost-pair enumerator and energy culler on the device.
//
// Replaces filter_ghost_pairs (ghostlight/src/ghost.cpp:105-138).  One block
// per enumerated pair traces the reference's probes — three axial rays at
// 650/550/450 nm for the intensity estimate (ghost.cpp:34-50) and the 8x8
// green probe for the area boost (ghost.cpp:53-102; the 52 of its points inside
// the unit disc) — in one launch instead of 55 host traces per pair.
//
// The launch is one wave whose time is one trace of up to three passes over the
// lens by IEEE-exact steps, so what is in that chain counts:
//   * all of a block's rays walk together through one call site, geometry only:
//     whether a probe lands and where does not depend on its weight;
//   * the axial rays note each bend; their coating weights are worked out
//     afterwards, all bends in parallel, and multiplied in path order;
//   * the graze test's three silhouettes (below) are checks along one walk,
//     with a mask of the variants still alive, not three walks.
// 24 surfaces, 253 pairs: 442 -> 107 us (three variants of three warps each,
// the weights in the chain and the axial rays walked apart from the probe).
//
// This translation unit is compiled IEEE-exact (-fmad=false, IEEE division
// and square root, no flush-to-zero), so its float arithmetic equals the
// reference host build's except inside cosf / atan2f / fmodf / sinf, which may
// differ in the last place.  Two guards make the results the reference's:
//  * a keep/drop decision whose estimate lies within a guard band of the
//    threshold is re-evaluated on the host with the identical code compiled
//    by the host compiler;
//  * the only libm-dependent tests of a probe ray are the silhouettes of
//    polygon and curved-blade apertures (atan2f, fmodf, cosf, sinf), so on a
//    lens that has one the probes also run with every such clear radius
//    scaled by 1 + 1e-6 and 1 - 1e-6; a pair whose probe outcome (which rays
//    land, their weights and landing box) changes between the two has a ray
//    grazing a silhouette and is traced again on the host.
// The surviving set, its order, the area boosts and the footprints are then
// the reference's bit for bit.
#include "gl_internal.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

namespace gl {

namespace {

constexpr int kProbeThreads = 64;   // 3 intensity rays + 52 spread probes, padded

using ProbeOut = FilterProbe;
constexpr float kGraze = 1e-6f;     // relative clear-radius perturbation of the graze test

bool has_silhouette(const gl_surface* s, int n)
{
    for (int i = 0; i < n; ++i)
        if (s[i].aperture_shape == GL_APERTURE_POLYGON && s[i].aperture_blades >= 3) return true;
    return false;
}

bool same_probe(const ProbeOut& x, const ProbeOut& y)
{
    return std::memcmp(&x, &y, sizeof(ProbeOut)) == 0;
}

// One bend of an axial ray: what its weight needs (surface_weight and
// surface_attenuator of step(), gl_trace.cuh).
struct Bend {
    V3 d, nrm, hit;
    float n1, n2;
    int surf_refl;                  // surface, bit 16: reflected
};

// Shared memory of a block for n surfaces and walks of up to L bends.
size_t probe_smem(int n, int L)
{
    return sizeof(SurfRec) * n + sizeof(float) * 6 * n + (sizeof(Bend) + sizeof(float2)) * 3 * L + 16;
}

// recs: nv variants of n records (exact, then the widened and narrowed
// silhouettes of the graze test); open: the exact records with the silhouette
// surfaces' apertures opened; silhouettes: bit per such surface (none: nv = 1).
__global__ void __launch_bounds__(kProbeThreads)
filter_probe_kernel(const SurfRec* __restrict__ recs, const SurfRec* __restrict__ open, int n, int nv,
                    uint64_t silhouettes, const float* __restrict__ ior_at3, const float* __restrict__ ior_bf3,
                    const int2* __restrict__ pairs, float front_R, float start_z, int lmax, ProbeOut* __restrict__ out)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Bend* bends = reinterpret_cast<Bend*>(smem_raw);                 // [axial ray][lmax]
    float2* factors = reinterpret_cast<float2*>(bends + 3 * lmax);   // weight, attenuator
    SurfRec* lens = reinterpret_cast<SurfRec*>(factors + 3 * lmax);
    float* at = reinterpret_cast<float*>(lens + n);
    float* bf = at + 3 * n;
    __shared__ float px[64], py[64];
    __shared__ int ok[64];                                           // variants that land
    __shared__ int points[64];                                       // probe points inside the disc
    __shared__ int n_points[2];
    __shared__ int n_bends[3], axial_ok[3], end[3][3];               // [ray], [ray], [ray][variant]
    const int tid = threadIdx.x;
    {
        const int words = n * (int)(sizeof(SurfRec) / 4);
        const int* src = reinterpret_cast<const int*>(open);
        int* dst = reinterpret_cast<int*>(lens);
        for (int i = tid; i < words; i += kProbeThreads) dst[i] = src[i];
        for (int i = tid; i < 3 * n; i += kProbeThreads) { at[i] = ior_at3[i]; bf[i] = ior_bf3[i]; }
    }
    const float gu = ((tid % 8 + 0.5f) / 8) * 2.0f - 1.0f, gv = ((tid / 8 + 0.5f) / 8) * 2.0f - 1.0f;
    const bool inside = !(gu * gu + gv * gv > 1.0f);
    const unsigned m = __ballot_sync(0xffffffffu, inside);
    if ((tid & 31) == 0) n_points[tid >> 5] = __popc(m);
    ok[tid] = 0;
    __syncthreads();
    if (inside) points[(tid >= 32 ? n_points[0] : 0) + __popc(m & ((1u << (tid & 31)) - 1u))] = tid;
    __syncthreads();
    const int2 p = pairs[blockIdx.x];
    const int a = p.x, b = p.y, L1 = b + 1, L2 = L1 + (b - a), L = L2 + (n - 1 - a);
    const bool axial = tid < 3;
    if (tid < 3 + n_points[0] + n_points[1])
    {
        const int k = axial ? 0 : points[tid - 3], li = axial ? tid : 1;
        const float u = ((k % 8 + 0.5f) / 8) * 2.0f - 1.0f;
        const float v = ((k / 8 + 0.5f) / 8) * 2.0f - 1.0f;
        V3 o = axial ? v3(0.0f, 0.0f, start_z) : v3(u * front_R, v * front_R, start_z);
        V3 d = v3(0.0f, 0.0f, 1.0f);
        const float* la = at + li * n;
        const float* lb = bf + li * n;
        float cur = 1.0f;
        int alive = (1 << nv) - 1, cnt = 0;
        #pragma unroll 1
        for (int q = 0; q < L && alive; ++q)
        {
            // the three legs of trace_ghost
            int s; bool refl, back = false;
            if (q < L1)      { s = q;                refl = (s == b); }
            else if (q < L2) { s = 2 * b - q;        refl = (s == a); back = true; }
            else             { s = a + 1 + (q - L2); refl = false; }
            const SurfRec& S = lens[s];
            if (!(S.flags & SF_ACTIVE)) continue;
            const float n1 = cur, n2 = back ? lb[s] : la[s];
            float t = 0.0f;
            V3 nrm, nd;
            int left = 0;
            if (intersect(o, d, S, t, nrm))
            {
                left = alive;
                if ((silhouettes >> s) & 1)
                {
                    // the hit in the surface's frame, as intersect() forms it
                    V3 lo = o, ld = d;
                    if (S.flags & SF_TRANSFORMED)
                    {
                        lo = m3tmul(S.rot, o - v3(S.dec_x, S.dec_y, S.z)) + v3(0.0f, 0.0f, S.z);
                        ld = m3tmul(S.rot, d);
                    }
                    const V3 hit = lo + ld * t;
                    for (int w = 0; w < nv; ++w)
                        if (((left >> w) & 1) && !check_aperture(hit, recs[w * n + s])) left &= ~(1 << w);
                }
                if (!refl && left && !refract(d, nrm, n1, n2, nd)) left = 0;
            }
            // a variant that ends here has the weight of the bends so far
            if (axial)
                for (int w = 0; w < nv; ++w)
                    if (((alive & ~left) >> w) & 1) end[tid][w] = cnt;
            alive = left;
            if (!alive) break;
            const V3 hit = o + d * t;
            if (axial)
            {
                Bend B;
                B.d = d; B.nrm = nrm; B.hit = hit; B.n1 = n1; B.n2 = n2;
                B.surf_refl = s | (refl ? 1 << 16 : 0);
                bends[tid * lmax + cnt] = B;
            }
            ++cnt;
            o = hit;
            if (refl)
            {
                d = reflect(d, nrm);
                cur = back ? la[a] : cur;
            }
            else
            {
                d = nd;
                cur = n2;
            }
        }
        TraceOut r;
        r.status = 1;
        if (alive) to_sensor(o, d, r);
        const int landed = r.status == 0 ? alive : 0;
        if (axial)
        {
            n_bends[tid] = cnt;
            axial_ok[tid] = landed;
            for (int w = 0; w < nv; ++w)
                if ((alive >> w) & 1) end[tid][w] = cnt;
        }
        else
        {
            ok[k] = landed;
            if (landed) { px[k] = r.x; py[k] = r.y; }
        }
    }
    __syncthreads();
    // the bends' weights, all at once
    const float lams[3] = {650.0f, 550.0f, 450.0f};
    for (int i = tid; i < 3 * lmax; i += kProbeThreads)
    {
        const int r = i / lmax;
        if (i - r * lmax >= n_bends[r]) continue;
        const Bend B = bends[i];
        const SurfRec& S = lens[B.surf_refl & 0xffff];
        factors[i] = make_float2(surface_weight(B.d, B.nrm, B.n1, B.n2, S, lams[r], (B.surf_refl >> 16) != 0),
                                 surface_attenuator(B.hit, S));
    }
    __syncthreads();
    if (tid < 3 * nv)
    {
        const int w = tid / 3, r = tid - 3 * w;
        ProbeOut* q = out + (size_t)w * gridDim.x + blockIdx.x;
        float weight = 1.0f;
        for (int i = 0; i < end[r][w]; ++i)
        {
            const float2 f = factors[r * lmax + i];
            weight *= f.x;
            weight *= f.y;
        }
        q->w[r] = weight;
        q->wok[r] = (axial_ok[r] >> w) & 1;
    }
    else if (tid >= 32 && tid < 32 + nv)
    {
        const int w = tid - 32;
        ProbeOut* q = out + (size_t)w * gridDim.x + blockIdx.x;
        float mnx = 1e30f, mxx = -1e30f, mny = 1e30f, mxy = -1e30f;
        int valid = 0;
        for (int k = 0; k < 64; ++k)
        {
            if (!((ok[k] >> w) & 1)) continue;
            mnx = fminf(mnx, px[k]); mxx = fmaxf(mxx, px[k]);
            mny = fminf(mny, py[k]); mxy = fmaxf(mxy, py[k]);
            ++valid;
        }
        q->mnx = mnx; q->mxx = mxx; q->mny = mny; q->mxy = mxy; q->valid = valid;
    }
}

}  // namespace
}  // namespace gl

using namespace gl;

// Device scratch of the filter, kept per device and grown on demand (never
// shrunk): a per-call cudaMalloc/cudaFree pair would cost a device-wide
// synchronisation each call, stalling whatever other streams have in flight
// (the reference keeps its ghost buffers in a leaked cache for the same
// reason, ghost_render.cu:505-510).  The mutex serialises callers; each call
// finishes its copies before it returns.
namespace {
std::mutex g_scratch_mu;
struct Scratch { void* ptr = nullptr; size_t bytes = 0; };
Scratch g_scratch[64];

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
}  // namespace

extern "C" int gl_filter_ghost_pairs(const gl_surface* surfaces, int n, float hw, float hh,
                                     const gl_filter_params* prm, gl_ghost_pair* out_pairs,
                                     float* out_boosts, float* out_fp, int cap, int* n_out,
                                     int* n_rechecked)
{
    if (!surfaces || n <= 0 || !prm || !n_out) return fail(GL_ERR_INVALID, "filter_ghost_pairs: bad arguments");
    std::vector<SurfRec> recs((size_t)n);
    int rc = pack_lens(surfaces, n, recs.data(), kTablesHost);     // the host re-check's records
    if (rc) return rc;

    // Enumerate (ghost.cpp:17-31) and apply the IOR-contrast test
    // (ghost.cpp:118-125) — exact float comparisons, done here.
    std::vector<int2> cand;
    for (int a = 0; a < n; ++a)
    {
        if (!surfaces[a].is_active) continue;
        for (int b = a + 1; b < n; ++b)
        {
            if (!surfaces[b].is_active) continue;
            float iba = ior_before_nd(surfaces, a), iaa = surfaces[a].ior;
            float ibb = ior_before_nd(surfaces, b), iab = surfaces[b].ior;
            if (std::abs(iba - iaa) < 0.001f || std::abs(ibb - iab) < 0.001f) continue;
            cand.push_back(make_int2(a, b));
        }
    }
    int rechecked = 0;
    int kept = 0;
    if (!cand.empty())
    {
        const float lams[3] = {650.0f, 550.0f, 450.0f};
        std::vector<float> at(3 * (size_t)n), bf(3 * (size_t)n);
        build_ior_tables(surfaces, n, lams, 3, at.data(), bf.data());
        const int np = (int)cand.size();
        const int nv = has_silhouette(surfaces, n) ? 3 : 1;         // record variants of the graze test
        std::vector<ProbeOut> res((size_t)np * nv);
        cudaError_t e = cudaSuccess;
        auto chk = [&](cudaError_t x) { if (e == cudaSuccess) e = x; };
        // one block: records of the variants and the opened set, tables, pairs; then the results
        const size_t o_at = align256(sizeof(SurfRec) * n * (nv + 1)), o_bf = o_at + align256(sizeof(float) * 3 * n);
        const size_t o_pairs = o_bf + align256(sizeof(float) * 3 * n);
        const size_t o_out = o_pairs + align256(sizeof(int2) * np);
        const size_t need = o_out + align256(sizeof(ProbeOut) * np * nv);
        int dev = 0;
        chk(cudaGetDevice(&dev));
        if (e == cudaSuccess && (dev < 0 || dev >= 64)) e = cudaErrorInvalidDevice;
        std::vector<SurfRec> drecs((size_t)n * (nv + 1));           // the device probes' records
        uint64_t silhouettes = 0;
        int lmax = 0;
        for (const int2& c : cand) lmax = std::max(lmax, (c.y + 1) + (c.y - c.x) + (n - 1 - c.x));
        if (e == cudaSuccess)
        {
            rc = pack_lens(surfaces, n, drecs.data(), dev);
            if (rc) return rc;
            for (int v = 1; v < nv; ++v)
            {
                std::vector<gl_surface> moved(surfaces, surfaces + n);
                const float f = v == 1 ? 1.0f + kGraze : 1.0f - kGraze;
                for (gl_surface& g : moved)
                    if (g.aperture_shape == GL_APERTURE_POLYGON && g.aperture_blades >= 3) g.semi_aperture *= f;
                rc = pack_lens(moved.data(), n, drecs.data() + (size_t)v * n, dev);
                if (rc) return rc;
            }
            for (int i = 0; i < n; ++i)
            {
                SurfRec& open = drecs[(size_t)nv * n + i];
                open = drecs[i];
                if (nv == 1 || surfaces[i].aperture_shape != GL_APERTURE_POLYGON || surfaces[i].aperture_blades < 3) continue;
                silhouettes |= (uint64_t)1 << i;
                open.shape = 0;
                open.semi_ap = INFINITY;
            }
        }
        std::unique_lock<std::mutex> lock(g_scratch_mu);
        Scratch& sc = g_scratch[e == cudaSuccess ? dev : 0];
        if (e == cudaSuccess && sc.bytes < need)
        {
            if (sc.ptr) cudaFree(sc.ptr);
            sc.ptr = nullptr;
            sc.bytes = 0;
            chk(cudaMalloc(&sc.ptr, need));
            if (e == cudaSuccess) sc.bytes = need;
        }
        char* base = static_cast<char*>(sc.ptr);
        SurfRec* d_recs = reinterpret_cast<SurfRec*>(base);
        float* d_at = reinterpret_cast<float*>(base + o_at);
        float* d_bf = reinterpret_cast<float*>(base + o_bf);
        int2* d_pairs = reinterpret_cast<int2*>(base + o_pairs);
        ProbeOut* d_out = reinterpret_cast<ProbeOut*>(base + o_out);
        if (e == cudaSuccess)
        {
            std::vector<char> host(o_out);
            std::memcpy(host.data(), drecs.data(), sizeof(SurfRec) * drecs.size());
            std::memcpy(host.data() + o_at, at.data(), sizeof(float) * 3 * n);
            std::memcpy(host.data() + o_bf, bf.data(), sizeof(float) * 3 * n);
            std::memcpy(host.data() + o_pairs, cand.data(), sizeof(int2) * np);
            chk(cudaMemcpy(base, host.data(), o_out, cudaMemcpyHostToDevice));
            const size_t smem = probe_smem(n, lmax);
            if (e == cudaSuccess && smem > 46 * 1024) chk((cudaError_t)raise_smem_limit((const void*)filter_probe_kernel, smem));
        }
        if (e == cudaSuccess)
        {
            const float front_R = surfaces[0].semi_aperture;
            const float start_z = surfaces[0].z - kSpawnOffset;
            filter_probe_kernel<<<np, kProbeThreads, probe_smem(n, lmax)>>>(d_recs, d_recs + (size_t)nv * n, n, nv,
                                                                          silhouettes, d_at, d_bf, d_pairs, front_R,
                                                                          start_z, lmax, d_out);
            chk(cudaGetLastError());
            chk(cudaMemcpy(res.data(), d_out, sizeof(ProbeOut) * np * nv, cudaMemcpyDeviceToHost));
        }
        lock.unlock();
        if (e != cudaSuccess)
            return fail(e == cudaErrorMemoryAllocation ? GL_ERR_OOM : GL_ERR_CUDA,
                        std::string("filter_ghost_pairs: ") + cudaGetErrorString(e));
        g_last_launches = 1;

        const float thr = prm->min_ghost_intensity;
        for (int i = 0; i < np; ++i)
        {
            ProbeOut r = res[i];
            if (nv == 3 && !(same_probe(res[(size_t)np + i], res[(size_t)2 * np + i]) &&
                             same_probe(res[i], res[(size_t)np + i])))
            {
                // a probe ray grazes a polygon / blade silhouette: trace the
                // pair's probes again on the host
                host_filter_probe(surfaces, recs.data(), n, cand[i].x, cand[i].y, &r);
                ++rechecked;
            }
            // estimate_ghost_intensity's sum order: total += w650, w550, w450
            float total = 0.0f;
            for (int ch = 0; ch < 3; ++ch)
                if (r.wok[ch]) total += r.w[ch];
            float est = total / 3.0f;
            const float band = 1e-4f * std::fabs(thr);
            if (!(std::fabs(est - thr) > band))
            {
                est = host_intensity_estimate(surfaces, recs.data(), n, cand[i].x, cand[i].y);
                ++rechecked;
            }
            if (est < thr) continue;
            float boost = 1.0f;
            if (prm->ghost_normalize)
            {
                if (r.valid >= 2)
                {
                    float gw = std::max(r.mxx - r.mnx, 0.01f), gh = std::max(r.mxy - r.mny, 0.01f);
                    float area = (gw * gh) / ((2.0f * hw) * (2.0f * hh));
                    boost = (area < 1.0f) ? 1.0f : (prm->max_area_boost < area) ? prm->max_area_boost : area;
                }
            }
            if (out_pairs && kept < cap)
            {
                out_pairs[kept] = {cand[i].x, cand[i].y};
                if (out_boosts) out_boosts[kept] = boost;
                if (out_fp)
                {
                    out_fp[2 * kept] = (r.valid >= 2) ? r.mxx - r.mnx : 0.0f;
                    out_fp[2 * kept + 1] = (r.valid >= 2) ? r.mxy - r.mny : 0.0f;
                }
            }
            ++kept;
        }
    }
    *n_out = kept;
    if (n_rechecked) *n_rechecked = rechecked;
    if (out_pairs && kept > cap) return fail(GL_ERR_INVALID, "filter_ghost_pairs: capacity too small");
    return GL_OK;
}
