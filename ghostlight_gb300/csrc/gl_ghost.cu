// gl_ghost.cu — batched ghost trace + splat (the scatter of
// launch_ghost_render, ghostlight/src/ghost_render.cu:209-491 and :630-1442).
//
// GB300 layout
//   * A render plan keeps everything the trace reads resident in HBM: packed
//     lens records, per-wavelength IOR slices, the spectral table, the pupil
//     grids (one per pair; grids may differ in size), per-source beam data and
//     a list of work items = (pair, source, 256-sample tile).
//   * ONE persistent launch covers every pair x source: each CTA stages the
//     lens table and IOR slices in shared memory once, then pops tasks from a
//     global counter until none is left.  The pairs that sample one grid are
//     walked as a tree that shares their common legs (ghost_tree_kernel).
//     Launch-bound per-ghost loops and their tail effects disappear; the plan
//     executes with kernel launches only, so it can be captured in a CUDA graph.
//   * The reference's per-pair launch loop (ghost_render.cu:1544-1557) is kept
//     as `plain_per_pair` — the same kernel, one launch per pair, no queue.
//   * Splat: the reference issues 12 scalar float atomics per surviving
//     ray-wavelength.  Here the accumulator is RGBA float4, one 16-byte vector
//     atomic per tap; a warp whose landings share one footprint sums them first.
//     The pair-by-pair walk carries its current 2x2 footprint across the
//     wavelength loop and flushes it when it moves.
//   * The flush kernel reads the RGBA accumulator once, applies the 3x3
//     spectral correction (ghost_render.cu:610-622, same rounding order) and
//     writes the three planar float32 outputs with coalesced vector stores.
#include "gl_disp.cuh"
#include "gl_render.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

namespace gl {

#ifndef GL_RENDER_MIN_BLOCKS
#define GL_RENDER_MIN_BLOCKS 8
#endif
constexpr int kRenderMinBlocks = GL_RENDER_MIN_BLOCKS;
constexpr unsigned kFull = 0xffffffffu;

// Per-lane splat footprint kept in shared memory (12 floats, stride 13 so the
// lanes of a warp fall in distinct banks) together with its 2x2 origin.
constexpr int kAccStride = 13;
constexpr int kLaneFloats = 14;      // a lane's shared memory: the footprint, or two ray states of the tree walk

__device__ __forceinline__ void flush_taps(float4* accum, int W, int H, int cx, int cy, const float* acc)
{
    #pragma unroll
    for (int k = 0; k < 4; ++k)
    {
        const int xi = cx + (k & 1), yi = cy + (k >> 1);
        if (xi < 0 || xi >= W || yi < 0 || yi >= H) continue;
        const float r = acc[3 * k], g = acc[3 * k + 1], b = acc[3 * k + 2];
        if (r == 0.0f && g == 0.0f && b == 0.0f) continue;
        atomicAdd(accum + ((size_t)yi * W + xi), make_float4(r, g, b, 0.0f));
    }
}

// ---- render-path surface interaction --------------------------------------
// Same physics as trace_surface_step (trace.cpp:84-135), arranged for the
// render kernel: the common case (untilted sphere or plane, round aperture,
// single-layer coating) is straight-line code; the general intersection
// (asphere Newton solve, cylinder, tilted/decentred frame) and the polygon
// stop are inlined behind warp-uniform branches (an out-of-line call saved
// and restored registers through local memory: measured 2% slower on the
// aspheric wide-angle frame, 8% on the decentred anamorphic sweep); other
// coating models stay out of line.

// Sphere or plane in the vertex-plane form c*|q|^2 - 2*q_z = 0 (q relative to
// the vertex, c = 1/R, c = 0 for a plane).  The ray is first moved to the
// vertex plane, then the root nearest to it is taken in the
// cancellation-free product form t = -C / (B + sign(B) sqrt(B^2 - A C)).
// Choosing the root with the smaller |t| is choosing the hit whose z lies
// nearer the vertex, which is the reference's root rule (trace_core.h:
// 505-515); unlike b^2 - 4ac about the centre of curvature, this form loses
// no precision for large radii or rays near the vertex.
//
// Every lane of the warp runs it (a lane whose ray is dead computes values
// nobody reads): it returns whether the ray hits instead of leaving early, so
// the lock-step walk pays for no divergent branches; the rare far-root case
// is a warp-uniform branch.
__device__ __forceinline__ bool sphere_hit(V3 o, V3 d, float z_s, float c, float& t_out, V3& q_out)
{
    const float t0 = (z_s - o.z) / d.z;
    const float px = o.x + d.x * t0, py = o.y + d.y * t0;
    const float A = c * (d.x * d.x + d.y * d.y + d.z * d.z);   // c |d|^2
    const float B = c * (px * d.x + py * d.y) - d.z;
    const float C = c * (px * px + py * py);
    const float disc = B * B - A * C;
    // den = B + sign(B) sqrt(disc) vanishes only when B = 0 and disc = 0,
    // i.e. A C = 0: A = 0 is a plane, whose B = -d_z, and C = 0 puts the
    // vertex-plane point on the axis, where B = -d_z too; with |d_z| >= 1e-12
    // neither can happen, so a live ray never divides by zero here
    const float den = B + copysignf(sqrtf(disc), B);
    const float ts = -C / den;
    float t = t0 + ts;
    bool ok = (fabsf(d.z) >= 1e-12f) & (disc >= 0.0f);
    const bool near = t > 1e-6f;
    if (__any_sync(kFull, ok & !near))
    {
        // the near root is behind the ray: the far root, if any, is the hit
        const float tb = t0 + (C / A) / ts;
        const bool far = (A != 0.0f) & (ts != 0.0f) & (tb > 1e-6f);
        ok = ok & (near | far);
        t = near ? t : tb;
    }
    t_out = t;
    q_out = v3(o.x + d.x * t, o.y + d.y * t, o.z + d.z * t - z_s);
    return ok;
}

__device__ __forceinline__ bool check_polygon(float hx, float hy, float h2, const SurfRec& s)
{
    float r = sqrtf(h2);
    if (r < 1e-9f) return true;
    if (s.blade.deformed) return r <= s.semi_ap * blade_radius_at(s.blade, atan2f(hy, hx));
    const float angle = atan2f(hy, hx) - s.rot_rad;
    float off = fmodf(angle, s.sector);
    if (off < 0.0f) off += s.sector;
    off -= 0.5f * s.sector;
    return r <= s.apothem / cosf(off);
}

__device__ __forceinline__ bool aperture_ok(float x, float y, const SurfRec& s)
{
    const float hx = x / s.aspect, hy = y;
    const float h2 = hx * hx + hy * hy;
    if (!(h2 <= s.semi_ap * s.semi_ap)) return false;
    if (s.shape == 1) return check_polygon(hx, hy, h2, s);
    if (s.shape == 2) return image_aperture_ok(x, y, s);
    return true;
}

// Everything but an untilted sphere/plane: the shared reference formulation.
__device__ __forceinline__ bool intersect_general(V3 o, V3 d, const SurfRec& s, float& t, V3& nrm)
{
    return intersect(o, d, s, t, nrm);
}

__device__ __noinline__ float weight_general(V3 d, V3 nrm, float n1, float n2, const SurfRec& s,
                                             float lam, bool reflecting)
{
    return surface_weight(d, nrm, n1, n2, s, lam, reflecting);
}

__device__ __noinline__ float attenuator_general(V3 hit, const SurfRec& s)
{
    return surface_attenuator(hit, s);
}

// The per-step fields of one surface packed into two 16-byte words (two
// vector shared-memory loads per step instead of a dozen scalar ones).
struct __align__(16) HotRec {
    float z, c, sa2, inv_aspect;
    int bits, ar_layers;
    float ar_scale;                 // 0.25^(ar_layers - 1): the extra AR layers of the SIMPLE model
    int pad;
};
// HB_FAST: the common surface — active, untilted sphere or plane, round or
// elliptical stop, single-layer coating with at least one layer, no
// attenuator — whose step is one straight-line path behind one test.
// HB_ROUND: an HB_FAST surface whose stop is round (aspect 1).
// HB_COMMON: a surface of any form and stop with HB_FAST's coating.
enum HotBits { HB_ACTIVE = 1, HB_GENERAL = 2, HB_POLYGON = 4, HB_SIMPLE = 8, HB_ATTEN = 16, HB_IMAGE = 32,
               HB_FAST = 64, HB_ROUND = 128, HB_COMMON = 256 };

__device__ __forceinline__ HotRec make_hot(const SurfRec& s)
{
    HotRec h;
    h.z = s.z;
    h.c = (fabsf(s.radius) < 1e-6f) ? 0.0f : s.inv_r;
    h.sa2 = s.semi_ap * s.semi_ap;
    h.inv_aspect = 1.0f / s.aspect;
    h.bits = ((s.flags & SF_ACTIVE) ? HB_ACTIVE : 0) |
             ((s.form != 0 || (s.flags & SF_TRANSFORMED)) ? HB_GENERAL : 0) |
             ((s.shape == 1) ? HB_POLYGON : 0) | ((s.coating == 0) ? HB_SIMPLE : 0) |
             ((s.coating == 4) ? HB_ATTEN : 0) | ((s.shape == 2) ? HB_IMAGE : 0);
    if (h.bits == (HB_ACTIVE | HB_SIMPLE) && s.ar_layers >= 1) h.bits |= HB_FAST | (s.aspect == 1.0f ? HB_ROUND : 0);
    if ((h.bits & (HB_ACTIVE | HB_SIMPLE | HB_ATTEN)) == (HB_ACTIVE | HB_SIMPLE) && s.ar_layers >= 1) h.bits |= HB_COMMON;
    h.ar_layers = s.ar_layers;
    h.ar_scale = 1.0f;
    for (int i = 1; i < s.ar_layers; ++i) h.ar_scale *= 0.25f;
    h.pad = 0;
    return h;
}

// Single-layer MgF2 reflectance (coating_reflectance / surface_reflectance,
// fresnel.h:92-178) with the film phase factor 2*pi*n_c*d/lambda supplied per
// wavelength (kdelta) and cos(2 delta) formed as 2 cos^2(delta) - 1: delta is
// below pi here, where the SFU cosine is accurate.
//
// The Airy sum R = (r01^2 + r12^2 + 2 r01 r12 c) / (1 + r01^2 r12^2 + 2 r01 r12 c)
// with r01 = A/B, r12 = C/D is evaluated as one quotient of the numerators
// and denominators scaled by (B D)^2 — one division where the textbook form
// has three.  cos_2 >= 0 is the substrate-side cosine when the caller already
// has it (a refraction's transmitted cosine: the film keeps n sin(theta), so
// it is the same angle); cos_2 < 0 computes it here.
// HAVE_COS2: cos_2 is the substrate-side cosine (a refraction's transmitted
// cosine); otherwise it is computed here.  The film-TIR fallbacks to the bare
// Fresnel reflectance are rare: they are taken as warp-uniform branches and
// selected per lane (every lane of the warp calls this).
// LAYERED: the caller knows the surface has at least one layer.
// Returns R before the extra layers' scale, which it leaves in `scale` (1 for
// the bare Fresnel fallbacks), so a refraction's weight 1 - scale R is one FMA.
template <bool HAVE_COS2, bool LAYERED = false>
__device__ __forceinline__ float mgf2_reflectance(float cos_i, float n1, float n2, int layers, float ar_scale,
                                                  float kdelta, float cos_2, float& scale)
{
    scale = 1.0f;
    if (!LAYERED && layers <= 0) return fresnel_reflectance(cos_i, n1, n2);
    const float cn = 1.38f;
    const float a1 = n1 * (1.0f / cn);
    const float sin2_c = a1 * a1 * (1.0f - cos_i * cos_i);
    const float cos_c = sqrtf(1.0f - sin2_c);
    bool bare = sin2_c >= 1.0f;
    if (!HAVE_COS2)
    {
        const float a2 = cn / n2;
        const float sin2_2 = a2 * a2 * (1.0f - cos_c * cos_c);
        bare = bare | (sin2_2 >= 1.0f);
        cos_2 = sqrtf(1.0f - sin2_2);
    }
    const float p1 = n1 * cos_i, pc = cn * cos_c, p2 = n2 * cos_2;
    const float A = p1 - pc, B = p1 + pc, Cn = pc - p2, D = pc + p2;
    const float AD = A * D, CB = Cn * B, BD = B * D, AC = A * Cn;
    const float cd = __cosf(kdelta * cos_c);
    const float c2d = 2.0f * cd * cd - 1.0f;
    const float x = 2.0f * AC * BD * c2d;
    float R = (AD * AD + CB * CB + x) / (BD * BD + AC * AC + x);
    R = fminf(fmaxf(R, 0.0f), 1.0f);
    scale = ar_scale;
    if (__any_sync(kFull, bare))
    {
        const float Rb = fresnel_reflectance(cos_i, n1, n2);
        R = bare ? Rb : R;
        scale = bare ? 1.0f : ar_scale;
    }
    return R;
}

// Snell's law as refract_ray (trace_core.h:533-552), renormalised like it:
// the walk's directions then stay unit to rounding over every interaction
// (a drift in |d| would bias the next surface's root and the landing).
// ci = -dot(nrm, d) >= 0; returns the transmitted cosine (for the coating)
// and clears ok on total internal reflection.
__device__ __forceinline__ float refract_unit(V3& d, V3 nrm, float ci, float n1, float n2, bool& ok)
{
    const float nr = n1 / n2;
    const float s2t = nr * nr * (1.0f - ci * ci);
    ok = ok & (s2t < 1.0f);
    const float ct = sqrtf(1.0f - s2t);
    d = d * nr + nrm * (nr * ci - ct);
    d = d * rsqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
    return ct;
}

// The step of an HB_FAST surface: the common path of surface_step below with
// none of its per-kind tests (same arithmetic, same result).
// ROUND: the stop is round (no aspect scaling).  reflect_ior is read only
// on a reflecting step: through ior_a (the IOR after surface a) when the walk
// runs backward, else it is the current medium.
// COMMON: any HB_COMMON surface (s: its record).  Other forms and stops take
// their own way to the hit and the normal and join the path there.
template <bool WEIGHT, bool ROUND, bool COMMON = false>
__device__ __forceinline__ bool surface_step_fast(V3& o, V3& d, const HotRec& h, float kdelta, float n2,
                                                  bool reflecting, bool back, const float2* ior_a, float& cur,
                                                  float& w, bool alive, const SurfRec* s = nullptr)
{
    bool ok;
    V3 nrm;
    if (!COMMON || (h.bits & HB_FAST))
    {
        const float c = h.c;
        V3 q;
        float t;
        ok = alive & sphere_hit(o, d, h.z, c, t, q);
        const float hx = ROUND ? q.x : q.x * h.inv_aspect, hy = q.y;
        ok = ok & (hx * hx + hy * hy <= h.sa2);
        nrm = v3(c * q.x, c * q.y, c * q.z - 1.0f);
        o = v3(q.x, q.y, q.z + h.z);
    }
    else if (h.bits & HB_GENERAL)
    {
        float t = 0.0f;
        ok = alive && intersect_general(o, d, *s, t, nrm);
        o = o + d * t;
    }
    else
    {
        const float c = h.c;
        V3 q;
        float t;
        ok = alive & sphere_hit(o, d, h.z, c, t, q);
        const float hx = q.x * h.inv_aspect, hy = q.y;
        const float h2 = hx * hx + hy * hy;
        ok = ok & (h2 <= h.sa2);
        if (h.bits & HB_POLYGON) ok = ok & check_polygon(hx, hy, h2, *s);
        else if ((h.bits & HB_IMAGE) && ok) ok = image_aperture_ok(q.x, q.y, *s);
        nrm = v3(c * q.x, c * q.y, c * q.z - 1.0f);
        o = v3(q.x, q.y, q.z + h.z);
    }
    // The normal is not turned to oppose the ray: with cr = -nrm.d, ci = |cr|
    // and sg the sign of cr, reflection d + (sg nrm)(2 ci) = d + nrm (2 cr)
    // and Snell's nr d + (sg nrm)(nr ci - ct) = nr d + nrm (nr cr - sg ct),
    // the signs cancelling exactly.
    const float cr = -dot(nrm, d);
    const float ci = fabsf(cr);
    const float n1 = cur;
    if (reflecting)
    {
        if (WEIGHT)
        {
            float sc;
            const float R = mgf2_reflectance<false, true>(ci, n1, n2, h.ar_layers, h.ar_scale, kdelta, -1.0f, sc);
            w *= R * sc;
        }
        d = d + nrm * (2.0f * cr);
        d = d * rsqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
        cur = back ? ior_a->x : cur;
    }
    else
    {
        const float nr = n1 / n2;
        const float s2t = nr * nr * (1.0f - ci * ci);
        ok = ok & (s2t < 1.0f);
        const float ct = sqrtf(1.0f - s2t);
        d = d * nr + nrm * fmaf(nr, cr, cr < 0.0f ? ct : -ct);
        d = d * rsqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
        if (WEIGHT)
        {
            float sc;
            const float R = mgf2_reflectance<true, true>(ci, n1, n2, h.ar_layers, h.ar_scale, kdelta, ct, sc);
            w *= fmaf(-R, sc, 1.0f);
        }
        cur = n2;
    }
    return ok;
}

// One surface interaction on the lane's ray; returns whether the ray lives
// on.  Every lane of the warp runs it, whether or not its ray is still alive
// (the walk is lock-step, so a lane leaving early saves no issue slot, only
// adds branch and reconvergence instructions): the geometry of the common
// path (untilted sphere or plane, round stop, single-layer coating) is
// straight-line code whose tests fold into the result, and the caller
// ignores the state of a lane whose ray died.  Branches are on the
// surface's kind (the same for every lane) or warp-uniform votes; the
// out-of-line weight models and bitmap stops, which index memory with the
// ray's values, run only for lanes whose ray is alive.
// WEIGHT = false skips the energy weight: whether a ray dies (missed,
// clipped, TIR) is geometry only (trace_cuda.h sets the status from geometry
// alone), so the off-sensor probe needs none of it.
template <bool WEIGHT>
__device__ __forceinline__ bool surface_step(V3& o, V3& d, const HotRec& h, const SurfRec& s, float lam,
                                             float kdelta, float n2, bool reflecting, float reflect_ior,
                                             float& cur, float& w, bool alive)
{
    V3 nrm, hit;
    bool ok;
    if (!(h.bits & HB_GENERAL))
    {
        const float c = h.c;
        V3 q;
        float t;
        ok = alive & sphere_hit(o, d, h.z, c, t, q);
        const float hx = q.x * h.inv_aspect, hy = q.y;
        const float h2 = hx * hx + hy * hy;
        ok = ok & (h2 <= h.sa2);
        // one test on the common path: plain circular / elliptical stops
        if (h.bits & HB_POLYGON) ok = ok & check_polygon(hx, hy, h2, s);
        else if ((h.bits & HB_IMAGE) && ok) ok = image_aperture_ok(q.x, q.y, s);
        // outward normal (c q_x, c q_y, c q_z - 1), turned to oppose the ray
        // (for a plane, c = 0, it is (0, 0, -1) as it stands)
        nrm = v3(c * q.x, c * q.y, c * q.z - 1.0f);
        hit = v3(q.x, q.y, q.z + h.z);
    }
    else
    {
        float t = 0.0f;
        ok = alive && intersect_general(o, d, s, t, nrm);
        hit = o + d * t;
    }
    float ci = -dot(nrm, d);
    if (ci < 0.0f) { nrm = -nrm; ci = -ci; }
    o = hit;
    const float n1 = cur;
    const bool simple = (h.bits & HB_SIMPLE) != 0;
    if (reflecting)
    {
        if (WEIGHT)
        {
            if (simple)
            {
                float sc;
                const float R = mgf2_reflectance<false>(ci, n1, n2, h.ar_layers, h.ar_scale, kdelta, -1.0f, sc);
                w *= R * sc;
            }
            else if (ok) w *= weight_general(d, nrm, n1, n2, s, lam, true);
            if (h.bits & HB_ATTEN) w *= attenuator_general(hit, s);
        }
        d = d + nrm * (2.0f * ci);
        d = d * rsqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
        cur = reflect_ior;
    }
    else
    {
        const V3 d_in = d;
        const float ct = refract_unit(d, nrm, ci, n1, n2, ok);
        if (WEIGHT)
        {
            if (simple)
            {
                float sc;
                const float R = mgf2_reflectance<true>(ci, n1, n2, h.ar_layers, h.ar_scale, kdelta, ct, sc);
                w *= fmaf(-R, sc, 1.0f);
            }
            else if (ok) w *= weight_general(d_in, nrm, n1, n2, s, lam, false);
            if (h.bits & HB_ATTEN) w *= attenuator_general(hit, s);
        }
        cur = n2;
    }
    return ok;
}

// The three legs of trace_ghost_ray (trace.cpp:196-233) flattened into one
// step sequence k = 0 .. L-1 with a single step site.  The warp walks the
// sequence in lock step for one wavelength at a time: the surface, its form,
// its aperture shape, reflect-or-refract and the IOR pair are the same for
// every lane (uniform branches, broadcast shared-memory reads); only the ray
// state differs.  The walk stops as soon as every lane's ray has died.
__device__ __forceinline__ void splat_ray(const RenderArgs& A, const PairDev& P, const SourceDev& S,
                                          const float4& sp, V3 o, V3 d, float w,
                                          int& cx, int& cy, float* acc)
{
    // propagate_to_sensor (trace.cpp:147-162), then the splat (ghost_render.cu:423-463)
    if (!(fabsf(d.z) >= 1e-12f)) return;
    const float ts = -o.z / d.z;
    if (!(ts >= 0.0f)) return;
    const float rx = o.x + d.x * ts, ry = o.y + d.y * ts;
    if (!isfinite(rx) || !isfinite(ry)) return;
    const float base = w * P.w_ray * A.gain * P.boost;
    if (base < 1e-14f) return;
    float px = (rx / A.hw2 + 0.5f) * A.fmt_w + A.fmt_x0;
    float py = (ry / A.hh2 + 0.5f) * A.fmt_h + A.fmt_y0;
    if (!isfinite(px) || !isfinite(py)) return;
    px = fmaxf(-2.0e9f, fminf(2.0e9f, px));
    py = fmaxf(-2.0e9f, fminf(2.0e9f, py));
    const int x0 = (int)floorf(px - 0.5f), y0 = (int)floorf(py - 0.5f);
    const float fx = (px - 0.5f) - (float)x0, fy = (py - 0.5f) - (float)y0;
    const float power = (S.r * sp.y + S.g * sp.z + S.b * sp.w) * base;
    const float c0 = power * sp.y, c1 = power * sp.z, c2 = power * sp.w;
    if (x0 != cx || y0 != cy)
    {
        if (cx != INT_MIN) flush_taps(A.accum, A.width, A.height, cx, cy, acc);
        cx = x0; cy = y0;
        #pragma unroll
        for (int q = 0; q < 12; ++q) acc[q] = 0.0f;
    }
    const float wt[4] = {(1.0f - fx) * (1.0f - fy), fx * (1.0f - fy), (1.0f - fx) * fy, fx * fy};
    #pragma unroll
    for (int q = 0; q < 4; ++q)
    {
        acc[3 * q] += c0 * wt[q];
        acc[3 * q + 1] += c1 * wt[q];
        acc[3 * q + 2] += c2 * wt[q];
    }
}

template <bool PROBE>
__device__ __forceinline__ void trace_warp(const RenderArgs& A, const SurfRec* lens, const HotRec* hot,
                                           const float2* ab, const float4* spec,
                                           const float* kdel, const PairDev& P, const SourceDev& S,
                                           float2 uv, bool active, float* acc, int pair, int li0, int li1)
{
    const int n = A.n_surf, a = P.a, b = P.b;
    const int L1 = b + 1, L2 = L1 + (b - a), L = L2 + (n - 1 - a);
    int cx = INT_MIN, cy = INT_MIN;

    const unsigned n_lanes = __popc(__ballot_sync(kFull, active));
    int n_lambda = 0;
    #pragma unroll 1
    for (int li = li0; li < li1; ++li)
    {
        // probe: stop once any warp has found the pair on the sensor (read
        // through L2, where the other warps' atomics land)
        if (PROBE && li > li0 && A.pair_hits != nullptr && __ldcg(A.pair_hits + pair) > 0) break;
        ++n_lambda;
        const float4 sp = spec[li];
        const float kdelta = kdel[li];
        const float2* abl = ab + li * n;
        V3 o = v3(uv.x * A.front_R + S.sdx, uv.y * A.front_R + S.sdy, A.start_z);
        V3 d = v3(S.dx, S.dy, S.dz);
        float w = 1.0f, cur = 1.0f;
        bool alive = active;
        #pragma unroll 1
        for (int k = 0; k < L; ++k)
        {
            if (!__any_sync(kFull, alive)) break;
            int s; float n2; bool refl; bool back = false;
            if (k < L1)      { s = k;                refl = (s == b); }
            else if (k < L2) { s = 2 * b - k;        refl = (s == a); back = true; }
            else             { s = a + 1 + (k - L2); refl = false; }
            const HotRec hr = hot[s];
            const float2 io = abl[s];
            n2 = back ? io.y : io.x;
            const float rior = (back && refl) ? abl[a].x : cur;
            // every lane steps (see surface_step); a dead lane's state is not
            // read; an inactive surface leaves the ray as it is
            bool ok;
            if (hr.bits & HB_ROUND)
                ok = surface_step_fast<!PROBE, true>(o, d, hr, kdelta, n2, refl, back, abl + a, cur, w, alive);
            else if (hr.bits & HB_FAST)
                ok = surface_step_fast<!PROBE, false>(o, d, hr, kdelta, n2, refl, back, abl + a, cur, w, alive);
            else if (hr.bits & HB_ACTIVE)
                ok = surface_step<!PROBE>(o, d, hr, lens[s], sp.x, kdelta, n2, refl, rior, cur, w, alive);
            else continue;
            alive = ok;
        }
        if (PROBE)
        {
            // Off-sensor probe (the STATS pass of ghost_render.cu:402-415 with
            // the 1.25 margin of :148): did this ray land inside the inflated
            // frame?  One hit anywhere keeps the pair, so the warp stops at
            // the first wavelength that produced one.
            bool hit = false, surv = false;
            if (alive && fabsf(d.z) >= 1e-12f)
            {
                const float ts = -o.z / d.z;
                if (ts >= 0.0f)
                {
                    const float sx = o.x + d.x * ts, sy = o.y + d.y * ts;
                    surv = isfinite(sx) && isfinite(sy);
                    const float spx = (sx / A.hw2 + 0.5f) * A.fmt_w + A.fmt_x0;
                    const float spy = (sy / A.hh2 + 0.5f) * A.fmt_h + A.fmt_y0;
                    hit = isfinite(spx) && isfinite(spy) && spx >= 0.0f && spx < (float)A.width &&
                          spy >= 0.0f && spy < (float)A.height;
                }
            }
            if (A.stats != nullptr)
            {
                // diagnostic pass (the STATS instantiation, ghost_render.cu:402-415):
                // count, never stop early
                const unsigned sv = __ballot_sync(kFull, surv), hv = __ballot_sync(kFull, hit);
                if ((threadIdx.x & 31) == 0)
                {
                    if (sv) atomicAdd(A.stats + 3 * pair + 1, (unsigned long long)__popc(sv));
                    if (hv) atomicAdd(A.stats + 3 * pair + 2, (unsigned long long)__popc(hv));
                }
                continue;
            }
            if (__any_sync(kFull, hit))
            {
                if ((threadIdx.x & 31) == 0)
                {
                    atomicAdd(A.pair_hits + pair, 1);
                    if (A.traced) atomicAdd(A.traced, (unsigned long long)n_lanes * n_lambda);
                }
                return;
            }
        }
        else if (alive)
        {
            splat_ray(A, P, S, sp, o, d, w, cx, cy, acc);
        }
    }
    if (!PROBE && cx != INT_MIN) flush_taps(A.accum, A.width, A.height, cx, cy, acc);
    if (A.traced && (threadIdx.x & 31) == 0) atomicAdd(A.traced, (unsigned long long)n_lanes * n_lambda);
    if (PROBE && A.stats && (threadIdx.x & 31) == 0)
        atomicAdd(A.stats + 3 * pair, (unsigned long long)n_lanes * n_lambda);
}

// A render CTA's tables in shared memory.
struct Staged {
    HotRec* hot;
    float4* spec;
    float2* ab;        // per (wavelength, surface): (IOR after the surface, IOR before it), one
                       // 8-byte shared load for either direction of the walk
    float* kdel;
    SurfRec* lens;
    float* lanes;      // kLaneFloats per lane
};

__device__ __forceinline__ Staged stage_tables(const RenderArgs& A, unsigned char* smem_raw)
{
    Staged T;
    T.hot = reinterpret_cast<HotRec*>(smem_raw);
    T.spec = reinterpret_cast<float4*>(T.hot + A.n_surf);
    T.ab = reinterpret_cast<float2*>(T.spec + A.n_spec);
    T.kdel = reinterpret_cast<float*>(T.ab + A.n_spec * A.n_surf);
    T.lens = reinterpret_cast<SurfRec*>(T.kdel + A.n_spec);
    T.lanes = reinterpret_cast<float*>(T.lens + A.n_surf);
    const int tid = threadIdx.x;
    const int words = A.n_surf * (int)(sizeof(SurfRec) / 4);
    const int* src = reinterpret_cast<const int*>(A.recs);
    int* dst = reinterpret_cast<int*>(T.lens);
    for (int i = tid; i < words; i += blockDim.x) dst[i] = src[i];
    for (int i = tid; i < A.n_spec; i += blockDim.x)
    {
        T.spec[i] = A.spec[i];
        // film phase factor of the MgF2 quarter-wave layer (fresnel.h:103, 168)
        T.kdel[i] = 2.0f * kPi * 1.38f * (550.0f / (4.0f * 1.38f)) / A.spec[i].x;
    }
    const int nt = A.n_spec * A.n_surf;
    for (int i = tid; i < nt; i += blockDim.x) T.ab[i] = make_float2(A.ior_at[i], A.ior_bf[i]);
    __syncthreads();
    for (int i = tid; i < A.n_surf; i += blockDim.x) T.hot[i] = make_hot(T.lens[i]);
    __syncthreads();
    return T;
}

template <bool PROBE>
__global__ void __launch_bounds__(kRenderThreads, kRenderMinBlocks) ghost_render_kernel(const RenderArgs A)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Staged T = stage_tables(A, smem_raw);
    const int tid = threadIdx.x;
    float* acc = T.lanes + tid * kAccStride;   // 13 floats per lane: conflict-free banks
    // Warp-granular work: each warp takes one task at a time — a (pair,
    // source, 32-sample) item and one of its l_chunks wavelength ranges — so
    // no CTA-wide barrier sits inside the loop, and splitting the wavelengths
    // shortens the tasks at the queue's tail.
    const int lane = tid & 31;
    const int gwarp = (int)((blockIdx.x * blockDim.x + tid) >> 5);
    const int nwarp = (int)((gridDim.x * blockDim.x) >> 5);
    const int chunks = A.l_chunks > 1 ? A.l_chunks : 1;
    const int l_size = (A.n_spec + chunks - 1) / chunks;
    const long long n_tasks = (long long)A.n_items * chunks;
    long long next_static = (long long)A.item_base * chunks + gwarp;
    for (;;)
    {
        long long task;
        if (A.counter != nullptr)
        {
            int v = 0;
            if (lane == 0) v = atomicAdd(A.counter, 1);
            task = __shfl_sync(kFull, v, 0);
        }
        else
        {
            task = next_static;
            next_static += nwarp;
        }
        if (task >= n_tasks) break;
        const int item = (int)(task / chunks);
        const int chunk = (int)(task - (long long)item * chunks);
        int li0 = chunk * l_size, li1 = min(A.n_spec, li0 + l_size);
        if (li0 >= li1) continue;
        int4 w;
        if (A.items != nullptr) w = A.items[item];
        else
        {
            int tiles = A.u_tiles, base = A.u_grid_base, gn = A.u_grid_n, local = item;
            if (A.u_npass > 0)
            {
                const int q = (item >= A.u_start[2]) ? 2 : (item >= A.u_start[1] ? 1 : 0);
                tiles = A.u_tl[q]; base = A.u_base[q]; gn = A.u_n[q]; local = item - A.u_start[q];
            }
            const int per_pair = tiles * A.u_n_src;
            const int pr = local / per_pair, rem = local - pr * per_pair;
            const int sr = rem / tiles, t = (rem - sr * tiles) * kTile;
            w = make_int4(pr, sr, base + t, min(kTile, gn - t));
        }
        if (A.pair_hits != nullptr)
        {
            // render: skip pairs the probe found off-sensor; probe passes
            // after the first: skip pairs already known to be on-sensor
            const int h = PROBE ? __ldcg(A.pair_hits + w.x) : A.pair_hits[w.x];
            if (PROBE ? (h > 0) : (h == 0)) continue;
        }
        PairDev P = A.pairs[w.x];
        if (A.items == nullptr) P.w_ray = A.w_uniform;
        const SourceDev S = A.sources[w.y];
        const bool active = lane < w.w;
        const float2 uv = active ? A.samples[w.z + lane] : make_float2(0.0f, 0.0f);
        trace_warp<PROBE>(A, T.lens, T.hot, T.ab, T.spec, T.kdel, P, S, uv, active, acc, w.x, li0, li1);
    }
}

// ---- shared legs ---------------------------------------------------------------
// Rays of one pupil sample, source and wavelength that belong to different
// pairs walk the same way as long as their pairs agree: every pair (a, b) goes
// forward through 0 .. b - 1, and every pair of one b turns there and comes back
// through b - 1, b - 2, ....  The pairs that sample the same grid are therefore
// walked as one tree: forward once, at each b back once, and from each a its
// own last leg to the sensor.  Each ray still sees the operations of its own
// walk in their order, so its landing and weight are the same.  All pairs of 24
// surfaces are 4924 steps that way against 11224 pair by pair.
//
// The tree is cut into segments of a few hundred steps (which repeat the
// forward leg up to their first b), a task is one segment of one 32-sample tile,
// source and wavelength.  A segment is a list of runs, each a straight walk over
// neighbouring surfaces with one step site; the ray states to come back to, before
// the last b and before the last a, wait in the lane's shared-memory slot
// (which the pair-by-pair walk uses for its splat footprint: a task has one
// wavelength, so there is nothing to carry).
// Bound by instruction issue and fetch: the warps of an SM stand at different
// surfaces, and with a copy of the step per kind of surface their instructions
// came from the cache of the whole GPC at 97% of its rate (82% hits in the SM's,
// 74% of the issue slots used; the probe, whose step has no weights, 98% and
// 87%).  So the round-stop copy is left out here and surfaces of other forms and
// stops join the common step behind their intersection (HB_COMMON).  24 surfaces,
// 253 pairs on adaptive grids, 31 wavelengths: the render 5.15 -> 1.50 ms; 120
// pairs x 5 sources, 64^2 x 16 wavelengths: 1.66 -> 0.47.
enum RunFlags { RUN_REFLECT = 1, RUN_BACK = 2, RUN_LOAD_F = 4, RUN_LOAD_B = 8, RUN_SAVE_F = 16, RUN_SAVE_B = 32,
                RUN_FORWARD = 64, RUN_LAST = 128 };

// A run is an int4 {s0 | s1 << 8, flags, pairs, skip}.  Walk from s0 to s1 (one
// surface at a time, backward with RUN_BACK), the first step reflecting with
// RUN_REFLECT.  pairs: the pairs of the segment (at most
// 32) that hang on the run, as their mask; skip: the run to go on with when none
// of them is wanted any more or every ray died on the way.  RUN_LAST: the last
// leg of one pair, splatted at its end.
struct TreeSegment { int run_begin, run_end, pair_begin, pair_end; };
struct TreeGrid { int task_begin, sample_base, n_samples, tiles, seg_base, n_segs; };

struct TreeArgs {
    const TreeGrid* grids;          // n_grids + 1 (the last: the task count)
    const TreeSegment* segments;
    const int4* runs;
    const int* pairs;               // pairs of the segments, in order
    int n_grids, n_src;
};

// splat_ray for a single ray-wavelength: straight to the accumulator.  Called by
// the whole warp; lanes whose ray did not land have valid = false.  Where all
// landings of the warp share one 2 x 2 footprint (a focused ghost) they are
// summed first, so that its pixels take one addition instead of 32.
__device__ __forceinline__ void splat_now(const RenderArgs& A, const PairDev& P, const SourceDev& S, const float4& sp,
                                          V3 o, V3 d, float w, bool valid)
{
    int x0 = 0, y0 = 0;
    float v[12];
    #pragma unroll
    for (int q = 0; q < 12; ++q) v[q] = 0.0f;
    const float ts = -o.z / d.z;
    const float rx = o.x + d.x * ts, ry = o.y + d.y * ts;
    const float base = w * P.w_ray * A.gain * P.boost;
    float px = (rx / A.hw2 + 0.5f) * A.fmt_w + A.fmt_x0;
    float py = (ry / A.hh2 + 0.5f) * A.fmt_h + A.fmt_y0;
    valid = valid && fabsf(d.z) >= 1e-12f && ts >= 0.0f && isfinite(rx) && isfinite(ry) && !(base < 1e-14f) &&
            isfinite(px) && isfinite(py);
    if (valid)
    {
        px = fmaxf(-2.0e9f, fminf(2.0e9f, px));
        py = fmaxf(-2.0e9f, fminf(2.0e9f, py));
        x0 = (int)floorf(px - 0.5f);
        y0 = (int)floorf(py - 0.5f);
        // off the frame altogether: nothing to add
        valid = x0 >= -1 && x0 < A.width && y0 >= -1 && y0 < A.height;
    }
    const unsigned m = __ballot_sync(kFull, valid);
    if (m == 0) return;
    if (valid)
    {
        const float fx = (px - 0.5f) - (float)x0, fy = (py - 0.5f) - (float)y0;
        const float power = (S.r * sp.y + S.g * sp.z + S.b * sp.w) * base;
        const float c0 = power * sp.y, c1 = power * sp.z, c2 = power * sp.w;
        const float wt[4] = {(1.0f - fx) * (1.0f - fy), fx * (1.0f - fy), (1.0f - fx) * fy, fx * fy};
        #pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            v[3 * q] = c0 * wt[q];
            v[3 * q + 1] = c1 * wt[q];
            v[3 * q + 2] = c2 * wt[q];
        }
    }
    const int lead = __ffs(m) - 1;
    const int lx = __shfl_sync(kFull, x0, lead), ly = __shfl_sync(kFull, y0, lead);
    if (__popc(m) > 3 && __all_sync(kFull, !valid || (x0 == lx && y0 == ly)))
    {
        #pragma unroll
        for (int q = 0; q < 12; ++q)
            for (int k = 16; k > 0; k >>= 1) v[q] += __shfl_xor_sync(kFull, v[q], k);
        valid = (int)(threadIdx.x & 31) == lead;
    }
    if (valid) flush_taps(A.accum, A.width, A.height, x0, y0, v);
}

// Whether the lane's ray landed inside the inflated frame (see trace_warp).
__device__ __forceinline__ bool probe_hit(const RenderArgs& A, V3 o, V3 d, bool alive)
{
    if (!alive || !(fabsf(d.z) >= 1e-12f)) return false;
    const float ts = -o.z / d.z;
    if (!(ts >= 0.0f)) return false;
    const float sx = o.x + d.x * ts, sy = o.y + d.y * ts;
    const float spx = (sx / A.hw2 + 0.5f) * A.fmt_w + A.fmt_x0;
    const float spy = (sy / A.hh2 + 0.5f) * A.fmt_h + A.fmt_y0;
    return isfinite(spx) && isfinite(spy) && spx >= 0.0f && spx < (float)A.width && spy >= 0.0f && spy < (float)A.height;
}

// PROBE: the off-sensor probe (see trace_warp).  Pairs with a hit are not wanted
// any more; wavelengths are the slowest index, so that the first finds most of
// them.  The frame above: the probe pair by pair in two stages (the second with
// its samples sorted by where the first wavelength's ray died) 0.95 ms, as a tree
// 0.44.
template <bool PROBE>
__global__ void __launch_bounds__(kRenderThreads, kRenderMinBlocks) ghost_tree_kernel(const RenderArgs A, const TreeArgs G)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Staged T = stage_tables(A, smem_raw);
    const int lane = threadIdx.x & 31;
    // the lane's slot: the state before the last b, then (7 fields on) before the last a
    float* slot = T.lanes + threadIdx.x;
    const int n_tasks = G.grids[G.n_grids].task_begin;
    for (;;)
    {
        int task = 0;
        if (lane == 0) task = atomicAdd(A.counter, 1);
        task = __shfl_sync(kFull, task, 0);
        if (task >= n_tasks) break;
        int lo = 0, hi = G.n_grids;
        while (hi - lo > 1)
        {
            const int mid = (lo + hi) >> 1;
            if (G.grids[mid].task_begin <= task) lo = mid;
            else hi = mid;
        }
        // tiles fastest: neighbouring tasks land on different pixels
        const TreeGrid g = G.grids[lo];
        int r = task - g.task_begin;
        const int tile = r % g.tiles;
        r /= g.tiles;
        const int si = r % G.n_src;
        r /= G.n_src;
        const int li = PROBE ? r / g.n_segs : r % A.n_spec;
        const TreeSegment seg = G.segments[g.seg_base + (PROBE ? r % g.n_segs : r / A.n_spec)];
        const bool active = tile * kTile + lane < g.n_samples;
        const unsigned n_lanes = (unsigned)min(kTile, g.n_samples - tile * kTile);
        // the pairs to walk: probe, those without a hit yet (read through L2,
        // where the other warps' atomics land); render, those with one
        bool on = seg.pair_begin + lane < seg.pair_end;
        if (on && A.pair_hits != nullptr)
        {
            const int* hit = A.pair_hits + G.pairs[seg.pair_begin + lane];
            on = PROBE ? __ldcg(hit) == 0 : *hit != 0;
        }
        unsigned want = __ballot_sync(kFull, on);
        if (want == 0) continue;
        if (A.traced && lane == 0) atomicAdd(A.traced, (unsigned long long)n_lanes * __popc(want));
        const SourceDev S = A.sources[si];
        const float2 uv = active ? A.samples[g.sample_base + tile * kTile + lane] : make_float2(0.0f, 0.0f);
        const float4 sp = T.spec[li];
        const float kdelta = T.kdel[li];
        const float2* abl = T.ab + li * A.n_surf;
        V3 o = v3(uv.x * A.front_R + S.sdx, uv.y * A.front_R + S.sdy, A.start_z);
        V3 d = v3(S.dx, S.dy, S.dz);
        float w = 1.0f, cur = 1.0f, cur_f = 1.0f, cur_b = 1.0f;
        bool alive = active;
        unsigned alive_f = 0, alive_b = 0;
        #pragma unroll 1
        for (int ri = seg.run_begin; ri < seg.run_end; ++ri)
        {
            const int4 run = __ldg(G.runs + ri);
            const int flags = run.y;
            if (((unsigned)run.z & want) == 0)
            {
                if (flags & RUN_FORWARD) break;          // nor anything after it
                if (!(flags & RUN_LAST)) ri = run.w - 1;
                continue;
            }
            if (flags & (RUN_LOAD_F | RUN_LOAD_B))
            {
                const bool f = (flags & RUN_LOAD_F) != 0;
                const float* q = slot + (f ? 0 : 7 * kRenderThreads);
                o = v3(q[0], q[kRenderThreads], q[2 * kRenderThreads]);
                d = v3(q[3 * kRenderThreads], q[4 * kRenderThreads], q[5 * kRenderThreads]);
                w = q[6 * kRenderThreads];
                cur = f ? cur_f : cur_b;
                alive = (((f ? alive_f : alive_b) >> lane) & 1u) != 0;
            }
            const int s0 = run.x & 0xff, s1 = (run.x >> 8) & 0xff;
            const int dir = (flags & RUN_BACK) ? -1 : 1;
            int left = (flags & RUN_BACK) ? s0 - s1 : s1 - s0;
            bool refl = (flags & RUN_REFLECT) != 0;
            #pragma unroll 1
            for (int s = s0; left >= 0; s += dir, --left, refl = false)
            {
                if (!__any_sync(kFull, alive)) break;
                // a turn is met in the direction before it
                const bool back = ((flags & RUN_BACK) != 0) != refl;
                const HotRec hr = T.hot[s];
                const float2 io = abl[s];
                const float n2 = back ? io.y : io.x;
                const float rior = (back && refl) ? io.x : cur;
                bool ok;
                if (hr.bits & HB_COMMON)        // (a round stop's aspect factor is exactly 1)
                    ok = surface_step_fast<!PROBE, false, true>(o, d, hr, kdelta, n2, refl, back, abl + s, cur, w, alive, T.lens + s);
                else if (hr.bits & HB_ACTIVE)
                    ok = surface_step<!PROBE>(o, d, hr, T.lens[s], sp.x, kdelta, n2, refl, rior, cur, w, alive);
                else continue;
                alive = ok;
            }
            const unsigned left_alive = __ballot_sync(kFull, alive);
            if (flags & RUN_LAST)
            {
                const int pair = G.pairs[seg.pair_begin + __ffs(run.z) - 1];
                if (PROBE)
                {
                    if (__any_sync(kFull, probe_hit(A, o, d, alive)))
                    {
                        if (lane == 0) atomicAdd(A.pair_hits + pair, 1);
                        want &= ~(unsigned)run.z;
                    }
                }
                else if (left_alive) splat_now(A, A.pairs[pair], S, sp, o, d, w, alive);
                continue;
            }
            if (left_alive == 0)
            {
                // nothing comes of the runs that start from here
                if (flags & RUN_FORWARD) break;
                ri = run.w - 1;
                continue;
            }
            if (flags & (RUN_SAVE_F | RUN_SAVE_B))
            {
                const bool f = (flags & RUN_SAVE_F) != 0;
                float* q = slot + (f ? 0 : 7 * kRenderThreads);
                q[0] = o.x; q[kRenderThreads] = o.y; q[2 * kRenderThreads] = o.z;
                q[3 * kRenderThreads] = d.x; q[4 * kRenderThreads] = d.y; q[5 * kRenderThreads] = d.z;
                q[6 * kRenderThreads] = w;
                if (f) { cur_f = cur; alive_f = left_alive; }
                else { cur_b = cur; alive_b = left_alive; }
            }
        }
    }
}

// RGBA accumulator -> planar r/g/b with the optional 3x3 correction, four
// pixels per thread (one 64-byte read, three 16-byte writes).
__global__ void ghost_flush_kernel(const float4* __restrict__ accum, size_t n_px, float* __restrict__ out_r,
                                   float* __restrict__ out_g, float* __restrict__ out_b, int apply,
                                   float c00, float c01, float c02, float c10, float c11, float c12,
                                   float c20, float c21, float c22)
{
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t p0 = q * 4;
    if (p0 >= n_px) return;
    float r[4], g[4], b[4];
    #pragma unroll
    for (int k = 0; k < 4; ++k)
    {
        float4 v = (p0 + k < n_px) ? accum[p0 + k] : make_float4(0, 0, 0, 0);
        if (apply)
        {
            r[k] = __fadd_rn(__fadd_rn(__fmul_rn(c00, v.x), __fmul_rn(c01, v.y)), __fmul_rn(c02, v.z));
            g[k] = __fadd_rn(__fadd_rn(__fmul_rn(c10, v.x), __fmul_rn(c11, v.y)), __fmul_rn(c12, v.z));
            b[k] = __fadd_rn(__fadd_rn(__fmul_rn(c20, v.x), __fmul_rn(c21, v.y)), __fmul_rn(c22, v.z));
        }
        else
        {
            r[k] = v.x; g[k] = v.y; b[k] = v.z;
        }
    }
    const bool vec = (p0 + 4 <= n_px) && ((((uintptr_t)(out_r + p0)) | ((uintptr_t)(out_g + p0)) |
                                          ((uintptr_t)(out_b + p0))) & 15) == 0;
    if (vec)
    {
        *reinterpret_cast<float4*>(out_r + p0) = make_float4(r[0], r[1], r[2], r[3]);
        *reinterpret_cast<float4*>(out_g + p0) = make_float4(g[0], g[1], g[2], g[3]);
        *reinterpret_cast<float4*>(out_b + p0) = make_float4(b[0], b[1], b[2], b[3]);
    }
    else
    {
        for (int k = 0; k < 4 && p0 + k < n_px; ++k) { out_r[p0 + k] = r[k]; out_g[p0 + k] = g[k]; out_b[p0 + k] = b[k]; }
    }
}

// ---------------------------------------------------------------------------
// Plan: resident device state of one ghost render request.
// ---------------------------------------------------------------------------
// A tree of shared legs (TreeArgs) on the device.
struct TreeDev {
    int n_tasks = 0, n_grids = 0;
    TreeGrid* grids = nullptr;
    TreeSegment* segments = nullptr;
    int4* runs = nullptr;
    int* pairs = nullptr;
};

struct GhostPlan {
    int device = 0;
    int n_surf = 0, n_spec = 0, n_pairs = 0, n_items = 0;
    int width = 0, height = 0;
    gl_ghost_render_params prm{};
    std::vector<int> pair_item_begin;   // first item of each pair (+ sentinel)
    // device
    SurfRec* recs = nullptr;
    float* ior_at = nullptr;
    float* ior_bf = nullptr;
    float4* spec = nullptr;
    int4* items = nullptr;
    PairDev* pairs = nullptr;
    SourceDev* sources = nullptr;
    float2* samples = nullptr;
    int* counter = nullptr;
    float4* accum = nullptr;            // RGBA scratch, width x height
    size_t smem = 0;
    int queue_ctas = 0;                 // CTAs of the persistent queue when there is work for all
    int per_sm = 0, n_sm = 0;           // resident render CTAs per SM, SM count
    int launch_ipw = 0;                 // 0: persistent queue; > 0: static chunks of this many items per warp
    int l_chunks = 1;                   // wavelength ranges per item (tasks per item)
    // shared legs (n_tasks > 0: used by the persistent queue, and by the probe)
    int n_src = 0;
    TreeDev tree, probe_tree;
    long long rays = 0;                 // ray-wavelength traces per execute
    float front_R = 0.0f, start_z = 0.0f;
    // off-sensor cull (probe passes)
    bool cull = false;
    int4* probe_items = nullptr;
    float2* probe_samples = nullptr;
    int probe_begin[4] = {0, 0, 0, 0};   // item range of each pass
    int* pair_hits = nullptr;
    int* probe_counters = nullptr;
    int* pair_hits_init = nullptr;          // 1 = not probed (always rendered), 0 = probed
    long long probe_rays = 0;
    unsigned long long* traced = nullptr;   // [render, probe] traces executed by the last execute
    // optional timing events recorded around the probe and render launches
    cudaEvent_t ev_probe = nullptr, ev_render = nullptr, ev_end = nullptr;
    // Device memory comes from the device's stream-ordered pool: creating and
    // destroying a plan then costs no device-wide synchronisation (a
    // cudaFree waits for every stream).  `done` is recorded after each
    // execute; destroy waits for it (or, after a stream capture, for the
    // device) and releases the blocks in stream order.
    cudaMemPool_t pool = nullptr;
    cudaStream_t own = nullptr;         // the device's plan stream (uploads, releases)
    cudaEvent_t done = nullptr;
    bool executed = false, captured = false;
};

// One non-blocking stream per device for plan uploads and releases.
static cudaStream_t plan_stream(int dev)
{
    static std::mutex mu;
    static cudaStream_t st[64] = {};
    if (dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lk(mu);
    if (!st[dev] && cudaStreamCreateWithFlags(&st[dev], cudaStreamNonBlocking) != cudaSuccess) st[dev] = nullptr;
    return st[dev];
}

static void plan_free(GhostPlan* p)
{
    if (!p) return;
    if (p->captured) cudaDeviceSynchronize();               // graph replays may still use the blocks
    else if (p->executed && p->done) cudaEventSynchronize(p->done);
    void* blocks[] = {p->recs, p->ior_at, p->ior_bf, p->spec, p->items, p->pairs, p->sources, p->samples,
                      p->counter, p->accum, p->probe_items, p->probe_samples, p->pair_hits, p->probe_counters,
                      p->traced, p->pair_hits_init, p->tree.grids, p->tree.segments, p->tree.runs, p->tree.pairs,
                      p->probe_tree.grids, p->probe_tree.segments, p->probe_tree.runs, p->probe_tree.pairs};
    for (void* b : blocks)
    {
        if (!b) continue;
        if (p->own) cudaFreeAsync(b, p->own);
        else cudaFree(b);
    }
    if (p->done) cudaEventDestroy(p->done);
    delete p;
}

template <class T>
static cudaError_t upload(T** dst, const T* src, size_t count, cudaMemPool_t pool, cudaStream_t st)
{
    cudaError_t e = cudaMallocFromPoolAsync(reinterpret_cast<void**>(dst), std::max<size_t>(count, 1) * sizeof(T),
                                            pool, st);
    if (e != cudaSuccess) return e;
    if (count) e = cudaMemcpyAsync(*dst, src, count * sizeof(T), cudaMemcpyHostToDevice, st);
    return e;
}

template <class T>
static cudaError_t alloc(T** dst, size_t bytes, cudaMemPool_t pool, cudaStream_t st)
{
    return cudaMallocFromPoolAsync(reinterpret_cast<void**>(dst), bytes, pool, st);
}

size_t render_smem(int n_surf, int n_spec)
{
    return (size_t)n_surf * 32 + (size_t)n_spec * 16 + (size_t)n_spec * 4 + 2 * (size_t)n_spec * n_surf * 4 +
           (size_t)n_surf * sizeof(SurfRec) + (size_t)kRenderThreads * kLaneFloats * 4;
}

// The opt-in only grows (per device and kernel), so a plan created earlier
// with a larger table keeps launching after a smaller one was prepared.
int raise_smem_limit(const void* kernel, size_t bytes)
{
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, size_t> limit;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    std::lock_guard<std::mutex> lk(mu);
    size_t& cur = limit[{dev, kernel}];
    if (bytes <= cur) return (int)cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) cur = bytes;
    return (int)e;
}

cudaError_t render_prepare(size_t smem, int* per_sm, int* n_sm)
{
    cudaError_t e = (cudaError_t)raise_smem_limit((const void*)ghost_render_kernel<false>, smem);
    if (e == cudaSuccess) e = (cudaError_t)raise_smem_limit((const void*)ghost_tree_kernel<false>, smem);
    if (e == cudaSuccess) e = (cudaError_t)raise_smem_limit((const void*)ghost_tree_kernel<true>, smem);
    if (e == cudaSuccess) e = (cudaError_t)raise_smem_limit((const void*)ghost_render_kernel<true>, smem);
    if (e == cudaSuccess && per_sm) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, ghost_render_kernel<false>, kRenderThreads, smem);
    int dev = 0;
    if (e == cudaSuccess && n_sm) e = cudaGetDevice(&dev);
    if (e == cudaSuccess && n_sm) e = cudaDeviceGetAttribute(n_sm, cudaDevAttrMultiProcessorCount, dev);
    return e;
}

cudaError_t render_launch(const RenderArgs& A, bool probe, int grid, size_t smem, cudaStream_t st)
{
    if (probe) ghost_render_kernel<true><<<grid, kRenderThreads, smem, st>>>(A);
    else ghost_render_kernel<false><<<grid, kRenderThreads, smem, st>>>(A);
    return cudaGetLastError();
}

cudaError_t flush_launch(const float4* accum, size_t n_px, float* r, float* g, float* b, int apply, const float* C,
                         cudaStream_t st)
{
    const size_t quads = (n_px + 3) / 4;
    const int fb = 256;
    ghost_flush_kernel<<<(unsigned)((quads + fb - 1) / fb), fb, 0, st>>>(accum, n_px, r, g, b, apply, C[0], C[1], C[2],
                                                                         C[3], C[4], C[5], C[6], C[7], C[8]);
    return cudaGetLastError();
}

SourceDev make_source(const gl_flare_source& s)
{
    const float bx = tanf(s.angle_x), by = tanf(s.angle_y);
    V3 dir = normalized(v3(bx, by, 1.0f));
    return {dir.x, dir.y, dir.z, -kSpawnOffset * bx, -kSpawnOffset * by, s.r, s.g, s.b};
}

// Pupil samples in Morton order over the unit square: 32 consecutive samples
// (one warp) then cover a compact patch of the pupil, whose rays tend to
// vignette together, instead of a strip across it.  The set of samples and
// each one's weight are unchanged.
static inline uint32_t morton_code(const gl_pupil_sample& p)
{
    auto spread = [](uint32_t x) {
        x &= 0x3ffu;
        x = (x | (x << 16)) & 0x030000ffu;
        x = (x | (x << 8)) & 0x0300f00fu;
        x = (x | (x << 4)) & 0x030c30c3u;
        x = (x | (x << 2)) & 0x09249249u;
        return x;
    };
    const float fu = std::min(std::max((p.u + 1.0f) * 512.0f, 0.0f), 1023.0f);
    const float fv = std::min(std::max((p.v + 1.0f) * 512.0f, 0.0f), 1023.0f);
    return (spread((uint32_t)fu) << 1) | spread((uint32_t)fv);
}

// A stable sort on the code: ordering an ordered grid again changes nothing,
// so a caller may hand in grids it has ordered (and cached) once, and the
// plan build then only checks them (one linear pass instead of a sort).
void morton_order(const gl_pupil_sample* in, int n, gl_pupil_sample* out)
{
    bool sorted = true;
    uint32_t prev = 0;
    for (int i = 0; i < n && sorted; ++i)
    {
        const uint32_t c = morton_code(in[i]);
        sorted = (i == 0) || c >= prev;
        prev = c;
    }
    if (sorted)
    {
        std::copy(in, in + n, out);
        return;
    }
    std::vector<std::pair<uint32_t, int>> key;
    key.reserve((size_t)n);
    for (int i = 0; i < n; ++i) key.push_back({morton_code(in[i]), i});
    std::stable_sort(key.begin(), key.end(),
                     [](const std::pair<uint32_t, int>& x, const std::pair<uint32_t, int>& y) { return x.first < y.first; });
    for (int i = 0; i < n; ++i) out[i] = in[key[i].second];
}

int probe_grids(const gl_surface* surfaces, int n_surf, int blades_override, float rotation_deg,
                std::vector<gl_pupil_sample>& out, int begin[4])
{
    out.clear();
    for (int pass = 0; pass < 3; ++pass)
    {
        gl_sampler_params sp;
        sp.ray_grid = 40;
        sp.pupil_jitter = 1;
        sp.jitter_seed = (int)(0x9E3779B9u * (unsigned)(pass + 1));
        sp.blades_override = blades_override;
        sp.rotation_deg = rotation_deg;
        std::vector<gl_pupil_sample> g;
        const int rc = build_aperture_samples(surfaces, n_surf, sp, g);
        if (rc) return rc;
        begin[pass] = (int)out.size();
        out.insert(out.end(), g.begin(), g.end());
    }
    begin[3] = (int)out.size();
    return GL_OK;
}

// Wavelength ranges per item by default: about eight wavelengths per task
// (31 -> 4, 16 -> 2, 8 -> 1), the split the autotuner picks on the
// 31-wavelength frames; set_lambda_split overrides it.
int default_lambda_split(int n_spec)
{
    return std::max(1, std::min(n_spec, (n_spec + 4) / 8));
}

// The tree walk's tables (see "shared legs").  tasks = 0: the pair-by-pair walk
// it is (a pair that turns at an inactive surface, or more tasks than a counter
// holds).  Otherwise the tree is taken even where little is shared: one pair
// alone, 128^2 x 31 wavelengths 51 us pair by pair, 48 as a tree; four pairs of
// one b 166 / 123; 66 pairs 16^2 x 8 45 / 46, 96^2 x 16 542 / 343.
struct TreeBuild {
    std::vector<TreeGrid> grids;
    std::vector<TreeSegment> segments;
    std::vector<int4> runs;
    std::vector<int> pairs;
    int tasks = 0;
};

// Groups of pairs with the samples [base, base + n) that each is traced on.
struct TreeGroup { std::vector<int> pairs; int base, n; };

static TreeBuild build_tree(const SurfRec* recs, int n, const gl_ghost_pair* pairs, std::vector<TreeGroup> groups,
                            int n_src, int n_spec, long long warps)
{
    // active surfaces before each
    std::vector<int> act((size_t)n + 1, 0);
    for (int i = 0; i < n; ++i) act[i + 1] = act[i] + ((recs[i].flags & SF_ACTIVE) ? 1 : 0);
    auto steps = [&](int from, int to) { return to >= from ? act[to + 1] - act[from] : 0; };     // surfaces from .. to
    for (const TreeGroup& g : groups)
        for (int i : g.pairs)       // the turn must be a step (an inactive surface is passed by unturned)
            if (!(recs[pairs[i].surf_a].flags & SF_ACTIVE) || !(recs[pairs[i].surf_b].flags & SF_ACTIVE)) return {};
    // steps of the whole tree over all tiles, sources and wavelengths
    double whole = 0.0;
    for (TreeGroup& g : groups)
    {
        std::sort(g.pairs.begin(), g.pairs.end(), [&](int x, int y) {
            return pairs[x].surf_b != pairs[y].surf_b ? pairs[x].surf_b < pairs[y].surf_b : pairs[x].surf_a > pairs[y].surf_a;
        });
        const double rays = (double)((g.n + kTile - 1) / kTile) * n_src * n_spec;
        int b0 = -1, a0 = 0, f = 0;
        for (int i : g.pairs)
        {
            const int a = pairs[i].surf_a, b = pairs[i].surf_b;
            if (b != b0)
            {
                whole += rays * (steps(f, b - 1) + 1);
                f = b;
                b0 = b;
                a0 = b - 1;
            }
            whole += rays * (steps(a + 1, a0) + steps(a, n - 1));
            a0 = a;
        }
    }
    // about 20 tasks per resident warp, of a few hundred steps
    const int target = (int)std::min(400.0, std::max(40.0, whole / (20.0 * (double)warps)));
    TreeBuild T;
    long long tasks = 0;
    for (const TreeGroup& g : groups)
    {
        if (g.n <= 0 || g.pairs.empty()) continue;
        TreeGrid G{(int)std::min<long long>(tasks, 1LL << 30), g.base, g.n, (g.n + kTile - 1) / kTile, (int)T.segments.size(), 0};
        int cost = 0, b0 = -1, a0 = 0, f = 0, last_f = -1, last_b = -1;
        // A segment's end: which pairs hang on each run (a forward run: all from
        // its b on; a backward run: those of its b from its a on), and where to
        // go on without it (the next forward run, or the end).
        auto close = [&] {
            if (T.segments.size() == (size_t)G.seg_base || T.segments.back().run_end >= 0) return;
            TreeSegment& seg = T.segments.back();
            seg.run_end = (int)T.runs.size();
            seg.pair_end = (int)T.pairs.size();
            int next = seg.run_end;
            unsigned after = 0, of_b = 0;
            for (int r = seg.run_end - 1; r >= seg.run_begin; --r)
            {
                int4& run = T.runs[r];
                run.w = next;
                if (run.y & RUN_LAST) of_b |= (unsigned)run.z;
                else if (run.y & RUN_FORWARD)
                {
                    after |= of_b;
                    of_b = 0;
                    run.z = (int)after;
                    next = r;
                }
                else run.z = (int)of_b;
            }
        };
        for (int i : g.pairs)
        {
            const int a = pairs[i].surf_a, b = pairs[i].surf_b;
            if (b0 < 0 || cost >= target || (int)T.pairs.size() - T.segments.back().pair_begin >= 32)
            {
                close();
                T.segments.push_back({(int)T.runs.size(), -1, (int)T.pairs.size(), 0});
                cost = 0;
                b0 = -1;
                f = 0;
                last_f = -1;
            }
            if (b != b0)
            {
                // forward from the last b (or the start) to b - 1
                if (last_f >= 0) T.runs[last_f].y |= RUN_SAVE_F;
                T.runs.push_back(make_int4(f | ((b - 1) << 8), RUN_FORWARD | (last_f >= 0 ? RUN_LOAD_F : 0), 0, 0));
                last_f = (int)T.runs.size() - 1;
                cost += steps(f, b - 1);
                // turn at b, back through b - 1 .. a + 1
                T.runs.push_back(make_int4(b | ((a + 1) << 8), RUN_REFLECT | RUN_BACK, 0, 0));
                cost += 1 + steps(a + 1, b - 1);
                f = b;
            }
            else
            {
                // on from the last a: back through a0 .. a + 1
                T.runs[last_b].y |= RUN_SAVE_B;
                T.runs.push_back(make_int4(a0 | ((a + 1) << 8), RUN_BACK | RUN_LOAD_B, 0, 0));
                cost += steps(a + 1, a0);
            }
            last_b = (int)T.runs.size() - 1;
            T.runs.push_back(make_int4(a | ((n - 1) << 8), RUN_REFLECT | RUN_LAST,
                                       (int)(1u << ((int)T.pairs.size() - T.segments.back().pair_begin)), 0));
            T.pairs.push_back(i);
            cost += steps(a, n - 1);
            b0 = b;
            a0 = a;
        }
        close();
        G.n_segs = (int)T.segments.size() - G.seg_base;
        T.grids.push_back(G);
        tasks += (long long)G.n_segs * G.tiles * n_src * n_spec;
    }
    if (tasks <= 0 || tasks >= (1LL << 30)) return {};
    T.grids.push_back({(int)tasks, 0, 0, 1, (int)T.segments.size(), 0});
    T.tasks = (int)tasks;
    return T;
}

int plan_create(const gl_surface* surfaces, int n_surf, const gl_ghost_pair* pairs, const float* boosts,
                const int32_t* pair_grid, int n_pairs, const gl_flare_source* sources, int n_src,
                const gl_pupil_sample* samples, const int32_t* grid_offsets, int n_grids,
                const gl_spectral_sample* spec, int n_spec, const gl_ghost_render_params* prm,
                GhostPlan** out)
{
    if (!surfaces || n_surf <= 0 || !prm || !out) return fail(GL_ERR_INVALID, "render_ghosts: bad arguments");
    if (n_pairs < 0 || n_src < 0 || n_grids < 0) return fail(GL_ERR_INVALID, "render_ghosts: negative count");
    if (n_pairs > 0 && (!pairs || !boosts)) return fail(GL_ERR_INVALID, "render_ghosts: missing pairs");
    if (n_src > 0 && !sources) return fail(GL_ERR_INVALID, "render_ghosts: missing sources");
    if (prm->width <= 0 || prm->height <= 0) return fail(GL_ERR_INVALID, "render_ghosts: width and height must be positive");
    if ((long long)prm->width * prm->height > (1LL << 31)) return fail(GL_ERR_INVALID, "render_ghosts: image has too many pixels");
    if (n_spec < 1 || n_spec > kMaxSpec || !spec) return fail(GL_ERR_INVALID, "render_ghosts: spectral table must hold 1..256 samples");
    if (!(prm->sensor_half_w > 0.0f) || !(prm->sensor_half_h > 0.0f))
        return fail(GL_ERR_INVALID, "render_ghosts: sensor half extents must be positive");
    if (n_grids > 0 && (!grid_offsets || !samples)) return fail(GL_ERR_INVALID, "render_ghosts: missing pupil grids");
    for (int i = 0; i < n_pairs; ++i)
    {
        const int a = pairs[i].surf_a, b = pairs[i].surf_b;
        if (a < 0 || b <= a || b >= n_surf) return fail(GL_ERR_INVALID, "render_ghosts: bounce indices must satisfy 0 <= a < b < n");
        const int g = pair_grid ? pair_grid[i] : 0;
        if (g < 0 || g >= n_grids) return fail(GL_ERR_INVALID, "render_ghosts: pair grid index out of range");
    }
    for (int g = 0; g < n_grids; ++g)
        if (grid_offsets[g + 1] < grid_offsets[g] || grid_offsets[g] < 0)
            return fail(GL_ERR_INVALID, "render_ghosts: grid offsets must be non-decreasing");

    int plan_dev = 0;
    GL_CUDA_TRY(cudaGetDevice(&plan_dev));
    std::vector<SurfRec> recs((size_t)n_surf);
    int rc = pack_lens(surfaces, n_surf, recs.data(), plan_dev);
    if (rc) return rc;

    GhostPlan* p = new GhostPlan();
    cudaGetDevice(&p->device);
    p->n_surf = n_surf; p->n_spec = n_spec; p->n_pairs = n_pairs;
    p->front_R = surfaces[0].semi_aperture;              // ghost_render.cu:738-739
    p->start_z = surfaces[0].z - kSpawnOffset;
    p->width = prm->width; p->height = prm->height; p->prm = *prm;
    // the per-pair form keeps the reference kernel's shape: every thread loops
    // over all wavelengths (ghost_render.cu:372)
    p->l_chunks = prm->plain_per_pair ? 1 : default_lambda_split(n_spec);

    std::vector<float> lams((size_t)n_spec), at((size_t)n_spec * n_surf), bf((size_t)n_spec * n_surf);
    std::vector<float4> sp((size_t)n_spec);
    for (int i = 0; i < n_spec; ++i)
    {
        lams[i] = spec[i].lambda;
        sp[i] = make_float4(spec[i].lambda, spec[i].cmf_r, spec[i].cmf_g, spec[i].cmf_b);
    }
    build_ior_tables(surfaces, n_surf, lams.data(), n_spec, at.data(), bf.data());

    // Per-source beam (ghost_render.cu:349-358): tanf slopes, the normalised
    // direction and the spawn-plane shift that follows the beam.
    std::vector<SourceDev> src((size_t)n_src);
    for (int i = 0; i < n_src; ++i) src[i] = make_source(sources[i]);

    const int n_samples_all = n_grids > 0 ? grid_offsets[n_grids] : 0;
    std::vector<gl_pupil_sample> ordered((size_t)n_samples_all);
    for (int g = 0; g < n_grids; ++g)
        morton_order(samples + grid_offsets[g], grid_offsets[g + 1] - grid_offsets[g], ordered.data() + grid_offsets[g]);

    std::vector<PairDev> pd((size_t)n_pairs);
    std::vector<int4> items;
    p->pair_item_begin.assign((size_t)n_pairs + 1, 0);
    for (int i = 0; i < n_pairs; ++i)
    {
        const int g = pair_grid ? pair_grid[i] : 0;
        const int g0 = grid_offsets[g], ng = grid_offsets[g + 1] - grid_offsets[g];
        pd[i] = {pairs[i].surf_a, pairs[i].surf_b, boosts[i], ng > 0 ? 1.0f / (float)ng : 0.0f};
        p->pair_item_begin[i] = (int)items.size();
        for (int s = 0; s < n_src; ++s)
            for (int t = 0; t < ng; t += kTile)
                items.push_back(make_int4(i, s, g0 + t, std::min(kTile, ng - t)));
        p->rays += (long long)ng * n_src * n_spec;
    }
    p->pair_item_begin[n_pairs] = (int)items.size();
    p->n_items = (int)items.size();

    // Off-sensor probe grids (ghost_render.cu:1022-1027): 40x40, wang-hash
    // jitter with a fixed seed per pass, the config's blade override.
    p->cull = prm->cull_dead_pairs && n_pairs > 1 && n_spec != 3 && !prm->plain_per_pair;
    std::vector<int4> pitems;
    std::vector<gl_pupil_sample> psamples;
    std::vector<int> hits_init((size_t)n_pairs, 1);
    if (p->cull)
    {
        // A pair is probed only when its own grid is larger than the three
        // probe passes: rendering a pair that lands nowhere costs less than
        // proving it, and never changes the image.
        int pbeg[4];
        {
            const int rcs = probe_grids(surfaces, n_surf, prm->blades_override, prm->rotation_deg, psamples, pbeg);
            if (rcs) { plan_free(p); return rcs; }
        }
        const int n_probe_samples = pbeg[3];
        for (int i = 0; i < n_pairs; ++i)
        {
            const int gi = pair_grid ? pair_grid[i] : 0;
            const int ng = grid_offsets[gi + 1] - grid_offsets[gi];
            hits_init[i] = (ng > n_probe_samples) ? 0 : 1;
        }
        for (int pass = 0; pass < 3; ++pass)
        {
            const int base = pbeg[pass], cnt = pbeg[pass + 1] - pbeg[pass];
            p->probe_begin[pass] = (int)pitems.size();
            for (int i = 0; i < n_pairs; ++i)
            {
                if (hits_init[i]) continue;
                for (int s = 0; s < n_src; ++s)
                    for (int t = 0; t < cnt; t += kTile)
                        pitems.push_back(make_int4(i, s, base + t, std::min(kTile, cnt - t)));
                p->probe_rays += (long long)cnt * n_src * n_spec;
            }
        }
        p->probe_begin[3] = (int)pitems.size();
    }
    const int n_samples = n_grids > 0 ? grid_offsets[n_grids] : 0;

    cudaError_t e = cudaSuccess;
    auto chk = [&](cudaError_t x) { if (e == cudaSuccess) e = x; };
    chk(shared_device_pool(p->device, &p->pool));
    p->own = plan_stream(p->device);
    if (e == cudaSuccess && !p->own) e = cudaErrorInvalidResourceHandle;
    if (e == cudaSuccess) chk(cudaEventCreateWithFlags(&p->done, cudaEventDisableTiming));
    if (e != cudaSuccess)
    {
        p->own = nullptr;
        plan_free(p);
        return fail(GL_ERR_CUDA, std::string("render_ghosts: ") + cudaGetErrorString(e));
    }
    cudaMemPool_t pool = p->pool;
    cudaStream_t ost = p->own;
    chk(upload(&p->recs, recs.data(), recs.size(), pool, ost));
    chk(upload(&p->ior_at, at.data(), at.size(), pool, ost));
    chk(upload(&p->ior_bf, bf.data(), bf.size(), pool, ost));
    chk(upload(&p->spec, sp.data(), sp.size(), pool, ost));
    chk(upload(&p->items, items.data(), items.size(), pool, ost));
    chk(upload(&p->pairs, pd.data(), pd.size(), pool, ost));
    chk(upload(&p->sources, src.data(), src.size(), pool, ost));
    chk(upload(&p->samples, reinterpret_cast<const float2*>(ordered.data()), (size_t)n_samples, pool, ost));
    chk(alloc(&p->counter, sizeof(int), pool, ost));
    chk(alloc(&p->traced, 2 * sizeof(unsigned long long), pool, ost));
    if (p->cull)
    {
        chk(upload(&p->probe_items, pitems.data(), pitems.size(), pool, ost));
        chk(upload(&p->probe_samples, reinterpret_cast<const float2*>(psamples.data()), psamples.size(), pool, ost));
        chk(alloc(&p->pair_hits, sizeof(int) * std::max(1, n_pairs), pool, ost));
        chk(upload(&p->pair_hits_init, hits_init.data(), hits_init.size(), pool, ost));
        chk(alloc(&p->probe_counters, sizeof(int) * 4, pool, ost));
    }
    TreeBuild trees[2];
    if (e == cudaSuccess && p->n_items > 0)
    {
        int n_sm = 0;
        chk(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, p->device));
        const long long warps = (long long)n_sm * kRenderMinBlocks * (kRenderThreads / 32);
        p->n_src = n_src;
        auto put = [&](TreeBuild& t, TreeDev& d, std::vector<TreeGroup> groups) {
            t = build_tree(recs.data(), n_surf, pairs, std::move(groups), n_src, n_spec, warps);
            if (t.tasks <= 0) return;
            d.n_tasks = t.tasks;
            d.n_grids = (int)t.grids.size() - 1;
            chk(upload(&d.grids, t.grids.data(), t.grids.size(), pool, ost));
            chk(upload(&d.segments, t.segments.data(), t.segments.size(), pool, ost));
            chk(upload(&d.runs, t.runs.data(), t.runs.size(), pool, ost));
            chk(upload(&d.pairs, t.pairs.data(), t.pairs.size(), pool, ost));
        };
        if (!prm->plain_per_pair)
        {
            std::vector<TreeGroup> groups((size_t)n_grids);
            for (int g = 0; g < n_grids; ++g) groups[g] = {{}, grid_offsets[g], grid_offsets[g + 1] - grid_offsets[g]};
            for (int i = 0; i < n_pairs; ++i) groups[pair_grid ? pair_grid[i] : 0].pairs.push_back(i);
            put(trees[0], p->tree, std::move(groups));
        }
        if (p->cull)
        {
            TreeGroup probed{{}, 0, (int)psamples.size()};
            for (int i = 0; i < n_pairs; ++i)
                if (hits_init[i] == 0) probed.pairs.push_back(i);
            put(trees[1], p->probe_tree, {std::move(probed)});
        }
    }
    chk(alloc(&p->accum, (size_t)prm->width * prm->height * sizeof(float4), pool, ost));
    if (e == cudaSuccess) chk(cudaMemsetAsync(p->accum, 0, (size_t)prm->width * prm->height * sizeof(float4), ost));
    // the host vectors above go out of scope: the uploads must have landed
    chk(cudaStreamSynchronize(ost));
    p->smem = render_smem(n_surf, n_spec);
    int per_sm = 0, n_sm = 0;
    if (e == cudaSuccess) chk(render_prepare(p->smem, &per_sm, &n_sm));
    if (e != cudaSuccess)
    {
        plan_free(p);
        return fail(e == cudaErrorMemoryAllocation ? GL_ERR_OOM : GL_ERR_CUDA,
                    std::string("render_ghosts: ") + cudaGetErrorString(e));
    }
    const int warps_per_block = kRenderThreads / 32;
    p->per_sm = std::max(1, per_sm);
    p->n_sm = n_sm;
    p->queue_ctas = p->per_sm * n_sm;
    // The pair-by-pair walk and the probes: a plan of few items splits its
    // wavelengths further, to about 20 tasks per resident warp; a task's chain of
    // steps is what such a frame waits for.  66 pairs pair by pair: 32^2 x 8
    // wavelengths 158 -> 64 us, 64^2 x 8 232 -> 139; 120 pairs x 5 sources, 42^2 x 8
    // 621 -> 463; above (180850 items x 31) the default's eight wavelengths per task
    // stay best (6128 us, 6326 with four).
    if (!prm->plain_per_pair && p->n_items > 0)
    {
        const long long want = (20LL * p->queue_ctas * warps_per_block + p->n_items - 1) / p->n_items;
        if (want > p->l_chunks)
        {
            const int l_size = std::max(1, (int)(n_spec / std::min<long long>(want, n_spec)));
            p->l_chunks = std::max(p->l_chunks, (n_spec + l_size - 1) / l_size);
        }
    }
    *out = p;
    return GL_OK;
}

// Launch shape of the batched render (the autotuner's knob): items_per_warp
// 0 = persistent work queue over ctas_per_sm CTAs per SM (0 = every resident
// slot); > 0 = one-shot CTAs of that many 32-sample items per warp.
int plan_set_launch(GhostPlan* p, int items_per_warp, int ctas_per_sm)
{
    if (items_per_warp < 0 || ctas_per_sm < 0) return fail(GL_ERR_INVALID, "ghost_plan_set_launch: negative value");
    const int cps = ctas_per_sm == 0 ? p->per_sm : std::min(ctas_per_sm, p->per_sm);
    p->launch_ipw = items_per_warp;
    p->queue_ctas = cps * p->n_sm;
    return GL_OK;
}

// CTAs of the persistent queue for `items` items of `chunks` tasks.
static int queue_grid(const GhostPlan* p, long long items, int chunks)
{
    const int warps_per_block = kRenderThreads / 32;
    const long long tasks = items * std::max(1, chunks);
    return (int)std::max<long long>(1, std::min<long long>((tasks + warps_per_block - 1) / warps_per_block, p->queue_ctas));
}

static TreeArgs tree_args(const GhostPlan* p, const TreeDev& t)
{
    return {t.grids, t.segments, t.runs, t.pairs, t.n_grids, p->n_src};
}

// An event recorded inside a stream capture becomes an event-record node
// (external), so a replayed graph records it too.
static cudaError_t record_event(cudaEvent_t ev, cudaStream_t st)
{
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(st, &cs);
    if (e != cudaSuccess) return e;
    return cs == cudaStreamCaptureStatusActive ? cudaEventRecordWithFlags(ev, st, cudaEventRecordExternal)
                                               : cudaEventRecord(ev, st);
}

int plan_execute(GhostPlan* p, float* d_out_r, float* d_out_g, float* d_out_b, cudaStream_t st)
{
    if (!p || !d_out_r || !d_out_g || !d_out_b) return fail(GL_ERR_INVALID, "render_ghosts: null output");
    const size_t n_px = (size_t)p->width * p->height;
    int launches = 0;
    GL_CUDA_TRY(cudaMemsetAsync(p->accum, 0, n_px * sizeof(float4), st));
    RenderArgs A{};
    A.recs = p->recs; A.ior_at = p->ior_at; A.ior_bf = p->ior_bf; A.spec = p->spec;
    A.items = p->items; A.pairs = p->pairs; A.sources = p->sources; A.samples = p->samples;
    A.counter = nullptr; A.accum = p->accum;
    A.n_surf = p->n_surf; A.n_spec = p->n_spec; A.n_items = p->n_items; A.item_base = 0;
    A.l_chunks = p->l_chunks;
    A.width = p->width; A.height = p->height;
    A.fmt_w = (float)p->prm.fmt_w; A.fmt_h = (float)p->prm.fmt_h;
    A.fmt_x0 = (float)p->prm.fmt_x0; A.fmt_y0 = (float)p->prm.fmt_y0;
    A.hw2 = 2.0f * p->prm.sensor_half_w; A.hh2 = 2.0f * p->prm.sensor_half_h;
    A.gain = p->prm.flare_gain;
    A.front_R = p->front_R; A.start_z = p->start_z;
    A.pair_hits = nullptr;
    A.traced = p->traced;
    GL_CUDA_TRY(cudaMemsetAsync(p->traced, 0, 2 * sizeof(unsigned long long), st));
    if (p->ev_probe) GL_CUDA_TRY(record_event(p->ev_probe, st));
    if (p->cull && p->n_items > 0)
    {
        // Probe passes: the frame inflated by CULL_MARGIN = 1.25
        // (ghost_render.cu:148).  The three passes are one persistent launch
        // without a boundary per pass: a pair is culled only when no ray of any
        // pass hits, and a pair that has a hit is not looked at again.  The tree
        // takes the passes' samples as one grid, wavelength by wavelength; pair
        // by pair the items come in pass order, so a later pass probes only the
        // pairs still without a hit (the reference's candidate rule).
        GL_CUDA_TRY(cudaMemcpyAsync(p->pair_hits, p->pair_hits_init, sizeof(int) * p->n_pairs,
                                    cudaMemcpyDeviceToDevice, st));
        GL_CUDA_TRY(cudaMemsetAsync(p->probe_counters, 0, sizeof(int) * 4, st));
        RenderArgs B = A;
        B.samples = p->probe_samples;
        B.pair_hits = p->pair_hits;
        B.traced = p->traced + 1;
        B.hw2 = 2.0f * (p->prm.sensor_half_w * 1.25f);
        B.hh2 = 2.0f * (p->prm.sensor_half_h * 1.25f);
        const int n_it = p->probe_begin[3];
        if (n_it > 0)
        {
            B.items = p->probe_items;
            B.n_items = n_it;
            B.counter = p->probe_counters;
            if (p->probe_tree.n_tasks > 0)
                ghost_tree_kernel<true><<<queue_grid(p, p->probe_tree.n_tasks, 1), kRenderThreads, p->smem, st>>>(
                    B, tree_args(p, p->probe_tree));
            else
                ghost_render_kernel<true><<<queue_grid(p, n_it, B.l_chunks), kRenderThreads, p->smem, st>>>(B);
            ++launches;
        }
        GL_CUDA_TRY(cudaGetLastError());
        A.pair_hits = p->pair_hits;
    }
    if (p->ev_render) GL_CUDA_TRY(record_event(p->ev_render, st));
    if (p->n_items > 0)
    {
        if (p->prm.plain_per_pair)
        {
            // The reference's per-ghost loop: one launch per pair, sized to it.
            for (int i = 0; i < p->n_pairs; ++i)
            {
                const int b0 = p->pair_item_begin[i], b1 = p->pair_item_begin[i + 1];
                if (b1 <= b0) continue;
                A.item_base = b0;
                A.n_items = b1;
                const int warps_per_block = kRenderThreads / 32;
                ghost_render_kernel<false><<<(b1 - b0 + warps_per_block - 1) / warps_per_block, kRenderThreads, p->smem, st>>>(A);
                ++launches;
            }
            GL_CUDA_TRY(cudaGetLastError());
        }
        else if (p->launch_ipw > 0)
        {
            const int per_cta = (kRenderThreads / 32) * p->launch_ipw;
            const int grid = std::max(1, (p->n_items + per_cta - 1) / per_cta);
            ghost_render_kernel<false><<<grid, kRenderThreads, p->smem, st>>>(A);
            GL_CUDA_TRY(cudaGetLastError());
            ++launches;
        }
        else
        {
            GL_CUDA_TRY(cudaMemsetAsync(p->counter, 0, sizeof(int), st));
            A.counter = p->counter;
            if (p->tree.n_tasks > 0)
                ghost_tree_kernel<false><<<queue_grid(p, p->tree.n_tasks, 1), kRenderThreads, p->smem, st>>>(
                    A, tree_args(p, p->tree));
            else
                ghost_render_kernel<false><<<queue_grid(p, p->n_items, A.l_chunks), kRenderThreads, p->smem, st>>>(A);
            GL_CUDA_TRY(cudaGetLastError());
            ++launches;
        }
    }
    if (p->ev_end) GL_CUDA_TRY(record_event(p->ev_end, st));
    const float* C = p->prm.correction;
    const size_t quads = (n_px + 3) / 4;
    const int fb = 256;
    ghost_flush_kernel<<<(unsigned)((quads + fb - 1) / fb), fb, 0, st>>>(
        p->accum, n_px, d_out_r, d_out_g, d_out_b, p->prm.apply_correction,
        C[0], C[1], C[2], C[3], C[4], C[5], C[6], C[7], C[8]);
    GL_CUDA_TRY(cudaGetLastError());
    ++launches;
    // completion marker for destroy (see GhostPlan::done)
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    GL_CUDA_TRY(cudaStreamIsCapturing(st, &cs));
    if (cs == cudaStreamCaptureStatusActive)
        p->captured = true;
    else
    {
        GL_CUDA_TRY(cudaEventRecord(p->done, st));
        p->executed = true;
    }
    g_last_launches = launches;
    return GL_OK;
}

// ---------------------------------------------------------------------------
// Batched ray trace (trace_ghost_ray / trace_primary_ray, trace.cpp:171,243)
// with an arbitrary wavelength per ray: the IOR of every surface is
// evaluated per ray from the dispersion data.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) trace_rays_kernel(const SurfRec* __restrict__ recs,
                                                         const DispRec* __restrict__ disp, int n,
                                                         int a, int b, const float* __restrict__ rays,
                                                         int n_rays, float* __restrict__ out)
{
    __shared__ SurfRec lens[kMaxSurfaces];
    __shared__ DispRec dr[kMaxSurfaces];
    {
        const int words = n * (int)(sizeof(SurfRec) / 4);
        for (int i = threadIdx.x; i < words; i += blockDim.x)
            reinterpret_cast<int*>(lens)[i] = reinterpret_cast<const int*>(recs)[i];
        const int dw = n * (int)(sizeof(DispRec) / 4);
        for (int i = threadIdx.x; i < dw; i += blockDim.x)
            reinterpret_cast<int*>(dr)[i] = reinterpret_cast<const int*>(disp)[i];
    }
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_rays) return;
    const float* r = rays + 7 * (size_t)i;
    const float lam = r[6];
    float at[kMaxSurfaces], bf[kMaxSurfaces];
    float last = 1.0f;
    for (int k = 0; k < n; ++k)
    {
        at[k] = disp_ior(dr[k], lam);
        bf[k] = last;
        if (lens[k].flags & SF_ACTIVE) last = at[k];
    }
    const V3 o = v3(r[0], r[1], r[2]), d = v3(r[3], r[4], r[5]);
    TraceOut t = (b < 0) ? trace_primary(lens, n, at, o, d, lam) : trace_ghost(lens, n, at, bf, o, d, lam, a, b);
    float* q = out + 5 * (size_t)i;
    q[0] = t.x; q[1] = t.y; q[2] = t.z; q[3] = t.w; q[4] = (float)t.status;
}

}  // namespace gl

using namespace gl;

struct gl_ghost_plan { GhostPlan* p; };

extern "C" {

int gl_ghost_plan_create(const gl_surface* surfaces, int n_surfaces, const gl_ghost_pair* pairs,
                         const float* area_boosts, const int32_t* pair_grid, int n_pairs,
                         const gl_flare_source* sources, int n_sources, const gl_pupil_sample* samples,
                         const int32_t* grid_offsets, int n_grids, const gl_spectral_sample* spec,
                         int n_spec, const gl_ghost_render_params* params, gl_ghost_plan** out)
{
    if (!out) return fail(GL_ERR_INVALID, "ghost_plan_create: null out");
    GhostPlan* p = nullptr;
    int rc = plan_create(surfaces, n_surfaces, pairs, area_boosts, pair_grid, n_pairs, sources, n_sources,
                         samples, grid_offsets, n_grids, spec, n_spec, params, &p);
    if (rc) return rc;
    *out = new gl_ghost_plan{p};
    return GL_OK;
}

int gl_ghost_plan_execute(gl_ghost_plan* plan, float* d_out_r, float* d_out_g, float* d_out_b, void* stream)
{
    if (!plan) return fail(GL_ERR_INVALID, "ghost_plan_execute: null plan");
    return plan_execute(plan->p, d_out_r, d_out_g, d_out_b, (cudaStream_t)stream);
}

int gl_morton_order(const gl_pupil_sample* in, int n, gl_pupil_sample* out)
{
    if (n < 0 || (n > 0 && (!in || !out))) return fail(GL_ERR_INVALID, "morton_order: bad arguments");
    morton_order(in, n, out);
    return GL_OK;
}

int gl_ghost_plan_set_launch(gl_ghost_plan* plan, int items_per_warp, int ctas_per_sm)
{
    if (!plan) return fail(GL_ERR_INVALID, "ghost_plan_set_launch: null plan");
    return plan_set_launch(plan->p, items_per_warp, ctas_per_sm);
}

int gl_ghost_plan_set_lambda_split(gl_ghost_plan* plan, int chunks)
{
    if (!plan) return fail(GL_ERR_INVALID, "ghost_plan_set_lambda_split: null plan");
    if (chunks < 1) return fail(GL_ERR_INVALID, "ghost_plan_set_lambda_split: chunks must be >= 1");
    plan->p->l_chunks = std::min(chunks, plan->p->n_spec);
    return GL_OK;
}

int gl_ghost_plan_info(const gl_ghost_plan* plan, long long* rays, int* n_items, int* grid)
{
    if (!plan) return fail(GL_ERR_INVALID, "ghost_plan_info: null plan");
    if (rays) *rays = plan->p->rays + plan->p->probe_rays;
    if (n_items) *n_items = plan->p->n_items;
    const GhostPlan* p = plan->p;
    if (grid) *grid = p->tree.n_tasks > 0 ? queue_grid(p, p->tree.n_tasks, 1) : queue_grid(p, p->n_items, p->l_chunks);
    return GL_OK;
}

int gl_ghost_plan_walk(const gl_ghost_plan* plan, int* render_tasks, int* probe_tasks)
{
    if (!plan) return fail(GL_ERR_INVALID, "ghost_plan_walk: null plan");
    if (render_tasks) *render_tasks = plan->p->tree.n_tasks;
    if (probe_tasks) *probe_tasks = plan->p->probe_tree.n_tasks;
    return GL_OK;
}

int gl_ghost_plan_traced(const gl_ghost_plan* plan, long long* out)
{
    if (!plan || !out) return fail(GL_ERR_INVALID, "ghost_plan_traced: bad arguments");
    unsigned long long v[2] = {0, 0};
    GL_CUDA_TRY(cudaMemcpy(v, plan->p->traced, sizeof(v), cudaMemcpyDeviceToHost));
    *out = (long long)(v[0] + v[1]);
    return GL_OK;
}

// The diagnostic stats pass (launch_ghost_render's collect_stats launch,
// ghost_render.cu:1357-1431): every render item of the plan traced again
// without weights or splat and without the off-sensor cull, counting per pair
// the ray-wavelength traces, the rays that left the lens and those landing
// inside the frame.  out: 3 x n_pairs host counters {traces, survived, on
// sensor}, pair-major.  Synchronises the stream.
int gl_ghost_plan_stats(gl_ghost_plan* plan, unsigned long long* out, void* stream)
{
    if (!plan || !out) return fail(GL_ERR_INVALID, "ghost_plan_stats: null argument");
    GhostPlan* p = plan->p;
    cudaStream_t st = (cudaStream_t)stream;
    const size_t bytes = sizeof(unsigned long long) * 3 * (size_t)std::max(1, p->n_pairs);
    unsigned long long* d = nullptr;
    GL_CUDA_TRY(cudaMallocAsync(reinterpret_cast<void**>(&d), bytes, st));
    cudaError_t e = cudaMemsetAsync(d, 0, bytes, st);
    if (e == cudaSuccess && p->n_items > 0)
    {
        RenderArgs A{};
        A.recs = p->recs; A.ior_at = p->ior_at; A.ior_bf = p->ior_bf; A.spec = p->spec;
        A.items = p->items; A.pairs = p->pairs; A.sources = p->sources; A.samples = p->samples;
        A.accum = p->accum;
        A.n_surf = p->n_surf; A.n_spec = p->n_spec; A.n_items = p->n_items; A.item_base = 0;
        A.l_chunks = 1;
        A.width = p->width; A.height = p->height;
        A.fmt_w = (float)p->prm.fmt_w; A.fmt_h = (float)p->prm.fmt_h;
        A.fmt_x0 = (float)p->prm.fmt_x0; A.fmt_y0 = (float)p->prm.fmt_y0;
        A.hw2 = 2.0f * p->prm.sensor_half_w; A.hh2 = 2.0f * p->prm.sensor_half_h;
        A.gain = p->prm.flare_gain;
        A.front_R = p->front_R; A.start_z = p->start_z;
        A.stats = d;
        const int warps_per_block = kRenderThreads / 32;
        ghost_render_kernel<true><<<(p->n_items + warps_per_block - 1) / warps_per_block, kRenderThreads, p->smem,
                                    st>>>(A);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, d, sizeof(unsigned long long) * 3 * p->n_pairs,
                                              cudaMemcpyDeviceToHost, st);
    cudaFreeAsync(d, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return fail(GL_ERR_CUDA, std::string("ghost_plan_stats: ") + cudaGetErrorString(e));
    g_last_launches = 1;
    return GL_OK;
}

int gl_ghost_plan_traced_split(const gl_ghost_plan* plan, long long* render, long long* probe)
{
    if (!plan) return fail(GL_ERR_INVALID, "ghost_plan_traced_split: null plan");
    unsigned long long v[2] = {0, 0};
    GL_CUDA_TRY(cudaMemcpy(v, plan->p->traced, sizeof(v), cudaMemcpyDeviceToHost));
    if (render) *render = (long long)v[0];
    if (probe) *probe = (long long)v[1];
    return GL_OK;
}

int gl_ghost_plan_set_timing(gl_ghost_plan* plan, void* ev_probe, void* ev_render, void* ev_end)
{
    if (!plan) return fail(GL_ERR_INVALID, "ghost_plan_set_timing: null plan");
    plan->p->ev_probe = (cudaEvent_t)ev_probe;
    plan->p->ev_render = (cudaEvent_t)ev_render;
    plan->p->ev_end = (cudaEvent_t)ev_end;
    return GL_OK;
}

int gl_ghost_plan_pair_hits(const gl_ghost_plan* plan, int32_t* out, int n)
{
    if (!plan || !out || n < plan->p->n_pairs) return fail(GL_ERR_INVALID, "ghost_plan_pair_hits: bad arguments");
    if (!plan->p->cull) { for (int i = 0; i < plan->p->n_pairs; ++i) out[i] = 1; return GL_OK; }
    GL_CUDA_TRY(cudaMemcpy(out, plan->p->pair_hits, sizeof(int) * plan->p->n_pairs, cudaMemcpyDeviceToHost));
    return GL_OK;
}

int gl_ghost_plan_destroy(gl_ghost_plan* plan)
{
    if (!plan) return GL_OK;
    plan_free(plan->p);
    delete plan;
    return GL_OK;
}

int gl_render_ghosts(const gl_surface* surfaces, int n_surfaces, const gl_ghost_pair* pairs,
                     const float* area_boosts, const int32_t* pair_grid, int n_pairs,
                     const gl_flare_source* sources, int n_sources, const gl_pupil_sample* samples,
                     const int32_t* grid_offsets, int n_grids, const gl_spectral_sample* spec, int n_spec,
                     const gl_ghost_render_params* params, float* d_out_r, float* d_out_g, float* d_out_b,
                     void* stream)
{
    GhostPlan* p = nullptr;
    int rc = plan_create(surfaces, n_surfaces, pairs, area_boosts, pair_grid, n_pairs, sources, n_sources,
                         samples, grid_offsets, n_grids, spec, n_spec, params, &p);
    if (rc) return rc;
    rc = plan_execute(p, d_out_r, d_out_g, d_out_b, (cudaStream_t)stream);
    cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
    plan_free(p);
    if (rc) return rc;
    if (e != cudaSuccess) return fail(GL_ERR_CUDA, std::string("render_ghosts: ") + cudaGetErrorString(e));
    return GL_OK;
}

int gl_trace_rays(const gl_surface* surfaces, int n, int bounce_a, int bounce_b, const float* d_rays,
                  int n_rays, float* d_out, void* stream)
{
    if (!surfaces || n <= 0) return fail(GL_ERR_INVALID, "trace_rays: lens has no surfaces");
    if (bounce_b >= 0 && (bounce_a < 0 || bounce_a >= bounce_b || bounce_b >= n))
        return fail(GL_ERR_INVALID, "bounce indices must satisfy 0 <= bounce_a < bounce_b < num_surfaces");
    if (n_rays < 0 || (n_rays > 0 && (!d_rays || !d_out))) return fail(GL_ERR_INVALID, "trace_rays: bad ray buffers");
    if (n_rays == 0) return GL_OK;
    int dev = 0;
    GL_CUDA_TRY(cudaGetDevice(&dev));
    std::vector<SurfRec> recs((size_t)n);
    int rc = pack_lens(surfaces, n, recs.data(), dev);
    if (rc) return rc;
    const std::vector<DispRec> disp = disp_records(surfaces, n);
    cudaStream_t st = (cudaStream_t)stream;
    // one block of the device's pool (kept, where the default pool gives its
    // memory back at every synchronisation: 0.2 ms of each call), one copy
    const size_t o_disp = (sizeof(SurfRec) * n + 255) & ~(size_t)255, bytes = o_disp + sizeof(DispRec) * n;
    std::vector<char> host(bytes);
    std::memcpy(host.data(), recs.data(), sizeof(SurfRec) * n);
    std::memcpy(host.data() + o_disp, disp.data(), sizeof(DispRec) * n);
    cudaMemPool_t pool;
    char* block = nullptr;
    GL_CUDA_TRY(shared_device_pool(dev, &pool));
    GL_CUDA_TRY(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&block), bytes, pool, st));
    cudaError_t e = cudaMemcpyAsync(block, host.data(), bytes, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
    {
        trace_rays_kernel<<<(n_rays + 127) / 128, 128, 0, st>>>(reinterpret_cast<SurfRec*>(block),
                                                                reinterpret_cast<DispRec*>(block + o_disp), n, bounce_a,
                                                                bounce_b, d_rays, n_rays, d_out);
        e = cudaGetLastError();
    }
    const cudaError_t f = cudaFreeAsync(block, st);
    // The host block must outlive the async copy.
    const cudaError_t w = cudaStreamSynchronize(st);
    GL_CUDA_TRY(e);
    GL_CUDA_TRY(f);
    GL_CUDA_TRY(w);
    g_last_launches = 1;
    return GL_OK;
}

}  // extern "C"

// ===========================================================================
// Allocation-free batched trace
//
// Some callers cannot allocate device memory while they run: a plug-in hosted
// by an application that owns the device heap through its own allocator, code
// on a real-time thread where an allocation's latency (and the device-wide
// synchronisation cudaMalloc may imply) is not allowed, or a host that has
// already reserved the whole device.  For them this entry point keeps the
// only scratch the trace needs — the packed lens records and dispersion
// terms — in one fixed array in device memory that is part of this library,
// sized for the largest lens the path accepts (64 surfaces).  The caller
// still passes the ray buffer and the result buffer.
//
// Every call looks up the array's device address with cudaGetSymbolAddress
// on the current device (the lookup allocates nothing), so the address is
// never stale, e.g. after a cudaDeviceReset.  A call ends with a
// cudaStreamSynchronize (the lens records are staged on its stack frame), so
// it must not be made while `stream` is being captured: it returns
// GL_ERR_INVALID there instead of breaking the caller's capture.  All calls
// share the array and it keeps whatever the last call wrote: each call
// overwrites the records it uses before launching, and calls that overlap on
// the GPU (other threads or streams) race on it.
// ===========================================================================
namespace gl {

constexpr int kNoAllocMaxSurfaces = 64;

struct NoAllocTables {
    SurfRec recs[kNoAllocMaxSurfaces];
    DispRec disp[kNoAllocMaxSurfaces];
};

static __device__ __align__(256) unsigned char g_trace_tables[sizeof(NoAllocTables)];

static int trace_tables_address(void** out)
{
    void* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&ptr, g_trace_tables);
    if (e != cudaSuccess || ptr == nullptr)
        return fail(GL_ERR_CUDA, std::string("trace_rays_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    *out = ptr;
    return GL_OK;
}

}  // namespace gl

extern "C" int gl_trace_rays_noalloc(const gl_surface* surfaces, int n, int bounce_a, int bounce_b,
                                     const float* d_rays, int n_rays, float* d_out, void* stream)
{
    if (!surfaces || n <= 0) return fail(GL_ERR_INVALID, "trace_rays_noalloc: lens has no surfaces");
    if (n > kNoAllocMaxSurfaces)
        return fail(GL_ERR_INVALID, "trace_rays_noalloc: lens has more than 64 surfaces, the size of the fixed table");
    if (bounce_b >= 0 && (bounce_a < 0 || bounce_a >= bounce_b || bounce_b >= n))
        return fail(GL_ERR_INVALID, "bounce indices must satisfy 0 <= bounce_a < bounce_b < num_surfaces");
    if (n_rays < 0 || (n_rays > 0 && (!d_rays || !d_out))) return fail(GL_ERR_INVALID, "trace_rays_noalloc: bad ray buffers");
    if (n_rays == 0) return GL_OK;
    cudaStream_t st = (cudaStream_t)stream;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    GL_CUDA_TRY(cudaStreamIsCapturing(st, &cap));
    if (cap != cudaStreamCaptureStatusNone)
        return fail(GL_ERR_INVALID, "trace_rays_noalloc: the call synchronises its stream and cannot be captured");
    int device = 0;
    GL_CUDA_TRY(cudaGetDevice(&device));
    void* base = nullptr;
    int rc = trace_tables_address(&base);
    if (rc) return rc;
    NoAllocTables host;   // staged on the stack: no heap, no device allocation
    rc = pack_lens(surfaces, n, host.recs, device, false);
    if (rc) return rc;
    for (int i = 0; i < n; ++i)
    {
        host.disp[i].model = surfaces[i].disp_model;
        host.disp[i].nd = surfaces[i].ior; host.disp[i].vd = surfaces[i].abbe_v; host.disp[i].pad = 0.0f;
        for (int k = 0; k < 3; ++k) { host.disp[i].B[k] = surfaces[i].sellmeier_B[k]; host.disp[i].C[k] = surfaces[i].sellmeier_C[k]; }
    }
    NoAllocTables* dev_tables = static_cast<NoAllocTables*>(base);
    GL_CUDA_TRY(cudaMemcpyAsync(dev_tables->recs, host.recs, sizeof(SurfRec) * n, cudaMemcpyHostToDevice, st));
    GL_CUDA_TRY(cudaMemcpyAsync(dev_tables->disp, host.disp, sizeof(DispRec) * n, cudaMemcpyHostToDevice, st));
    trace_rays_kernel<<<(n_rays + 127) / 128, 128, 0, st>>>(dev_tables->recs, dev_tables->disp, n, bounce_a,
                                                            bounce_b, d_rays, n_rays, d_out);
    GL_CUDA_TRY(cudaGetLastError());
    // The staging copy lives on this stack frame until the copies are done.
    GL_CUDA_TRY(cudaStreamSynchronize(st));
    g_last_launches = 1;
    return GL_OK;
}
