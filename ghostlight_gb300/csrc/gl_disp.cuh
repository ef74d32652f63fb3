// gl_disp.cuh — a surface's dispersion terms on the device, for the traces whose
// wavelength comes with the ray (the renders carry per-wavelength tables).
#pragma once

#include "gl_internal.h"

#include <vector>

namespace gl {

struct DispRec {
    int model;
    float nd, vd, pad;
    float B[3], C[3];
};

__device__ __forceinline__ float disp_ior(const DispRec& d, float lam)
{
    if (d.model == GL_DISP_SELLMEIER)
    {
        float l = lam * 1e-3f;
        float l2 = l * l;
        float n2 = 1.0f;
        n2 += d.B[0] * l2 / (l2 - d.C[0]);
        n2 += d.B[1] * l2 / (l2 - d.C[1]);
        n2 += d.B[2] * l2 / (l2 - d.C[2]);
        return (n2 > 0.0f) ? sqrtf(n2) : 1.0f;
    }
    const float n_d = d.nd, V_d = d.vd;
    if (V_d < 0.1f || n_d <= 1.0001f) return n_d;
    const float lF = 486.13f, lC = 656.27f, ld = 587.56f;
    float dn = (n_d - 1.0f) / V_d;
    float iF = 1.0f / (lF * lF), iC = 1.0f / (lC * lC), id = 1.0f / (ld * ld);
    float B = dn / (iF - iC);
    float Aa = n_d - B * id;
    return Aa + B / (lam * lam);
}

inline std::vector<DispRec> disp_records(const gl_surface* surfaces, int n)
{
    std::vector<DispRec> disp((size_t)n);
    for (int i = 0; i < n; ++i)
    {
        disp[i].model = surfaces[i].disp_model;
        disp[i].nd = surfaces[i].ior; disp[i].vd = surfaces[i].abbe_v; disp[i].pad = 0.0f;
        for (int k = 0; k < 3; ++k) { disp[i].B[k] = surfaces[i].sellmeier_B[k]; disp[i].C[k] = surfaces[i].sellmeier_C[k]; }
    }
    return disp;
}

}  // namespace gl
