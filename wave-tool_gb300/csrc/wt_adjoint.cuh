// wt_adjoint.cuh — the adjoint at one vertex, shared by the recurrence kernel
// (wt_adjoint.cu) and the matrix-product kernel (wt_adjoint_mma.cu).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "wt_device.cuh"
#include "wt_internal.h"

namespace wt {
namespace dev {

// Adjoints of the eight sums at one vertex from dL/dpos (gp) and dL/dnrm (gn,
// with has_nrm).  Order: dx, dy, dz, jx, jz, sxx,
// sxz, szz.  See oracle/gerstner_f64.c:wto_adjoint_f64 for the same algebra.
__device__ __forceinline__ void vertex_adjoint(const VertexSums& s, float xl, float zl, const PatchAux& a,
                                               const HmDev& hm, bool pow2, float3 gp, float3 gn, bool has_nrm,
                                               float g[8]) {
    const float a1 = 1.0f - s.sxx, a3 = -s.sxz, b1 = -s.sxz, b3 = 1.0f - s.szz;
    HmSample h = {0.0f, 0.0f, 0.0f, 0.0f};
    if (hm.present) h = hm_sample(hm, a, xl + s.dx, zl + s.dz, pow2);
    const float px0 = a1, px1 = fmaf(h.hx, a1, fmaf(h.hz, a3, s.jx)), px2 = a3;
    const float pz0 = b1, pz1 = fmaf(h.hx, b1, fmaf(h.hz, b3, s.jz)), pz2 = b3;
    const float gpx_ = gp.x, gpy_ = gp.y, gpz_ = gp.z;
    float gPx0 = 0.0f, gPx1 = 0.0f, gPx2 = 0.0f, gPz0 = 0.0f, gPz1 = 0.0f, gPz2 = 0.0f;
    if (has_nrm) {
        const float N0 = pz1 * px2 - pz2 * px1, N1 = pz2 * px0 - pz0 * px2, N2 = pz0 * px1 - pz1 * px0;
        const float inv = rsqrtf(fmaf(N0, N0, fmaf(N1, N1, N2 * N2)));
        const float n0 = N0 * inv, n1 = N1 * inv, n2 = N2 * inv;
        const float d = fmaf(n0, gn.x, fmaf(n1, gn.y, n2 * gn.z));
        const float gN0 = (gn.x - n0 * d) * inv, gN1 = (gn.y - n1 * d) * inv, gN2 = (gn.z - n2 * d) * inv;
        // N = Pz x Px:  g_Pz = Px x gN,  g_Px = gN x Pz
        gPz0 = px1 * gN2 - px2 * gN1;
        gPz1 = px2 * gN0 - px0 * gN2;
        gPz2 = px0 * gN1 - px1 * gN0;
        gPx0 = gN1 * pz2 - gN2 * pz1;
        gPx1 = gN2 * pz0 - gN0 * pz2;
        gPx2 = gN0 * pz1 - gN1 * pz0;
    }
    const float g_a1 = fmaf(gPx1, h.hx, gPx0), g_a3 = fmaf(gPx1, h.hz, gPx2);
    const float g_b1 = fmaf(gPz1, h.hx, gPz0), g_b3 = fmaf(gPz1, h.hz, gPz2);
    const float g_hx = fmaf(gPx1, a1, gPz1 * b1), g_hz = fmaf(gPx1, a3, gPz1 * b3);
    const float g_X = fmaf(gpy_, h.hx, g_hz * h.hxz), g_Z = fmaf(gpy_, h.hz, g_hx * h.hxz);
    g[0] = gpx_ + g_X;        // dx
    g[1] = gpy_;              // dy
    g[2] = gpz_ + g_Z;        // dz
    g[3] = gPx1;              // jx
    g[4] = gPz1;              // jz
    g[5] = -g_a1;             // sxx
    g[6] = -g_a3 - g_b1;      // sxz
    g[7] = -g_b3;             // szz
}

}  // namespace dev
}  // namespace wt
