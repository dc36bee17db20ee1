// wt_prep.cuh — validation and the FP64 constants of a patch table, shared by
// the prep kernels (wt_displace.cu) and the one-patch kernel (wt_single.cu).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "wt_device.cuh"
#include "wt_internal.h"

namespace wt {
namespace dev {

constexpr uint32_t kNoPatch = 0xffffffffu;

__device__ __forceinline__ bool finitef(float x) { return isfinite(x); }

// Wave i; wide: the array is on a 16-byte boundary (else eight loads a wave, of
// which each touches as many lines as these two: with them one block took 18.8 us
// to read and check the 9000 waves of 300 patches).
__device__ __forceinline__ bool waves_wide(const wt_wave* waves) {
    return (reinterpret_cast<uintptr_t>(waves) & 15u) == 0;
}
__device__ __forceinline__ wt_wave load_wave(const wt_wave* __restrict__ waves, uint32_t i, bool wide) {
    if (!wide) return waves[i];
    const float4* f = reinterpret_cast<const float4*>(waves) + 2ull * i;
    const float4 a = __ldg(f), b = __ldg(f + 1);
    return wt_wave{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
}

__device__ __forceinline__ bool wave_ok(const wt_wave& w) {
    bool lam_ok = (w.wavelength > 0.0f) && !isnan(w.wavelength);  // +inf allowed (k = 0)
    return lam_ok && finitef(w.amplitude) && finitef(w.dir_x) && finitef(w.dir_z) &&
           finitef(w.steepness_q) && finitef(w.speed) && finitef(w.phase);
}

__device__ __forceinline__ bool patch_ok(const wt_patch& P, uint32_t n_waves, uint64_t out_capacity) {
    const uint64_t verts = (uint64_t)P.cols * P.rows;
    return P.cols >= 2 && P.rows >= 2 && P.cols <= (1u << 20) && P.rows <= (1u << 20) && verts < (1ull << 31) &&
           P.flags == 0 && (uint64_t)P.wave_offset + P.wave_count <= n_waves && P.out_offset <= out_capacity &&
           verts <= out_capacity - P.out_offset && finitef(P.bl[0]) && finitef(P.bl[1]) && finitef(P.br[0]) &&
           finitef(P.br[1]) && finitef(P.tl[0]) && finitef(P.tl[1]) && finitef(P.tr[0]) && finitef(P.tr[1]) &&
           (__double2hiint(P.time_s) & 0x7ff00000) != 0x7ff00000 && finitef(P.y_offset);
}

// turns mod 1 as 64-bit fixed point
__device__ __forceinline__ unsigned long long to_fixed_turns(double turns) {
    return __double2ull_rz((turns - floor(turns)) * 18446744073709551616.0);
}

// positive remainder of x by m (FP64)
__device__ __forceinline__ double pmod(double x, double m) {
    double r = x - m * floor(x / m);
    return r >= m ? r - m : (r < 0.0 ? r + m : r);
}

__device__ __forceinline__ double inv_wavelength(const wt_wave& w) {  // k / 2pi
    const double lam = w.wavelength;
    return isinf(lam) ? 0.0 : 1.0 / lam;
}

// theta / 2pi of wave w at (col, row) of patch Pt is t00 + col*ta + row*tb +
// col*row*tg; which = 0..3 gives that constant, in turns mod 1.  (Fused
// multiply-adds spelt out: every kernel forms the same bits.)
__device__ __forceinline__ unsigned long long phase_turns(int which, const wt_patch& Pt, const wt_wave& w) {
    const double inv_lam = inv_wavelength(w);
    const double Dx = w.dir_x, Dz = w.dir_z;
    const double blx = Pt.bl[0], blz = Pt.bl[1];
    double t;
    if (which == 0) {
        t = fma((double)w.phase, 1.0 / kTwoPi,
                fma(fma(Dx, blx, Dz * blz), inv_lam, __dmul_rn(__dmul_rn((double)w.speed, Pt.time_s), inv_lam)));
    } else {
        double ex, ez, inv;
        if (which == 1) {
            ex = (double)Pt.br[0] - blx;
            ez = (double)Pt.br[1] - blz;
            inv = 1.0 / (double)(Pt.cols - 1);
        } else if (which == 2) {
            ex = (double)Pt.tl[0] - blx;
            ez = (double)Pt.tl[1] - blz;
            inv = 1.0 / (double)(Pt.rows - 1);
        } else {
            ex = (double)Pt.tr[0] - Pt.tl[0] - Pt.br[0] + blx;
            ez = (double)Pt.tr[1] - Pt.tl[1] - Pt.br[1] + blz;
            if (ex == 0.0 && ez == 0.0) return 0ull;  // a parallelogram: no cross term
            inv = __dmul_rn(1.0 / (double)(Pt.cols - 1), 1.0 / (double)(Pt.rows - 1));
        }
        t = __dmul_rn(__dmul_rn(fma(Dx, ex, __dmul_rn(Dz, ez)), inv_lam), inv);
    }
    return to_fixed_turns(t);
}

// The FP32 coefficients of the eight sums.
__device__ __forceinline__ void sum_coefs(const wt_wave& w, PairCoef& c) {
    const double k = kTwoPi * inv_wavelength(w);
    const double Dx = w.dir_x, Dz = w.dir_z, A = w.amplitude, Q = w.steepness_q;
    c.qadx = (float)(Q * A * Dx);
    c.a = (float)A;
    c.qadz = (float)(Q * A * Dz);
    c.akdx = (float)(A * k * Dx);
    c.akdz = (float)(A * k * Dz);
    c.qakxx = (float)(Q * A * k * Dx * Dx);
    c.qakxz = (float)(Q * A * k * Dx * Dz);
    c.qakzz = (float)(Q * A * k * Dz * Dz);
}

// FP64 constants of wave w on patch Pt (the phase on the patch's bilinear grid
// as 64-bit fixed-point turns, and the FP32 coefficients of the eight sums).
__device__ __forceinline__ PairCoef make_pair_coef(const wt_patch& Pt, const wt_wave& w) {
    PairCoef c;
    c.t00 = phase_turns(0, Pt, w);
    c.ta = phase_turns(1, Pt, w);
    c.tb = phase_turns(2, Pt, w);
    c.tg = phase_turns(3, Pt, w);
    sum_coefs(w, c);
    return c;
}

// Texel coordinate of the world point X on an axis of n texels:
// scale * n * X - 0.5, the BL part reduced by the wrap period in FP64.
__device__ __forceinline__ float texel_origin(const HmDev& hm, double n, double scale, double x) {
    const double period = hm.wrap == WT_WRAP_MIRRORED_REPEAT ? 2.0 * n : n;
    return (float)(pmod(scale * n * x, period) - 0.5);
}

// Per-patch constants: local frame, steps, texel origin reduced by the wrap
// period in FP64, bounce, first coefficient slot.
__device__ __forceinline__ PatchAux make_patch_aux(const wt_patch& Pt, const HmDev& hm, uint32_t pair_offset) {
    double blx = Pt.bl[0], blz = Pt.bl[1];
    PatchAux a;
    a.e1x = (float)((double)Pt.br[0] - blx);
    a.e1z = (float)((double)Pt.br[1] - blz);
    a.e2x = (float)((double)Pt.tl[0] - blx);
    a.e2z = (float)((double)Pt.tl[1] - blz);
    a.e3x = (float)((double)Pt.tr[0] - Pt.tl[0] - Pt.br[0] + blx);
    a.e3z = (float)((double)Pt.tr[1] - Pt.tl[1] - Pt.br[1] + blz);
    a.blx = Pt.bl[0];
    a.blz = Pt.bl[1];
    a.inv_cm1 = Pt.cols > 1 ? 1.0f / (float)(Pt.cols - 1) : 0.0f;
    a.inv_rm1 = Pt.rows > 1 ? 1.0f / (float)(Pt.rows - 1) : 0.0f;
    if (hm.present) {
        const double W = hm.width, H = hm.height;
        a.hu0 = texel_origin(hm, W, (double)hm.sample_scale, blx);
        a.hv0 = texel_origin(hm, H, -(double)hm.sample_scale, blz);
        a.su = (float)((double)hm.sample_scale * W);
        a.sv = (float)(-(double)hm.sample_scale * H);
    } else {
        a.hu0 = a.hv0 = a.su = a.sv = 0.0f;
    }
    a.y_offset = Pt.y_offset;
    a.pair_offset = pair_offset;
    return a;
}

}  // namespace dev
}  // namespace wt
