// wt_forward.cuh — one tile of the forward's recurrence kernels: k_forward
// (wt_displace.cu) takes tiles of any table from a queue, k_single
// (wt_single.cu) those of a one-patch table.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "wt_device.cuh"
#include "wt_internal.h"

namespace wt {
namespace dev {

// A patch in the forward's shared-memory tile table (queue order).
struct QInfo {
    uint32_t cols, nwaves, pair_offset, p;
    uint64_t out0;
};
constexpr uint32_t kTabPatches = 1024;
// Per warp in the forward's shared memory (float4 units): the wave staging
// and, for the shared-memory epilogue, the parked sums.
__host__ __device__ constexpr int fwd_warp_f4(int epi, int smax) { return 32 * kStage + epi * smax * 2 * 32; }
__host__ __device__ constexpr size_t tab_bytes(uint32_t n) {
    return n <= kTabPatches ? sizeof(QInfo) * n + 4 * (n + 1) : 0;
}

// The tile of 32 * SMAX columns from c0 in one row (fewer at the row's end).
// coef: the patch's constants per wave; smem: the warp's part (the wave staging,
// 32 x kStage float4, then the parked sums of the tile's vertices, [j][half][lane]
// float4, conflict-free); su: the view (kModeStage).
// EPI = 0: epilogue unrolled over the lane's vertices straight from the
// accumulator registers; EPI = 1: the sums are parked in shared memory and a
// single rolled copy of the epilogue runs (smaller code, larger smem carve-out).
// MODE (FwdMode): kModeSave also stores each vertex's eight wave sums to `sums`,
// kModeStage the vertex-stage outputs of `view` (a compile-time switch: a
// run-time null test of the sums pointer in the epilogue cost 4 % of the
// kernel).
template <int SMAX, int EPI, int MODE>
__device__ __forceinline__ void forward_tile(const PairCoef* __restrict__ coef, uint32_t nwaves, uint32_t cols,
                                             uint64_t out0, uint32_t row, uint32_t c0, const PatchAux* aux,
                                             const HmDev& hm, bool pow2, bool fast, float* __restrict__ pos,
                                             float* __restrict__ nrm, uint32_t flags, uint32_t chunk,
                                             float4* __restrict__ sums, float4* smem, const float* su,
                                             const StageOut& so) {
    const int lane = threadIdx.x & 31;
    float4* const wst = smem;
    float4* const ebuf = smem + 32 * kStage;
    const uint32_t S = min((uint32_t)SMAX, (cols - c0 + 31u) / 32u);  // the row's last tile is narrower

    // the patch's constants are loaded after the wave loop (held across it
    // they would take 15 registers), except for the saving forward, which
    // spills less with them loaded here
    constexpr bool kLateAux = MODE != kModeSave;
    PatchAux a;
    if (!kLateAux) a = *aux;

    float2 acc[SMAX][4];
#pragma unroll
    for (int j = 0; j < SMAX; ++j)
#pragma unroll
        for (int m = 0; m < 4; ++m) acc[j][m] = make_float2(0.0f, 0.0f);

    for (uint32_t w0 = 0; w0 < nwaves; w0 += chunk) {
        const uint32_t nw = min(chunk, nwaves - w0);
        __syncwarp();
        if ((uint32_t)lane < nw) {
            stage_wave(coef[w0 + lane], c0, row, wst + kStage * lane);
        }
        __syncwarp();
        wave_loop_dispatch<SMAX>(S, acc, wst, nw, lane);
    }
    if (kLateAux) a = *aux;

    // grid position along the row: x(col) = col * du * (e1 + v e3) + v e2
    const float v = (float)row * a.inv_rm1;
    const float gx = (a.e1x + v * a.e3x) * a.inv_cm1, gz = (a.e1z + v * a.e3z) * a.inv_cm1;
    const float colf = (float)(c0 + lane);
    const float xb = fmaf(colf, gx, v * a.e2x), zb = fmaf(colf, gz, v * a.e2z);
    const uint64_t rowbase = out0 + (uint64_t)row * cols;
    if (EPI == 1) {
        // park the sums, then one rolled copy of the per-vertex epilogue
        // (each lane reads back only its own slots)
#pragma unroll
        for (int j = 0; j < SMAX; ++j) {
            if ((uint32_t)j < S) {
                ebuf[(2 * j) * 32 + lane] = make_float4(acc[j][0].x, acc[j][0].y, acc[j][1].x, acc[j][1].y);
                ebuf[(2 * j + 1) * 32 + lane] = make_float4(acc[j][2].x, acc[j][2].y, acc[j][3].x, acc[j][3].y);
            }
        }
#pragma unroll 1
        for (uint32_t j = 0; j < S; ++j) {
            const uint32_t col = c0 + lane + 32 * j;
            if (col < cols) {
                const float4 s0 = ebuf[(2 * j) * 32 + lane], s1 = ebuf[(2 * j + 1) * 32 + lane];
                const float xl = fmaf(32.0f * (float)j, gx, xb);
                const float zl = fmaf(32.0f * (float)j, gz, zb);
                const float2 pr[4] = {make_float2(s0.x, s0.y), make_float2(s0.z, s0.w), make_float2(s1.x, s1.y),
                                      make_float2(s1.z, s1.w)};
                if (MODE == kModePlain && fast)
                    finish_vertex<MODE, true>(sums_of(pr), xl, zl, a, hm, pow2, rowbase + col, pos, nrm, flags,
                                              sums, su, so);
                else
                    finish_vertex<MODE>(sums_of(pr), xl, zl, a, hm, pow2, rowbase + col, pos, nrm, flags, sums,
                                        su, so);
            }
        }
    } else {
        // kB vertices at a time: their texel loads are all issued before
        // the first of them is used (half the lane's vertices: 1.079 ->
        // 1.059 ms on 256 uneven patches at 8 per lane, 4 and 1 measured
        // the same; the saving and staging epilogues, with more outputs
        // live, take one at a time: more would spill)
        constexpr int kB = MODE == kModePlain ? SMAX / 2 : 1;
#pragma unroll
        for (int jb = 0; jb < SMAX; jb += kB) {
            HmTexels T[kB];
#pragma unroll
            for (int u = 0; u < kB; ++u) {
                const int j = jb + u;
                const uint32_t col = c0 + lane + 32 * j;
                T[u] = HmTexels{};
                if ((uint32_t)j < S && col < cols && hm.present) {
                    const float xd = fmaf(32.0f * j, gx, xb) + acc[j][0].x;
                    const float zd = fmaf(32.0f * j, gz, zb) + acc[j][1].x;
                    if (MODE == kModePlain && fast) T[u] = hm_fetch<true>(hm, a, xd, zd, pow2);
                    else T[u] = hm_fetch<false>(hm, a, xd, zd, pow2);
                }
            }
#pragma unroll
            for (int u = 0; u < kB; ++u) {
                const int j = jb + u;
                const uint32_t col = c0 + lane + 32 * j;
                if ((uint32_t)j < S && col < cols) {
                    const float xl = fmaf(32.0f * j, gx, xb);
                    const float zl = fmaf(32.0f * j, gz, zb);
                    finish_vertex_t<MODE>(sums_of(acc[j]), xl, zl, a, hm, T[u], rowbase + col, pos, nrm, flags,
                                          sums, su, so);
                }
            }
        }
    }
}

}  // namespace dev
}  // namespace wt
