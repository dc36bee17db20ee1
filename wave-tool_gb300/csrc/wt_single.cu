// wt_single.cu — the forward of a one-patch table in one kernel.
//
// A call on one patch (a frame's projected grid, a scene patch, a fit step) is
// short, and a prep kernel in front of it costs as much as the sums: one block
// working through FP64 latencies while the GPU idles, then a launch.  Here
// every block forms the patch's constants itself, in shared memory (at most
// kSingleWaves waves: 8 KB), its warps taking one kind of constant each so that
// the FP64 chains run side by side, and then runs its share of the row tiles,
// dealt round-robin (the tiles are alike: no queue).  The same device functions
// as the general path (wt_prep.cuh, wt_forward.cuh), so the same bits.
// Measured back to back (before: prep + forward kernels): 128^2 x 4 waves
// 14.3 -> 8.0 us, 1024^2 x 32 34.8 -> 22.5 us, projected grid + vertex stage
// 513^2 x 4 50.4 -> 32.8 us and 1024^2 x 32 with the noise layer 69.6 -> 56.5 us.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "wt_device.cuh"
#include "wt_forward.cuh"
#include "wt_internal.h"
#include "wt_prep.cuh"

namespace wt {
namespace {

using namespace wt::dev;

constexpr int kThreads = 512;
constexpr uint32_t kWarps = kThreads / 32;

struct Single {
    PairCoef coef[kSingleWaves];
    wt_wave waves[kSingleWaves];
    PatchAux aux;
    alignas(8) wt_patch patch;
    float view[36];
};

template <int EPI>
constexpr size_t smem_bytes() {
    return sizeof(float4) * kWarps * fwd_warp_f4(EPI, 8) + sizeof(Single);
}

template <int EPI, int MODE>
__global__ void __launch_bounds__(kThreads, 1)
k_single(const wt_patch* __restrict__ patches, const wt_wave* __restrict__ waves, uint32_t n_waves, HmDev hm,
         float* __restrict__ pos, float* __restrict__ nrm, uint64_t out_capacity, uint64_t coef_capacity,
         uint32_t flags, char* __restrict__ ws, uint32_t chunk, float4* __restrict__ sums,
         const wt_view* __restrict__ view, StageOut so) {
    extern __shared__ float4 smem[];
    Single& sh = *reinterpret_cast<Single*>(smem + kWarps * fwd_warp_f4(EPI, 8));
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    cudaGridDependencySynchronize();
    // the patch and every wave (the patch says which) in one round of loads
    if (tid >= kThreads - 32) {
        if (lane < sizeof(wt_patch) / 4)
            reinterpret_cast<uint32_t*>(&sh.patch)[lane] = reinterpret_cast<const uint32_t*>(patches)[lane];
    }
    for (uint32_t i = tid; i < n_waves * 8u; i += kThreads)
        reinterpret_cast<uint32_t*>(sh.waves)[i] = reinterpret_cast<const uint32_t*>(waves)[i];
    if (MODE == kModeStage && tid < 36) sh.view[tid] = reinterpret_cast<const float*>(view)[tid];
    __syncthreads();
    const wt_patch& P = sh.patch;
    const bool ok = patch_ok(P, n_waves, out_capacity);
    const uint32_t nw = ok ? P.wave_count : 0u;
    const wt_wave* const pw = sh.waves + (ok ? P.wave_offset : 0u);
    // kinds of constants, 32 waves a warp: the four phase constants, the
    // coefficients, and the patch's own
    const uint32_t tasks = 5u * ((nw + 31u) / 32u) + 1u;
    bool bad = !ok;
    for (uint32_t t = warp; t < tasks; t += kWarps) {
        if (t + 1u == tasks) {
            if (lane == 0) sh.aux = make_patch_aux(P, hm, 0);
            continue;
        }
        const uint32_t kind = t % 5u, i = t / 5u * 32u + lane;
        if (i >= nw) continue;
        const wt_wave w = pw[i];
        PairCoef& c = sh.coef[i];
        if (kind < 4u) {
            (&c.t00)[kind] = phase_turns((int)kind, P, w);
        } else {
            bad |= !wave_ok(w);
            sum_coefs(w, c);
        }
    }
    bad = __syncthreads_or(bad);
    const bool nomem = nw > coef_capacity;  // the workspace is short of wave slots: refused, as in the prep
    const uint32_t cols = P.cols, tpr = bad || nomem ? 0u : tiles_per_row(cols, 8), total = P.rows * tpr;
    if (blockIdx.x == 0 && tid == 0) {
        WsHeader* hdr = reinterpret_cast<WsHeader*>(ws);
        hdr->status = bad ? (uint32_t)WT_ERR_INVALID_ARG : (nomem ? (uint32_t)WT_ERR_NOMEM : 0u);
        hdr->bad_patch = bad ? 0u : kNoPatch;
        hdr->n_patches = 1;
        hdr->total_tiles = total;
    }
    const bool pow2 = hm.present && (hm.width & (hm.width - 1)) == 0 && (hm.height & (hm.height - 1)) == 0;
    const bool fast = pow2 && hm.wrap == WT_WRAP_REPEAT;
    const uint64_t out0 = P.out_offset;
    // a block's warps take tiles gridDim.x apart: few tiles spread over the SMs
    for (uint32_t t = blockIdx.x + gridDim.x * warp; t < total; t += gridDim.x * kWarps) {
        const uint32_t row = t / tpr, c0 = (t - row * tpr) * 256u;
        forward_tile<8, EPI, MODE>(sh.coef, nw, cols, out0, row, c0, &sh.aux, hm, pow2, fast, pos, nrm, flags, chunk,
                                   sums, smem + warp * fwd_warp_f4(EPI, 8), sh.view, so);
    }
}

template <int EPI, int MODE>
cudaError_t launch_t(const FwdConfig& cfg, const wt_patch* patches, const wt_wave* waves, uint32_t n_waves,
                     const HmDev& hm, float* pos, float* nrm, uint64_t out_capacity, uint32_t flags, void* ws,
                     const WsLayout& L, const FwdExtra& x, cudaStream_t s) {
    static std::atomic<int> ready[64];  // shared-memory attribute set, per device
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    const int sms = sm_count();
    if (sms <= 0) return cudaErrorInvalidDevice;
    if (!ready[dev].load(std::memory_order_relaxed)) {
        const cudaError_t e = cudaFuncSetAttribute(k_single<EPI, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)smem_bytes<EPI>());
        if (e != cudaSuccess) return e;
        ready[dev].store(1, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)sms);
    lc.blockDim = dim3(kThreads);
    lc.dynamicSmemBytes = smem_bytes<EPI>();
    lc.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    const uint64_t coef_cap = (L.end - L.coef) / sizeof(PairCoef);
    return cudaLaunchKernelEx(&lc, k_single<EPI, MODE>, patches, waves, n_waves, hm, pos, nrm, out_capacity, coef_cap,
                              flags, static_cast<char*>(ws), (uint32_t)cfg.chunk, reinterpret_cast<float4*>(x.sums),
                              x.view, x.stage);
}

}  // namespace

cudaError_t launch_single(const FwdConfig& cfg, const wt_patch* patches, const wt_wave* waves, uint32_t n_waves,
                          const HmDev& hm, float* pos, float* nrm, uint64_t out_capacity, uint32_t flags, void* ws,
                          const WsLayout& L, const FwdExtra& x, cudaStream_t s) {
    if (x.sums && x.view) return cudaErrorInvalidValue;
    if (x.sums)
        return launch_t<0, kModeSave>(cfg, patches, waves, n_waves, hm, pos, nrm, out_capacity, flags, ws, L, x, s);
    // (the vertex stage through the rolled epilogue: 56.5 against 57.3 us on a
    // 1024^2 frame; the plain one from registers: 22.5 against 22.7 us)
    if (x.view)
        return launch_t<1, kModeStage>(cfg, patches, waves, n_waves, hm, pos, nrm, out_capacity, flags, ws, L, x, s);
    return launch_t<0, kModePlain>(cfg, patches, waves, n_waves, hm, pos, nrm, out_capacity, flags, ws, L, x, s);
}

}  // namespace wt
