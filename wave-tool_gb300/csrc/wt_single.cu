// wt_single.cu — the forward of a one-patch table in one kernel.
//
// A call on one patch (a frame's projected grid, a scene patch, a fit step) is
// short, and a prep kernel in front of it costs as much as the sums: one block
// working through FP64 latencies while the GPU idles, then a launch.  Here
// every block forms the patch's constants itself, in shared memory (at most
// kSingleWaves waves: 8 KB), its warps taking one kind of constant each so that
// the FP64 chains run side by side, and then runs its share of the row tiles,
// dealt round-robin (the tiles are alike: no queue); or, where the patch is a
// parallelogram (mma_patch), its sums as matrix products (wt_mma.cuh) over
// runs of rows dealt in advance, with twelve warps on epilogues, three forming
// operands (all warps form the first tile's) and the last issuing.  The same
// device functions as the general path (wt_prep.cuh, wt_forward.cuh,
// wt_mma.cuh), so the same bits.
// Measured back to back (before: prep + forward kernels): 128^2 x 4 waves 14.3 -> 8.4
// us, 1024^2 x 32 34.8 -> 13.5 as products (22.5 by recurrence), 2048^2 x 128 244 ->
// 75; projected grid + vertex stage (10 us of it the grid's kernel) 513^2 x 4 49 ->
// 24.6 us and 1024^2 x 32 with the noise layer 69.7 -> 49.0.  From 64 waves on two
// million vertices the general path's launches, with six warps for the operands,
// take less (2048^2 x 128 72): the autotuner finds that.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "wt_device.cuh"
#include "wt_forward.cuh"
#include "wt_internal.h"
#include "wt_mma.cuh"
#include "wt_prep.cuh"

namespace wt {
namespace {

using namespace wt::dev;

constexpr int kThreads = 512;
constexpr uint32_t kWarps = kThreads / 32;
// the matrix products' warps: epilogues, then operands, then the issuer
constexpr uint32_t kProd = 3, kIssuer = mma::kEpi + kProd;
static_assert(kIssuer + 1 == kWarps, "warp roles");

struct Single {
    PairCoef coef[kSingleWaves];
    wt_wave waves[kSingleWaves];
    PatchAux aux;
    alignas(8) wt_patch patch;
    float view[36];
};

// What the matrix products need besides: behind Single, only in launches
// whose patch can qualify (`mma`).
struct Products {
    mma::Table table;
    unsigned long long full[2], done[2];          // a step's operands are written / its products complete
    unsigned long long acc_full[2], acc_free[2];  // a tile's sums are complete / read
    unsigned long long last;                      // all products issued are complete
    mma::PerSum scales;
    float4 inv[2];  // their inverses
    uint32_t tmem;
    int fail;
};

// Shared memory: the row tiles' staging, or, with `mma`, the operands (1024-byte
// aligned; the staging lies over them); then Single (and Products).
template <int EPI>
__host__ __device__ constexpr size_t stage_bytes() {
    return sizeof(float4) * kWarps * fwd_warp_f4(EPI, 8);
}
template <int EPI>
constexpr size_t smem_bytes(bool mma) {
    return mma ? 1024 + mma::kOperands + sizeof(Single) + sizeof(Products) : stage_bytes<EPI>() + sizeof(Single);
}
static_assert(stage_bytes<1>() <= mma::kOperands && sizeof(Single) % 16 == 0, "shared memory layout");

// Items (a column block's runs of rows) per column block for `ct` blocks over
// `grid` blocks of threads: the count, of one to four items per block of
// threads, with the least work on the fullest one, an item costing its rows and
// the forming of operand A (about 4 + N / 8 rows' time).
__device__ __forceinline__ uint32_t items_per_block(uint32_t rows, uint32_t ct, uint32_t nw, uint32_t grid) {
    uint32_t best = 1, cost = 0xffffffffu;
    for (uint32_t w = 1; w <= 4; ++w) {
        const uint32_t ni = min(max(grid * w / ct, 1u), (rows + 1u) / 2u);
        const uint32_t c = (ct * ni + grid - 1u) / grid * ((rows + ni - 1u) / ni + 4u + nw / 8u);
        if (c < cost) {
            cost = c;
            best = ni;
        }
    }
    return best;
}

// A block's items of a parallelogram patch.  Returns false when a wait ran out.
template <int MODE, int HM>
__device__ __forceinline__ bool run_products(Single& sh, Products& pr, char* op, uint32_t nw, const HmDev& hm, bool pow2,
                                             const mma::Output& o, unsigned long long limit_ns) {
    using namespace mma;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t cols = sh.patch.cols, rows = sh.patch.rows, ct = (cols + 127u) / 128u;
    const uint32_t ni = items_per_block(rows, ct, nw, gridDim.x);
    if (blockIdx.x >= ct * ni) return true;
    // the scales, a sum a warp, and the wave table
    if (warp < 8) {
        float m = 0.0f;
        for (uint32_t i = lane; i < nw; i += 32u) m = fmaxf(m, fabsf((&sh.coef[i].qadx)[warp]));
        const float scale = warp_scale(m);
        if (lane == 0) (&pr.scales.a.x)[warp] = scale;
    }
    __syncthreads();
    const float4* coef = reinterpret_cast<const float4*>(sh.coef);
    if (tid < ((nw + 7u) & ~7u)) {
        float4 v[4];
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) v[e] = tid < nw ? coef[4u * tid + e] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        table_entry(pr.table, tid, v, pr.scales);
    }
    if (tid == 0) {
        for (uint32_t i = 0; i < 2; ++i) {
            mbar_init(&pr.full[i], kProd);
            mbar_init(&pr.done[i], 1);
            mbar_init(&pr.acc_full[i], 1);
            mbar_init(&pr.acc_free[i], kEpi);
        }
        mbar_init(&pr.last, 1);
        pr.fail = limit_ns == 0;
        write_inverses(pr.inv, pr.scales, mean_loss(nw, nw > kOneAccWaves));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kWarps - 1) tmem_alloc(&pr.tmem);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = pr.tmem, op_s = smem_u32(op), rb = tile_rows(nw), chunks = (nw + kChunk - 1u) / kChunk;
    const uint32_t items = ct * ni;
    const auto first_row = [&](uint32_t ri) { return (uint32_t)((uint64_t)rows * ri / ni); };
    // the first item's A and first step, by all warps
    {
        const uint32_t cb = blockIdx.x / ni, ri = blockIdx.x - cb * ni, i0 = first_row(ri), i1 = first_row(ri + 1u);
        uint32_t dealt = 0;
        write_a(op, pr.table, nw, 128u * cb, warp, kWarps, lane);
        write_b(op_s, 0, rb, pr.table, nw, 0, i0, min(rb, i1 - i0), warp, kWarps, lane, dealt);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
    }
    const Limit limit{&pr.fail, limit_ns};
    uint32_t s = 0, tile = 0;  // steps and tiles
    bool ok = true;
    if (warp == kIssuer) {
        if (lane == 0) {
            for (uint32_t item = blockIdx.x; item < items && ok; item += gridDim.x) {
                const uint32_t ri = item % ni, i0 = first_row(ri), i1 = first_row(ri + 1u);
                for (uint32_t r0 = i0; r0 < i1 && ok; r0 += rb, ++tile) {
                    if (tile >= 2u) ok = mbar_wait(&pr.acc_free[tile & 1u], ((tile >> 1) - 1u) & 1u, limit);
                    for (uint32_t ch = 0; ch < chunks && ok; ++ch, ++s) {
                        ok = mbar_wait(&pr.full[s & 1u], (s >> 1) & 1u, limit);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        issue_step(op_s, tmem + (tile & 1u) * 256u, nw, rb, min(rb, i1 - r0), ch, s & 1u);
                        commit(&pr.done[s & 1u]);
                    }
                    if (ok) commit(&pr.acc_full[tile & 1u]);
                }
            }
            drain(&pr.last, &pr.fail);
        }
        __syncwarp();
    } else if (warp >= kEpi) {
        uint32_t dealt = 0;
        for (uint32_t item = blockIdx.x; item < items && ok; item += gridDim.x) {
            const uint32_t cb = item / ni, ri = item - cb * ni, i0 = first_row(ri), i1 = first_row(ri + 1u);
            const uint32_t s0 = s;
            if (s > 0) {
                // the previous item's products no longer read the operands
                ok = warp_wait(&pr.done[(s - 1u) & 1u], ((s - 1u) >> 1) & 1u, limit);
                if (!ok) break;
                write_a(op, pr.table, nw, 128u * cb, warp - kEpi, kProd, lane);
            }
            for (uint32_t r0 = i0; r0 < i1 && ok; r0 += rb) {
                for (uint32_t ch = 0; ch < chunks; ++ch, ++s) {
                    // the stage: its products of two steps ago are complete
                    if (s >= s0 + 2u) ok = warp_wait(&pr.done[s & 1u], ((s - 2u) >> 1) & 1u, limit);
                    if (!ok) break;
                    if (s > 0) {
                        write_b(op_s, s & 1u, rb, pr.table, nw, ch * kChunk, r0, min(rb, i1 - r0), warp - kEpi, kProd, lane,
                                dealt);
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                    }
                    if (lane == 0) mbar_arrive(&pr.full[s & 1u]);
                }
            }
        }
    } else {
        const PatchAux a = sh.aux;
        const uint32_t quad = warp & 3u;
        for (uint32_t item = blockIdx.x; item < items && ok; item += gridDim.x) {
            const uint32_t cb = item / ni, ri = item - cb * ni, i0 = first_row(ri), i1 = first_row(ri + 1u);
            Tile t{0, cols, 128u * cb, i0, sh.patch.out_offset + (uint64_t)i0 * cols, pr.inv, nw > kOneAccWaves};
            for (uint32_t r0 = i0; r0 < i1; r0 += rb, ++tile) {
                ok = warp_wait(&pr.acc_full[tile & 1u], (tile >> 1) & 1u, limit);
                if (!ok) break;
                t.acc = tmem + (tile & 1u) * 256u;
                if (t.c0 + 32u * quad < cols)
                    tile_epilogue<MODE, HM>(t, a, hm, pow2, o, quad, lane, ((warp >> 2) + tile) % (kEpi / 4u), kEpi / 4u, min(rb, i1 - r0));
                __syncwarp();
                if (lane == 0) mbar_arrive(&pr.acc_free[tile & 1u]);
                t.row0 += rb;
                t.out0 += (uint64_t)rb * cols;
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kWarps - 1) tmem_free(tmem);
    return pr.fail == 0;
}

template <int EPI, int MODE, int HM>
__global__ void __launch_bounds__(kThreads, 1)
k_single(const wt_patch* __restrict__ patches, const wt_wave* __restrict__ waves, uint32_t n_waves, HmDev hm,
         float* __restrict__ pos, float* __restrict__ nrm, uint64_t out_capacity, uint64_t coef_capacity,
         uint32_t flags, char* __restrict__ ws, uint32_t chunk, float4* __restrict__ sums,
         const wt_view* __restrict__ view, StageOut so, uint32_t mma, unsigned long long limit_ns) {
    extern __shared__ float4 raw[];
    float4* const smem = mma ? raw + ((1024u - (mma::smem_u32(raw) & 1023u)) & 1023u) / 16u : raw;
    Single& sh = *reinterpret_cast<Single*>(reinterpret_cast<char*>(smem) + (mma ? mma::kOperands : stage_bytes<EPI>()));
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    cudaGridDependencySynchronize();
    // (before the constants are formed, so well before a block can report a wait)
    WsHeader* const hdr = reinterpret_cast<WsHeader*>(ws);
    if (blockIdx.x == 0 && tid == 0) hdr->status = 0;
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
    bool bad = !ok, wild = false;
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
            wild |= !mma_wave(w);
            sum_coefs(w, c);
        }
    }
    bad = __syncthreads_or(bad);
    wild = __syncthreads_or(wild);
    const bool nomem = nw > coef_capacity;  // the workspace is short of wave slots: refused, as in the prep
    const uint32_t cols = P.cols, tpr = bad || nomem ? 0u : tiles_per_row(cols, 8), total = P.rows * tpr;
    const bool products = mma && total > 0 && !wild && mma_patch(P, kMmaMaxWaves);
    if (blockIdx.x == 0 && tid == 0) {
        if (bad || nomem) hdr->status = bad ? (uint32_t)WT_ERR_INVALID_ARG : (uint32_t)WT_ERR_NOMEM;
        hdr->bad_patch = bad ? 0u : kNoPatch;
        hdr->n_patches = 1;
        hdr->total_tiles = total;
        hdr->mma_items = products ? total : 0u;  // (the autotuner: no tile runs by the recurrence)
    }
    const bool pow2 = hm.present && (hm.width & (hm.width - 1)) == 0 && (hm.height & (hm.height - 1)) == 0;
    const bool fast = pow2 && hm.wrap == WT_WRAP_REPEAT;
    const uint64_t out0 = P.out_offset;
    if (products) {
        Products& pr = *reinterpret_cast<Products*>(&sh + 1);
        const mma::Output o{pos, nrm, sums, sh.view, so, flags};
        if (!run_products<MODE, HM>(sh, pr, reinterpret_cast<char*>(smem), nw, hm, pow2, o, limit_ns) && tid == 0)
            atomicCAS(&hdr->status, 0u, (uint32_t)WT_ERR_TIMEOUT);
        return;
    }
    // a block's warps take tiles gridDim.x apart: few tiles spread over the SMs
    for (uint32_t t = blockIdx.x + gridDim.x * warp; t < total; t += gridDim.x * kWarps) {
        const uint32_t row = t / tpr, c0 = (t - row * tpr) * 256u;
        forward_tile<8, EPI, MODE>(sh.coef, nw, cols, out0, row, c0, &sh.aux, hm, pow2, fast, pos, nrm, flags, chunk,
                                   sums, smem + warp * fwd_warp_f4(EPI, 8), sh.view, so);
    }
}

template <int EPI, int MODE, int HM>
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
        const cudaError_t e = cudaFuncSetAttribute(k_single<EPI, MODE, HM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)smem_bytes<EPI>(true));
        if (e != cudaSuccess) return e;
        ready[dev].store(1, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)sms);
    lc.blockDim = dim3(kThreads);
    const bool mma = n_waves >= kMmaMinWaves;  // fewer: the patch cannot qualify
    lc.dynamicSmemBytes = smem_bytes<EPI>(mma);
    lc.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    const uint64_t coef_cap = (L.end - L.coef) / sizeof(PairCoef);
    return cudaLaunchKernelEx(&lc, k_single<EPI, MODE, HM>, patches, waves, n_waves, hm, pos, nrm, out_capacity, coef_cap,
                              flags, static_cast<char*>(ws), (uint32_t)cfg.chunk, reinterpret_cast<float4*>(x.sums),
                              x.view, x.stage, mma ? 1u : 0u, wait_limit());
}

template <int EPI, int MODE>
cudaError_t launch_hm(const FwdConfig& cfg, const wt_patch* patches, const wt_wave* waves, uint32_t n_waves,
                      const HmDev& hm, float* pos, float* nrm, uint64_t out_capacity, uint32_t flags, void* ws,
                      const WsLayout& L, const FwdExtra& x, cudaStream_t s) {
    const auto f = hm_kind(hm) == 0   ? launch_t<EPI, MODE, 0>
                   : hm_kind(hm) == 1 ? launch_t<EPI, MODE, 1>
                                      : launch_t<EPI, MODE, 2>;
    return f(cfg, patches, waves, n_waves, hm, pos, nrm, out_capacity, flags, ws, L, x, s);
}

}  // namespace

cudaError_t launch_single(const FwdConfig& cfg, const wt_patch* patches, const wt_wave* waves, uint32_t n_waves,
                          const HmDev& hm, float* pos, float* nrm, uint64_t out_capacity, uint32_t flags, void* ws,
                          const WsLayout& L, const FwdExtra& x, cudaStream_t s) {
    if (x.sums && x.view) return cudaErrorInvalidValue;
    if (x.sums)
        return launch_hm<0, kModeSave>(cfg, patches, waves, n_waves, hm, pos, nrm, out_capacity, flags, ws, L, x, s);
    // (the vertex stage through the rolled epilogue: 56.5 against 57.3 us on a
    // 1024^2 frame; the plain one from registers: 22.5 against 22.7 us)
    if (x.view)
        return launch_hm<1, kModeStage>(cfg, patches, waves, n_waves, hm, pos, nrm, out_capacity, flags, ws, L, x, s);
    return launch_hm<0, kModePlain>(cfg, patches, waves, n_waves, hm, pos, nrm, out_capacity, flags, ws, L, x, s);
}

}  // namespace wt
