// wt_mma.cu — the forward of the parallelogram patches of a table as matrix
// products (wt_mma.cuh), one block of 20 warps per SM:
//   warps 0-11   epilogues;
//   warps 12-17  form the operands in shared memory;
//   warp 18      issues the products and commits them;
//   warp 19      takes items from the queue and stages their wave tables, one
//                or two items ahead.
// An item is 128 columns of one patch by a run of rows (mma_item_rows).  The
// warps are coupled by barriers in shared memory only.  Every wait is bounded;
// one that runs out records WT_ERR_TIMEOUT and ends the block.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "wt_device.cuh"
#include "wt_internal.h"
#include "wt_mma.cuh"

namespace wt {
namespace {

using namespace wt::dev;
using namespace wt::mma;

constexpr uint32_t kProd = 6;  // warps that form operands
constexpr uint32_t kIssuer = kEpi + kProd, kQueue = kIssuer + 1;
constexpr uint32_t kThreads = 32 * (kQueue + 1);
constexpr uint32_t kRing = 3;  // items in flight

struct Item {
    PatchAux aux;
    uint64_t out0;  // output index of (row0, column 0)
    uint32_t cols, c0, row0, nrows;
    uint32_t nwaves;
    float4 inv[2];  // the sums' inverse scales
};

struct Shared {
    Table table[kRing];
    Item item[kRing];
    unsigned long long full[2], done[2];          // a step's operands are written / its products complete
    unsigned long long acc_full[2], acc_free[2];  // a tile's sums are complete / read
    unsigned long long item_full[kRing], item_free[kRing];
    unsigned long long last;                       // all products issued are complete
    uint32_t tmem;
    int fail;
    float view[36];
};

constexpr size_t kSmemBytes = 1024 + kOperands + sizeof(Shared);

template <int MODE, int HM>
__global__ void __launch_bounds__(kThreads, 1)
k_forward_mma(const wt_patch* __restrict__ patches, HmDev hm, float* __restrict__ pos, float* __restrict__ nrm,
              uint32_t flags, char* __restrict__ ws, WsLayout L, float4* __restrict__ sums,
              const wt_view* __restrict__ view, StageOut so, unsigned long long limit_ns) {
    cudaTriggerProgrammaticLaunchCompletion();  // the next kernel waits for this one's end
    cudaGridDependencySynchronize();
    WsHeader* hdr = reinterpret_cast<WsHeader*>(ws);
    const uint32_t n_items = hdr->mma_items;
    if (blockIdx.x >= n_items) return;
    extern __shared__ char raw[];
    char* const op = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
    Shared& sh = *reinterpret_cast<Shared*>(op + kOperands);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    if (MODE == kModeStage && threadIdx.x < 36) sh.view[threadIdx.x] = reinterpret_cast<const float*>(view)[threadIdx.x];
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < 2; ++i) {
            mbar_init(&sh.full[i], kProd);
            mbar_init(&sh.done[i], 1);
            mbar_init(&sh.acc_full[i], 1);
            mbar_init(&sh.acc_free[i], kEpi);
        }
        for (uint32_t i = 0; i < kRing; ++i) {
            mbar_init(&sh.item_full[i], 1);
            mbar_init(&sh.item_free[i], kEpi + kProd + 1);
        }
        mbar_init(&sh.last, 1);
        sh.fail = limit_ns == 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kQueue) tmem_alloc(&sh.tmem);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sh.tmem;
    const uint32_t op_s = smem_u32(op);
    const Limit limit{&sh.fail, limit_ns};

    if (warp == kQueue) {
        // ---- the queue: items and their wave tables
        const uint32_t* sorted = reinterpret_cast<const uint32_t*>(ws + L.sorted);
        const uint32_t* tile_pre = reinterpret_cast<const uint32_t*>(ws + L.tile_pre);
        const PatchAux* aux = reinterpret_cast<const PatchAux*>(ws + L.aux);
        const float4* coef = reinterpret_cast<const float4*>(ws + L.coef);
        const uint32_t n = hdr->n_patches, item_rows = hdr->mma_rows;
        uint32_t t = blockIdx.x, q = 0;
        for (uint32_t k = 0;; ++k) {
            const uint32_t slot = k % kRing;
            uint32_t t_next = 0;
            if (t < n_items && lane == 0) t_next = atomicAdd(&hdr->mma_counter, 1u) + gridDim.x;
            if (k >= kRing && !warp_wait(&sh.item_free[slot], (k / kRing - 1u) & 1u, limit)) break;
            Item& it = sh.item[slot];
            if (t >= n_items) {
                if (lane == 0) {
                    it.nrows = 0;
                    mbar_arrive(&sh.item_full[slot]);
                }
                break;
            }
            // the last q with tile_pre[q] <= t, 32 probes at a time
            uint32_t hi = n;
            while (hi - q > 1) {
                const uint32_t step = (hi - q + 31u) / 32u;
                const uint32_t at = min(q + (lane + 1u) * step, hi);
                const uint32_t c = __popc(__ballot_sync(0xffffffffu, at < hi && tile_pre[at] <= t));
                hi = min(q + (c + 1u) * step, hi);
                q += c * step;
            }
            const uint32_t p = sorted[q];
            const uint32_t lt = t - tile_pre[q];
            const uint32_t rows = patches[p].rows, cols = patches[p].cols, nw = patches[p].wave_count;
            const uint64_t out = patches[p].out_offset;
            const PatchAux& pa = aux[p];
            const uint32_t first = pa.pair_offset;
            if (lane < 16) reinterpret_cast<uint32_t*>(&it.aux)[lane] = reinterpret_cast<const uint32_t*>(&pa)[lane];
            PerSum m{};
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c)
                if (32u * c + lane < nw) {
                    max8(m, coef[4ull * (first + 32u * c + lane) + 2], coef[4ull * (first + 32u * c + lane) + 3]);
                }
            const PerSum scales = warp_scales(m);
            const uint32_t pad = min((nw + 7u) & ~7u, kMmaMaxWaves);  // zero waves up to a multiple of 8
#pragma unroll 2
            for (uint32_t i = lane; i < pad; i += 32u) {
                float4 v[4];
#pragma unroll
                for (uint32_t e = 0; e < 4; ++e)
                    v[e] = i < nw ? coef[4ull * (first + i) + e] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                table_entry(sh.table[slot], i, v, scales);
            }
            if (lane == 0) {
                // rows split evenly over the patch's items of this column block
                const uint32_t ni = (rows + item_rows - 1u) / item_rows;
                const uint32_t ct = lt / ni, ri = lt - ct * ni;
                const uint32_t r0 = (uint32_t)((uint64_t)rows * ri / ni), r1 = (uint32_t)((uint64_t)rows * (ri + 1u) / ni);
                it.cols = cols;
                it.c0 = 128u * ct;
                it.row0 = r0;
                it.nrows = r1 - r0;
                it.nwaves = nw;
                it.out0 = out + (uint64_t)r0 * cols;
                write_inverses(it.inv, scales, mean_loss(nw, nw > kOneAccWaves));
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.item_full[slot]);
            t = __shfl_sync(0xffffffffu, t_next, 0);
        }
    } else if (warp == kIssuer) {
        // ---- the tensor core
        if (lane == 0) {
            uint32_t s = 0, tile = 0;
            bool ok = true;
            for (uint32_t k = 0; ok; ++k) {
                const uint32_t slot = k % kRing;
                ok = mbar_wait(&sh.item_full[slot], (k / kRing) & 1u, limit);
                if (!ok) break;
                const Item& it = sh.item[slot];
                const uint32_t nrows = it.nrows, nw = it.nwaves, rb = tile_rows(nw);
                if (nrows == 0) break;
                for (uint32_t r0 = 0; r0 < nrows && ok; r0 += rb, ++tile) {
                    if (tile >= 2u) ok = mbar_wait(&sh.acc_free[tile & 1u], ((tile >> 1) - 1u) & 1u, limit);
                    for (uint32_t ch = 0; ch * kChunk < nw && ok; ++ch, ++s) {
                        ok = mbar_wait(&sh.full[s & 1u], (s >> 1) & 1u, limit);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        issue_step(op_s, tmem + (tile & 1u) * 256u, nw, rb, min(rb, nrows - r0), ch, s & 1u);
                        commit(&sh.done[s & 1u]);
                    }
                    if (ok) commit(&sh.acc_full[tile & 1u]);
                }
                mbar_arrive(&sh.item_free[slot]);
            }
            drain(&sh.last, &sh.fail);
        }
        __syncwarp();
    } else if (warp >= kEpi) {
        // ---- operands
        uint32_t s = 0, dealt = 0;  // steps written
        bool ok = true;
        for (uint32_t k = 0; ok; ++k) {
            const uint32_t slot = k % kRing;
            ok = warp_wait(&sh.item_full[slot], (k / kRing) & 1u, limit);
            if (!ok) break;
            const Item& it = sh.item[slot];
            const Table& T = sh.table[slot];
            const uint32_t nrows = it.nrows, nw = it.nwaves, rb = tile_rows(nw), row0 = it.row0;
            if (nrows == 0) break;
            // the previous item's products no longer read the operands
            if (s > 0) ok = warp_wait(&sh.done[(s - 1u) & 1u], ((s - 1u) >> 1) & 1u, limit);
            if (!ok) break;
            const uint32_t s0 = s;
            write_a(op, T, nw, it.c0, warp - kEpi, kProd, lane);
            for (uint32_t r0 = 0; r0 < nrows && ok; r0 += rb) {
                for (uint32_t w0 = 0; w0 < nw; w0 += kChunk, ++s) {
                    // the stage: its products of two steps ago are complete
                    if (s >= s0 + 2u) ok = warp_wait(&sh.done[s & 1u], ((s - 2u) >> 1) & 1u, limit);
                    if (!ok) break;
                    write_b(op_s, s & 1u, rb, T, nw, w0, row0 + r0, min(rb, nrows - r0), warp - kEpi, kProd, lane, dealt);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.full[s & 1u]);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.item_free[slot]);
        }
    } else {
        // ---- epilogues
        const bool pow2 = hm.present && (hm.width & (hm.width - 1)) == 0 && (hm.height & (hm.height - 1)) == 0;
        const Output o{pos, nrm, sums, sh.view, so, flags};
        uint32_t tile = 0;
        bool ok = true;
        for (uint32_t k = 0; ok; ++k) {
            const uint32_t slot = k % kRing;
            ok = warp_wait(&sh.item_full[slot], (k / kRing) & 1u, limit);
            if (!ok) break;
            const Item& it = sh.item[slot];
            const uint32_t nrows = it.nrows, rb = tile_rows(it.nwaves);
            if (nrows == 0) break;
            const PatchAux a = it.aux;
            Tile t{0, it.cols, it.c0, it.row0, it.out0, it.inv, it.nwaves > kOneAccWaves};
            for (uint32_t r0 = 0; r0 < nrows; r0 += rb, ++tile) {
                ok = warp_wait(&sh.acc_full[tile & 1u], (tile >> 1) & 1u, limit);
                if (!ok) break;
                t.acc = tmem + (tile & 1u) * 256u;
                if (t.c0 + 32u * (warp & 3u) < t.cols)
                    tile_epilogue<MODE, HM>(t, a, hm, pow2, o, warp & 3u, lane, ((warp >> 2) + tile) % (kEpi / 4u), kEpi / 4u, min(rb, nrows - r0));
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.acc_free[tile & 1u]);
                t.row0 += rb;
                t.out0 += (uint64_t)rb * t.cols;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.item_free[slot]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (sh.fail && threadIdx.x == 0) atomicCAS(&hdr->status, 0u, (uint32_t)WT_ERR_TIMEOUT);
    if (warp == kQueue) tmem_free(tmem);
}

template <int MODE, int HM>
cudaError_t launch_mma_t(const wt_patch* patches, const HmDev& hm, float* pos, float* nrm, uint32_t flags, void* ws, const WsLayout& L,
                         const FwdExtra& x, cudaStream_t s) {
    static std::atomic<int> ready[64];  // shared-memory attribute set, per device
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    const int sms = sm_count();
    if (sms <= 0) return cudaErrorInvalidDevice;
    if (!ready[dev].load(std::memory_order_relaxed)) {
        const cudaError_t e =
            cudaFuncSetAttribute(k_forward_mma<MODE, HM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
        if (e != cudaSuccess) return e;
        ready[dev].store(1, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)sms);
    lc.blockDim = dim3(kThreads);
    lc.dynamicSmemBytes = kSmemBytes;
    lc.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, k_forward_mma<MODE, HM>, patches, hm, pos, nrm, flags, static_cast<char*>(ws), L,
                              reinterpret_cast<float4*>(x.sums), x.view, x.stage, wait_limit());
}

template <int MODE>
cudaError_t launch_mma_hm(const wt_patch* patches, const HmDev& hm, float* pos, float* nrm, uint32_t flags, void* ws,
                          const WsLayout& L, const FwdExtra& x, cudaStream_t s) {
    switch (hm_kind(hm)) {
        case 0: return launch_mma_t<MODE, 0>(patches, hm, pos, nrm, flags, ws, L, x, s);
        case 1: return launch_mma_t<MODE, 1>(patches, hm, pos, nrm, flags, ws, L, x, s);
        default: return launch_mma_t<MODE, 2>(patches, hm, pos, nrm, flags, ws, L, x, s);
    }
}

}  // namespace

cudaError_t launch_forward_mma(const wt_patch* patches, const HmDev& hm, float* pos, float* nrm, uint32_t flags,
                               void* ws, const WsLayout& L, const FwdExtra& x, cudaStream_t s) {
    if (x.sums && x.view) return cudaErrorInvalidValue;
    if (x.sums) return launch_mma_hm<kModeSave>(patches, hm, pos, nrm, flags, ws, L, x, s);
    if (x.view) return launch_mma_hm<kModeStage>(patches, hm, pos, nrm, flags, ws, L, x, s);
    return launch_mma_hm<kModePlain>(patches, hm, pos, nrm, flags, ws, L, x, s);
}

}  // namespace wt
