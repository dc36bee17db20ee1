// wt_adjoint_mma.cu — the adjoint's per-wave moments of parallelogram patches as
// matrix products on the tensor cores (wt_mma.cuh has the forward's).
//
// With g_q the adjoints of a vertex's eight sums and the phase x_i(col) + y_i(row)
// of wave i, every moment follows from
//   Z_q = sum g_q e^{i theta} = sum_row e^{i y} Y_q(row),   Y_q(row) = sum_col g_q e^{i x},
// and the same sums weighted with u = col / (cols - 1) and v = row / (rows - 1).
// The column sums are the products: for 128 columns, 8 rows and up to 64 waves
//   D[(wave, cos | sin)][row, weight, q] = sum_col E[col][wave, cos | sin] G[col][row, weight, q],
// weight = 1, u.  E is the forward's operand A as it lies in shared memory, read
// with the columns as the contracted direction; G is written by the epilogue that
// turns a vertex's sums into its adjoints.  The row sums (a paired FMA per row, q
// and weight) stay in the registers of the threads that read D, one thread per
// wave and part, over an item's rows, and end in one record per item and wave.
// A term costs 16 / 8 multiply-adds for each weight on the tensor pipe instead of
// 22 on the FMA pipe.
//
// FP16 hi + lo operands and three products, as in the forward, cross products
// first; G is scaled by powers of two, one per half tile and sum (its largest
// value to [2^13, 2^14)), so that no sum loses bits to a larger one.
//
// One block of 24 warps per SM: 0-15 vertex adjoints, 16-19 row sums, 20-21
// operands, 22 issues the products, 23 the queue and the rows' sines.  A tile is
// 16 rows (the forward's products), a half tile 8 (the adjoint's).  Every wait is
// bounded.
//
// What bounds it: issue slots (61 % busy), two thirds of them the vertex adjoints
// (about 400 instructions per 32 vertices: the normal's adjoint, the scales, 16
// values split into hi and lo); the products take 30 % of the tensor pipe,
// DRAM 19 % (dL/dpos and dL/dnrm once).  Measured, 64 patches of 64-1024 side
// with 8-64 waves, 16 M vertices, the whole call: 433 us against 1056 with the
// recurrence.  On the way: 8 vertex warps and 6 for operands 587 us; 16 and 2 of
// them, gradients loaded a half tile ahead 490; the next tile's operand B before
// this tile's sines 466; the sines in the queue's warp 445.  One scale for the
// position's three sums and one for the slopes' five cost as much as eight.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "wt_adjoint.cuh"
#include "wt_device.cuh"
#include "wt_internal.h"
#include "wt_mma.cuh"

namespace wt {
namespace {

using namespace wt::dev;
using namespace wt::mma;

constexpr uint32_t kVert = 16, kSums = 4, kProd = 2;  // warps
constexpr uint32_t kEach = 32 / kVert;                // a vertex warp's rows of a half tile
constexpr uint32_t kProd0 = kVert + kSums, kIssuer = kProd0 + kProd, kQueue = kIssuer + 1;
constexpr uint32_t kThreads = 32 * (kQueue + 1);
constexpr uint32_t kRing = 2;                   // items in flight
constexpr uint32_t kTileRows = 16, kHalf = 8;
constexpr uint32_t kOffB = 2 * kSlotA, kStageB = 2 * kTileRows * kRowB;  // the forward's operand B: two stages
constexpr uint32_t kOffG = kOffB + 2 * kStageB;  // G: [hi | lo][64 of (row, weight, q)][128 columns][128 B]
constexpr uint32_t kGroupG = 16384, kPartG = 2 * kGroupG;
constexpr uint32_t kBytes = kOffG + 2 * kPartG;
static_assert(kEach == 2 && kBytes == kOperands && kMmaAdjMaxWaves == 64, "shared memory layout");

struct Item {
    PatchAux aux;
    uint64_t out0;  // output index of (row0, column 0)
    uint64_t rec0;  // first record
    uint32_t cols, c0, row0, nrows;
    uint32_t nwaves, first;
    float4 inv[2];  // the forward sums' inverse scales
};

struct Shared {
    Table table[kRing];
    Item item[kRing];
    float2 trig[2][kTileRows][kMmaAdjMaxWaves];  // (cos y, sin y) of a tile's rows
    float4 scale[4][2];                          // 1 / G's scales of a half tile, one per sum
    uint4 top[4][2];                             // largest |g| of a half tile (bits)
    unsigned long long full[2], done[2];           // forward: operand B written / its products complete
    unsigned long long acc_full[2], acc_free[2];   // forward: a tile's sums complete / read
    unsigned long long trig_full[2], trig_free[2];
    unsigned long long top_full;                   // every vertex warp has added to `top`
    unsigned long long g_full, g_free;             // G written / its products complete
    unsigned long long d_full[2], d_free[2];       // D complete / read
    unsigned long long a_full, drained;            // an item's E written / its last product complete
    unsigned long long item_full[kRing], item_free[kRing];
    unsigned long long last;                       // all products issued are complete
    uint32_t tmem;
    int fail;
};

constexpr size_t kSmemBytes = 1024 + kBytes + sizeof(Shared);
static_assert(kSmemBytes <= 227 * 1024, "shared memory");

// The power of two that takes a largest value (its bits) to [2^13, 2^14), and its inverse.
__device__ __forceinline__ float scale_of(uint32_t top) {
    return __uint_as_float((267u << 23) - (max(top, 14u << 23) & 0x7f800000u));
}
__device__ __forceinline__ float inverse(float scale) { return __uint_as_float((254u << 23) - __float_as_uint(scale)); }

__device__ __forceinline__ float3 load_grad(const float* p, uint64_t i, bool vec3, bool wide) {
    if (wide) {
        const float4 v = __ldcs(reinterpret_cast<const float4*>(p) + i);
        return make_float3(v.x, v.y, v.z);
    }
    const float* q = p + (vec3 ? 3 : 4) * i;
    return make_float3(q[0], q[1], q[2]);
}

// wide: dL/dpos and dL/dnrm are float4 on 16-byte boundaries
template <bool SAVED>
__global__ void __launch_bounds__(kThreads, 1)
k_adjoint_mma(const wt_patch* __restrict__ patches, HmDev hm, const float* __restrict__ gpos,
              const float* __restrict__ gnrm, uint32_t flags, char* __restrict__ ws, AdjLayout L,
              const float4* __restrict__ sums, uint32_t wide, unsigned long long limit_ns) {
    cudaTriggerProgrammaticLaunchCompletion();  // the next kernel waits for this one's end
    cudaGridDependencySynchronize();
    WsHeader* hdr = reinterpret_cast<WsHeader*>(ws);
    const uint32_t n_items = hdr->mma_items;
    if (blockIdx.x >= n_items) return;
    extern __shared__ char raw[];
    char* const op = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
    Shared& sh = *reinterpret_cast<Shared*>(op + kBytes);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < 2; ++i) {
            mbar_init(&sh.full[i], kProd);
            mbar_init(&sh.done[i], 1);
            mbar_init(&sh.acc_full[i], 1);
            mbar_init(&sh.acc_free[i], kVert);
            mbar_init(&sh.trig_full[i], 1);
            mbar_init(&sh.trig_free[i], kSums);
            mbar_init(&sh.d_full[i], 1);
            mbar_init(&sh.d_free[i], kSums);
        }
        mbar_init(&sh.top_full, kVert);
        mbar_init(&sh.g_full, kVert);
        mbar_init(&sh.g_free, 1);
        mbar_init(&sh.a_full, kProd);
        mbar_init(&sh.drained, 1);
        for (uint32_t i = 0; i < kRing; ++i) {
            mbar_init(&sh.item_full[i], 1);
            mbar_init(&sh.item_free[i], kVert + kSums + kProd + 1);
        }
        for (uint32_t i = 0; i < 8; ++i) (&sh.top[0][0])[i] = make_uint4(0, 0, 0, 0);
        mbar_init(&sh.last, 1);
        sh.fail = limit_ns == 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kQueue) tmem_alloc(&sh.tmem);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sh.tmem;          // columns 0-127 and 128-255: the forward's sums; 256-383, 384-511: D
    const uint32_t op_s = smem_u32(op);
    const Limit limit{&sh.fail, limit_ns};

    if (warp == kQueue) {
        // ---- the queue: items and their wave tables; the sines of an item's rows
        const uint32_t* sorted = reinterpret_cast<const uint32_t*>(ws + L.f.sorted);
        const uint32_t* tile_pre = reinterpret_cast<const uint32_t*>(ws + L.f.tile_pre);
        const PatchAux* aux = reinterpret_cast<const PatchAux*>(ws + L.f.aux);
        const float4* coef = reinterpret_cast<const float4*>(ws + L.f.coef);
        const uint32_t* part_off = reinterpret_cast<const uint32_t*>(ws + L.part_off);
        const uint32_t n = hdr->n_patches, item_rows = hdr->mma_rows;
        uint32_t t = blockIdx.x, q = 0, tile = 0;
        const auto sines = [&](uint32_t slot, uint32_t from, uint32_t to) {
            const Item& it = sh.item[slot];
            const Table& T = sh.table[slot];
            const uint32_t nrows = it.nrows, nw = it.nwaves, row0 = it.row0;
            const uint32_t lanes = nw > 16u ? 32u : (nw > 8u ? 16u : 8u), each = 32u / lanes;  // of a row; rows at a time
            for (uint32_t r0 = from; r0 < min(nrows, to); r0 += kTileRows, ++tile) {
                if (tile >= 2u && !warp_wait(&sh.trig_free[tile & 1u], ((tile >> 1) - 1u) & 1u, limit)) return false;
                const uint32_t rt = min(kTileRows, nrows - r0);
                for (uint32_t w = lane & (lanes - 1u); w < nw; w += lanes) {
                    const ulonglong2 y = T.y[(w & ~31u) + ((w & 31u) >> 1) + 16u * (w & 1u)];
                    const unsigned long long step = each * y.y;
                    unsigned long long ph = y.x + (unsigned long long)(row0 + r0 + lane / lanes) * y.y;
#pragma unroll 4
                    for (uint32_t r = lane / lanes; r < rt; r += each, ph += step) {
                        float sn, cs;
                        sincos_turns((uint32_t)(ph >> 32), sn, cs);
                        sh.trig[tile & 1u][r][w] = make_float2(cs, sn);
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh.trig_full[tile & 1u]);
            }
            return true;
        };
        for (uint32_t k = 0;; ++k) {
            const uint32_t slot = k % kRing;
            uint32_t t_next = 0;
            if (t < n_items && lane == 0) t_next = atomicAdd(&hdr->mma_counter, 1u) + gridDim.x;
            // the last item's first two tiles before the next item, which is not needed
            // as early and may have to wait for its place
            if (k > 0 && !sines((k - 1u) % kRing, 0, 2u * kTileRows)) break;
            if (k >= kRing && !warp_wait(&sh.item_free[slot], (k / kRing - 1u) & 1u, limit)) break;
            Item& it = sh.item[slot];
            if (t >= n_items) {
                if (lane == 0) {
                    it.nrows = 0;
                    mbar_arrive(&sh.item_full[slot]);
                }
                if (k > 0) sines((k - 1u) % kRing, 2u * kTileRows, 0xffffffffu);
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
            for (uint32_t i = lane; i < nw; i += 32u) {
                max8(m, coef[4ull * (first + i) + 2], coef[4ull * (first + i) + 3]);
            }
            const PerSum scales = warp_scales(m);
            const uint32_t pad = (nw + 7u) & ~7u;  // zero waves up to a multiple of 8
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
                it.first = first;
                it.out0 = out + (uint64_t)r0 * cols;
                write_inverses(it.inv, scales, mean_loss(nw, false));
                it.rec0 = part_off[q] + (uint64_t)lt * nw;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.item_full[slot]);
            if (k > 0 && !sines((k - 1u) % kRing, 2u * kTileRows, 0xffffffffu)) break;
            t = __shfl_sync(0xffffffffu, t_next, 0);
        }
    } else if (warp == kIssuer) {
        // ---- the tensor core
        if (lane == 0) {
            uint32_t s = 0, tile = 0, half = 0;  // forward steps and tiles issued, half tiles
            bool ok = true;
            for (uint32_t k = 0; ok; ++k) {
                const uint32_t slot = k % kRing;
                ok = mbar_wait(&sh.item_full[slot], (k / kRing) & 1u, limit);
                if (!ok) break;
                const Item& it = sh.item[slot];
                const uint32_t nrows = it.nrows, nw = it.nwaves;
                if (nrows == 0) break;
                ok = mbar_wait(&sh.a_full, k & 1u, limit);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                // the forward's products of one tile (one accumulator: at most 64 waves)
                const auto forward = [&](uint32_t rt) {
                    if (tile >= 2u) ok = mbar_wait(&sh.acc_free[tile & 1u], ((tile >> 1) - 1u) & 1u, limit);
                    const uint32_t d = tmem + (tile & 1u) * 128u, rn = (rt + 1u) & ~1u;
                    const uint32_t idesc = (1u << 4) | (rn << 17) | ((128u / 16u) << 24);
                    for (uint32_t ch = 0; ch * kChunk < nw && ok; ++ch, ++s) {
                        ok = mbar_wait(&sh.full[s & 1u], (s >> 1) & 1u, limit);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t ks = (min(kChunk, nw - ch * kChunk) + 7u) / 8u;
                        const uint64_t ah = operand_desc(op_s + ch * kSlotA), al = operand_desc(op_s + ch * kSlotA + kSlotA / 2);
                        const uint32_t bs = op_s + kOffB + (s & 1u) * kStageB;
                        const uint64_t bh = operand_desc(bs), bl = operand_desc(bs + kStageB / 2);
                        for (uint32_t i = 0; i < ks; ++i) mma_f16(d, al + 2u * i, bh + 2u * i, idesc, (ch | i) != 0u);
                        for (uint32_t i = 0; i < ks; ++i) mma_f16(d, ah + 2u * i, bl + 2u * i, idesc, 1u);
                        for (uint32_t i = 0; i < ks; ++i) mma_f16(d, ah + 2u * i, bh + 2u * i, idesc, 1u);
                        commit(&sh.done[s & 1u]);
                    }
                    if (ok) commit(&sh.acc_full[tile & 1u]);
                    ++tile;
                };
                // the columns that exist, in steps of 16
                const uint32_t kc = (min(128u, it.cols - it.c0) + 15u) / 16u;
                const uint64_t eh = transposed_desc(op_s, kSlotA), el = transposed_desc(op_s + kSlotA / 2, kSlotA);
                const uint64_t gh = transposed_desc(op_s + kOffG, kGroupG), gl = transposed_desc(op_s + kOffG + kPartG, kGroupG);
                // fp16 operands, both read across their rows; FP32 sums; M = N = 128
                const uint32_t idesc = (1u << 4) | (1u << 15) | (1u << 16) | ((128u / 8u) << 17) | ((128u / 16u) << 24);
                if (!SAVED) forward(min(kTileRows, nrows));
                for (uint32_t r0 = 0; r0 < nrows && ok; r0 += kTileRows) {
                    if (!SAVED && r0 + kTileRows < nrows) forward(min(kTileRows, nrows - r0 - kTileRows));
                    for (uint32_t r = r0; r < min(r0 + kTileRows, nrows) && ok; r += kHalf, ++half) {
                        if (half >= 2u) ok = mbar_wait(&sh.d_free[half & 1u], ((half >> 1) - 1u) & 1u, limit);
                        const uint32_t d = tmem + 256u + (half & 1u) * 128u;
                        if (ok) ok = mbar_wait(&sh.g_full, half & 1u, limit);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        // 16 columns: 2048 bytes on; cross products first
                        for (uint32_t i = 0; i < kc; ++i) mma_f16(d, el + 128u * i, gh + 128u * i, idesc, i != 0u);
                        for (uint32_t i = 0; i < kc; ++i) mma_f16(d, eh + 128u * i, gl + 128u * i, idesc, 1u);
                        for (uint32_t i = 0; i < kc; ++i) mma_f16(d, eh + 128u * i, gh + 128u * i, idesc, 1u);
                        commit(&sh.g_free);
                        commit(&sh.d_full[half & 1u]);
                    }
                }
                commit(&sh.drained);
                mbar_arrive(&sh.item_free[slot]);
            }
            drain(&sh.last, &sh.fail);
        }
        __syncwarp();
    } else if (warp >= kProd0) {
        // ---- operands: E (which is the forward's A) and the forward's B
        uint32_t s = 0, dealt = 0;
        const uint32_t pw = warp - kProd0;
        bool ok = true;
        for (uint32_t k = 0; ok; ++k) {
            const uint32_t slot = k % kRing;
            ok = warp_wait(&sh.item_full[slot], (k / kRing) & 1u, limit);
            if (!ok) break;
            const Item& it = sh.item[slot];
            const Table& T = sh.table[slot];
            const uint32_t nrows = it.nrows, nw = it.nwaves, row0 = it.row0;
            if (nrows == 0) break;
            const auto rows_b = [&](uint32_t r0) {
                for (uint32_t w0 = 0; w0 < nw; w0 += kChunk, ++s) {
                    // the stage: its products of two steps ago are complete
                    if (s >= 2u) ok = warp_wait(&sh.done[s & 1u], ((s - 2u) >> 1) & 1u, limit);
                    if (!ok) return;
                    write_b<kTileRows>(op_s + kOffB + (s & 1u) * kStageB, T, nw, w0, row0 + r0, min(kTileRows, nrows - r0), pw, kProd,
                                       lane, dealt);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.full[s & 1u]);
                }
            };
            if (!SAVED) rows_b(0);
            // the previous item's products no longer read E
            if (ok && k > 0) ok = warp_wait(&sh.drained, (k - 1u) & 1u, limit);
            if (!ok) break;
            write_a(op, T, nw, it.c0, pw, kProd, lane);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.a_full);
            for (uint32_t r0 = kTileRows; !SAVED && r0 < nrows && ok; r0 += kTileRows) rows_b(r0);
            if (!ok) break;
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.item_free[slot]);
        }
    } else if (warp >= kVert) {
        // ---- row sums: a thread has one part (cosine or sine) of one wave
        const PairCoef* coef = reinterpret_cast<const PairCoef*>(ws + L.f.coef);
        float* partials = reinterpret_cast<float*>(ws + L.partials);
        const uint32_t quad = warp & 3u, wave = 16u * quad + (lane >> 1);
        uint32_t tile = 0, half = 0;
        bool ok = true;
        for (uint32_t k = 0; ok; ++k) {
            const uint32_t slot = k % kRing;
            ok = warp_wait(&sh.item_full[slot], (k / kRing) & 1u, limit);
            if (!ok) break;
            const Item& it = sh.item[slot];
            const uint32_t nrows = it.nrows, nw = it.nwaves, row0 = it.row0;
            if (nrows == 0) break;
            const float inv_rm1 = it.aux.inv_rm1;
            // The tensor core cuts each step's sum off towards zero: half a unit of the
            // last place (2^-24) for each of an item's steps of the leading product, of
            // a partial sum half as large as the whole on average.  The mean loss is
            // given back; without it the gradients of all cases measured were short by
            // 1.5e-7 to 3.8e-7, with it and with the recurrence by up to 1.2e-7.
            const float mean_loss = (float)((min(128u, it.cols - it.c0) + 15u) / 16u) * 0x1p-25f;
            float2 P[8], V[8], U[8];  // sums of (cos y, sin y) times Y_q, plain, times v, and of the u-weighted Y_q
#pragma unroll
            for (int i = 0; i < 8; ++i) P[i] = V[i] = U[i] = make_float2(0.0f, 0.0f);
            for (uint32_t r0 = 0; r0 < nrows && ok; r0 += kTileRows, ++tile) {
                ok = warp_wait(&sh.trig_full[tile & 1u], (tile >> 1) & 1u, limit);
                for (uint32_t r1 = r0; r1 < min(r0 + kTileRows, nrows) && ok; r1 += kHalf, ++half) {
                    ok = warp_wait(&sh.d_full[half & 1u], (half >> 1) & 1u, limit);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t at = tmem + 256u + (half & 1u) * 128u + ((32u * quad) << 16);
                    const float4 s0 = sh.scale[half & 3u][0], s1 = sh.scale[half & 3u][1];
                    float sc[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
                    for (int i = 0; i < 8; ++i) sc[i] = fmaf(sc[i], mean_loss, sc[i]);
                    const uint32_t rows = min(kHalf, nrows - r1);
#pragma unroll 1
                    for (uint32_t r = 0; r < rows; ++r) {
                        float y[8], z[8];  // plain, u-weighted
                        tmem_ld8(at + 16u * r, y);
                        tmem_ld8(at + 16u * r + 8u, z);
                        const float2 cs = sh.trig[tile & 1u][r1 - r0 + r][wave];
                        const float v = (float)(row0 + r1 + r) * inv_rm1;
                        tmem_wait(y, z);
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float p = y[i] * sc[i], w = p * v, q = z[i] * sc[i];
                            P[i] = __ffma2_rn(make_float2(p, p), cs, P[i]);
                            V[i] = __ffma2_rn(make_float2(w, w), cs, V[i]);
                            U[i] = __ffma2_rn(make_float2(q, q), cs, U[i]);
                        }
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.d_free[half & 1u]);
                }
                __syncwarp();
                if (ok && lane == 0) mbar_arrive(&sh.trig_free[tile & 1u]);
            }
            if (!ok) break;
            // sum g cos theta = (cos part, cos y) - (sin part, sin y), sum g sin
            // theta = (cos part, sin y) + (sin part, cos y): even lanes hold the
            // cosine part, the next lane the sine part
            const auto both = [&](const float2& own, float& c, float& sn) {
                const float ox = __shfl_xor_sync(0xffffffffu, own.x, 1), oy = __shfl_xor_sync(0xffffffffu, own.y, 1);
                c = own.x - oy;
                sn = own.y + ox;
            };
            float C[8], S[8], Cu[8], Su[8], Cv[8], Sv[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                both(P[i], C[i], S[i]);
                both(U[i], Cu[i], Su[i]);
                both(V[i], Cv[i], Sv[i]);
            }
            if ((lane & 1u) == 0u && wave < nw) {
                const PairCoef& c = coef[it.first + wave];
                const float kc[4] = {c.qadx, c.qadz, c.akdx, c.akdz}, ks[4] = {c.a, c.qakxx, c.qakxz, c.qakzz};
                // order of the sums: dx, dy, dz, jx, jz, sxx, sxz, szz; dx, dz, jx, jz
                // go with the cosine
                const auto phase = [&](const float (&cc)[8], const float (&ss)[8]) {
                    const float u = fmaf(ks[0], cc[1], fmaf(ks[1], cc[5], fmaf(ks[2], cc[6], ks[3] * cc[7])));
                    return u - fmaf(kc[0], ss[0], fmaf(kc[1], ss[2], fmaf(kc[2], ss[3], kc[3] * ss[4])));
                };
                const float t0 = phase(C, S), tu = phase(Cu, Su), tv = phase(Cv, Sv);
                float* r = partials + (size_t)kAdjRecord * (it.rec0 + wave);
                r[0] = C[0];
                r[1] = S[1];
                r[2] = C[2];
                r[3] = C[3];
                r[4] = C[4];
                r[5] = S[5];
                r[6] = S[6];
                r[7] = S[7];
                r[8] = t0;
                r[9] = fmaf(it.aux.e1x, tu, it.aux.e2x * tv);
                r[10] = fmaf(it.aux.e1z, tu, it.aux.e2z * tv);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&sh.item_free[slot]);
        }
    } else {
        // ---- vertex adjoints
        const bool pow2 = hm.present && (hm.width & (hm.width - 1)) == 0 && (hm.height & (hm.height - 1)) == 0;
        const bool vec3 = (flags & WT_LAYOUT_VEC3) != 0;
        const uint32_t quad = warp & 3u, group = warp >> 2, cl = 32u * quad + lane;
        const uint32_t g_at = op_s + kOffG + (cl >> 3) * 1024u + (cl & 7u) * 128u;
        uint32_t tile = 0, half = 0;
        bool ok = true;
        for (uint32_t k = 0; ok; ++k) {
            const uint32_t slot = k % kRing;
            ok = warp_wait(&sh.item_full[slot], (k / kRing) & 1u, limit);
            if (!ok) break;
            const Item& it = sh.item[slot];
            const uint32_t nrows = it.nrows, cols = it.cols, row0 = it.row0;
            if (nrows == 0) break;
            const PatchAux a = it.aux;
            const uint32_t col = it.c0 + cl;
            const float u = (float)col * a.inv_cm1;
            const float xc = (float)col * (a.e1x * a.inv_cm1), zc = (float)col * (a.e1z * a.inv_cm1);
            // the upstream gradients of the warp's vertices of a half tile, loaded while
            // the half tile before is scaled and written
            float3 gp[kEach], gn[kEach];
            const auto load_half = [&](uint32_t r1) {
#pragma unroll
                for (uint32_t i = 0; i < kEach; ++i) {
                    const uint32_t r = r1 + group + kVert / 4u * i;
                    gp[i] = gn[i] = make_float3(0.0f, 0.0f, 0.0f);
                    if (r < nrows && col < cols) {
                        const uint64_t v = it.out0 + (uint64_t)r * cols + col;
                        gp[i] = load_grad(gpos, v, vec3, wide != 0u);
                        if (gnrm) gn[i] = load_grad(gnrm, v, vec3, wide != 0u);
                    }
                }
            };
            load_half(0);
            const bool writes = it.c0 + 32u * quad < ((cols + 15u) & ~15u);  // columns past the last step of 16 are not read
            for (uint32_t r0 = 0; r0 < nrows && ok; r0 += kTileRows, ++tile) {
                if (!SAVED) {
                    ok = warp_wait(&sh.acc_full[tile & 1u], (tile >> 1) & 1u, limit);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                }
                const uint32_t acc = tmem + (tile & 1u) * 128u + ((32u * quad) << 16);
                for (uint32_t r1 = r0; r1 < min(r0 + kTileRows, nrows) && ok; r1 += kHalf, ++half) {
                    // the warp's four vertices: their sums, then in place their adjoints
                    float g[kEach][8];
                    if (SAVED) {
#pragma unroll
                        for (uint32_t i = 0; i < kEach; ++i) {
                            const uint32_t r = r1 + group + kVert / 4u * i;
                            const uint64_t v = r < nrows && col < cols ? it.out0 + (uint64_t)r * cols + col : it.out0;
                            const float4 s0 = __ldcs(sums + 2 * v), s1 = __ldcs(sums + 2 * v + 1);
                            g[i][0] = s0.x; g[i][1] = s0.y; g[i][2] = s0.z; g[i][3] = s0.w;
                            g[i][4] = s1.x; g[i][5] = s1.y; g[i][6] = s1.z; g[i][7] = s1.w;
                        }
                    } else {
#pragma unroll
                        for (uint32_t i = 0; i < kEach; ++i) tmem_ld8(acc + 8u * (r1 - r0 + group + kVert / 4u * i), g[i]);
                        tmem_wait(g[0], g[1]);
                    }
                    const float4 i0 = it.inv[0], i1 = it.inv[1];
#pragma unroll
                    for (uint32_t i = 0; i < kEach; ++i) {
                        const uint32_t r = r1 + group + kVert / 4u * i;
                        const float f[8] = {g[i][0], g[i][1], g[i][2], g[i][3], g[i][4], g[i][5], g[i][6], g[i][7]};
                        // (the forward's accumulator order: dx, dz, jx, jz, dy, sxx, sxz, szz)
                        const VertexSums sm =
                            SAVED ? VertexSums{f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7]}
                                  : scaled_sums(f, i0, i1);
                        const float vv = (float)(row0 + r) * a.inv_rm1;
                        vertex_adjoint(sm, fmaf(vv, a.e2x, xc), fmaf(vv, a.e2z, zc), a, hm, pow2, gp[i], gn[i], gnrm != nullptr,
                                       g[i]);
                        if (!(r < nrows && col < cols))
#pragma unroll
                            for (int e = 0; e < 8; ++e) g[i][e] = 0.0f;
                    }
                    load_half(r1 + kHalf);
                    if (!SAVED && (r1 + kHalf >= nrows || r1 + kHalf >= r0 + kTileRows)) {
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&sh.acc_free[tile & 1u]);
                    }
                    // each sum's largest adjoint of the half tile sets its scale
                    uint32_t mine = 0;
#pragma unroll
                    for (uint32_t e = 0; e < 8; ++e) {
                        const uint32_t b = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(fabsf(g[0][e]), fabsf(g[1][e]))));
                        if (lane == e) mine = b;
                    }
                    uint4* const top = sh.top[half & 3u];
                    if (lane < 8) atomicMax(reinterpret_cast<uint32_t*>(top) + lane, mine);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.top_full);
                    ok = warp_wait(&sh.top_full, half & 1u, limit);
                    if (!ok) break;
                    // G: the previous half tile's products no longer read it
                    if (half >= 1u) ok = warp_wait(&sh.g_free, (half - 1u) & 1u, limit);
                    if (!ok) break;
                    const uint4 t0 = top[0], t1 = top[1];
                    const float f[8] = {scale_of(t0.x), scale_of(t0.y), scale_of(t0.z), scale_of(t0.w),
                                        scale_of(t1.x), scale_of(t1.y), scale_of(t1.z), scale_of(t1.w)};
                    if (threadIdx.x == 0) {
                        sh.top[(half + 2u) & 3u][0] = sh.top[(half + 2u) & 3u][1] = make_uint4(0, 0, 0, 0);
                        sh.scale[half & 3u][0] = make_float4(inverse(f[0]), inverse(f[1]), inverse(f[2]), inverse(f[3]));
                        sh.scale[half & 3u][1] = make_float4(inverse(f[4]), inverse(f[5]), inverse(f[6]), inverse(f[7]));
                    }
                    if (writes) {
#pragma unroll
                        for (uint32_t i = 0; i < kEach; ++i) {
                            const uint32_t r = group + kVert / 4u * i;  // in the half tile: its 16 values are two 16-byte pieces
                            const uint32_t d0 = g_at + (r >> 2) * kGroupG;
#pragma unroll
                            for (uint32_t e = 0; e < 8; ++e) g[i][e] *= f[e];
#pragma unroll
                            for (uint32_t w = 0; w < 2; ++w) {
                                const float c = w ? u : 1.0f;
                                uint4 h, l;
                                split2(make_float2(g[i][0] * c, g[i][1] * c), h.x, l.x);
                                split2(make_float2(g[i][2] * c, g[i][3] * c), h.y, l.y);
                                split2(make_float2(g[i][4] * c, g[i][5] * c), h.z, l.z);
                                split2(make_float2(g[i][6] * c, g[i][7] * c), h.w, l.w);
                                const uint32_t d = d0 + ((((r & 3u) * 2u + w) ^ (cl & 7u)) << 4);
                                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(d), "r"(h.x), "r"(h.y), "r"(h.z),
                                             "r"(h.w)
                                             : "memory");
                                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(d + kPartG), "r"(l.x), "r"(l.y),
                                             "r"(l.z), "r"(l.w)
                                             : "memory");
                            }
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh.g_full);
                }
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

template <bool SAVED>
cudaError_t launch_t(const wt_patch* patches, const HmDev& hm, const float* gpos, const float* gnrm, uint32_t flags,
                     void* ws, const AdjLayout& L, const float* sums, cudaStream_t s) {
    static std::atomic<int> ready[64];  // shared-memory attribute set, per device
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    const int sms = sm_count();
    if (sms <= 0) return cudaErrorInvalidDevice;
    if (!ready[dev].load(std::memory_order_relaxed)) {
        const cudaError_t e =
            cudaFuncSetAttribute(k_adjoint_mma<SAVED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes);
        if (e != cudaSuccess) return e;
        ready[dev].store(1, std::memory_order_relaxed);
    }
    const auto on16 = [](const float* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
    const uint32_t wide = !(flags & WT_LAYOUT_VEC3) && on16(gpos) && on16(gnrm) ? 1u : 0u;
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
    return cudaLaunchKernelEx(&lc, k_adjoint_mma<SAVED>, patches, hm, gpos, gnrm, flags, static_cast<char*>(ws), L,
                              reinterpret_cast<const float4*>(sums), wide, wait_limit());
}

}  // namespace

cudaError_t launch_adjoint_mma(const wt_patch* patches, const HmDev& hm, const float* gpos, const float* gnrm,
                               uint32_t flags, void* ws, const AdjLayout& L, const float* sums, cudaStream_t s) {
    return sums ? launch_t<true>(patches, hm, gpos, gnrm, flags, ws, L, sums, s)
                : launch_t<false>(patches, hm, gpos, gnrm, flags, ws, L, nullptr, s);
}

}  // namespace wt
