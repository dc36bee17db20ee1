// wt_displace.cu — forward Gerstner path on sm_103a.
//
// Replaces the per-vertex work of assets/shaders/water-grid.vert:114-194
// (grid bilerp :87-91, Gerstner sum :74-85, heightmap :93-111 sampled at the
// displaced point :141-144, bounce :147, normal :164-190) and the uniform
// upload of src/render-engine.cpp:1057-1110 (steepness already normalised by
// the caller, :1073).
//
// Three launches (two when the scan kernel forms the constants: small tables), and
// before or after the last one (launch_displace) the matrix products of parallelogram
// patches (wt_mma.cu) when the call has 8 waves or more; one launch for one patch (wt_single.cu).  All
// stream-ordered and graph-capturable:
//   k_prep_scan              validate patches and waves, prefix sums, LPT sort
//                            of patches by wave count, tile queue reset (one
//                            block; the constants of small tables by others)
//   k_prep_coef  (grid)      FP64 per-(patch, wave) phase constants in 64-bit
//                            fixed-point turns + FP32 sum coefficients;
//                            per-patch local frame; runs alongside the scan
//   k_forward    (persistent) one tile = one patch row segment of 32*S
//                            vertices per warp; lane l owns columns
//                            c0 + l + 32 j, j < S.  Per wave: one MUFU sincos
//                            per lane, an exact rotation to the second vertex,
//                            then the Chebyshev recurrence on the FMA pipe; 8
//                            FMAs, issued as 4 paired FP32 FMAs, accumulate
//                            displacement and the surface Jacobian.  Epilogue:
//                            heightmap bilerp + gradient, exact normal,
//                            streaming stores (and, by variant, the wave sums
//                            or the vertex stage).
#include <cuda_runtime.h>

#include <algorithm>

#include <atomic>
#include <cstdint>

#include "wt_device.cuh"
#include "wt_forward.cuh"
#include "wt_prep.cuh"
#include "wt_internal.h"

namespace wt {
namespace {

using namespace wt::dev;

constexpr uint32_t kWaveBins = 1024;     // wave counts >= 1023 share the last bin
constexpr uint32_t kSortBins = 2 * kWaveBins;  // matrix-product patches (mma_patch) above the others
constexpr uint32_t kMmaFlag = 0x80000000u;     // in the tile counts: the patch qualifies
constexpr uint32_t kWaveMaskWords = 512;  // waves validated into a shared bitmask up to 16384
constexpr uint32_t kRankSortMax = 64;


// Sort key of a patch: larger keys run first.
__device__ __forceinline__ uint32_t sort_key(uint32_t wave_count, bool mma) {
    return min(wave_count, kWaveBins - 1u) + (mma ? kWaveBins : 0u);
}

__device__ __forceinline__ void flag_error(WsHeader* h, uint32_t code, uint32_t patch) {
    atomicCAS(&h->status, 0u, code);
    atomicMin(&h->bad_patch, patch);
}

// ---- stage 1: validation, prefix sums, LPT order ---------------------------
// Tables of at most kSmallPrep patches, in one launch: the first block does the
// scans through shared memory, with two dependent global loads (the patches, then
// each pair's wave) instead of the general path's chain of global-memory scans,
// and the others form the constants.  Writes what the general path writes:
// header, pair and tile prefixes, the order, tiles, the constants and, for the
// adjoint, its queue (adj_scan_body's arrays).
constexpr uint32_t kSmallPrep = 32;

// The constants of such a table, by the blocks after the first: one kind of
// constant for 32 pairs (or the patches' own) is a task, and a block takes four at
// a time, one warp per scheduler.  An FP64 operation holds a scheduler's pipe for
// 64 cycles, so the five kinds of a pair one after another on one SM, beside the
// scans, were most of this kernel (7 patches of 106 pairs, the whole call 19.9 us, now
// 15.7).
constexpr uint32_t kSmallTasks = 4;  // per block and round
constexpr uint32_t kSmallPairs = 1u << 17;  // patches x waves (the pairs are mostly far fewer)

__device__ void prep_small_constants(const wt_patch* __restrict__ patches, uint32_t n, const wt_wave* __restrict__ waves,
                                     uint32_t n_waves, uint64_t out_capacity, uint64_t coef_capacity, char* ws,
                                     const WsLayout& L, const HmDev& hm) {
    constexpr unsigned kAll = 0xffffffffu;
    PatchAux* aux = reinterpret_cast<PatchAux*>(ws + L.aux);
    PairCoef* coef = reinterpret_cast<PairCoef*>(ws + L.coef);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (warp >= kSmallTasks) return;
    // the pairs' offsets, as the first block finds them
    uint32_t end = lane < n && patch_ok(patches[lane], n_waves, out_capacity) ? patches[lane].wave_count : 0u;
    const uint32_t count = end;
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kAll, end, o);
        if (lane >= o) end += y;
    }
    const uint32_t total = __shfl_sync(kAll, end, 31);
    if (total > coef_capacity) return;
    const bool wide = waves_wide(waves);
    const uint32_t tasks = 5u * ((total + 31u) / 32u) + 1u;
    for (uint32_t t = (blockIdx.x - 1u) * kSmallTasks + warp; t < tasks; t += (gridDim.x - 1u) * kSmallTasks) {
        if (t == 0) {
            if (lane < n) aux[lane] = make_patch_aux(patches[lane], hm, end - count);
            continue;
        }
        const uint32_t kind = (t - 1u) % 5u, P = 32u * ((t - 1u) / 5u) + lane;
        uint32_t p = 0, before = 0;  // the patch of pair P, and the pairs before it
        for (uint32_t q = 0; q < n; ++q) {
            const uint32_t e = __shfl_sync(kAll, end, q);
            if (e <= P) {
                p = q + 1u;
                before = e;
            }
        }
        if (P >= total) continue;
        const wt_patch& Pt = patches[p];
        const wt_wave w = load_wave(waves, Pt.wave_offset + (P - before), wide);
        if (kind < 4u) (&coef[P].t00)[kind] = phase_turns((int)kind, Pt, w);
        else sum_coefs(w, coef[P]);
    }
}

// Validates the waves pair by pair (where the pairs are fewer than the waves: a
// pool that the table uses a part of), four at a time: wave_of gives the wave of
// pair i and its patch, found from the last one's, and fails hears of those that
// do not pass.
template <typename WaveOf, typename Fails>
__device__ __forceinline__ void for_pairs(uint32_t total, bool wide, const wt_wave* __restrict__ waves, WaveOf wave_of,
                                          Fails fails) {
    uint32_t p = 0;
    for (uint32_t i0 = threadIdx.x; i0 < total; i0 += 4u * blockDim.x) {
        wt_wave w[4];
        uint32_t at[4];
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
            const uint32_t i = i0 + e * blockDim.x;
            if (i < total) {
                const uint32_t k = wave_of(i, p);
                w[e] = load_wave(waves, k, wide);
            }
            at[e] = p;
        }
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
            if (i0 + e * blockDim.x >= total) continue;
            const bool good = wave_ok(w[e]), tame = mma_wave(w[e]);
            if (!(good && tame)) fails(at[e], good, tame);
        }
    }
}

__device__ void prep_small(const wt_patch* __restrict__ patches, uint32_t n, const wt_wave* __restrict__ waves,
                           uint32_t n_waves, uint64_t out_capacity, uint64_t coef_capacity, uint32_t tile_cols,
                           char* ws, const WsLayout& L, const HmDev& hm, uint32_t mma_sms, const MmaRule& rule, int do_adj,
                           const AdjLayout& AL, uint32_t adj_chunk_max, uint32_t adj_min_tiles) {
    __shared__ wt_patch sp[kSmallPrep];
    __shared__ uint32_t s_sorted[kSmallPrep];      // patch at each sorted rank
    __shared__ uint32_t s_off[kSmallPrep + 1];     // pair prefix over the structurally valid patches
    __shared__ uint32_t s_rank_tiles[kSmallPrep];  // tiles of the patch at each sorted rank
    __shared__ uint32_t s_struct_bad, s_wave_bad;  // bit p: patch p fails that check
    __shared__ uint32_t s_wave_wild;               // bit p: a wave of patch p is no mma_wave
    __shared__ uint32_t s_choices[kItemChoices];
    WsHeader* hdr = reinterpret_cast<WsHeader*>(ws);
    uint32_t* sorted = reinterpret_cast<uint32_t*>(ws + L.sorted);
    uint32_t* tile_pre = reinterpret_cast<uint32_t*>(ws + L.tile_pre);
    uint32_t* pair_off = reinterpret_cast<uint32_t*>(ws + L.pair_off);
    uint32_t* tiles_g = reinterpret_cast<uint32_t*>(ws + L.tiles);
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    constexpr unsigned kAll = 0xffffffffu;

    if (tid < n) sp[tid] = patches[tid];
    if (tid == 0) s_wave_bad = s_wave_wild = 0;
    __syncthreads();
    uint32_t tiles_p = 0;  // warp 0: lane p's patch
    bool mma_p = false;
    if (tid < 32) {
        bool ok = false;
        uint32_t wc = 0;
        if (tid < n) {
            const wt_patch& P = sp[tid];
            ok = patch_ok(P, n_waves, out_capacity);
            wc = ok ? P.wave_count : 0u;
            tiles_p = ok ? P.rows * tiles_per_row(P.cols, tile_cols / 32) : 0u;
            mma_p = ok && mma_patch(P, rule.max_waves);
        }
        uint32_t x = wc;  // inclusive prefix of the pair counts
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kAll, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        if (tid < n) s_off[tid + 1] = x;
        if (tid == 0) s_off[0] = 0;
        const unsigned bad = __ballot_sync(kAll, tid < n && !ok);
        if (tid == 0) s_struct_bad = bad;
    }
    __syncthreads();
    const uint32_t total_pairs = s_off[n];
    const bool nomem = total_pairs > coef_capacity;
    const bool wide = waves_wide(waves);
    if (total_pairs <= max(blockDim.x, n_waves / 4u)) {
        for_pairs(total_pairs, wide, waves, [&](uint32_t i, uint32_t& p) {
            while (s_off[p + 1] <= i) ++p;
            return sp[p].wave_offset + (i - s_off[p]);
        }, [&](uint32_t p, bool good, bool tame) {
            if (!good) atomicOr(&s_wave_bad, 1u << p);
            if (!tame) atomicOr(&s_wave_wild, 1u << p);
        });
    } else {
        // each wave once (patches share them); the patches of one that fails
#pragma unroll 4
        for (uint32_t i = tid; i < n_waves; i += blockDim.x) {
            const wt_wave w = load_wave(waves, i, wide);
            const bool good = wave_ok(w), tame = mma_wave(w);
            for (uint32_t p = 0; !(good && tame) && p < n; ++p) {
                if (i - sp[p].wave_offset >= s_off[p + 1] - s_off[p]) continue;  // (none of an invalid patch's)
                if (!good) atomicOr(&s_wave_bad, 1u << p);
                if (!tame) atomicOr(&s_wave_wild, 1u << p);
            }
        }
    }
    __syncthreads();
    if (tid >= 32) return;
    const unsigned bad = s_struct_bad | s_wave_bad;
    if (tid < n && ((s_wave_bad >> tid) & 1u)) tiles_p = 0;
    mma_p = mma_p && tiles_p > 0 && !((s_wave_wild >> tid) & 1u);
    uint32_t mma_rows = 0, mma_items = 0;
    unsigned long long rowct = 0;  // rows x 128-column blocks of the matrix-product patches
    const unsigned mma_set = __ballot_sync(kAll, mma_p);
    if (mma_set) {
        const uint32_t ct = mma_p ? (sp[tid].cols + 127u) / 128u : 0u;
        const uint32_t rows = mma_p ? sp[tid].rows : 0u;
        rowct = (unsigned long long)rows * ct;
        for (int o = 16; o > 0; o >>= 1) rowct += __shfl_xor_sync(kAll, rowct, o);
        const auto count = [&](uint32_t h) { return __reduce_add_sync(kAll, ct * ((rows + h - 1u) / h)); };
        mma_rows = mma_item_rows(rowct, mma_sms, 0);
        mma_items = count(mma_rows);
        if (mma_compares(rule, rowct, mma_items, mma_sms)) {
#pragma unroll 1
            for (uint32_t k = 0; k < kItemChoices; ++k) {
                const uint32_t items = count(mma_item_rows(rowct, mma_sms, k));
                if (tid == 0) s_choices[k] = items;
            }
            __syncwarp();
            mma_rows = mma_item_rows(rowct, mma_sms, mma_item_choice(rowct, mma_sms, s_choices));
            mma_items = count(mma_rows);
        }
        if (mma_p) tiles_p = ct * ((rows + mma_rows - 1u) / mma_rows);
    }
    if (tid < n) {
        pair_off[tid] = s_off[tid];
        tiles_g[tid] = tiles_p;
    }
    bool adj_nomem = false;  // lane 0
    if (nomem) {
        // workspace too small for the wave slots: run nothing
        if (tid < n) tile_pre[tid] = 0;
        if (tid == 0) {
            tile_pre[n] = 0;
            pair_off[n] = 0;
            if (do_adj) hdr->total_chunks = 0;
        }
    } else {
        // descending wave count, ties by index (as the general path's rank sort)
        const uint32_t key = tid < n ? sort_key(sp[tid].wave_count, mma_p) : 0u;
        uint32_t rank = 0;
        for (uint32_t q = 0; q < n; ++q) {
            const uint32_t kq = __shfl_sync(kAll, key, q);
            rank += kq > key || (kq == key && q < tid);
        }
        if (tid < n) {
            sorted[rank] = tid;
            s_rank_tiles[rank] = tiles_p;
        }
        __syncwarp();
        const uint32_t tq = tid < n ? s_rank_tiles[tid] : 0u;
        uint32_t x = tq;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kAll, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        const uint32_t total_tiles = __shfl_sync(kAll, x, 31);
        if (tid < n) tile_pre[tid] = x - tq;
        if (tid == 0) {
            tile_pre[n] = total_tiles;
            pair_off[n] = total_pairs;
        }
        if (tid == 0) hdr->total_tiles = total_tiles;
        if (do_adj) {
            // the adjoint's queue: each patch's rank, its chunks of tiles and
            // the prefixes of chunks and of records (chunks x waves) over the
            // sorted order, summed in 32 bits as the general path does
            uint32_t* rank_g = reinterpret_cast<uint32_t*>(ws + AL.rank);
            uint32_t* part_off = reinterpret_cast<uint32_t*>(ws + AL.part_off);
            uint32_t* chunk_pre = reinterpret_cast<uint32_t*>(ws + AL.chunk_pre);
            if (tid < n) s_sorted[rank] = tid;
            __syncwarp();
            const uint32_t chunk = total_tiles - mma_items + rowct / 2u >= adj_min_tiles ? adj_chunk_max : 1u;
            const uint32_t each = tid < (uint32_t)__popc(mma_set) ? 1u : chunk;  // an item is a chunk
            uint32_t chunks = 0, rec = 0;
            if (tid < n) {
                const uint32_t pq = s_sorted[tid];
                chunks = (tq + each - 1) / each;
                const uint64_t r = (uint64_t)chunks * (s_off[pq + 1] - s_off[pq]);
                rec = r > 0xffffffffull ? 0xffffffffu : (uint32_t)r;
                rank_g[pq] = tid;
            }
            uint32_t xr = rec, xc = chunks;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t yr = __shfl_up_sync(kAll, xr, o), yc = __shfl_up_sync(kAll, xc, o);
                if (lane >= (uint32_t)o) {
                    xr += yr;
                    xc += yc;
                }
            }
            const uint32_t total_rec = __shfl_sync(kAll, xr, 31), total_chunks = __shfl_sync(kAll, xc, 31);
            if (tid < n) {
                part_off[tid] = xr - rec;
                chunk_pre[tid] = xc - chunks;
            }
            if (tid == 0) {
                part_off[n] = total_rec;
                chunk_pre[n] = total_chunks;
                hdr->adj_chunk = chunk;
                const bool over = (uint64_t)total_rec > AL.cap_records || total_rec == 0xffffffffu || total_tiles == 0;
                hdr->total_chunks = over ? 0u : total_chunks;
                adj_nomem = over && total_tiles != 0;
            }
        }
    }
    if (tid == 0) {
        hdr->status = bad ? (uint32_t)WT_ERR_INVALID_ARG : (nomem || adj_nomem ? (uint32_t)WT_ERR_NOMEM : 0u);
        hdr->bad_patch = bad ? (uint32_t)(__ffs(bad) - 1) : kNoPatch;
        hdr->tile_counter = nomem ? 0u : mma_items;  // the recurrence kernel's tiles follow the items
        hdr->n_patches = n;
        hdr->tile_cols = tile_cols;
        hdr->mma_items = nomem || adj_nomem ? 0u : mma_items;
        hdr->mma_rows = mma_rows;
        hdr->mma_counter = 0;
        hdr->mma_patches = (uint32_t)__popc(mma_set);
        if (nomem) hdr->total_tiles = 0;
    }
}

// Tables of 33 to kMediumPrep patches and up to 16384 waves: a thread has a
// patch, in registers, and what the threads share is in shared memory, instead of
// the general path's round trips to global memory between its steps (256 patches
// of 64-128 side, the whole call 60 us, now 49).  Writes what the general path
// writes.  The next kernel forms the constants: with 1024 pairs or fewer this
// block did, and for 64 patches sharing 16 waves that was 34 of its 41 us.
constexpr uint32_t kMediumPrep = 1024;
constexpr uint32_t kRankPrep = 512;  // ordered by ranks up to here (n^2 comparisons), by counting above

// Exclusive prefix of v over the block's 1024 threads, and the total.
__device__ __forceinline__ uint32_t block_prefix(uint32_t v, uint32_t* part, uint32_t& total) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t x = v;
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();  // the last prefix's readers are done
    if (lane == 31) part[warp] = x;
    __syncthreads();
    uint32_t w = part[lane];
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
    }
    total = __shfl_sync(0xffffffffu, w, 31);
    const uint32_t before = __shfl_sync(0xffffffffu, w, (warp + 31u) & 31u);
    return (warp > 0 ? before : 0u) + x - v;
}

// Each wave once: its bits in good_wave and tame_wave, a warp's 32 waves a word.
template <bool WIDE>
__device__ __forceinline__ void each_wave(const wt_wave* __restrict__ waves, uint32_t n_waves, uint32_t* good_wave,
                                          uint32_t* tame_wave) {
    const uint32_t round = (n_waves + 31u) & ~31u;
#pragma unroll 4
    for (uint32_t w = threadIdx.x; w < round; w += blockDim.x) {
        bool good = false, tame = false;
        if (w < n_waves) {
            const wt_wave v = load_wave(waves, w, WIDE);
            good = wave_ok(v);
            tame = mma_wave(v);
        }
        const uint32_t word = __ballot_sync(0xffffffffu, good), tword = __ballot_sync(0xffffffffu, tame);
        if ((threadIdx.x & 31u) == 0) {
            good_wave[w >> 5] = word;
            tame_wave[w >> 5] = tword;
        }
    }
}

// What few tables take is out of line: the kernel runs once, from instructions
// that no earlier launch left in the cache (48 patches: 0.5 us the whole call).
__device__ __noinline__ void wave_masks(const wt_wave* __restrict__ waves, uint32_t n_waves, uint32_t* good_wave,
                                          uint32_t* tame_wave) {
    if (waves_wide(waves)) each_wave<true>(waves, n_waves, good_wave, tame_wave);
    else each_wave<false>(waves, n_waves, good_wave, tame_wave);
}

// A pool's pairs: sets a patch's bits in `fails`, 1 for a wave that is not valid, 2
// for one that is no mma_wave.
__device__ __noinline__ void medium_pairs(uint32_t total, bool wide, const wt_wave* __restrict__ waves, uint32_t n,
                                          const uint32_t* off, const uint32_t* w0, uint32_t* fails) {
    for_pairs(total, wide, waves, [&](uint32_t i, uint32_t& q) {
        uint32_t hi = n;  // the last q with off[q] <= i
        while (hi - q > 1u) {
            const uint32_t mid = (q + hi) >> 1;
            if (off[mid] <= i) q = mid; else hi = mid;
        }
        return w0[q] + (i - off[q]);
    }, [&](uint32_t q, bool good, bool tame) { atomicOr(&fails[q], (good ? 0u : 1u) | (tame ? 0u : 2u)); });
}

// Rows per item, compared over the block's patches (of rows rows, 0 where it is not
// queued, in ct column blocks), and the items' count.
__device__ __noinline__ uint32_t medium_item_rows(uint64_t rowct, uint32_t sms, uint32_t rows, uint32_t ct, uint32_t* count,
                                                  uint32_t& items) {
#pragma unroll 1
    for (uint32_t k = 0; k < kItemChoices; ++k) {
        const uint32_t h = mma_item_rows(rowct, sms, k), n = __reduce_add_sync(0xffffffffu, ct * ((rows + h - 1u) / h));
        if ((threadIdx.x & 31u) == 0 && n > 0) atomicAdd(&count[k], n);
    }
    __syncthreads();
    const uint32_t k = mma_item_choice(rowct, sms, count);
    items = count[k];
    return mma_item_rows(rowct, sms, k);
}

// Ranks by counting: descending keys, ties in any order (the order only schedules).
__device__ __noinline__ void medium_count_order(uint32_t n, uint32_t key, uint32_t* bins, uint32_t* part, uint32_t* rank) {
    const uint32_t p = threadIdx.x, at = kSortBins - 1u - key;
    bins[p] = bins[p + blockDim.x] = 0;
    __syncthreads();
    if (p < n) atomicAdd(&bins[at], 1u);
    __syncthreads();
    const uint2 c = reinterpret_cast<const uint2*>(bins)[p];
    uint32_t all;
    const uint32_t first = block_prefix(c.x + c.y, part, all);
    reinterpret_cast<uint2*>(bins)[p] = make_uint2(first, first + c.x);
    __syncthreads();
    if (p < n) rank[p] = atomicAdd(&bins[at], 1u);
}

__device__ void prep_medium(const wt_patch* __restrict__ patches, uint32_t n, const wt_wave* __restrict__ waves,
                            uint32_t n_waves, uint64_t out_capacity, uint64_t coef_capacity, uint32_t tile_cols, char* ws,
                            const WsLayout& L, uint32_t mma_sms, const MmaRule& rule, int do_adj, const AdjLayout& AL,
                            uint32_t adj_chunk_max, uint32_t adj_min_tiles, uint4* s_keys, uint32_t* s_tiles,
                            uint32_t* s_rank, uint32_t* good_wave, uint32_t* tame_wave) {
    __shared__ uint32_t part[32], s_bad, s_items, s_mma, s_choices[kItemChoices];
    __shared__ unsigned long long part64[32];
    constexpr unsigned kAll = 0xffffffffu;
    WsHeader* hdr = reinterpret_cast<WsHeader*>(ws);
    uint32_t* sorted = reinterpret_cast<uint32_t*>(ws + L.sorted);
    uint32_t* tile_pre = reinterpret_cast<uint32_t*>(ws + L.tile_pre);
    uint32_t* pair_off = reinterpret_cast<uint32_t*>(ws + L.pair_off);
    uint32_t* tiles_g = reinterpret_cast<uint32_t*>(ws + L.tiles);
    const uint32_t p = threadIdx.x, lane = p & 31u, warp = p >> 5;
    if (p == 0) {
        s_bad = kNoPatch;
        s_items = s_mma = 0;
    }
    if (p < kItemChoices) s_choices[p] = 0;
    if (p < n) s_rank[p] = 0;
    uint32_t count = 0, tl = 0, rows = 0, ct = 0, w0 = 0, waves_p = 0;
    bool ok = false, mma = false;
    if (p < n) {
        const wt_patch P = patches[p];
        ok = patch_ok(P, n_waves, out_capacity);
        mma = ok && mma_patch(P, rule.max_waves);
        count = ok ? P.wave_count : 0u;
        tl = ok ? P.rows * tiles_per_row(P.cols, tile_cols / 32) : 0u;
        rows = P.rows;
        ct = (P.cols + 127u) / 128u;
        w0 = P.wave_offset;
        waves_p = P.wave_count;
    }
    // The waves: each once, a warp's 32 waves a word, beside the patches' loads;
    // or, where the table has a pool of more than 32 a patch, when the pairs are
    // known, and pair by pair if they are few (a pool of 16000 waves, 33 patches of
    // 4 waves: 27 us the whole call with each wave once, 14 pair by pair).
    const bool wide = waves_wide(waves);
    const bool pool = n_waves > 32u * n;
    if (!pool && wide) each_wave<true>(waves, n_waves, good_wave, tame_wave);
    uint32_t total_pairs;
    const uint32_t off = block_prefix(count, part, total_pairs);  // (and the bits are written)
    const bool nomem = total_pairs > coef_capacity;
    const bool by_pair = pool && total_pairs <= n_waves / 4u;
    if (by_pair) {
        uint32_t *const s_w0 = reinterpret_cast<uint32_t*>(s_keys), *const s_off = s_w0 + kMediumPrep;
        if (p < n) {
            s_w0[p] = w0;
            s_off[p] = off;
            s_tiles[p] = 0;
        }
        __syncthreads();
        medium_pairs(total_pairs, wide, waves, n, s_off, s_w0, s_tiles);
        __syncthreads();
    } else if (pool || !wide) {
        wave_masks(waves, n_waves, good_wave, tame_wave);
        __syncthreads();
    }
    if (p < n) {
        pair_off[p] = off;
        bool bad = false, wild = false;
        if (by_pair) {
            bad = s_tiles[p] & 1u;
            wild = s_tiles[p] & 2u;
        } else {
            for (uint32_t w = w0, w1 = w0 + count; w < w1 && !bad;) {
                const uint32_t bit = w & 31u, take = min(32u - bit, w1 - w);
                const uint32_t want = (take == 32u ? 0xffffffffu : ((1u << take) - 1u)) << bit;
                bad = (good_wave[w >> 5] & want) != want;
                wild |= (tame_wave[w >> 5] & want) != want;
                w += take;
            }
        }
        if (bad) tl = 0;
        mma = mma && !bad && !wild;
        if (!ok || bad) atomicMin(&s_bad, p);
    }
    // the matrix-product patches' items
    unsigned long long rowct = mma ? (unsigned long long)rows * ct : 0ull;
    for (int o = 16; o > 0; o >>= 1) rowct += __shfl_xor_sync(kAll, rowct, o);
    if (lane == 0) part64[warp] = rowct;
    __syncthreads();
    rowct = part64[lane];
    for (int o = 16; o > 0; o >>= 1) rowct += __shfl_xor_sync(kAll, rowct, o);
    uint32_t item_rows = 0, n_items = 0;
    if (rowct > 0) {
        item_rows = mma_item_rows(rowct, mma_sms, 0);
        const uint32_t items = __reduce_add_sync(kAll, mma ? ct * ((rows + item_rows - 1u) / item_rows) : 0u);
        const uint32_t some = __popc(__ballot_sync(kAll, mma));
        if (lane == 0 && some > 0) {
            atomicAdd(&s_items, items);
            atomicAdd(&s_mma, some);
        }
        __syncthreads();
        n_items = s_items;
        if (mma_compares(rule, rowct, n_items, mma_sms))
            item_rows = medium_item_rows(rowct, mma_sms, mma ? rows : 0u, ct, s_choices, n_items);
        if (mma) tl = ct * ((rows + item_rows - 1u) / item_rows);
    }
    const uint32_t key = p < n ? sort_key(waves_p, mma) : 0u;
    uint32_t* const bins = reinterpret_cast<uint32_t*>(s_keys);  // kSortBins of them
    if (n <= kRankPrep) {
        // ranks: keys descending, ties by index; each patch's comparisons shared out
        // over as many threads as there are
        const uint32_t n4 = (n + 3u) / 4u;
        if (p < 4u * n4) bins[p] = key;
        __syncthreads();
        const uint32_t shares = blockDim.x / n, share = p / n, mine = p - share * n;
        if (share < shares) {
            const uint32_t k = bins[mine];
            uint32_t rank = 0;
            for (uint32_t q = share * n4 / shares; q < (share + 1u) * n4 / shares; ++q) {
                const uint4 v = s_keys[q];
                rank += v.x > k || (v.x == k && 4u * q < mine);
                rank += v.y > k || (v.y == k && 4u * q + 1u < mine);
                rank += v.z > k || (v.z == k && 4u * q + 2u < mine);
                rank += v.w > k || (v.w == k && 4u * q + 3u < mine);
            }
            atomicAdd(&s_rank[mine], rank);
        }
    } else {
        medium_count_order(n, key, bins, part, s_rank);
    }
    __syncthreads();
    if (p < n) {
        tiles_g[p] = tl;
        const uint32_t rank = s_rank[p];
        s_tiles[rank] = tl;
        if (!nomem) sorted[rank] = p;
    }
    __syncthreads();
    const uint32_t tq = p < n && !nomem ? s_tiles[p] : 0u;
    uint32_t total_tiles;
    const uint32_t before = block_prefix(tq, part, total_tiles);
    if (p < n) tile_pre[p] = before;
    if (p == 0) {
        const bool any_bad = s_bad != kNoPatch;
        const uint32_t items = nomem ? 0u : n_items;
        hdr->status = any_bad ? (uint32_t)WT_ERR_INVALID_ARG : (nomem ? (uint32_t)WT_ERR_NOMEM : 0u);
        hdr->bad_patch = s_bad;
        hdr->tile_counter = items;  // the recurrence kernel's tiles follow the items
        hdr->n_patches = n;
        hdr->tile_cols = tile_cols;
        hdr->mma_items = items;
        hdr->mma_rows = item_rows;
        hdr->mma_counter = 0;
        hdr->mma_patches = nomem ? 0u : s_mma;
        hdr->total_tiles = total_tiles;
        tile_pre[n] = total_tiles;
        // bounds every coefficient write of the next kernel
        pair_off[n] = nomem ? 0u : total_pairs;
        if (nomem && do_adj) hdr->total_chunks = 0;
    }
    if (do_adj && !nomem) {
        __syncthreads();  // sorted, tile_pre and the header are complete
        adj_scan_body(ws, AL, n, adj_chunk_max, adj_min_tiles, rowct / 2u);
    }
}

// small: a table of at most kSmallPrep patches whose constants are formed here too,
// by the blocks after the first (prep_small_constants), so that no second prep
// kernel runs.
__global__ void __launch_bounds__(1024) k_prep_scan(const wt_patch* __restrict__ patches, uint32_t n,
                                                    const wt_wave* __restrict__ waves, uint32_t n_waves,
                                                    uint64_t out_capacity, uint64_t coef_capacity,
                                                    uint32_t tile_cols, char* ws, WsLayout L, HmDev hm,
                                                    int small, uint32_t mma_sms, MmaRule rule, int do_adj,
                                                    AdjLayout AL,
                                                    uint32_t adj_chunk_max, uint32_t adj_min_tiles) {
#if __CUDA_ARCH__ >= 900
    // the coefficient kernel does not read what this one writes (it forms its
    // own offsets and waits for this grid before it completes): let it start
    // (with the constants formed here the next kernel is the forward, which
    // waits at its start anyway)
    if (!small) cudaTriggerProgrammaticLaunchCompletion();
#endif
    if (blockIdx.x > 0) {
        prep_small_constants(patches, n, waves, n_waves, out_capacity, coef_capacity, ws, L, hm);
        return;
    }
    if (small) {
        prep_small(patches, n, waves, n_waves, out_capacity, coef_capacity, tile_cols, ws, L, hm, mma_sms, rule, do_adj, AL,
                   adj_chunk_max, adj_min_tiles);
        return;
    }
    WsHeader* hdr = reinterpret_cast<WsHeader*>(ws);
    uint32_t* sorted = reinterpret_cast<uint32_t*>(ws + L.sorted);
    uint32_t* tile_pre = reinterpret_cast<uint32_t*>(ws + L.tile_pre);
    uint32_t* pair_off = reinterpret_cast<uint32_t*>(ws + L.pair_off);
    uint32_t* tiles = reinterpret_cast<uint32_t*>(ws + L.tiles);
    __shared__ __align__(16) uint32_t bins[kSortBins];
    constexpr uint32_t kScanSmemOffsets = 4096;
    __shared__ uint32_t off_s[kScanSmemOffsets];
    __shared__ uint32_t good_wave[kWaveMaskWords];  // bit w: wave w passes wave_ok
    __shared__ uint32_t tame_wave[kWaveMaskWords];  // bit w: wave w is an mma_wave
    __shared__ unsigned long long s_rowct;          // rows x 128-column blocks of the matrix-product patches
    __shared__ uint32_t s_mma_n, s_choices[kItemChoices + 1];

    if (n <= kMediumPrep && n_waves <= 32u * kWaveMaskWords) {
        prep_medium(patches, n, waves, n_waves, out_capacity, coef_capacity, tile_cols, ws, L, mma_sms, rule, do_adj, AL,
                    adj_chunk_max, adj_min_tiles, reinterpret_cast<uint4*>(bins), off_s, off_s + kMediumPrep, good_wave,
                    tame_wave);
        return;
    }
    if (threadIdx.x == 0) {
        hdr->status = 0;
        hdr->bad_patch = kNoPatch;
        hdr->tile_counter = 0;
        hdr->n_patches = n;
        hdr->tile_cols = tile_cols;
        hdr->mma_items = 0;
        hdr->mma_counter = 0;
        hdr->mma_patches = 0;
        s_rowct = 0;
        s_mma_n = 0;
    }
    if (threadIdx.x <= kItemChoices) s_choices[threadIdx.x] = 0;
    // up to kRankSortMax patches are ordered by rank (their keys in bins[]),
    // more by a counting sort over the bins
    const bool rank_sort = n <= kRankSortMax;
    if (!rank_sort)
        for (uint32_t i = threadIdx.x; i < kSortBins; i += blockDim.x) bins[i] = 0;
    __syncthreads();

    // structural validation; pair_off <- wave counts of the patches that pass
    const auto row_blocks = [](const wt_patch& P) { return (unsigned long long)P.rows * ((P.cols + 127u) / 128u); };
    {
        unsigned long long rowct = 0;
        for (uint32_t p = threadIdx.x; p < n; p += blockDim.x) {
            const wt_patch P = patches[p];
            const bool ok = patch_ok(P, n_waves, out_capacity), mma = ok && mma_patch(P, rule.max_waves);
            if (!ok) flag_error(hdr, WT_ERR_INVALID_ARG, p);
            pair_off[p] = ok ? P.wave_count : 0u;
            tiles[p] = ok ? P.rows * tiles_per_row(P.cols, tile_cols / 32) | (mma ? kMmaFlag : 0u) : 0u;
            if (mma) rowct += row_blocks(P);
        }
        for (int o = 16; o > 0; o >>= 1) rowct += __shfl_xor_sync(0xffffffffu, rowct, o);
        // one a warp: a 64-bit sum in shared memory is a loop of compare-and-swaps
        if ((threadIdx.x & 31u) == 0 && rowct > 0) atomicAdd(&s_rowct, rowct);
    }
    __syncthreads();
    // a patch that turns out not to qualify (keep: what stays of its tiles)
    const auto clear_tiles = [&](uint32_t p, uint32_t keep) {
        if (atomicAnd(&tiles[p], keep) & kMmaFlag) atomicAdd(&s_rowct, 0ull - row_blocks(patches[p]));
    };
    const uint32_t total_pairs = block_exclusive_scan(pair_off, n);
    if (threadIdx.x == 0) pair_off[n] = total_pairs;
    __syncthreads();
    // wave validation; a patch with a bad wave runs no tiles.  More pairs
    // than threads and up to 16384 waves: each wave once, coalesced, into a
    // shared bitmask (a warp's 32 waves are one word), then each patch tests
    // its range of bits.  Otherwise one pair per thread, the owning patch
    // found by binary search.
    const bool off_in_smem = n + 1 <= kScanSmemOffsets;
    if (off_in_smem)
        for (uint32_t i = threadIdx.x; i <= n; i += blockDim.x) off_s[i] = pair_off[i];
    const uint32_t* off = off_in_smem ? off_s : pair_off;
    const bool wide = waves_wide(waves);
    if (total_pairs > blockDim.x && n_waves <= 32u * kWaveMaskWords) {
        wave_masks(waves, n_waves, good_wave, tame_wave);
        __syncthreads();
        for (uint32_t p = threadIdx.x; p < n; p += blockDim.x) {
            if (off[p + 1] == off[p]) continue;  // invalid patch (or no waves)
            const uint32_t w0 = patches[p].wave_offset, w1 = w0 + (off[p + 1] - off[p]);
            bool bad = false, wild = false;
            for (uint32_t w = w0; w < w1 && !bad;) {
                const uint32_t bit = w & 31u, take = min(32u - bit, w1 - w);
                const uint32_t want = (take == 32u ? 0xffffffffu : ((1u << take) - 1u)) << bit;
                bad = (good_wave[w >> 5] & want) != want;
                wild |= (tame_wave[w >> 5] & want) != want;
                w += take;
            }
            if (bad) {
                flag_error(hdr, WT_ERR_INVALID_ARG, p);
                clear_tiles(p, 0u);
            } else if (wild) {
                clear_tiles(p, ~kMmaFlag);
            }
        }
    } else {
        __syncthreads();
        for (uint32_t P = threadIdx.x; P < total_pairs; P += blockDim.x) {
            uint32_t lo = 0, hi = n + 1;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (off[mid] <= P) lo = mid + 1; else hi = mid;
            }
            const uint32_t p = lo - 1;
            const wt_wave w = load_wave(waves, patches[p].wave_offset + (P - off[p]), wide);
            if (!wave_ok(w)) {
                flag_error(hdr, WT_ERR_INVALID_ARG, p);
                clear_tiles(p, 0u);
            } else if (!mma_wave(w)) {
                clear_tiles(p, ~kMmaFlag);
            }
        }
    }
    const bool nomem = total_pairs > coef_capacity;
    __syncthreads();
    if (nomem) {
        // workspace too small for the wave slots: run nothing.  pair_off[n]
        // bounds every coefficient write of the next kernel.
        if (threadIdx.x == 0) {
            atomicCAS(&hdr->status, 0u, (uint32_t)WT_ERR_NOMEM);
            hdr->total_tiles = 0;
            pair_off[n] = 0;
            if (do_adj) hdr->total_chunks = 0;
        }
        for (uint32_t p = threadIdx.x; p <= n; p += blockDim.x) tile_pre[p] = 0;
        return;
    }
    // the matrix-product patches' items, then the sort keys
    if (s_rowct > 0) {
        // the items with at most h rows, into the patches' tiles and summed
        const auto count_items = [&](uint32_t h, uint32_t* sum) {
            uint32_t items = 0, some = 0;
            for (uint32_t p = threadIdx.x; p < n; p += blockDim.x) {
                if (!(tiles[p] & kMmaFlag)) continue;
                const uint32_t it = (patches[p].cols + 127u) / 128u * ((patches[p].rows + h - 1u) / h);
                tiles[p] = it | kMmaFlag;
                items += it;
                ++some;
            }
            items = __reduce_add_sync(0xffffffffu, items);
            some = __reduce_add_sync(0xffffffffu, some);
            if ((threadIdx.x & 31u) == 0 && some > 0) {
                atomicAdd(sum, items);
                atomicAdd(&s_mma_n, some);
            }
            __syncthreads();
        };
        uint32_t k = 0;
        count_items(mma_item_rows(s_rowct, mma_sms, 0), &s_choices[0]);
        const uint32_t n_mma = s_mma_n;
        if (mma_compares(rule, s_rowct, s_choices[0], mma_sms)) {
            __syncthreads();  // every thread has read the count
#pragma unroll 1
            for (k = 1; k < kItemChoices; ++k) count_items(mma_item_rows(s_rowct, mma_sms, k), &s_choices[k]);
            k = mma_item_choice(s_rowct, mma_sms, s_choices);
            count_items(mma_item_rows(s_rowct, mma_sms, k), &s_choices[kItemChoices]);
        }
        if (threadIdx.x == 0) {
            hdr->mma_items = s_choices[k];
            hdr->mma_patches = n_mma;
            hdr->mma_rows = mma_item_rows(s_rowct, mma_sms, k);
            hdr->tile_counter = s_choices[k];  // the recurrence kernel's tiles follow the items
        }
    }
    for (uint32_t p = threadIdx.x; p < n; p += blockDim.x) {
        const uint32_t key = sort_key(off[p + 1] - off[p], tiles[p] & kMmaFlag);
        if (rank_sort) bins[p] = key;
        else atomicAdd(&bins[kSortBins - 1 - key], 1u);  // descending
    }
    __syncthreads();
    // sort by descending key, ties in any order: the order only schedules
    // tiles, results do not depend on it
    if (rank_sort) {
        for (uint32_t p = threadIdx.x; p < n; p += blockDim.x) {
            const uint32_t key = bins[p];
            uint32_t rank = 0;
            for (uint32_t q = 0; q < n; ++q) rank += bins[q] > key || (bins[q] == key && q < p);
            sorted[rank] = p;
        }
    } else {
        const uint32_t used = s_mma_n > 0 ? 0u : kSortBins - kWaveBins;  // (larger keys are matrix products')
        block_exclusive_scan(bins + used, kSortBins - used);
        __syncthreads();
        for (uint32_t p = threadIdx.x; p < n; p += blockDim.x) {
            const uint32_t key = sort_key(off[p + 1] - off[p], tiles[p] & kMmaFlag);
            sorted[atomicAdd(&bins[kSortBins - 1 - key], 1u)] = p;
        }
    }
    __syncthreads();
    for (uint32_t q = threadIdx.x; q < n; q += blockDim.x) tile_pre[q] = tiles[sorted[q]] & ~kMmaFlag;
    __syncthreads();
    const uint32_t total_tiles = block_exclusive_scan(tile_pre, n);
    if (threadIdx.x == 0) {
        tile_pre[n] = total_tiles;
        hdr->total_tiles = total_tiles;
    }
    if (do_adj) {
        __syncthreads();  // sorted, tile_pre and the header's total_tiles are complete
        adj_scan_body(ws, AL, n, adj_chunk_max, adj_min_tiles, s_rowct / 2u);
    }
}

// ---- stage 2: FP64 constants per (patch, wave) and per patch ---------------
// Up to kSmemOffsets - 1 patches each block forms the wave-count prefix of
// the structurally valid patches itself, so this kernel runs alongside the
// scan kernel and waits for it only before it completes (the forward kernel
// waits for this one); with more patches it waits first and reads the scan's
// prefix.
__global__ void __launch_bounds__(256) k_prep_coef(const wt_patch* __restrict__ patches, uint32_t n,
                                                   const wt_wave* __restrict__ waves, uint32_t n_waves,
                                                   uint64_t out_capacity, uint64_t coef_capacity, HmDev hm,
                                                   char* ws, WsLayout L) {
    const uint32_t* pair_off_g = reinterpret_cast<const uint32_t*>(ws + L.pair_off);
    PatchAux* aux = reinterpret_cast<PatchAux*>(ws + L.aux);
    PairCoef* coef = reinterpret_cast<PairCoef*>(ws + L.coef);
    constexpr uint32_t kSmemOffsets = 4096;
    __shared__ uint32_t off_s[kSmemOffsets];
    const bool own = n + 1 <= kSmemOffsets;
    uint32_t total;
    if (own) {
        for (uint32_t p = threadIdx.x; p < n; p += blockDim.x) {
            const wt_patch P = patches[p];
            off_s[p] = patch_ok(P, n_waves, out_capacity) ? P.wave_count : 0u;
        }
        __syncthreads();
        total = block_exclusive_scan(off_s, n);
        if (threadIdx.x == 0) off_s[n] = total;
        __syncthreads();
        if (total > coef_capacity) total = 0;  // the scan kernel reports the shortfall
    } else {
#if __CUDA_ARCH__ >= 900
        cudaGridDependencySynchronize();
#endif
        total = pair_off_g[n];  // 0 when the workspace is short
    }
    const uint32_t* pair_off = own ? off_s : pair_off_g;
    // One kind of constant of 32 pairs per warp task (the four phase constants,
    // the sum coefficients), and the constants of 32 patches: neighbouring tasks
    // on different SMs, so that the FP64 chains (a warp-wide operation holds the
    // pipe for about 64 cycles) run side by side.  One thread per pair doing all
    // of it in consecutive warps: 14.0 us for 48 patches of 0-40 waves, 6.5 us
    // this way.  All kinds in one task from two rounds of tasks on, since every
    // kind divides by the wavelength again (16000 pairs:
    // 13.4 us by kinds, now 10.7; 45000 pairs 25.0, now 17.2).
    const uint32_t lane = threadIdx.x & 31u, warps = gridDim.x * (blockDim.x >> 5);
    const bool wide = waves_wide(waves);
    const uint32_t groups = (total + 31u) / 32u, kinds = 5u * groups <= 8u * gridDim.x ? 5u : 1u;
    const uint32_t tasks = kinds * groups + (n + 31u) / 32u;
    for (uint32_t t = blockIdx.x + gridDim.x * (threadIdx.x >> 5); t < tasks; t += warps) {
        if (t >= kinds * groups) {
            const uint32_t p = 32u * (t - kinds * groups) + lane;
            if (p < n) aux[p] = make_patch_aux(patches[p], hm, pair_off[p]);
            continue;
        }
        const uint32_t kind = t % kinds, P = 32u * (t / kinds) + lane;
        if (P >= total) continue;
        // owning patch: last p with pair_off[p] <= P
        uint32_t lo = 0, hi = n + 1;
        while (lo < hi) {
            uint32_t mid = (lo + hi) >> 1;
            if (pair_off[mid] <= P) lo = mid + 1; else hi = mid;
        }
        const uint32_t p = lo - 1;
        const wt_patch& Pt = patches[p];
        const wt_wave w = load_wave(waves, Pt.wave_offset + (P - pair_off[p]), wide);
        if (kinds == 1u) coef[P] = make_pair_coef(Pt, w);
        else if (kind < 4u) (&coef[P].t00)[kind] = phase_turns((int)kind, Pt, w);
        else sum_coefs(w, coef[P]);
    }
#if __CUDA_ARCH__ >= 900
    // complete only after the scan kernel: whatever waits for this grid then
    // sees both (a no-op when already waited for above)
    if (own) cudaGridDependencySynchronize();
#endif
}

// ---- stage 3: the persistent forward kernel (its tile: wt_forward.cuh) ------
template <int THREADS, int MINB, int SMAX, int EPI, int MODE>
__global__ void __launch_bounds__(THREADS, MINB)
k_forward(const wt_patch* __restrict__ patches, HmDev hm, float* __restrict__ pos,
          float* __restrict__ nrm, uint32_t flags, char* __restrict__ ws, WsLayout L, uint32_t chunk,
          float4* __restrict__ sums_arg, const wt_view* __restrict__ view, StageOut so, uint32_t tab_in_smem) {
#if __CUDA_ARCH__ >= 900
    cudaGridDependencySynchronize();
#endif
    float4* const sums = MODE == kModeSave ? sums_arg : nullptr;
    // per warp: wave staging (32 x kStage float4), then the parked sums of
    // the tile's vertices ([j][half][lane] float4, conflict-free); after the
    // warps' parts, the 36 floats of the view (kModeStage)
    extern __shared__ float4 fwd_smem[];
    float4* const wbase = fwd_smem + (threadIdx.x >> 5) * fwd_warp_f4(EPI, SMAX);
    float* const su = reinterpret_cast<float*>(fwd_smem + (THREADS / 32) * fwd_warp_f4(EPI, SMAX));
    if (MODE == kModeStage) {
        if (threadIdx.x < 36) su[threadIdx.x] = reinterpret_cast<const float*>(view)[threadIdx.x];
        __syncthreads();
    }
    WsHeader* hdr = reinterpret_cast<WsHeader*>(ws);
    const uint32_t* sorted = reinterpret_cast<const uint32_t*>(ws + L.sorted);
    const uint32_t* tile_pre = reinterpret_cast<const uint32_t*>(ws + L.tile_pre);
    const PatchAux* aux = reinterpret_cast<const PatchAux*>(ws + L.aux);
    const PairCoef* coef = reinterpret_cast<const PairCoef*>(ws + L.coef);
    const int lane = threadIdx.x & 31;
    const uint32_t n = hdr->n_patches;
    const uint32_t total = hdr->total_tiles;
    const bool pow2 = hm.present && (hm.width & (hm.width - 1)) == 0 && (hm.height & (hm.height - 1)) == 0;
    // the plain epilogue's mask-only texel wrap (the other modes keep one
    // general copy of the epilogue: two would spill their extra outputs)
    const bool fast = pow2 && hm.wrap == WT_WRAP_REPEAT;

    // The tile table: with at most kTabPatches patches each block copies, in
    // queue (sorted) order, the tile prefix and each patch's columns, wave
    // count, first coefficient slot and output offset into shared memory,
    // so a tile's look-up reads no global memory (1.0594 -> 1.0547 ms on 256
    // uneven patches at 8 vertices per lane, 1.0777 -> 1.0680 at 4).
    QInfo* const tab = reinterpret_cast<QInfo*>(su + (MODE == kModeStage ? 36 : 0));
    uint32_t* const tab_pre = reinterpret_cast<uint32_t*>(tab + (tab_in_smem ? n : 0));
    // nothing to run: a table the prep refused (no order to copy), or one whose
    // patches all ran as matrix products
    if (total <= hdr->mma_items) return;
    if (tab_in_smem) {
        for (uint32_t qq = threadIdx.x; qq < n; qq += THREADS) {
            const uint32_t pp = sorted[qq];
            tab[qq] = QInfo{patches[pp].cols, patches[pp].wave_count, aux[pp].pair_offset, pp,
                            patches[pp].out_offset};
        }
        for (uint32_t qq = threadIdx.x; qq <= n; qq += THREADS) tab_pre[qq] = tile_pre[qq];
        __syncthreads();
    }
    const bool ts = tab_in_smem != 0;
    const uint32_t* const tpre = ts ? tab_pre : tile_pre;

    // The queue index of the next tile is fetched while the current one runs;
    // the tile's patch is searched forward from the previous tile's (tiles
    // come out of the queue in increasing order), galloping when it is far.
    uint32_t t_a = 0;
    if (lane == 0) t_a = atomicAdd(&hdr->tile_counter, 1u);
    uint32_t t = __shfl_sync(0xffffffffu, t_a, 0);
    uint32_t q = 0;
    while (t < total) {
        if (lane == 0) t_a = atomicAdd(&hdr->tile_counter, 1u);
        if (tpre[q + 1] <= t) {
            uint32_t step = 1, lo = q + 1, hi = q + 2;
            while (hi <= n && tpre[hi] <= t) { lo = hi; step <<= 1; hi = lo + step; }
            hi = min(hi, n + 1);
            while (hi - lo > 1) {  // tile_pre[lo] <= t < tile_pre[hi]
                const uint32_t mid = (lo + hi) >> 1;
                if (tpre[mid] <= t) lo = mid; else hi = mid;
            }
            q = lo;
        }
        uint32_t p, cols, nwaves, pair_offset;
        uint64_t out0;
        if (ts) {
            const QInfo e = tab[q];
            p = e.p;
            cols = e.cols;
            nwaves = e.nwaves;
            pair_offset = e.pair_offset;
            out0 = e.out0;
        } else {
            p = sorted[q];
            cols = patches[p].cols;
            nwaves = patches[p].wave_count;
            out0 = patches[p].out_offset;
            pair_offset = aux[p].pair_offset;
        }
        const uint32_t lt = t - tpre[q];
        const uint32_t tpr = tiles_per_row(cols, SMAX);
        const uint32_t row = lt / tpr;
        const uint32_t c0 = (lt - row * tpr) * 32u * SMAX;
        forward_tile<SMAX, EPI, MODE>(coef + pair_offset, nwaves, cols, out0, row, c0, aux + p, hm, pow2, fast, pos,
                                      nrm, flags, chunk, sums, wbase, su, so);
        t = __shfl_sync(0xffffffffu, t_a, 0);
    }
}

// ---- FP32-naive phase (precision studies only) -----------------------------
// The reference's arithmetic: theta = w*dot(D, xz) + phi*t in FP32 with world
// xz (water-grid.vert:78), accurate sinf/cosf so that only the phase
// representation differs from the default path.
__global__ void __launch_bounds__(256) k_forward_naive(const wt_patch* __restrict__ patches, uint32_t n,
                                                       const wt_wave* __restrict__ waves, HmDev hm,
                                                       float* __restrict__ pos, float* __restrict__ nrm,
                                                       uint32_t flags, const char* __restrict__ ws, WsLayout L) {
    const PatchAux* aux = reinterpret_cast<const PatchAux*>(ws + L.aux);
    const uint32_t* tile_pre = reinterpret_cast<const uint32_t*>(ws + L.tile_pre);
    const uint32_t* sorted = reinterpret_cast<const uint32_t*>(ws + L.sorted);
    const bool pow2 = hm.present && (hm.width & (hm.width - 1)) == 0 && (hm.height & (hm.height - 1)) == 0;
    for (uint32_t q = 0; q < n; ++q) {
        if (tile_pre[q + 1] == tile_pre[q]) continue;  // invalid patch
        const uint32_t p = sorted[q];
        const wt_patch P = patches[p];
        const PatchAux a = aux[p];
        const uint64_t nv = (uint64_t)P.cols * P.rows;
        const float t = (float)P.time_s;
        for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < nv;
             v += (uint64_t)gridDim.x * blockDim.x) {
            uint32_t row = (uint32_t)(v / P.cols), col = (uint32_t)(v - (uint64_t)row * P.cols);
            float u = (float)col * a.inv_cm1, vv = (float)row * a.inv_rm1, uv = u * vv;
            float xl = fmaf(u, a.e1x, fmaf(vv, a.e2x, uv * a.e3x));
            float zl = fmaf(u, a.e1z, fmaf(vv, a.e2z, uv * a.e3z));
            float xw = a.blx + xl, zw = a.blz + zl;
            VertexSums s{0, 0, 0, 0, 0, 0, 0, 0};
            for (uint32_t i = 0; i < P.wave_count; ++i) {
                const wt_wave w = waves[P.wave_offset + i];
                float k = isinf(w.wavelength) ? 0.0f : (float)(kTwoPi / (double)w.wavelength);
                float phi = w.speed * k;
                float th = k * (w.dir_x * xw + w.dir_z * zw) + phi * t + w.phase;
                float sn, c;
                sincosf(th, &sn, &c);
                float A = w.amplitude, Q = w.steepness_q;
                s.dx += Q * A * w.dir_x * c; s.dy += A * sn; s.dz += Q * A * w.dir_z * c;
                s.jx += A * k * w.dir_x * c; s.jz += A * k * w.dir_z * c;
                s.sxx += Q * A * k * w.dir_x * w.dir_x * sn;
                s.sxz += Q * A * k * w.dir_x * w.dir_z * sn;
                s.szz += Q * A * k * w.dir_z * w.dir_z * sn;
            }
            finish_vertex<kModePlain>(s, xl, zl, a, hm, pow2, P.out_offset + v, pos, nrm, flags, nullptr, nullptr,
                                  StageOut{});
        }
    }
}

template <int THREADS, int MINB, int SMAX, int EPI, int MODE>
cudaError_t launch_fwd_t(const FwdConfig& cfg, const wt_patch* patches, uint32_t n_patches, const HmDev& hm,
                         float* pos, float* nrm, uint32_t flags, void* ws, const WsLayout& L, const FwdExtra& x,
                         cudaStream_t s) {
    constexpr int kMaxDev = 64;
    static std::atomic<int> occ_cache[kMaxDev];  // resident blocks per SM, per device
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= kMaxDev) return cudaErrorInvalidDevice;
    const int sm = sm_count();
    if (sm <= 0) return cudaErrorInvalidDevice;
    constexpr size_t smem_base =
        sizeof(float4) * ((THREADS / 32) * fwd_warp_f4(EPI, SMAX) + (MODE == kModeStage ? 9 : 0));
    // the tile table of up to kTabPatches patches follows; occupancy is
    // taken at its largest size
    constexpr size_t smem_max = smem_base + tab_bytes(kTabPatches);
    const uint32_t tab_in_smem = n_patches <= kTabPatches ? 1u : 0u;
    const size_t smem = smem_base + (tab_in_smem ? tab_bytes(n_patches) : 0);
    int occ = occ_cache[dev].load(std::memory_order_relaxed);
    if (occ == 0) {
        int o = 0;
        cudaError_t e = cudaFuncSetAttribute(k_forward<THREADS, MINB, SMAX, EPI, MODE>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max);
        if (e != cudaSuccess) return e;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_forward<THREADS, MINB, SMAX, EPI, MODE>, THREADS,
                                                          smem_max);
        if (e != cudaSuccess) return e;
        occ = o < 1 ? 1 : o;
        occ_cache[dev].store(occ, std::memory_order_relaxed);
    }
    const int bps = cfg.blocks_per_sm > 0 ? (cfg.blocks_per_sm < occ ? cfg.blocks_per_sm : occ) : occ;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)(sm * bps));
    lc.blockDim = dim3(THREADS);
    lc.dynamicSmemBytes = smem;
    lc.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    const uint32_t chunk = cfg.chunk >= 1 && cfg.chunk <= 32 ? (uint32_t)cfg.chunk : 32u;
    return cudaLaunchKernelEx(&lc, k_forward<THREADS, MINB, SMAX, EPI, MODE>, patches, hm, pos, nrm, flags,
                              static_cast<char*>(ws), L, chunk, reinterpret_cast<float4*>(x.sums), x.view, x.stage,
                              tab_in_smem);
}

}  // namespace

cudaError_t launch_prep(const wt_patch* patches, uint32_t n_patches, const wt_wave* waves, uint32_t n_waves,
                        const HmDev& hm, uint64_t out_capacity, uint32_t tile_cols, void* ws,
                        const WsLayout& L, cudaStream_t s, const MmaRule& rule,
                        const AdjScanArgs* adj) {
    char* w = static_cast<char*>(ws);
    // coefficient capacity = what the caller's workspace holds past the fixed part
    // (the header records the real total; the scan refuses to overflow it)
    uint64_t coef_cap = (L.end - L.coef) / sizeof(PairCoef);
    // few patches, and (patch, wave) pairs by the most that the table can have: the scan
    // kernel forms the constants too
    const uint64_t pairs = (uint64_t)n_patches * n_waves;
    const int small = n_patches <= kSmallPrep && pairs <= kSmallPairs;
    const AdjScanArgs none{};
    const AdjScanArgs& A = adj ? *adj : none;
    const int sms = sm_count();
    if (sms <= 0) return cudaErrorInvalidDevice;
    const unsigned more = small
                              ? std::min((unsigned)sms - 1u, (unsigned)((5u * ((pairs + 31u) / 32u) + kSmallTasks) / kSmallTasks))
                              : 0u;
    k_prep_scan<<<1u + more, 1024, 0, s>>>(patches, n_patches, waves, n_waves, out_capacity, coef_cap, tile_cols, w, L,
                                   hm, small, (uint32_t)sms, rule, adj ? 1 : 0, A.L, A.chunk_max, A.min_tiles);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    if (small) return cudaSuccess;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)sms);
    lc.blockDim = dim3(256);
    lc.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, k_prep_coef, patches, n_patches, waves, n_waves, out_capacity, coef_cap, hm, w,
                              L);
}

bool forward_config_supported(const FwdConfig& c) {
    if (c.epi != 0 && c.epi != 1) return false;
    if (c.s == 8) return c.warps == 8 || c.warps == 16 || (c.warps == 20 && c.epi == 0);
    if (c.s == 4) return c.warps == 8 && c.epi == 0;
    return false;
}

// The epilogue variants beyond the plain one exist with the register
// epilogue only: a tuning with the shared-memory epilogue runs them through
// the register one, same shape; 20 warps (the plain forward's 96-register
// shape) run as 16.
template <int MODE>
cudaError_t launch_forward_mode(const FwdConfig& cfg, const wt_patch* patches, uint32_t n_patches, const HmDev& hm,
                                float* pos, float* nrm, uint32_t flags, void* ws, const WsLayout& L,
                                const FwdExtra& x, cudaStream_t s) {
    if (cfg.s == 4 && cfg.warps == 8)
        return launch_fwd_t<256, 3, 4, 0, MODE>(cfg, patches, n_patches, hm, pos, nrm, flags, ws, L, x, s);
    if (cfg.s == 8 && cfg.warps == 8)
        return launch_fwd_t<256, 2, 8, 0, MODE>(cfg, patches, n_patches, hm, pos, nrm, flags, ws, L, x, s);
    if (cfg.s == 8 && (cfg.warps == 16 || cfg.warps == 20))
        return launch_fwd_t<512, 1, 8, 0, MODE>(cfg, patches, n_patches, hm, pos, nrm, flags, ws, L, x, s);
    return cudaErrorInvalidValue;
}

cudaError_t launch_forward(const FwdConfig& cfg, const wt_patch* patches, uint32_t n_patches, const HmDev& hm,
                           float* pos, float* nrm, uint32_t flags, void* ws, const WsLayout& L, const FwdExtra& x,
                           cudaStream_t s) {
    if (x.sums && x.view) return cudaErrorInvalidValue;
    if (x.sums) return launch_forward_mode<kModeSave>(cfg, patches, n_patches, hm, pos, nrm, flags, ws, L, x, s);
    if (x.view) return launch_forward_mode<kModeStage>(cfg, patches, n_patches, hm, pos, nrm, flags, ws, L, x, s);
    // warps per block; the minimum-blocks hint sets the register budget
    if (cfg.s == 4 && cfg.warps == 8 && cfg.epi == 0)
        return launch_fwd_t<256, 3, 4, 0, kModePlain>(cfg, patches, n_patches, hm, pos, nrm, flags, ws, L, x, s);  // 80 regs
    if (cfg.s == 8 && cfg.epi == 0) {
        if (cfg.warps == 8) return launch_fwd_t<256, 2, 8, 0, kModePlain>(cfg, patches, n_patches, hm, pos, nrm, flags, ws, L, x, s);
        if (cfg.warps == 16) return launch_fwd_t<512, 1, 8, 0, kModePlain>(cfg, patches, n_patches, hm, pos, nrm, flags, ws, L, x, s);
        // 20 warps at 96 registers (a few bytes spilled): more warps to hide
        // the wave loop's latencies (256 uneven patches: 1.041 against 1.054
        // ms for 16 warps; 18 and 24 warps were slower)
        if (cfg.warps == 20) return launch_fwd_t<640, 1, 8, 0, kModePlain>(cfg, patches, n_patches, hm, pos, nrm, flags, ws, L, x, s);
    }
    if (cfg.s == 8 && cfg.epi == 1) {
        if (cfg.warps == 8) return launch_fwd_t<256, 2, 8, 1, kModePlain>(cfg, patches, n_patches, hm, pos, nrm, flags, ws, L, x, s);
        if (cfg.warps == 16) return launch_fwd_t<512, 1, 8, 1, kModePlain>(cfg, patches, n_patches, hm, pos, nrm, flags, ws, L, x, s);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_displace(const FwdConfig& cfg, const wt_patch* patches, uint32_t n_patches, const wt_wave* waves,
                            uint32_t n_waves, const HmDev& hm, float* pos, float* nrm, uint64_t out_capacity,
                            uint32_t flags, void* ws, const WsLayout& L, const FwdExtra& x, cudaStream_t s) {
    const bool naive = (flags & WT_PHASE_FP32_NAIVE) != 0;
    // one patch at the built-in launch shape (another shape, set or autotuned,
    // is run as asked for)
    if (!naive && n_patches == 1 && n_waves <= kSingleWaves && cfg.s == 8 && cfg.warps == 16 && cfg.epi == 1 &&
        cfg.blocks_per_sm == 0)
        return launch_single(cfg, patches, waves, n_waves, hm, pos, nrm, out_capacity, flags, ws, L, x, s);
    // with fewer waves than mma_patch asks for, no patch can qualify
    const bool mma = !naive && n_waves >= kMmaMinWaves;
    cudaError_t e = launch_prep(patches, n_patches, waves, n_waves, hm, out_capacity, 32u * cfg.s, ws, L, s,
                                MmaRule{mma ? kMmaMaxWaves : 0u, x.sums ? 64u : 0u});
    if (e != cudaSuccess) return e;
    if (naive) return launch_forward_naive(patches, n_patches, waves, hm, pos, nrm, flags, ws, L, out_capacity, s);
    const auto recurrence = [&] { return launch_forward(cfg, patches, n_patches, hm, pos, nrm, flags, ws, L, x, s); };
    const auto products = [&] {
        return mma ? launch_forward_mma(patches, hm, pos, nrm, flags, ws, L, x, s) : cudaSuccess;
    };
    // The products' kernel takes nearly all of an SM's shared memory, also for a table
    // without a patch of theirs, and what follows it starts later and with less cache.
    // Tables too large for the recurrence kernel's table in shared memory look their
    // tiles up through that cache: recurrence first (5000 skewed patches of 24 x 24, 9
    // waves, 231.8 -> 225.5 us, saving 252.6 -> 240.2; 1200 of 16 x 16 55.5 -> 53.5).  The
    // others the other way round (200 parallelograms of 200 x 100, 8 waves, saving, 63.1
    // against 67.5; 64 of 64-128 side 25.7 against 27.2; 700 skewed 43.4 and 43.3).
    const bool first = n_patches <= kTabPatches;
    e = first ? products() : recurrence();
    if (e != cudaSuccess) return e;
    return first ? recurrence() : products();
}

cudaError_t launch_forward_naive(const wt_patch* patches, uint32_t n_patches, const wt_wave* waves,
                                 const HmDev& hm, float* pos, float* nrm, uint32_t flags, void* ws,
                                 const WsLayout& L, uint64_t, cudaStream_t s) {
    const int sms = sm_count();
    if (sms <= 0) return cudaErrorInvalidDevice;
    k_forward_naive<<<sms * 4, 256, 0, s>>>(patches, n_patches, waves, hm, pos, nrm, flags,
                                            static_cast<const char*>(ws), L);
    return cudaGetLastError();
}

}  // namespace wt
