// wt_mma.cuh — the forward's wave sums of parallelogram patches as matrix
// products on the tensor cores (tcgen05): the pieces shared by the kernel of
// many-patch tables (wt_mma.cu) and the one-patch kernel (wt_single.cu).
//
// On a patch whose corners span a parallelogram the phase of wave i is
// x_i(col) + y_i(row) exactly, so with cos(x + y) = cos x cos y - sin x sin y
// (and the sine's form) each of the eight sums of a vertex is a dot product
// over (cos x_i, sin x_i): for 128 columns and R rows,
//   D[col][row, q] = sum_k A[col][k] B[row, q][k],   k = (wave, cos | sin),
//   A = (cos x_i, sin x_i),  B = the sum's coefficient times (cos y_i, -+sin y_i).
// A term (vertex x wave) costs 16 multiply-adds here against the 10 of the
// recurrence in forward_tile, but on the tensor pipe, and sines and cosines are
// only taken per column and per row.
//
// FP32 products from FP16 operands: every operand is split into hi + lo
// (11 + 11 bits) and lo*hi + hi*lo + hi*hi is accumulated in FP32; what is
// dropped is 2^-24 of the product.  B is scaled by a power of two per patch and
// sum (the sum's largest coefficient to [2^13, 2^14)) and the sums are scaled
// back, exactly; a scale for all eight would take bits from those whose
// coefficients are small beside another's (slopes beside displacements 2^26 as
// large: normals off by 5e-4, now 1e-7).  Sines and cosines are formed from the
// 64-bit fixed-point phases to 1e-7 (the recurrence starts from MUFU's 5e-7).
// Each product step truncates the accumulator, a bias of about 2^-25 of it
// towards zero: above 48 waves the cross products (2^-11 of the whole, two
// thirds of the steps) get an accumulator of their own, and above 32 the mean of
// what is lost is given back in the inverse scales (mean_loss; 128 waves were
// short by 2.6e-7 without it, 4.8e-7 with the largest waves first).  Relative
// displacement error (2-norm) against 64 bits on 500 x 400 vertices, mean of six
// tables, recurrence / products: 8 waves 2.9e-7 / 0.9e-7, 32 waves 3.3e-7 /
// 1.3e-7, 48 waves 3.1e-7 / 1.9e-7, 64 waves 3.1e-7 / 1.4e-7, 128 waves 3.9e-7 /
// 2.2e-7, and with the largest waves first 4.0e-7 / 3.2e-7.
//
// A step is 32 waves (64 fp16: one 128-byte row) of one tile: 128 columns by
// 32 rows (above 48 waves 16).  A stays in shared memory for a run of rows, B
// is formed per tile in two alternating stages, and two sets of accumulators
// (tensor memory holds 512 columns) let a tile's epilogue run during the next
// tile's products.  In the epilogue a warp reads the sums of 32 consecutive
// columns of a row, so its stores are whole lines.  Forming operands and
// epilogues are separate warps' work: done in turn by all 16 warps the two
// added up (256 patches 400 us, of which 235 without any epilogue: the
// chain form - product - form of two stages is latency), 385 us apart.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstdint>

#include "wt_device.cuh"
#include "wt_internal.h"

namespace wt {
namespace mma {

using namespace wt::dev;

constexpr uint32_t kEpi = 12;              // epilogue warps: three for each quarter of tensor memory
constexpr uint32_t kChunk = 32;            // waves per step
constexpr uint32_t kOneAccWaves = 48;      // above: cross products in an accumulator of their own
constexpr uint32_t kSlotA = 32768;         // a chunk of A: 128 rows x 128 B, hi and lo
constexpr uint32_t kRowB = 1024;           // a row's eight sums in a chunk of B: 8 x 128 B
constexpr uint32_t kOperands = 6 * kSlotA; // A (2 or 4 chunks) and two stages of B

// The waves of a patch, chunk by chunk; even waves of a chunk first, then odd.
struct Table {
    ulonglong2 y[kMmaMaxWaves];          // t00, tb
    float4 k0[kMmaMaxWaves];             // scaled Q*A*Dx, Q*A*Dz, A*k*Dx, A*k*Dz (cosine sums)
    float4 k1[kMmaMaxWaves];             // scaled A, Q*A*k*Dx^2, Q*A*k*Dx*Dz, Q*A*k*Dz^2 (sine sums)
    unsigned long long x[kMmaMaxWaves];  // ta (in wave order)
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
// What a wait needs besides its barrier: the block's flag that one ran out, and the
// limit (nanoseconds; 0: it has run out from the start).
struct Limit {
    int* fail;
    unsigned long long ns;
};
// Bounded wait for the phase of the given parity; false when it ran out here
// or in another warp (`fail`).
__device__ __forceinline__ bool mbar_wait(unsigned long long* b, uint32_t parity, const Limit& limit) {
    const uint32_t a = smem_u32(b);
    unsigned long long t0 = 0, t1 = 0;
    do {
        uint32_t ok;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
        if (*(volatile int*)limit.fail) return false;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        if (t0 == 0) t0 = t1;
    } while (t1 - t0 < limit.ns);
    *(volatile int*)limit.fail = 1;
    return false;
}
// The same by a whole warp, with one answer.
__device__ __forceinline__ bool warp_wait(unsigned long long* b, uint32_t parity, const Limit& limit) {
    return __all_sync(0xffffffffu, mbar_wait(b, parity, limit));
}

// K-major operand, 128-byte swizzle: rows of 128 B in groups of eight (1024 B).
// Read the other way (M- or N-major), the 64 elements of a row are the M or N
// direction, the rows K, and `lead` bytes further lie the next 64.
__device__ __forceinline__ uint64_t transposed_desc(uint32_t addr, uint32_t lead) {
    return (uint64_t)((addr & 0x3ffffu) >> 4) | ((uint64_t)(lead >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3ffffu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

// Eight columns of the warp's lanes: the sums of a row.
__device__ __forceinline__ void tmem_ld8(uint32_t addr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr));
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// All of tensor memory (one block per SM holds it), by one warp.
__device__ __forceinline__ void tmem_alloc(uint32_t* at) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(at)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t tmem) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// Ends tmem_ld8 loads; a and b are used after it (tied to the statement so that
// their uses stay behind it).
__device__ __forceinline__ void tmem_wait(float (&a)[8], float (&b)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(a[0]), "+f"(a[1]), "+f"(a[2]), "+f"(a[3]), "+f"(a[4]), "+f"(a[5]), "+f"(a[6]), "+f"(a[7])::"memory");
    asm volatile(""
                 : "+f"(b[0]), "+f"(b[1]), "+f"(b[2]), "+f"(b[3]), "+f"(b[4]), "+f"(b[5]), "+f"(b[6]), "+f"(b[7])::"memory");
}

__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }

// p as fp16 pairs hi + lo
__device__ __forceinline__ void split2(float2 p, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(p.x, p.y);
    const float2 d = __ffma2_rn(__half22float2(h), make_float2(-1.0f, -1.0f), p);
    hi = h2_bits(h);
    lo = h2_bits(__floats2half2_rn(d.x, d.y));
}

// Rows per tile, and the offset of the stages of B behind the chunks of A.
__device__ __forceinline__ uint32_t tile_rows(uint32_t nwaves) { return nwaves <= kOneAccWaves ? 32u : 16u; }
__device__ __forceinline__ uint32_t stage_offset(uint32_t rb, uint32_t stage) {
    return (rb == 32u ? 2u : 4u) * kSlotA + stage * (2u * rb * kRowB);
}

// Power of two that takes a sum's largest coefficient (bits mb of its magnitude)
// to [2^13, 2^14): fp16's hi + lo then hold every coefficient of the sum to 2^-22
// of itself or 2^-38 of the largest, whichever is more.
__device__ __forceinline__ int scale_exponent(uint32_t mb) {
    return mb == 0u ? 0 : min(max(13 - ((int)(mb >> 23) - 127), -110), 110);
}
__device__ __forceinline__ float pow2f(int e) { return __uint_as_float((uint32_t)(127 + e) << 23); }

// A value for each of the eight sums, in the order of PairCoef's coefficients.
struct PerSum {
    float4 a, b;
};
__device__ __forceinline__ void max8(PerSum& m, const float4& a, const float4& b) {
    const auto max4 = [](float4& m, const float4& v) {
        m = make_float4(fmaxf(m.x, fabsf(v.x)), fmaxf(m.y, fabsf(v.y)), fmaxf(m.z, fabsf(v.z)), fmaxf(m.w, fabsf(v.w)));
    };
    max4(m.a, a);
    max4(m.b, b);
}
// A patch's scales from its largest coefficients, by a whole warp whose lanes share them out.
__device__ __forceinline__ float warp_scale(float v) {
    return pow2f(scale_exponent(__reduce_max_sync(0xffffffffu, __float_as_uint(v))));
}
__device__ __forceinline__ PerSum warp_scales(const PerSum& m) {
    return PerSum{make_float4(warp_scale(m.a.x), warp_scale(m.a.y), warp_scale(m.a.z), warp_scale(m.a.w)),
                  make_float4(warp_scale(m.b.x), warp_scale(m.b.y), warp_scale(m.b.z), warp_scale(m.b.w))};
}
// The mean of what truncation takes from the sums of nw waves, as a part of them:
// about 2^-25 of the partial sum at each step that adds to it, which are the
// leading products (with one accumulator also the second chunk's cross products),
// and the partial sums of waves in no order are as far as the waves added so far.
// Up to a chunk it is less than FP32 holds beside 1.
__device__ __forceinline__ float mean_loss(uint32_t nw, bool two_acc) {
    if (nw <= kChunk) return 0.0f;
    const float steps = (float)((nw + 7u) / 8u), first = (float)(kChunk / 8u);
    return 0x1p-25f * (0.5f * (steps + 1.0f) + (two_acc ? 0.0f : 2.0f * (steps - first) * first / steps));
}
// The scales' inverses, with the mean loss given back, in the accumulators' order
// (the cosine sums dx, dz, jx, jz, then dy, sxx, sxz, szz), for scaled_sums.
__device__ __forceinline__ void write_inverses(float4 (&inv)[2], const PerSum& s, float loss) {
    const auto of = [&](float scale) {
        const float i = __uint_as_float((254u << 23) - __float_as_uint(scale));
        return fmaf(i, loss, i);
    };
    inv[0] = make_float4(of(s.a.x), of(s.a.z), of(s.a.w), of(s.b.x));
    inv[1] = make_float4(of(s.a.y), of(s.b.y), of(s.b.z), of(s.b.w));
}
// A vertex's sums from its accumulators and their inverse scales (no power of two
// above 32 waves: rounded here, whatever follows, so that every mode has the same
// bits).
__device__ __forceinline__ VertexSums scaled_sums(const float (&f)[8], const float4& i0, const float4& i1) {
    return VertexSums{__fmul_rn(f[0], i0.x), __fmul_rn(f[4], i1.x), __fmul_rn(f[1], i0.y), __fmul_rn(f[2], i0.z),
                      __fmul_rn(f[3], i0.w), __fmul_rn(f[5], i1.y), __fmul_rn(f[6], i1.z), __fmul_rn(f[7], i1.w)};
}

// Wave i's entry: c = its PairCoef as four float4.
__device__ __forceinline__ void table_entry(Table& T, uint32_t i, const float4 (&c)[4], const PerSum& s) {
    const uint32_t at = (i & ~31u) + ((i & 31u) >> 1) + 16u * (i & 1u);
    const uint4 u0 = *reinterpret_cast<const uint4*>(&c[0]), u1 = *reinterpret_cast<const uint4*>(&c[1]);
    T.y[at] = make_ulonglong2(((unsigned long long)u0.y << 32) | u0.x, ((unsigned long long)u1.y << 32) | u1.x);
    T.x[i] = ((unsigned long long)u0.w << 32) | u0.z;
    T.k0[at] = make_float4(c[2].x * s.a.x, c[2].z * s.a.z, c[2].w * s.a.w, c[3].x * s.b.x);
    T.k1[at] = make_float4(c[2].y * s.a.y, c[3].y * s.b.y, c[3].z * s.b.z, c[3].w * s.b.w);
}

// A of the 128 columns from c0, by `warps` warps: a thread forms four waves of
// one column (16 bytes of its row).
__device__ __forceinline__ void write_a(char* op, const Table& T, uint32_t nw, uint32_t c0, uint32_t warp,
                                        uint32_t warps, uint32_t lane) {
    for (uint32_t i = warp; i < ((nw + 7u) >> 3) * 8u; i += warps) {  // 32 columns by four waves
        const uint32_t cl = 32u * (i & 3u) + lane, c = c0 + cl, g = i >> 2;
        uint32_t h[4], l[4];
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
            const unsigned long long ta = T.x[4u * g + e];
            float sn, cs;
            sincos_turns(__umulhi(c, (uint32_t)ta) + c * (uint32_t)(ta >> 32), sn, cs);
            split2(make_float2(cs, sn), h[e], l[e]);
        }
        char* d = op + (g >> 3) * kSlotA + cl * 128u + (((g & 7u) ^ (cl & 7u)) << 4);
        *reinterpret_cast<uint4*>(d) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4*>(d + kSlotA / 2) = make_uint4(l[0], l[1], l[2], l[3]);
    }
}

// B of rows row0 .. row0 + rt - 1 and the chunk of waves from w0 into the stage
// at b, by `warps` warps: a thread forms two waves of one row, a warp the rows
// its 32 threads cover.  `dealt` counts the row groups handed out so far, so
// that short tiles load all warps in turn.
template <uint32_t RB>
__device__ __forceinline__ void write_b(uint32_t b, const Table& T, uint32_t nw, uint32_t w0, uint32_t row0, uint32_t rt,
                                        uint32_t warp, uint32_t warps, uint32_t lane, uint32_t& dealt) {
    const uint32_t pairs = (min(kChunk, nw - w0) + 7u) / 8u * 4u;
    const uint32_t shl = pairs <= 4u ? 2u : (pairs <= 8u ? 3u : 4u);
    const uint32_t per = 32u >> shl, groups = (rt + per - 1u) / per;  // rows per warp and the groups of them
    const uint32_t j = lane & ((1u << shl) - 1u);
    const uint32_t first = (warp + warps - dealt) % warps;
    dealt = (dealt + groups) % warps;
    if (j >= pairs) return;
    const uint32_t at0 = w0 + j;
    for (uint32_t r = first * per + (lane >> shl); r < rt; r += warps * per) {
        float2 cc[2], ss[2];  // (cos, -sin), (sin, cos)
        float4 k0[2], k1[2];
#pragma unroll
        for (uint32_t e = 0; e < 2; ++e) {
            const ulonglong2 y = T.y[at0 + 16u * e];
            float sn, cs;
            sincos_turns((uint32_t)((y.x + (unsigned long long)(row0 + r) * y.y) >> 32), sn, cs);
            cc[e] = make_float2(cs, -sn);
            ss[e] = make_float2(sn, cs);
            k0[e] = T.k0[at0 + 16u * e];
            k1[e] = T.k1[at0 + 16u * e];
        }
        // row i of the group, 16-byte piece (j >> 1) ^ i: bits 4-6 of the group's
        // address are free
        const uint32_t d0 = b + r * kRowB + ((j >> 1) << 4) + (j & 1u) * 8u;
        const float ka[2][8] = {{k0[0].x, k0[0].y, k0[0].z, k0[0].w, k1[0].x, k1[0].y, k1[0].z, k1[0].w},
                                {k0[1].x, k0[1].y, k0[1].z, k0[1].w, k1[1].x, k1[1].y, k1[1].z, k1[1].w}};
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) {
            uint2 h, l;
            const float2 p0 = __fmul2_rn(make_float2(ka[0][i], ka[0][i]), i < 4 ? cc[0] : ss[0]);
            const float2 p1 = __fmul2_rn(make_float2(ka[1][i], ka[1][i]), i < 4 ? cc[1] : ss[1]);
            split2(p0, h.x, l.x);
            split2(p1, h.y, l.y);
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"((d0 ^ (i << 4)) + i * 128u), "r"(h.x), "r"(h.y) : "memory");
            asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"((d0 ^ (i << 4)) + i * 128u + RB * kRowB), "r"(l.x), "r"(l.y) : "memory");
        }
    }
}

// The same with the rows per tile known at run time.
__device__ __forceinline__ void write_b(uint32_t op, uint32_t stage, uint32_t rb, const Table& T, uint32_t nw, uint32_t w0,
                                        uint32_t row0, uint32_t rt, uint32_t warp, uint32_t warps, uint32_t lane,
                                        uint32_t& dealt) {
    if (rb == 32u) write_b<32>(op + stage_offset(32, stage), T, nw, w0, row0, rt, warp, warps, lane, dealt);
    else write_b<16>(op + stage_offset(16, stage), T, nw, w0, row0, rt, warp, warps, lane, dealt);
}

__device__ __forceinline__ void commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// By the issuing thread when it issues no more, on every path: all its products and
// their arrivals on barriers are complete before the block's memory goes.  A
// limit of its own: a wait that ran out elsewhere does not end this one.
__device__ __forceinline__ void drain(unsigned long long* bar, int* fail) {
    commit(bar);
    int late = 0;
    if (!mbar_wait(bar, 0, Limit{&late, kWaitNs})) *(volatile int*)fail = 1;
}

// The products of chunk ch (ks steps of 8 waves) of a tile of rt rows.  op: the operands' shared address; acc: the tile's
// accumulators.  One thread.
__device__ __forceinline__ void issue_step(uint32_t op, uint32_t acc, uint32_t nw, uint32_t rb, uint32_t rt, uint32_t ch,
                                           uint32_t stage) {
    const uint32_t n = (rt + 1u) & ~1u;  // N = 8 n, a multiple of 16
    const uint32_t base = (1u << 4) | ((128u / 16u) << 24);  // fp16 operands, FP32 sums, M = 128
    const uint32_t ks = (min(kChunk, nw - ch * kChunk) + 7u) / 8u;
    const uint64_t ah = operand_desc(op + ch * kSlotA), al = operand_desc(op + ch * kSlotA + kSlotA / 2);
    const uint32_t bs = op + stage_offset(rb, stage);
    const uint64_t bh = operand_desc(bs), bl = operand_desc(bs + rb * kRowB);
    if (nw <= kOneAccWaves) {
        // cross products first
        const uint32_t idesc = base | (n << 17);
        for (uint32_t i = 0; i < ks; ++i) mma_f16(acc, al + 2u * i, bh + 2u * i, idesc, (ch | i) != 0u);
        for (uint32_t i = 0; i < ks; ++i) mma_f16(acc, ah + 2u * i, bl + 2u * i, idesc, 1u);
        for (uint32_t i = 0; i < ks; ++i) mma_f16(acc, ah + 2u * i, bh + 2u * i, idesc, 1u);
    } else {
        // hi(A) by hi and lo(B), which follow one another, in one product of
        // N = 256 (a product takes about 120 cycles at N = 128 and at 256): the
        // sums in 16 x 8 columns of the accumulator, the cross part in the next
        const uint32_t wide = base | (32u << 17), idesc = base | (n << 17);
        for (uint32_t i = 0; i < ks; ++i) mma_f16(acc, ah + 2u * i, bh + 2u * i, wide, (ch | i) != 0u);
        for (uint32_t i = 0; i < ks; ++i) mma_f16(acc + 128u, al + 2u * i, bh + 2u * i, idesc, 1u);
    }
}

// A tile whose products are complete, and how its vertices are written.
struct Tile {
    uint32_t acc;                // its accumulators
    uint32_t cols, c0, row0;     // the patch's columns; columns from c0, rows from row0
    uint64_t out0;               // output index of (row0, column 0)
    const float4* inv;           // the sums' inverse scales
    bool two_acc;
};
struct Output {
    float* pos;
    float* nrm;
    float4* sums;
    const float* view;
    StageOut so;
    uint32_t flags;
};

// One vertex from its sums and texels (world: the position in the world, else the
// displacement alone, whatever the grid point: a patch may span more than FP32's
// largest number; whole: every lane of the warp has a vertex).  Roundings spelt out
// where a multiply-add could be fused one way in one output mode and another way in
// the next: every mode writes the same bits.
template <int MODE, int HM>
__device__ __forceinline__ void finish(const VertexSums& s, float xl, float zl, bool world, const PatchAux& a,
                                       const HmDev& hm, const HmTexels& T, uint64_t v, const Output& o, bool whole) {
    if (MODE == kModeSave) {
        // 16 bytes a lane; where the warp's 32 columns all exist, two lanes exchange
        // halves first, so that each store writes whole 32-byte sectors (a vertex's eight
        // sums) instead of half ones.  Half sectors / one 32-byte store a lane / exchanged,
        // us: 64 patches of 64-1024 side 230 / 215 / 204, 40 of 520 x 200, 8 waves, 71 / 66 /
        // 64, 1100 of 128 x 100, 8 waves, 158 / 171 / 158, 24 waves 189 / 192 / 180.  Not in
        // patches of up to 64 columns, where half of the epilogue's warps have no column and
        // the others' instructions count: 1500 of 64 x 64, 16 waves, 107 / 117 / 117.
        float4* const at = o.sums + 2 * v;
        const float4 a4 = make_float4(s.dx, s.dy, s.dz, s.jx), b4 = make_float4(s.jz, s.sxx, s.sxz, s.szz);
        if (whole) {
            const bool odd = threadIdx.x & 1u;
            float4 other = odd ? a4 : b4;
            other.x = __shfl_xor_sync(0xffffffffu, other.x, 1);
            other.y = __shfl_xor_sync(0xffffffffu, other.y, 1);
            other.z = __shfl_xor_sync(0xffffffffu, other.z, 1);
            other.w = __shfl_xor_sync(0xffffffffu, other.w, 1);
            __stcs(odd ? at - 1 : at, odd ? other : a4);
            __stcs(odd ? at + 1 : at + 2, odd ? b4 : other);
        } else {
            __stcs(at, a4);
            __stcs(at + 1, b4);
        }
    }
    const float px0 = 1.0f - s.sxx, px2 = -s.sxz, pz0 = -s.sxz, pz2 = 1.0f - s.szz;
    float px1 = s.jx, pz1 = s.jz, dy = s.dy;
    if (HM != 0) {
        const HmSample g = hm_combine(hm, a, T);
        dy = __fadd_rn(dy, g.h);
        px1 = fmaf(g.hx, px0, fmaf(g.hz, px2, px1));
        pz1 = fmaf(g.hx, pz0, fmaf(g.hz, pz2, pz1));
    }
    dy = __fadd_rn(dy, a.y_offset);
    const float ox = world ? __fadd_rn(a.blx, __fadd_rn(xl, s.dx)) : s.dx;
    const float oz = world ? __fadd_rn(a.blz, __fadd_rn(zl, s.dz)) : s.dz;
    float n0 = fmaf(pz1, px2, -__fmul_rn(pz2, px1)), n1 = fmaf(pz2, px0, -__fmul_rn(pz0, px2)),
          n2 = fmaf(pz0, px1, -__fmul_rn(pz1, px0));
    const float inv = rsqrtf(fmaf(n0, n0, fmaf(n1, n1, n2 * n2)));
    n0 *= inv;
    n1 *= inv;
    n2 *= inv;
    if (o.flags & WT_LAYOUT_VEC3) {
        if (MODE != kModeStage || o.pos) {
            float* P = o.pos + 3 * v;
            __stcs(P, ox); __stcs(P + 1, dy); __stcs(P + 2, oz);
        }
        if (o.nrm) {
            float* N = o.nrm + 3 * v;
            __stcs(N, n0); __stcs(N + 1, n1); __stcs(N + 2, n2);
        }
    } else {
        if (MODE != kModeStage || o.pos) __stcs(reinterpret_cast<float4*>(o.pos) + v, make_float4(ox, dy, oz, world ? 1.0f : 0.0f));
        if (o.nrm) __stcs(reinterpret_cast<float4*>(o.nrm) + v, make_float4(n0, n1, n2, 0.0f));
    }
    if (MODE == kModeStage) stage_vertex<false>(o.view, make_float3(ox, dy, oz), make_float3(n0, n1, n2), v, o.so);
}

// Rows first, first + step, ... of a tile of rt rows, by one warp: 32 columns,
// the quarter of tensor memory the warp may read (quad).  HM: 0 no heightmap
// layer, 1 the mask-only wrap, 2 the general one (a kernel each: with the three
// in one kernel 256 patches took 15 us more, in instruction fetches).
template <int MODE, int HM>
__device__ __forceinline__ void tile_epilogue(const Tile& t, const PatchAux& a, const HmDev& hm, bool pow2,
                                              const Output& o, uint32_t quad, uint32_t lane, uint32_t first,
                                              uint32_t step, uint32_t rt) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const bool world = !(o.flags & WT_OUT_DISPLACEMENT);
    const float gx = a.e1x * a.inv_cm1, gz = a.e1z * a.inv_cm1;
    const uint32_t col = t.c0 + 32u * quad + lane;
    const float xc = (float)col * gx, zc = (float)col * gz;
    const uint32_t at = t.acc + ((32u * quad) << 16);
    const uint64_t v0 = t.out0 + col;
    const bool in = col < t.cols;
    const bool whole = MODE == kModeSave && t.cols > 64u && t.c0 + 32u * quad + 32u <= t.cols;  // the warp's columns
    const float4 i0 = t.inv[0], i1 = t.inv[1];
    float rowf = (float)(t.row0 + first);
    // two rows at a time: their texel loads are issued before the first is used
    // (four rows by one wider load: 394 against 386 us on 256 patches, in
    // registers)
#pragma unroll 1
    for (uint32_t r = first; r < rt; r += 2u * step) {
        float f[2][8];
        HmTexels T[2];
        VertexSums v[2];
        float xl[2], zl[2];
        const bool second = r + step < rt;
        const uint32_t at0 = at + 8u * r, at1 = at + 8u * (second ? r + step : r);
        tmem_ld8(at0, f[0]);
        tmem_ld8(at1, f[1]);
        tmem_wait(f[0], f[1]);
        if (t.two_acc) {
            float g[2][8];
            tmem_ld8(at0 + 128u, g[0]);
            tmem_ld8(at1 + 128u, g[1]);
            tmem_wait(g[0], g[1]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                f[0][i] += g[0][i];
                f[1][i] += g[1][i];
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const float vv = rowf * a.inv_rm1;
            rowf += (float)step;
            xl[u] = fmaf(vv, a.e2x, xc);
            zl[u] = fmaf(vv, a.e2z, zc);
            v[u] = scaled_sums(f[u], i0, i1);
            if (HM != 0) T[u] = hm_fetch<HM == 1>(hm, a, xl[u] + v[u].dx, zl[u] + v[u].dz, pow2);
            else T[u] = HmTexels{};
        }
        if (in) {
            finish<MODE, HM>(v[0], xl[0], zl[0], world, a, hm, T[0], v0 + r * t.cols, o, whole);
            if (second) finish<MODE, HM>(v[1], xl[1], zl[1], world, a, hm, T[1], v0 + (r + step) * t.cols, o, whole);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

}  // namespace mma
}  // namespace wt
