// wt_misc.cu — index buffer, noise heightmap synthesis, peak-rate probes.
#include <cuda_runtime.h>
#include <cstdint>

#include "wt_device.cuh"
#include "wt_internal.h"

namespace wt {
namespace {

// ---- projected-grid index buffer (src/program.cpp:686-717) ----------------
// One thread per output index: k = 6*cell + m, cell = row*(cols-1) + col,
// triangles (r,c) (r+1,c+1) (r+1,c) and (r,c) (r,c+1) (r+1,c+1).
// Coalesced 4-byte stores; the buffer is HBM-write-bound.
__global__ void __launch_bounds__(256) k_indices(uint32_t cols, uint32_t rows, uint32_t base, uint32_t* __restrict__ out,
                                                 uint64_t total) {
    const uint32_t cm1 = cols - 1;
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < total;
         k += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t cell = k / 6;
        uint32_t m = (uint32_t)(k - cell * 6);
        uint32_t row = (uint32_t)(cell / cm1);
        uint32_t col = (uint32_t)(cell - (uint64_t)row * cm1);
        // m:      0     1       2     3     4     5
        // dr:     0     1       1     0     0     1
        // dc:     0     1       0     0     1     1
        uint32_t dr = (0x26u >> m) & 1u;  // bits 1,2,5
        uint32_t dc = (0x32u >> m) & 1u;  // bits 1,4,5
        __stcs(out + k, base + (row + dr) * cols + col + dc);
    }
}

// ---- 8-bit heightmap ingestion -------------------------------------------
// texel (i, j) = R of pixel (i, row j counted from the bottom when flipped)
// as UNORM8 -> float: c / 255, correctly rounded (GL's conversion of an
// RGBA8 texel's red channel, sampled by water-grid.vert:106).
__global__ void __launch_bounds__(256) k_unorm8(const uint8_t* __restrict__ px, uint32_t w, uint32_t h,
                                                uint32_t channels, uint64_t stride, uint32_t flip,
                                                float* __restrict__ out) {
    const uint64_t n = (uint64_t)w * h;
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < n; k += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t j = (uint32_t)(k / w);
        const uint32_t i = (uint32_t)(k - (uint64_t)j * w);
        const uint32_t src = flip ? h - 1 - j : j;
        out[k] = (float)px[(uint64_t)src * stride + (uint64_t)i * channels] / 255.0f;
    }
}

// ---- noise heightmap -------------------------------------------------------
constexpr size_t kNoiseHeader = 256;
__device__ __forceinline__ uint32_t ordered(float f) {
    uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float unordered(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// h(i, j) = sum_m a_m sin(x_m(i) + y_m(j)),
//   x_m(i) = 2 pi (kx_m i mod W) / W,  y_m(j) = 2 pi (ky_m j mod H) / H + psi_m + rate_m t,
// is separable: sin(x + y) = sin x cos y + cos x sin y.  A block forms, per tile
// of texels and chunk of terms, the factors (sin x, cos x) of its columns and
// a (cos y, sin y) of its rows in shared memory (phases as 32-bit fixed-point
// turns, so that the wrap-around is the reduction; the time-shifted phase reduced
// in FP64 once per term), then spends one paired FMA per texel and term.  Each block leaves its
// minimum and maximum in the workspace, and k_noise_norm reduces those and
// normalises.  Two dependent launches: the layer of 512^2 texels and 64 terms
// took 23.4 us as four (min / max reset, factor tables through global memory,
// tiles, normalise), 10.0 us this way; what is left is launches and latency
// (33 MFMA, 2 MB).
// A tile is 16 x 16 threads of M x M texels: M = 2 for layers that fill the GPU
// only so, 4 where there are tiles enough (half of the factors and of the
// shared-memory reads per texel: 1024^2 x 64 terms 22.6 against 26.2 us,
// 2048^2 x 128 105 against 143 us).
constexpr uint32_t kNoiseBlocks = 608; // resident blocks at most (4 per SM)
__host__ __device__ constexpr uint32_t noise_tile(int m) { return 16u * (uint32_t)m; }

template <int M>
__global__ void __launch_bounds__(256) k_noise_tiles(const wt_noise_term* __restrict__ terms, uint32_t n_terms,
                                                     const float* __restrict__ rates, double t, uint32_t W, uint32_t H,
                                                     unsigned long long inv_w, unsigned long long inv_h,
                                                     float* __restrict__ out, uint2* __restrict__ mm) {
    cudaTriggerProgrammaticLaunchCompletion();  // the normalising pass waits for this grid's end
    constexpr uint32_t kNoiseTile = noise_tile(M), kNoiseChunk = 128u / M;  // terms at a time
    __shared__ __align__(16) float2 sc[kNoiseChunk][kNoiseTile], sr[kNoiseChunk][kNoiseTile];
    __shared__ uint4 term[kNoiseChunk];  // kx mod W, ky mod H, phase (turns * 2^32), amplitude
    __shared__ uint32_t s_lo, s_hi;
    const uint32_t tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const uint32_t tiles_x = (W + kNoiseTile - 1) / kNoiseTile, tiles = tiles_x * ((H + kNoiseTile - 1) / kNoiseTile);
    if (threadIdx.x == 0) {
        s_lo = 0xffffffffu;
        s_hi = 0u;
    }
    float lo = INFINITY, hi = -INFINITY;
    cudaGridDependencySynchronize();
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint32_t j0 = tile / tiles_x * kNoiseTile, i0 = (tile % tiles_x) * kNoiseTile;
        float2 h[M][M];  // (sine, cosine) parts
#pragma unroll
        for (int b = 0; b < M; ++b)
#pragma unroll
            for (int a = 0; a < M; ++a) h[b][a] = make_float2(0.0f, 0.0f);
        for (uint32_t m0 = 0; m0 < n_terms; m0 += kNoiseChunk) {
            const uint32_t nm = min(kNoiseChunk, n_terms - m0);
            __syncthreads();
            if (threadIdx.x < nm) {
                const wt_noise_term tm = terms[m0 + threadIdx.x];
                const int32_t x = (int32_t)((int64_t)tm.kx % (int64_t)W), y = (int32_t)((int64_t)tm.ky % (int64_t)H);
                // (psi + rate t) / 2 pi, reduced mod 1 in FP64 (t may be large)
                double turns = ((double)tm.phase + (rates ? (double)rates[m0 + threadIdx.x] * t : 0.0)) *
                               (0.5 / 3.14159265358979323846);
                turns -= floor(turns);
                term[threadIdx.x] = make_uint4((uint32_t)(x < 0 ? x + (int32_t)W : x), (uint32_t)(y < 0 ? y + (int32_t)H : y),
                                               (uint32_t)__double2ull_rn(turns * 4294967296.0),
                                               __float_as_uint(isfinite(turns) ? tm.amplitude : NAN));
            }
            __syncthreads();
            for (uint32_t e = threadIdx.x; e < nm * 2u * kNoiseTile; e += blockDim.x) {
                const uint32_t m = e / (2u * kNoiseTile), q = e % kNoiseTile;
                const uint4 tm = term[m];
                float sn, cs;
                if ((e & kNoiseTile) == 0u) {
                    dev::sincos_turns((uint32_t)((tm.x * (unsigned long long)(i0 + q) * inv_w) >> 32), sn, cs);
                    sc[m][q] = make_float2(sn, cs);
                } else {
                    dev::sincos_turns((uint32_t)((tm.y * (unsigned long long)(j0 + q) * inv_h) >> 32) + tm.z, sn, cs);
                    const float a = __uint_as_float(tm.w);
                    sr[m][q] = make_float2(a * cs, a * sn);
                }
            }
            __syncthreads();
#pragma unroll 4
            for (uint32_t m = 0; m < nm; ++m) {
                float2 x[M], y[M];
#pragma unroll
                for (int a = 0; a < M; a += 2) {
                    const float4 v = *reinterpret_cast<const float4*>(&sc[m][M * tx + a]);
                    const float4 w = *reinterpret_cast<const float4*>(&sr[m][M * ty + a]);
                    x[a] = make_float2(v.x, v.y);
                    x[a + 1] = make_float2(v.z, v.w);
                    y[a] = make_float2(w.x, w.y);
                    y[a + 1] = make_float2(w.z, w.w);
                }
#pragma unroll
                for (int b = 0; b < M; ++b)
#pragma unroll
                    for (int a = 0; a < M; ++a) h[b][a] = __ffma2_rn(x[a], y[b], h[b][a]);
            }
        }
#pragma unroll
        for (int b = 0; b < M; ++b)
#pragma unroll
            for (int a = 0; a < M; ++a) {
                const uint32_t i = i0 + M * tx + a, j = j0 + M * ty + b;
                if (i < W && j < H) {
                    const float v = h[b][a].x + h[b][a].y;
                    lo = fminf(lo, v);
                    hi = fmaxf(hi, v);
                    out[(size_t)j * W + i] = v;
                }
            }
    }
    const uint32_t wlo = __reduce_min_sync(0xffffffffu, ordered(lo)), whi = __reduce_max_sync(0xffffffffu, ordered(hi));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&s_lo, wlo);
        atomicMax(&s_hi, whi);
    }
    __syncthreads();
    if (threadIdx.x == 0) mm[blockIdx.x] = make_uint2(s_lo, s_hi);
}

__global__ void __launch_bounds__(256) k_noise_norm(float* __restrict__ out, size_t n, const uint2* __restrict__ mm,
                                                    uint32_t blocks) {
    __shared__ uint32_t s_lo, s_hi;
    if (threadIdx.x == 0) {
        s_lo = 0xffffffffu;
        s_hi = 0u;
    }
    cudaGridDependencySynchronize();
    __syncthreads();
    uint32_t a = 0xffffffffu, b = 0u;
    for (uint32_t i = threadIdx.x; i < blocks; i += blockDim.x) {
        const uint2 v = mm[i];
        a = min(a, v.x);
        b = max(b, v.y);
    }
    a = __reduce_min_sync(0xffffffffu, a);
    b = __reduce_max_sync(0xffffffffu, b);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&s_lo, a);
        atomicMax(&s_hi, b);
    }
    __syncthreads();
    const float lo = unordered(s_lo), hi = unordered(s_hi);
    const float span = hi - lo;
    // a correctly rounded division maps the extremes to exactly 0 and 1
    for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < n; v += (size_t)gridDim.x * blockDim.x)
        out[v] = span > 0.0f ? (out[v] - lo) / span : 0.0f;
}

// ---- peak probes -----------------------------------------------------------
// Eight independent dependent chains per thread: issue-bound FP32 FMA and
// MUFU sine, the two pipes the Gerstner sum can run on.
__global__ void __launch_bounds__(256) k_peak_fma(float* out, int iters, float a, float b) {
    float x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = threadIdx.x * 1e-3f + j;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = fmaf(x[j], a, b);
    }
    float s = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) s += x[j];
    out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

__global__ void __launch_bounds__(256) k_peak_sin(float* out, int iters) {
    float x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = threadIdx.x * 1e-3f + j;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = __sinf(x[j]);
    }
    float s = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) s += x[j];
    out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

int device_sms() { return sm_count(); }

}  // namespace

cudaError_t launch_indices(uint32_t cols, uint32_t rows, uint32_t base, uint32_t* out, cudaStream_t s) {
    uint64_t total = 6ull * (cols - 1) * (rows - 1);
    if (total == 0) return cudaSuccess;
    uint64_t want = (total + 255) / 256;
    unsigned blocks = (unsigned)(want < (uint64_t)device_sms() * 16 ? want : (uint64_t)device_sms() * 16);
    k_indices<<<blocks, 256, 0, s>>>(cols, rows, base, out, total);
    return cudaGetLastError();
}

cudaError_t launch_unorm8(const uint8_t* px, uint32_t w, uint32_t h, uint32_t channels, uint64_t stride,
                          uint32_t flip, float* out, cudaStream_t s) {
    const uint64_t n = (uint64_t)w * h;
    const uint64_t want = (n + 255) / 256;
    const unsigned blocks = (unsigned)(want < (uint64_t)device_sms() * 16 ? want : (uint64_t)device_sms() * 16);
    k_unorm8<<<blocks, 256, 0, s>>>(px, w, h, channels, stride, flip, out);
    return cudaGetLastError();
}

cudaError_t launch_noise(const wt_noise_term* terms, uint32_t n_terms, const float* rates, double t, uint32_t w,
                         uint32_t h, float* out, void* ws, cudaStream_t s) {
    // a block's minimum and maximum: the workspace holds 8 (256 + terms * (w + h))
    // bytes or more of them, never fewer than min(tiles, kNoiseBlocks) with a
    // term, and 32 without any (all texels are then zero)
    const auto tiles_of = [&](uint32_t side) { return (uint64_t)((w + side - 1) / side) * ((h + side - 1) / side); };
    const bool wide = tiles_of(noise_tile(4)) >= 256;
    const uint64_t tiles = tiles_of(noise_tile(wide ? 4 : 2));
    const uint32_t cap = n_terms > 0 ? kNoiseBlocks : (uint32_t)(kNoiseHeader / sizeof(uint2));
    const uint32_t blocks = (uint32_t)(tiles < cap ? tiles : cap);
    uint2* mm = static_cast<uint2*>(ws);
    cudaLaunchConfig_t lc = {};
    lc.blockDim = dim3(256);
    lc.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    lc.gridDim = dim3(blocks);
    // 2^64 / size, rounded down: a product with k j < 2^30 is off by less than
    // 2^-34 turns
    const auto inverse = [](uint32_t n) { return n > 1u ? ~0ull / n : 0ull; };
    cudaError_t e = cudaLaunchKernelEx(&lc, wide ? k_noise_tiles<4> : k_noise_tiles<2>, terms, n_terms, rates, t, w, h, inverse(w), inverse(h), out, mm);
    if (e != cudaSuccess) return e;
    const size_t n = (size_t)w * h;
    lc.gridDim = dim3((unsigned)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096));
    return cudaLaunchKernelEx(&lc, k_noise_norm, out, n, static_cast<const uint2*>(mm), blocks);
}

size_t noise_workspace_bytes(uint32_t n_terms, uint32_t w, uint32_t h) {
    return kNoiseHeader + sizeof(float2) * (size_t)n_terms * ((size_t)w + h);
}

cudaError_t measure_peaks(void* scratch, size_t bytes, double* fma, double* sin_rate, cudaStream_t s) {
    const int sms = device_sms();
    const int blocks = sms * 8, threads = 256;
    if ((size_t)blocks * threads * sizeof(float) > bytes) return cudaErrorInvalidValue;
    float* out = static_cast<float*>(scratch);
    cudaEvent_t e0, e1;
    cudaError_t e = cudaEventCreate(&e0);
    if (e != cudaSuccess) return e;
    e = cudaEventCreate(&e1);
    if (e != cudaSuccess) { cudaEventDestroy(e0); return e; }
    const int it_fma = 1 << 15, it_sin = 1 << 12;
    float best_fma = 1e30f, best_sin = 1e30f;
    for (int rep = 0; rep < 4; ++rep) {
        float ms = 0.0f;
        cudaEventRecord(e0, s);
        k_peak_fma<<<blocks, threads, 0, s>>>(out, it_fma, 0.999f, 0.001f);
        cudaEventRecord(e1, s);
        cudaEventSynchronize(e1);
        cudaEventElapsedTime(&ms, e0, e1);
        if (rep > 0 && ms < best_fma) best_fma = ms;
        cudaEventRecord(e0, s);
        k_peak_sin<<<blocks, threads, 0, s>>>(out, it_sin);
        cudaEventRecord(e1, s);
        cudaEventSynchronize(e1);
        cudaEventElapsedTime(&ms, e0, e1);
        if (rep > 0 && ms < best_sin) best_sin = ms;
    }
    e = cudaGetLastError();
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (e != cudaSuccess) return e;
    const double lanes = (double)blocks * threads;
    *fma = lanes * 8.0 * it_fma / (best_fma * 1e-3);
    *sin_rate = lanes * 8.0 * it_sin / (best_sin * 1e-3);
    return cudaSuccess;
}

}  // namespace wt
