// RFI excision kernels for sm_100a.
//
// The cleaner's decisions (masks, time flags, cell states) must agree bit for
// bit with frost's CPU cleaner, so every threshold-deciding sum keeps the
// reference's summation order: per (window, channel) over time for the
// bandpass refinement, moments and Welford statistics; per row over channels
// for the detection series; per (chunk, channel) over time for zdot and
// Kadane-along-time. Parallelism comes from the many independent
// (window, channel), row and (chunk, channel) sequences instead of from
// splitting any one of them. This file is compiled with --fmad=false so no
// multiply-add is contracted and each float/double operation rounds exactly
// as the IEEE host build does.
//
// Packed samples are decoded on the fly from the raw time-major block (LSB
// first below 8 bits, lib/prepare/sample_codec.hpp:18-109), so the 1/4-byte
// raw block is what every statistics pass reads from HBM.

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cstdint>
#include <cstring>
#include <type_traits>

#include <cuda_runtime.h>

#include "common.hpp"
#include "rfi_columns.cuh"
#include "rfi_kernels.hpp"
#include "rfi_stage.cuh"

namespace fb::rfi {

namespace {

// ---- sample decoding --------------------------------------------------

template <int D> __device__ __forceinline__ float rd(const uint8_t* __restrict__ row, uint64_t c) {
    if constexpr (D == FROST_UINT8) {
        return static_cast<float>(row[c]);
    } else if constexpr (D == FROST_UINT16) {
        return static_cast<float>(reinterpret_cast<const uint16_t*>(row)[c]);
    } else if constexpr (D == FROST_UINT32) {
        return static_cast<float>(reinterpret_cast<const uint32_t*>(row)[c]);
    } else if constexpr (D == FROST_FLOAT32) {
        return reinterpret_cast<const float*>(row)[c];
    } else {
        constexpr unsigned kBits = D == FROST_UINT1 ? 1U : D == FROST_UINT2 ? 2U : 4U;
        constexpr unsigned kMask = (1U << kBits) - 1U;
        const uint64_t bit       = c * kBits;
        return static_cast<float>((row[bit >> 3U] >> (bit & 7U)) & kMask);
    }
}

// The integer code of sample c of an integer dtype D (rd<D> is its float).
template <int D> __device__ __forceinline__ uint32_t rdi(const uint8_t* __restrict__ row, uint64_t c) {
    if constexpr (D == FROST_UINT8) {
        return row[c];
    } else if constexpr (D == FROST_UINT16) {
        return reinterpret_cast<const uint16_t*>(row)[c];
    } else if constexpr (D == FROST_UINT32) {
        return reinterpret_cast<const uint32_t*>(row)[c];
    } else {
        static_assert(D != FROST_FLOAT32, "rdi: integer dtypes only");
        constexpr unsigned kBits = D == FROST_UINT1 ? 1U : D == FROST_UINT2 ? 2U : 4U;
        constexpr unsigned kMask = (1U << kBits) - 1U;
        const uint64_t bit       = c * kBits;
        return (row[bit >> 3U] >> (bit & 7U)) & kMask;
    }
}

// Bits per packed sample of dtype D (usable in device code).
template <int D>
constexpr uint64_t kBitsOf = D == FROST_UINT1 ? 1 : D == FROST_UINT2 ? 2 : D == FROST_UINT4 ? 4
                           : D == FROST_UINT8 ? 8 : D == FROST_UINT16 ? 16 : 32;

#define FB_DTYPE_CASE(DT, ...)                                                                    \
    case DT: {                                                                                    \
        constexpr int D = DT;                                                                     \
        __VA_ARGS__;                                                                              \
    } break;

#define FB_DISPATCH(dtype, ...)                                                                   \
    switch (dtype) {                                                                              \
        FB_DTYPE_CASE(FROST_UINT1, __VA_ARGS__)                                                   \
        FB_DTYPE_CASE(FROST_UINT2, __VA_ARGS__)                                                   \
        FB_DTYPE_CASE(FROST_UINT4, __VA_ARGS__)                                                   \
        FB_DTYPE_CASE(FROST_UINT8, __VA_ARGS__)                                                   \
        FB_DTYPE_CASE(FROST_UINT16, __VA_ARGS__)                                                  \
        FB_DTYPE_CASE(FROST_UINT32, __VA_ARGS__)                                                  \
        FB_DTYPE_CASE(FROST_FLOAT32, __VA_ARGS__)                                                 \
    default: throw ::fb::Error(FROST_ERR_INVALID_ARGUMENT, "unsupported dtype");                 \
    }

// Rows fetched ahead per thread in the time-ordered (window or chunk,
// channel) loops: the loads are independent, only the sums are sequential.
constexpr int kBlock = 16;

// The float of a sample's stored bits (codes of 16 bits or less by the
// exponent of 2^23 and one subtraction: the conversion unit is left to the
// widening).
template <int D> __device__ __forceinline__ float sample_of(uint32_t v) {
    if constexpr (D == FROST_FLOAT32)
        return __uint_as_float(v);
    else if constexpr (D == FROST_UINT32)
        return static_cast<float>(v);
    else
        return __uint_as_float(0x4B000000U | v) - 8388608.0F;
}

// ---- order-exact helpers ------------------------------------------------

// std::min / std::max semantics (first argument kept on ties), which the
// remedian's median network relies on for bit-identical results.
template <class T> __device__ __forceinline__ T smin(T a, T b) { return (b < a) ? b : a; }
template <class T> __device__ __forceinline__ T smax(T a, T b) { return (a < b) ? b : a; }

__device__ __forceinline__ float median3(float a, float b, float c) {
    return a < b ? (b < c ? b : (a < c ? c : a)) : (a < c ? a : (b < c ? c : b));
}

// Median of five: drop the extremes of the first four, then the median of
// the remaining pair and the fifth value.
__device__ __forceinline__ float median5(float a, float b, float c, float d, float e) {
    const float f = smax(smin(a, b), smin(c, d));
    const float g = smin(smax(a, b), smax(c, d));
    return median3(e, f, g);
}

__device__ __forceinline__ float clampf(float v, float lo, float hi) {
    return (v < lo) ? lo : (hi < v) ? hi : v;
}

__device__ __forceinline__ uint64_t window_of(uint64_t t, uint64_t window, uint64_t nwin) {
    // a 32-bit division when both fit (a 64-bit one is a long software
    // sequence, paid per thread and row in the row-parallel kernels)
    const uint64_t w = (t | window) < (uint64_t{1} << 32)
                           ? static_cast<uint64_t>(static_cast<uint32_t>(t) / static_cast<uint32_t>(window))
                           : t / window;
    return w < nwin - 1 ? w : nwin - 1;
}

__device__ __forceinline__ uint64_t window_begin(uint64_t w, uint64_t window) { return w * window; }
__device__ __forceinline__ uint64_t window_end(uint64_t w, const Dims& d) {
    return w + 1 == d.nwin ? d.nsamps : (w + 1) * d.window;
}

__device__ __forceinline__ float normal_deviate(uint64_t h) {
    constexpr double kTwoPi = 6.283185307179586;
    const double u1         = uniform_open(h);
    const double u2         = uniform_open(splitmix64(h));
    return static_cast<float>(sqrt(-2.0 * log(u1)) * cos(kTwoPi * u2));
}

__device__ __forceinline__ uint64_t draw(const ApplyParams& p, uint64_t stream, uint64_t t,
                                         uint64_t c, uint64_t attempt) {
    return hash5(p.seed, p.block_index, (stream << 56U) ^ t, c, attempt);
}

// ---- finite check ---------------------------------------------------------

// Four 16-byte loads in flight a thread (1024 channels x 65 536: one word a
// thread in turn took 119 us, 65 so); the first `head` words lead up to a
// 16-byte boundary.
__global__ void __launch_bounds__(256)
    k_check_finite(const uint32_t* __restrict__ w, uint64_t n, uint64_t head, unsigned long long* first_bad) {
    const uint64_t id     = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    auto test             = [&](uint32_t x, uint64_t i) {
        if ((x & 0x7F800000U) == 0x7F800000U)
            atomicMin(first_bad, static_cast<unsigned long long>(i));
    };
    const uint64_t vecs = (n - head) / 4;
    const uint4* v      = reinterpret_cast<const uint4*>(w + head);
    for (uint64_t i = id; i < vecs; i += 4 * stride) {
        uint4 x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            x[k] = i + k * stride < vecs ? v[i + k * stride] : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint64_t at = head + 4 * (i + k * stride);
            test(x[k].x, at);
            test(x[k].y, at + 1);
            test(x[k].z, at + 2);
            test(x[k].w, at + 3);
        }
    }
    const uint64_t tail = head + 4 * vecs;
    if (id < head)
        test(w[id], id);
    if (id < n - tail)
        test(w[tail + id], tail + id);
}

// ---- a gulp's start and end ---------------------------------------------------

// Everything a cleaning pass counts or marks from zero, in one launch (six
// memsets of a few KB took 3 us each).
__global__ void __launch_bounds__(256)
    k_begin(unsigned long long* __restrict__ counters, uint64_t nslots, uint32_t* __restrict__ unmeasured,
            uint8_t* __restrict__ kchan_any, uint64_t nchans, uint8_t* __restrict__ time_flags,
            uint8_t* __restrict__ row_kchan, uint64_t nsamps, unsigned int* __restrict__ nslow) {
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    const uint64_t id     = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
    if (id < nslots)
        counters[id] = 0;
    if (id == 0)
        *nslow = 0;
    for (uint64_t i = id; i < nchans; i += stride) {
        unmeasured[i] = 0;
        kchan_any[i]  = 0;
    }
    for (uint64_t i = id; i < nsamps; i += stride) {
        time_flags[i] = 0;
        row_kchan[i]  = 0;
    }
}

// The last window's constants, kept for short tails.
__global__ void __launch_bounds__(256)
    k_keep_tail(uint64_t nchans, const float* __restrict__ loc, const float* __restrict__ scale,
                const float* __restrict__ out_loc, const float* __restrict__ out_scale, float* __restrict__ tail_loc,
                float* __restrict__ tail_scale, float* __restrict__ tail_out_loc, float* __restrict__ tail_out_scale) {
    const uint64_t c = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
    if (c >= nchans)
        return;
    tail_loc[c]       = loc[c];
    tail_scale[c]     = scale[c];
    tail_out_loc[c]   = out_loc[c];
    tail_out_scale[c] = out_scale[c];
}

// ---- bandpass -------------------------------------------------------------

// The evenly spaced sample rows of each window (row i of window w is block
// row b + i * len / m, lib/cpu/spectra_cpu.cpp:96-104), decoded to float:
// one CTA per (row, window), its threads across the channels.
template <int D>
__global__ void k_sample_rows(Dims d, const uint8_t* __restrict__ raw, float* __restrict__ out) {
    const uint64_t i   = blockIdx.x;
    const uint64_t w   = blockIdx.y;
    const uint64_t b   = window_begin(w, d.window);
    const uint64_t len = window_end(w, d) - b;
    const uint64_t m   = largest_power_of_five_leq(len < kMaxBandpassRows ? len : kMaxBandpassRows);
    if (i >= m)
        return;
    const uint64_t t  = b + (i * len) / m;
    const uint8_t* in = raw + t * d.row_bytes;
    float* dst        = out + (w * kMaxBandpassRows + i) * d.nchans;
    for (uint64_t c = threadIdx.x; c < d.nchans; c += blockDim.x)
        dst[c] = rd<D>(in, c);
}

// The remedian is a fixed tree (medians of five consecutive values, level by
// level), so its groups are independent: k_remedian evaluates it in
// parallel. One CTA covers 32 channels (a lane each) of one window; each
// warp reduces 125-row blocks (three tree levels in registers) to one value
// per channel, and warp 0 finishes the tree over the <= 25 block values. The
// level goes to loc and a flat flag (every sampled value of the channel
// compares equal) to inv; a second sweep takes the scale, remedian(|x -
// level|) x 1.4826 (lib/cpu/spectra_cpu.cpp:73-130). 25 warps, one a block:
// load latency bounds them (64 channels 33 + 20 us with 8 warps and two
// launches, 16 here; 1024 channels x 32 windows 297 us with 8 warps, 168 here).
constexpr int kRemedianWarps = 25;

// The remedian of 25 values p[0], p[stride], ... (medians of five
// consecutive values, then their median): the 25 loads are issued together
// before any is used, then lo / hi track the range of the raw values.
template <bool ABS>
__device__ __forceinline__ float remedian25(const float* __restrict__ p, uint64_t stride, float level, float& lo,
                                            float& hi) {
    float x[25];
#pragma unroll
    for (int i = 0; i < 25; ++i)
        x[i] = p[i * stride];
    float v[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        float y[5];
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            const float r = x[5 * j + i];
            if constexpr (ABS) {
                y[i] = fabsf(r - level);
            } else {
                lo   = fminf(lo, r);
                hi   = fmaxf(hi, r);
                y[i] = r;
            }
        }
        v[j] = median5(y[0], y[1], y[2], y[3], y[4]);
    }
    return median5(v[0], v[1], v[2], v[3], v[4]);
}

template <bool ABS>
__device__ __forceinline__ float remedian5(const float* __restrict__ p, uint64_t stride, float level, float& lo,
                                           float& hi) {
    float y[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const float r = p[i * stride];
        if constexpr (ABS) {
            y[i] = fabsf(r - level);
        } else {
            lo   = fminf(lo, r);
            hi   = fmaxf(hi, r);
            y[i] = r;
        }
    }
    return median5(y[0], y[1], y[2], y[3], y[4]);
}

// 125 values: five 25-value subtrees in turn (25 loads in flight per lane),
// their results shifted through registers in order.
template <bool ABS>
__device__ __forceinline__ float remedian125(const float* __restrict__ p, uint64_t stride, float level, float& lo,
                                             float& hi) {
    float a = 0.0F, b = 0.0F, c = 0.0F, d = 0.0F, e = 0.0F;
#pragma unroll 1
    for (int j = 0; j < 5; ++j) {
        const float t = remedian25<ABS>(p + 25 * j * stride, stride, level, lo, hi);
        a = b;
        b = c;
        c = d;
        d = e;
        e = t;
    }
    return median5(a, b, c, d, e);
}

/** The 32 channels' remedian over the window's sampled rows (ABS: of |x -
 * level|) in warp 0's lanes; lo, hi the range of this warp's values. */
template <bool ABS>
__device__ __forceinline__ float remedian_rows(const float* __restrict__ src, uint64_t n, int levels, bool in,
                                               float level, float (&part)[25][32], float& lo, float& hi) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int kb       = levels < 3 ? levels : 3; // tree levels inside a block
    const int up       = levels - kb;             // levels over the blocks (0..2)
    const int nblk     = up == 0 ? 1 : up == 1 ? 5 : 25;
    const uint64_t blk = kb == 1 ? 5 : kb == 2 ? 25 : 125; // a window has 5 rows or more
    for (int b = warp; b < nblk; b += kRemedianWarps) {
        const float* p = src + static_cast<uint64_t>(b) * blk * n;
        float v        = 0.0F;
        if (in) {
            switch (kb) {
            case 1: v = remedian5<ABS>(p, n, level, lo, hi); break;
            case 2: v = remedian25<ABS>(p, n, level, lo, hi); break;
            default: v = remedian125<ABS>(p, n, level, lo, hi); break;
            }
        }
        part[b][lane] = v;
    }
    __syncthreads();
    float r = part[0][lane];
    if (warp == 0 && up == 1) {
        r = median5(part[0][lane], part[1][lane], part[2][lane], part[3][lane], part[4][lane]);
    } else if (warp == 0 && up == 2) {
        float v[5];
#pragma unroll
        for (int j = 0; j < 5; ++j)
            v[j] = median5(part[5 * j][lane], part[5 * j + 1][lane], part[5 * j + 2][lane],
                           part[5 * j + 3][lane], part[5 * j + 4][lane]);
        r = median5(v[0], v[1], v[2], v[3], v[4]);
    }
    return r;
}

__global__ void __launch_bounds__(32 * kRemedianWarps)
    k_remedian(Dims d, const float* __restrict__ samples, float* __restrict__ loc, float* __restrict__ scale,
               float* __restrict__ flat_out) {
    __shared__ float part[25][32];
    __shared__ float plo[kRemedianWarps][32], phi[kRemedianWarps][32];
    __shared__ float level_of[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t n = d.nchans;
    const uint64_t c = static_cast<uint64_t>(blockIdx.x) * 32 + lane;
    const uint64_t w = blockIdx.y;
    const bool in    = c < n;
    const uint64_t len = window_end(w, d) - window_begin(w, d.window);
    const uint64_t m   = largest_power_of_five_leq(len < kMaxBandpassRows ? len : kMaxBandpassRows);
    int levels = 0;
    for (uint64_t q = m; q > 1; q /= 5)
        ++levels;
    const uint64_t o = w * n + c;
    const float* src = samples + w * kMaxBandpassRows * n + (in ? c : 0);
    float lo = FLT_MAX, hi = -FLT_MAX, ignored_lo = 0.0F, ignored_hi = 0.0F;
    const float level = remedian_rows<false>(src, n, levels, in, 0.0F, part, lo, hi);
    plo[warp][lane]   = lo;
    phi[warp][lane]   = hi;
    if (warp == 0)
        level_of[lane] = level;
    __syncthreads();
    const float r = remedian_rows<true>(src, n, levels, in, level_of[lane], part, ignored_lo, ignored_hi);
    if (warp != 0 || !in)
        return;
    float a = plo[0][lane], z = phi[0][lane];
#pragma unroll
    for (int k = 1; k < kRemedianWarps; ++k) {
        a = fminf(a, plo[k][lane]);
        z = fmaxf(z, phi[k][lane]);
    }
    loc[o]      = level;
    flat_out[o] = z > a ? 0.0F : 1.0F;
    scale[o]    = r * kMadToStd;
}

// The clipped refinement of the bandpass (lib/cpu/bandpass_kernels.hpp:17-76)
// after the two remedian passes: a lane per channel, a CTA per 32 channels
// of a window. Up to six passes over the sampled rows, each one chain of
// dependent FP64 additions in row order, streamed as rfi_columns.cuh says.
// 1024 channels, 2 windows: 124 us (172 with a warp that copies for itself
// and a loop the compiler orders); 4096 channels, 8 windows: 330 us (240 so,
// with fewer feeders in the walkers' way; 1056 with block-wide stages).
// Each channel updates only while its own sequence of steps is still
// running, so every channel takes the reference's steps whatever the others
// of its warp do. A flat channel (every sampled value equal) keeps its first
// sampled value as its level, as the sequential minimum does.
template <int U, int G> using SampleRing = cols::Ring<32, U, G == 1 ? 64 : 32, 4>;

// The sum over a column, in row order, of d = x - centre where |d| <= cut
// (SQUARE: of (d - shift)^2 there), and how many they are. A sum from +0 is
// never -0, so the +0 of a sample that is not kept leaves it as it is.
template <bool SQUARE, class R>
__device__ __forceinline__ double clipped_sum(const R& rows, double centre, double cut, double shift, uint32_t& kept) {
    constexpr int A = cols::kAhead;
    double sum      = 0.0;
    uint32_t count  = 0;
    uint32_t raw[A];          // row j in raw[j % A], read A rows ahead
    double x[4], d[4], v[2];  // widened 4 rows ahead, differences 3, terms 1
    uint32_t one[2];
    auto term = [&](double& t, uint32_t& o, double dv) {
        if constexpr (SQUARE) {
            double e;
            cols::sub(e, dv, shift);
            cols::mul(e, e, e);
            asm volatile("{\n\t.reg .pred p;\n\t.reg .f64 a;\n\tabs.f64 a, %1;\n\tsetp.le.f64 p, a, %2;\n\t"
                         "selp.f64 %0, %3, 0d0000000000000000, p;\n\t}"
                         : "=d"(t)
                         : "d"(dv), "d"(cut), "d"(e));
            o = 1;
        } else {
            cols::keep(t, o, dv, cut);
        }
    };
    rows.walk(
        [&](uint32_t a) {
#pragma unroll
            for (int j = 0; j < A; ++j)
                raw[j] = rows.bits(a + j * R::kPitch, j);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                cols::widen(x[j], __uint_as_float(raw[j]));
#pragma unroll
            for (int j = 0; j < 3; ++j)
                cols::sub(d[j], x[j], centre);
            term(v[0], one[0], d[0]);
        },
        [&](int r, uint32_t a, uint32_t b) {
#pragma unroll
            for (int j = 0; j < cols::kBatch; ++j) {
                cols::add(sum, sum, v[j & 1]);
                count += one[j & 1];
                raw[j % A] = rows.bits(j + A < cols::kBatch ? a + (j + A) * R::kPitch
                                                            : b + (j + A - cols::kBatch) * R::kPitch, r + j + A);
                cols::sub(d[(j + 3) & 3], x[(j + 3) & 3], centre);
                term(v[(j + 1) & 1], one[(j + 1) & 1], d[(j + 1) & 3]);
                cols::widen(x[j & 3], __uint_as_float(raw[(j + 4) % A]));
            }
        },
        [&](int r, uint32_t a) {
            double dv, t;
            uint32_t o;
            cols::widen(dv, __uint_as_float(rows.bits(a, r)));
            cols::sub(dv, dv, centre);
            term(t, o, dv);
            cols::add(sum, sum, t);
            count += o;
        });
    kept = count;
    return sum;
}

template <int U, int G>
__global__ void __launch_bounds__(32 * (G + 1))
    k_bandpass_refine(Dims d, const float* __restrict__ samples, float* __restrict__ loc_out,
                      float* __restrict__ scale_out, float* __restrict__ inv_out,
                      uint32_t* __restrict__ unmeasured) {
    using R = SampleRing<U, G>;
    extern __shared__ __align__(16) uint8_t rings[]; // [G][R::kBytes]
    const bool feeder    = threadIdx.x < 32;
    const uint64_t first = static_cast<uint64_t>(blockIdx.x) * 32 * G;
    const uint64_t w     = blockIdx.y;
    const uint64_t len   = window_end(w, d) - window_begin(w, d.window);
    const uint64_t m     = largest_power_of_five_leq(len < kMaxBandpassRows ? len : kMaxBandpassRows);
    const uint64_t n     = d.nchans;
    auto ring            = [&](int g) {
        const uint64_t c0 = first + 32 * static_cast<uint64_t>(g);
        return R(rings + g * R::kBytes, reinterpret_cast<const uint8_t*>(samples + w * kMaxBandpassRows * n + c0),
                 n * sizeof(float), c0 < n ? (n - c0) * sizeof(float) : 0, m);
    };
    const uint64_t c = first + threadIdx.x - 32;
    const bool in    = !feeder && c < n;
    const R rows     = ring(feeder ? 0 : static_cast<int>(threadIdx.x >> 5U) - 1);

    const uint64_t o  = w * n + c;
    const float level = in ? loc_out[o] : 0.0F;
    const float rms   = in ? scale_out[o] : 0.0F;
    const bool flat   = in && inv_out[o] != 0.0F;
    if (flat) {
        loc_out[o]   = samples[w * kMaxBandpassRows * n + c];
        scale_out[o] = 0.0F;
        inv_out[o]   = 0.0F;
        atomicAdd(&unmeasured[c], 1U);
    }
    bool live            = in && !flat;
    double centre        = level;
    double sd            = rms;
    const double dm      = static_cast<double>(m);
    const bool need_mean = live && !(sd > 0.0);
    const double all     = __longlong_as_double(0x7FF0000000000000LL); // keeps every sample
    uint32_t kept        = 0;
    if (__syncthreads_or(need_mean)) {
        if (feeder) {
            R::template feed<G>(ring);
            R::template feed<G>(ring);
        } else {
            const double mean = clipped_sum<false>(rows, 0.0, all, 0.0, kept) / dm;
            const double ss   = clipped_sum<true>(rows, 0.0, all, mean, kept);
            if (need_mean)
                sd = sqrt(ss / dm);
        }
    }
    for (int it = 0; it < kClipIterations; ++it) {
        if (!__syncthreads_or(live))
            break;
        const double cut = kClipSigma * sd;
        double sum = 0.0, ss = 0.0;
        if (feeder)
            R::template feed<G>(ring);
        else
            sum = clipped_sum<false>(rows, centre, cut, 0.0, kept);
        const double count = static_cast<double>(kept);
        if (live && count < 2.0)
            live = false;
        const double shift = live ? sum / count : 0.0;
        if (!__syncthreads_or(live))
            break;
        if (feeder) {
            R::template feed<G>(ring);
        } else {
            uint32_t ignored;
            ss = clipped_sum<true>(rows, centre, cut, shift, ignored);
        }
        if (live) {
            const double clipped = sqrt(ss / count);
            if (!(clipped > 0.0)) {
                live = false;
            } else {
                centre += shift;
                sd = clipped;
            }
        }
    }
    if (in && !flat) {
        const float fl = static_cast<float>(centre);
        const float fs = static_cast<float>(sd);
        loc_out[o]     = fl;
        scale_out[o]   = fs;
        inv_out[o]     = 1.0F / fs;
    }
}

// ---- moments --------------------------------------------------------------

// The moments of a window's channels in time order
// (lib/cpu/rfi_cpu_measure.cpp:91-138): nine running sums of z, its powers,
// its product with the previous z and the clipped sums, a lane per channel
// and 32 channels a CTA, streamed as rfi_columns.cuh says. Every sum is its
// own chain of FP64 additions, so ROLES warps of a CTA can keep them apart,
// each reading the same columns: with ROLES = 3 (where groups are few) a
// warp carries two or three sums (z and z^2 are formed again in each), with
// 1 all of them. 1024 float32 channels x 65 536 rows, 2 windows: 425 us
// (1611 with one warp's sums behind block-wide stages); 4096 uint8 channels,
// 8 windows: 1416 us (1976), where 12 FP64 operations a sample bound it.

template <int ROLES, int ROLE, class R, class Z>
__device__ __forceinline__ void moments_walk(const R& rows, Z&& z_of, float clip, MomentSums& out) {
    constexpr bool kLow  = ROLES == 1 || ROLE == 0; // s1, s2, lag
    constexpr bool kHigh = ROLES == 1 || ROLE == 1; // s3, s4
    constexpr bool kClip = ROLES == 1 || ROLE == 2; // nc, c1, c2
    constexpr int A      = cols::kAhead;
    double s1 = 0.0, s2 = 0.0, s3 = 0.0, s4 = 0.0, lag = 0.0, c1 = 0.0, c2 = 0.0;
    uint32_t nc = 0;
    uint32_t raw[A];
    double z[4];                // widened 3 rows ahead
    double z2[2], z3[2], lp[2]; // z^2, z^3 and the lag product a row ahead
    const double wide_clip = clip;
    // the products of row j (z of row j - 1 given) into slot k
    auto products = [&](int k, double zj, double before, bool first) {
        cols::mul(z2[k], zj, zj);
        if constexpr (kLow) {
            cols::mul(lp[k], zj, before);
            if (first)
                lp[k] = 0.0;
        }
        if constexpr (kHigh)
            cols::mul(z3[k], z2[k], zj);
    };
    auto sums = [&](double zj, double q2, double q3, double l) {
        if constexpr (kLow) {
            cols::add(s1, s1, zj);
            cols::add(s2, s2, q2);
            cols::add(lag, lag, l);
        }
        if constexpr (kHigh) {
            double q4;
            cols::mul(q4, q2, q2);
            cols::add(s3, s3, q3);
            cols::add(s4, s4, q4);
        }
        if constexpr (kClip) {
            // sums from +0 are never -0, so adding +0 leaves them as they are
            double k1, k2;
            uint32_t one;
            cols::keep(k1, one, zj, wide_clip);
            k2 = one != 0 ? q2 : 0.0;
            nc += one;
            cols::add(c1, c1, k1);
            cols::add(c2, c2, k2);
        }
    };
    double tail_prev = 0.0;
    rows.walk(
        [&](uint32_t a) {
#pragma unroll
            for (int j = 0; j < A; ++j)
                raw[j] = rows.bits(a + j * R::kPitch, j);
#pragma unroll
            for (int j = 0; j < 3; ++j)
                cols::widen(z[j], z_of(raw[j]));
            products(0, z[0], 0.0, true);
        },
        [&](int r, uint32_t a, uint32_t b) {
#pragma unroll
            for (int j = 0; j < cols::kBatch; ++j) {
                const float ahead = z_of(raw[(j + 3) % A]);
                raw[j % A] = rows.bits(j + A < cols::kBatch ? a + (j + A) * R::kPitch
                                                            : b + (j + A - cols::kBatch) * R::kPitch, r + j + A);
                products((j + 1) & 1, z[(j + 1) & 3], z[j & 3], false);
                cols::widen(z[(j + 3) & 3], ahead);
                sums(z[j & 3], z2[j & 1], z3[j & 1], lp[j & 1]);
            }
            tail_prev = z[(cols::kBatch - 1) & 3];
        },
        [&](int r, uint32_t a) {
            double zj;
            cols::widen(zj, z_of(rows.bits(a, r)));
            products(0, zj, tail_prev, r == 0);
            sums(zj, z2[0], z3[0], lp[0]);
            tail_prev = zj;
        });
    if constexpr (kLow) {
        out.s1  = s1;
        out.s2  = s2;
        out.lag = lag;
    }
    if constexpr (kHigh) {
        out.s3 = s3;
        out.s4 = s4;
    }
    if constexpr (kClip) {
        out.nc = static_cast<double>(nc);
        out.c1 = c1;
        out.c2 = c2;
    }
}

template <int D, int U, int G>
using MomentRing = cols::Ring<static_cast<int>(kBitsOf<D>), U, kBitsOf<D> < 32 ? 128 : G == 1 ? 64 : 32, 4>;

template <int D, int U, int G>
__global__ void __launch_bounds__(G == 1 ? 128 : 32 * (G + 1))
    k_moments(Dims d, const uint8_t* __restrict__ raw, const float* __restrict__ loc, const float* __restrict__ inv,
              const uint8_t* __restrict__ static_mask, float clip, MomentSums* __restrict__ out) {
    using R = MomentRing<D, U, G>;
    constexpr int kRoles = G == 1 ? 3 : 1;
    extern __shared__ __align__(16) uint8_t rings[]; // [G][R::kBytes]
    const int warp       = static_cast<int>(threadIdx.x >> 5U);
    const uint64_t first = static_cast<uint64_t>(blockIdx.x) * 32 * G;
    const uint64_t w     = blockIdx.y;
    const uint64_t b = window_begin(w, d.window), e = window_end(w, d);
    auto ring = [&](int g) {
        const uint64_t c0 = first + 32 * static_cast<uint64_t>(g), off = c0 * kBitsOf<D> / 8;
        return R(rings + g * R::kBytes, raw + b * d.row_bytes + off, d.row_bytes,
                 c0 < d.nchans ? d.row_bytes - off : 0, e - b);
    };
    const int group   = warp == 0 || G == 1 ? 0 : warp - 1;
    const uint64_t c  = first + 32 * static_cast<uint64_t>(group) + (threadIdx.x & 31U);
    const bool in     = warp != 0 && c < d.nchans;
    const uint64_t o  = w * d.nchans + c;
    const float l     = in ? loc[o] : 0.0F;
    const float iv    = in ? inv[o] : 0.0F;
    const bool active = in && static_mask[c] != 0 && iv != 0.0F;
    MomentSums s{0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (__syncthreads_or(active)) {
        if (warp == 0) {
            R::template feed<G>(ring);
            return;
        }
        const R rows = ring(group);
        auto z_of    = [&](uint32_t v) { return (sample_of<D>(v) - l) * iv; };
        if (kRoles == 1 || warp == 1)
            moments_walk<kRoles, 0>(rows, z_of, clip, s);
        else if (warp == 2)
            moments_walk<kRoles, 1>(rows, z_of, clip, s);
        else
            moments_walk<kRoles, 2>(rows, z_of, clip, s);
        if (!active)
            s = MomentSums{0, 0, 0, 0, 0, 0, 0, 0, 0};
    }
    if (!in)
        return;
    MomentSums& to = out[o];
    if (kRoles == 1 || warp == 1) {
        to.n   = active ? static_cast<double>(e - b) : 0.0;
        to.s1  = s.s1;
        to.s2  = s.s2;
        to.lag = s.lag;
    }
    if (kRoles == 1 || warp == 2) {
        to.s3 = s.s3;
        to.s4 = s.s4;
    }
    if (kRoles == 1 || warp == 3) {
        to.nc = s.nc;
        to.c1 = s.c1;
        to.c2 = s.c2;
    }
}

// Channels of a staged segment of the column scan (rfi_stage.cuh).
constexpr int kStageChans = 128;

// ---- row scan ---------------------------------------------------------------

constexpr int kScanRows = 128; // rows per CTA (one thread each)

template <int D> constexpr bool kIntRow = D != FROST_FLOAT32 && kBitsOf<D> <= 16;

// One row of the row scan (lib/cpu/rfi_cpu_measure.cpp:305-446), fed its
// channels in ascending order: the detection series sums and the Kadane
// states across frequency.
// With integer samples of at most 16 bits (INT) the row's sum and sum of
// squares are kept as integers: every partial double sum of such values is
// an integer below 2^53, so the reference's double sums are exact and equal
// the integer ones whatever the order.
template <bool INT, bool W32, bool KSPEC>
struct ScanRowAcc {
    double sum_det = 0.0, sum_keep = 0.0, sx = 0.0, sxx = 0.0;
    uint64_t isx = 0, isxx = 0;
    uint32_t tsx = 0, tsxx = 0;      // W32: the current tile's integer sums
    uint32_t n_keep = 0, n_meas = 0; // counts (exact as doubles when used)
    KadaneBest sp, sn; // rows are scanned whole: only the best runs are needed
    // Channel c, x its sample and xi the integer code (INT: x == xi exactly).
    // A channel that is not used adds 0 everywhere: no branch stands between
    // one channel's sums and the next one's, and a sum that starts at +0 is
    // never -0, so +0 leaves it as it is. A kept cell is not clamped, so one
    // widening serves both sums.
    __device__ __forceinline__ void step(uint32_t c, bool use, float x, uint32_t xi, float l, float ic, float clip) {
        const float zc  = (x - l) * ic;
        const float cl  = clampf(zc, -clip, clip);
        const bool keep = use && fabsf(zc) <= clip;
        const double u  = use ? cl : 0.0F;
        n_meas += use ? 1U : 0U;
        n_keep += keep ? 1U : 0U;
        sum_det += u;
        sum_keep += keep ? u : 0.0;
        if constexpr (INT && W32) {
            const uint32_t v = use ? xi : 0U;
            tsx += v;
            tsxx += v * v;
        } else if constexpr (INT) {
            const uint32_t v = use ? xi : 0U;
            isx += v;
            isxx += static_cast<uint64_t>(v) * v;
        } else {
            const double v = use ? x : 0.0F;
            sx += v;
            sxx += v * v;
        }
        if constexpr (KSPEC) {
            sp.append(static_cast<int32_t>(c), u);
            sn.append(static_cast<int32_t>(c), -u);
        }
    }
    __device__ __forceinline__ void resume() {
        sp.resume();
        sn.resume();
    }
    // W32: moves the tile's integer sums into the 64-bit ones (exact: a tile
    // of at most 1024 codes of at most 8 bits sums below 2^32 even squared)
    __device__ __forceinline__ void flush() {
        isx += tsx;
        isxx += tsxx;
        tsx  = 0;
        tsxx = 0;
    }
    __device__ void finish(const Dims& d, uint64_t t, const KspecParams& kp,
                           const uint64_t* __restrict__ good_prefix, float* __restrict__ s_det,
                           double* __restrict__ s_keep_d, float* __restrict__ s_keep_f,
                           float* __restrict__ row_std, Span32* __restrict__ kspec_pos,
                           Span32* __restrict__ kspec_neg, uint8_t* __restrict__ kspec_whole,
                           uint8_t* __restrict__ row_clip) const {
        const double dn     = n_meas > 1 ? static_cast<double>(n_meas) : 1.0;
        const double s_keep = n_keep > 0 ? sum_keep / static_cast<double>(n_keep) : 0.0;
        const double sx     = INT ? static_cast<double>(isx + tsx) : this->sx;
        const double sxx    = INT ? static_cast<double>(isxx + tsxx) : this->sxx;
        s_det[t]            = static_cast<float>(sum_det / dn);
        s_keep_f[t]         = static_cast<float>(s_keep);
        s_keep_d[t]         = s_keep;
        // a measured cell of this row is past the clip (a narrow-band cell
        // for the apply pass, which computes the same z from the same row,
        // constants and clip)
        row_clip[t] = n_keep != n_meas ? 1 : 0;
        const double mx     = sx / dn;
        const double var    = (sxx / dn) - (mx * mx);
        row_std[t]          = static_cast<float>(sqrt(var < 0.0 ? 0.0 : var));
        if (kp.enabled) {
            // accept_span (lib/cpu/rfi_cpu_measure.cpp:335-349)
            auto accept = [&](const Run& r, Span32& out) -> bool {
                out = {-1, -1};
                if (r.length() <= 0)
                    return false;
                const uint64_t lo    = static_cast<uint64_t>(r.start);
                const uint64_t hi    = static_cast<uint64_t>(r.end);
                const uint64_t count = good_prefix[hi + 1] - good_prefix[lo];
                const double nspan   = static_cast<double>(hi - lo + 1);
                const double snr     = r.sum / sqrt(static_cast<double>(count));
                if (snr > kp.threshold && nspan >= kp.min_bw_chans) {
                    out = {static_cast<int32_t>(lo), static_cast<int32_t>(hi)};
                    return nspan > kp.whole_chans;
                }
                return false;
            };
            Span32 a, b;
            bool whole     = accept(sp.best(), a);
            whole          = accept(sn.best(), b) || whole;
            kspec_pos[t]   = a;
            kspec_neg[t]   = b;
            kspec_whole[t] = whole ? 1 : 0;
        }
    }
};

// 128-byte column tiles of all 128 rows are copied into shared memory
// (cp.async, two tiles deep, three of 32-bit samples), each thread reading
// its own row 16 bytes at a time: rows of any pitch, 16-byte copies where
// the rows are multiples of 16 bytes (U = 16, rows padded to 144 bytes), else
// 4-byte ones from the word the row starts in (U = 4, rows of 33 words, each
// thread shifting its row's bytes into place). A row is one chain over its
// channels; 16 of them are taken at a time, without a branch on the mask.
// Bound by that chain where rows are few and by issue where they are many:
// 1912 uint8 channels (pitch no multiple of 16) x 4289 rows 540 -> 99 us,
// 1536 2-bit x 40 001: 236 -> 122, against a branch a channel and rows
// decoded one sample at a time; 4096 x 262 144 with Kadane across frequency
// 2550 -> 2427 (selects on the integer pipe bound it).
template <int U> constexpr int kRowStride = U == 16 ? 144 : 132;
constexpr int kRowTileBytes = 128;
template <int D> constexpr int kRowTiles = kBitsOf<D> == 32 ? 3 : 2;

template <int D, int U, bool KSPEC>
__global__ void __launch_bounds__(kScanRows)
    k_scan_rows(Dims d, const uint8_t* __restrict__ raw, const float* __restrict__ loc,
                const float* __restrict__ inv, const uint8_t* __restrict__ mask, float clip,
                KspecParams kp, const uint64_t* __restrict__ good_prefix,
                float* __restrict__ s_det, double* __restrict__ s_keep_d,
                float* __restrict__ s_keep_f, float* __restrict__ row_std,
                Span32* __restrict__ kspec_pos, Span32* __restrict__ kspec_neg,
                uint8_t* __restrict__ kspec_whole, uint8_t* __restrict__ row_clip) {
    extern __shared__ __align__(16) uint8_t tiles[]; // [kRowTiles][kScanRows][kRowStride]
    constexpr int kBits   = static_cast<int>(kBitsOf<D>);
    constexpr int kTileCh = kRowTileBytes * 8 / kBits;
    constexpr int kGroup  = kBits == 32 ? 4 : 16;           // channels a step of the loop below
    constexpr int kWords  = kGroup * kBits >= 32 ? kGroup * kBits / 32 : 1; // of packed samples
    constexpr int NT      = kRowTiles<D>;
    const uint64_t t0 = static_cast<uint64_t>(blockIdx.x) * kScanRows;
    const uint64_t t  = t0 + threadIdx.x;
    const bool active = t < d.nsamps;
    const uint32_t n  = static_cast<uint32_t>(d.nchans);
    const uint64_t w  = active ? window_of(t, d.window, d.nwin) : 0;
    const float* lw   = loc + w * n;
    const float* iw   = inv + w * n;
    // 16-byte loads of the window constants and mask need 16-byte aligned rows
    const bool vec = (reinterpret_cast<uintptr_t>(lw) | reinterpret_cast<uintptr_t>(iw) |
                      reinterpret_cast<uintptr_t>(mask)) % 16 == 0;
    const int nrows   = static_cast<int>(d.nsamps - t0 < kScanRows ? d.nsamps - t0 : kScanRows);
    const int ntiles  = static_cast<int>((d.row_bytes + kRowTileBytes - 1) / kRowTileBytes);
    auto issue = [&](int j) {
        if (j < ntiles) {
            const uint64_t b0 = static_cast<uint64_t>(j) * kRowTileBytes;
            const int bytes   = static_cast<int>(d.row_bytes - b0 < kRowTileBytes ? d.row_bytes - b0 : kRowTileBytes);
            uint8_t* dst      = tiles + (j % NT) * kScanRows * kRowStride<U>;
            if constexpr (U == 16) {
                const int chunks = bytes / 16;
                for (int i = threadIdx.x; i < nrows * chunks; i += kScanRows) {
                    const int r = i / chunks, v = i - r * chunks;
                    stage::cp_async16(dst + r * kRowStride<U> + v * 16, raw + (t0 + r) * d.row_bytes + b0 + v * 16);
                }
            } else {
                for (int i = threadIdx.x; i < nrows * 33; i += kScanRows) {
                    const int r      = i / 33, v = i - r * 33;
                    const uint8_t* a = raw + (t0 + r) * d.row_bytes + b0;
                    const int m      = static_cast<int>(reinterpret_cast<uintptr_t>(a) & 3U);
                    const int left   = m + bytes - 4 * v;
                    if (left > 0)
                        cols::cp_async4(dst + r * kRowStride<U> + v * 4, a - m + v * 4, left < 4 ? left : 4);
                }
            }
        }
        stage::commit();
    };
    for (int j = 0; j < NT - 1; ++j)
        issue(j);
    // 8-bit and narrower samples: the integer sums of a tile in 32 bits
    constexpr bool kW32 = kIntRow<D> && kBits <= 8;
    ScanRowAcc<kIntRow<D>, kW32, KSPEC> acc;
    const uint32_t shift = U == 16 ? 0U
                                   : static_cast<uint32_t>((reinterpret_cast<uintptr_t>(raw) + t * (d.row_bytes & 3U)) & 3U) * 8U;
    for (int j = 0; j < ntiles; ++j) {
        issue(j + NT - 1); // into the tile read before the last barrier
        stage::wait_pending<NT - 1>();
        __syncthreads();
        if (active) {
            const uint32_t* row =
                reinterpret_cast<const uint32_t*>(tiles + ((j % NT) * kScanRows + threadIdx.x) * kRowStride<U>);
            const uint32_t cb = static_cast<uint32_t>(j) * kTileCh; // channel indices fit 32 bits
            const uint32_t ce = n - cb < kTileCh ? n : cb + kTileCh;
#pragma unroll 1
            for (uint32_t q = cb; q < ce; q += kGroup) {
                uint32_t words[kWords];
                if constexpr (kGroup * kBits >= 32) {
                    const uint32_t* src = row + (q - cb) * kBits / 32;
                    if constexpr (U == 16 && kWords % 4 == 0) {
#pragma unroll
                        for (int k = 0; k < kWords; k += 4) {
                            const uint4 v = *reinterpret_cast<const uint4*>(src + k);
                            words[k] = v.x, words[k + 1] = v.y, words[k + 2] = v.z, words[k + 3] = v.w;
                        }
                    } else {
#pragma unroll
                        for (int k = 0; k < kWords; ++k)
                            words[k] = U == 16 ? src[k] : __funnelshift_r(src[k], src[k + 1], shift);
                    }
                } else { // 16 1-bit samples: half a word
                    const uint32_t bit = (q - cb) * kBits + shift;
                    words[0] = __funnelshift_r(row[bit >> 5], (bit & 31U) > 16U ? row[(bit >> 5) + 1] : 0U, bit & 31U);
                }
                float ls[kGroup], is[kGroup];
                uint32_t used = 0; // bit e: channel q + e counts
                const uint32_t live = ce - q;
                if (vec && live >= kGroup) {
                    // whole groups: the mask bytes and window constants as vector
                    // loads (the same for every row of the CTA)
#pragma unroll
                    for (int v4 = 0; v4 < kGroup / 4; ++v4) {
                        const float4 x = reinterpret_cast<const float4*>(lw + q)[v4];
                        const float4 y = reinterpret_cast<const float4*>(iw + q)[v4];
                        const uint32_t m = reinterpret_cast<const uint32_t*>(mask + q)[v4];
                        ls[4 * v4] = x.x, ls[4 * v4 + 1] = x.y, ls[4 * v4 + 2] = x.z, ls[4 * v4 + 3] = x.w;
                        is[4 * v4] = y.x, is[4 * v4 + 1] = y.y, is[4 * v4 + 2] = y.z, is[4 * v4 + 3] = y.w;
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            used |= (m >> (8 * e) & 0xFFU) != 0 ? 1U << (4 * v4 + e) : 0U;
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < kGroup; ++e) {
                        const bool in = static_cast<uint32_t>(e) < live;
                        ls[e]         = in ? lw[q + e] : 0.0F;
                        is[e]         = in ? iw[q + e] : 0.0F;
                        used |= in && mask[q + e] != 0 ? 1U << e : 0U;
                    }
                }
                acc.resume();
#pragma unroll
                for (int e = 0; e < kGroup; ++e) {
                    const uint32_t code = kBits == 32 ? words[e]
                                                      : words[e * kBits / 32] >> (e * kBits % 32) & ((1U << (kBits % 32)) - 1U);
                    acc.step(q + e, (used >> e & 1U) != 0 && is[e] != 0.0F, sample_of<D>(code), code, ls[e], is[e], clip);
                }
            }
            if constexpr (kW32)
                acc.flush();
        }
        __syncthreads(); // every thread is done with this tile
    }
    if (active)
        acc.finish(d, t, kp, good_prefix, s_det, s_keep_d, s_keep_f, row_std, kspec_pos, kspec_neg,
                   kspec_whole, row_clip);
}

// One (chunk, channel) sequence of the column scan
// (lib/cpu/rfi_cpu_measure.cpp:305-446): the block min/max of unmeasured
// cells, zdot sums and Kadane-along-time states. The per-(window, channel)
// constants are reloaded only when the window changes; rows are taken a few
// at a time, without a branch where they lie in one window and the channel is
// measured there.
// With Kadane: 4096 uint8 channels x 262 144 rows 3150 -> 2029 us, 479 float32
// channels x 12 734 rows 193 -> 70.
template <bool ZDOT, bool KCHAN>
struct ScanColAcc {
    const Dims* d;
    const float* loc;
    const float* inv;
    const float* clip_mean;
    const float* clip_inv_std;
    const double* s_keep_d;
    uint64_t c;
    float clip;
    uint64_t w = 0, wend = 0; // current window and its end (0: none yet)
    float l = 0.0F, iv = 0.0F, cm = 0.0F, ci = 0.0F;
    float cmin = FLT_MAX, cmax = -FLT_MAX;
    ZdotSums zs{0, 0, 0, 0, 0};
    uint32_t zn = 0;
    KadanePair32 kk; // Kadane along time of u and -u, widened when stored
    // the first sample of an active channel's chunk (every later sample of
    // the chunk follows in order)
    __device__ __forceinline__ void begin(uint64_t t0) {
        if constexpr (KCHAN)
            kk.begin(static_cast<int32_t>(t0));
    }
    __device__ __forceinline__ void enter(uint64_t t) {
        if (t >= wend) {
            w                = window_of(t, d->window, d->nwin);
            wend             = window_end(w, *d);
            const uint64_t o = w * d->nchans + c;
            l                = loc[o];
            iv               = inv[o];
            if constexpr (KCHAN) {
                cm = clip_mean[o];
                ci = clip_inv_std[o];
            }
        }
    }
    /** z's part of the sums; an outlier adds 0 (sums from +0 are never -0). */
    __device__ __forceinline__ void cell(float z, bool measured, uint64_t t) {
        const bool outlier = fabsf(z) > clip;
        if constexpr (ZDOT) {
            const double sk = s_keep_d[t];
            const bool on   = !outlier && measured;
            zn += on ? 1U : 0U; // the count, exact as an integer (stored as a double)
            const double zd = z;
            zs.sz += on ? zd : 0.0;
            zs.ss += on ? sk : 0.0;
            zs.sss += on ? sk * sk : 0.0;
            zs.szs += on ? zd * sk : 0.0;
        }
        if constexpr (KCHAN)
            kk.append(static_cast<int32_t>(t), outlier ? 0.0F : (z - cm) * ci);
    }
    /** N rows from t on, x(j) the j-th sample. */
    template <int N, class X> __device__ __forceinline__ void rows(X&& x, uint64_t t) {
        enter(t);
        if (t + N <= wend && iv != 0.0F) {
#pragma unroll
            for (int j = 0; j < N; ++j)
                cell((x(j) - l) * iv, true, t + j);
            return;
        }
#pragma unroll 1
        for (int j = 0; j < N; ++j) {
            enter(t + j);
            const float v = x(j);
            if (iv == 0.0F) {
                cmin = smin(cmin, v);
                cmax = smax(cmax, v);
            }
            cell(iv == 0.0F ? 0.0F : (v - l) * iv, iv != 0.0F, t + j);
        }
    }
    __device__ __forceinline__ void store(uint64_t k, float* cmin_out, float* cmax_out,
                                          ZdotSums* zs_out, KadaneState* kp_out,
                                          KadaneState* kn_out) const {
        const uint64_t o = k * d->nchans + c;
        cmin_out[o]      = cmin;
        cmax_out[o]      = cmax;
        if constexpr (ZDOT) {
            ZdotSums z = zs;
            z.n        = static_cast<double>(zn);
            zs_out[o]  = z;
        }
        if constexpr (KCHAN) {
            // an active channel appended every sample of the chunk
            const uint64_t t1   = (k + 1) * d->chunk < d->nsamps ? (k + 1) * d->chunk : d->nsamps;
            const int32_t last  = static_cast<int32_t>(t1) - 1;
            kp_out[o] = kk.widen_pos(last);
            kn_out[o] = kk.widen_neg(last);
        }
    }
};

// Without zdot and Kadane the column scan only looks for the range of
// unmeasured cells: whether any of the block's active channels has one in the
// chunk's windows. A whole pass over the raw block is left out where none
// has (64 channels x 4096 samples: 71 us of a 450 us clean, 744 4-bit
// channels x 229 009: 662 us of 3430; the check takes 3).
__device__ __forceinline__ bool block_has_unmeasured(const Dims& d, const float* __restrict__ inv, uint64_t c,
                                                     bool active, uint64_t t0, uint64_t t1) {
    bool some = false;
    if (active && t0 < t1) {
        const uint64_t w1 = window_of(t1 - 1, d.window, d.nwin);
        for (uint64_t w = window_of(t0, d.window, d.nwin); w <= w1; ++w)
            some |= inv[w * d.nchans + c] == 0.0F;
    }
    return __syncthreads_or(some) != 0;
}

template <int D, bool ZDOT, bool KCHAN>
__global__ void k_scan_cols(Dims d, const uint8_t* __restrict__ raw, const float* __restrict__ loc,
                            const float* __restrict__ inv, const uint8_t* __restrict__ mask,
                            float clip, const double* __restrict__ s_keep_d, const float* __restrict__ clip_mean,
                            const float* __restrict__ clip_inv_std, float* __restrict__ cmin_out,
                            float* __restrict__ cmax_out, ZdotSums* __restrict__ zs_out,
                            KadaneState* __restrict__ kp_out, KadaneState* __restrict__ kn_out) {
    const uint64_t c = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
    const uint64_t k = blockIdx.y;
    const bool in    = c < d.nchans;
    const uint64_t t0 = k * d.chunk;
    const uint64_t t1 = (t0 + d.chunk < d.nsamps) ? t0 + d.chunk : d.nsamps;
    const bool walk = ZDOT || KCHAN || block_has_unmeasured(d, inv, c, in && mask[c] != 0, t0, t1);
    if (!in)
        return;
    ScanColAcc<ZDOT, KCHAN> acc{&d, loc, inv, clip_mean, clip_inv_std, s_keep_d, c, clip};
    if (walk && mask[c] != 0) {
        if (t0 < t1)
            acc.begin(t0);
        for (uint64_t tb = t0; tb < t1; tb += kBlock) {
            // fetch kBlock rows ahead of their sequential use
            float xs[kBlock];
#pragma unroll
            for (int q = 0; q < kBlock; ++q)
                xs[q] = tb + q < t1 ? rd<D>(raw + (tb + q) * d.row_bytes, c) : 0.0F;
            if (tb + kBlock <= t1) {
                acc.template rows<kBlock>([&](int j) { return xs[j]; }, tb);
            } else {
#pragma unroll
                for (int q = 0; q < kBlock; ++q)
                    if (tb + q < t1)
                        acc.template rows<1>([&](int) { return xs[q]; }, tb + q);
            }
        }
    }
    acc.store(k, cmin_out, cmax_out, zs_out, kp_out, kn_out);
}

template <int D, bool ZDOT, bool KCHAN>
__global__ void __launch_bounds__(kStageChans)
    k_scan_cols_staged(Dims d, const uint8_t* __restrict__ raw, const float* __restrict__ loc,
                       const float* __restrict__ inv, const uint8_t* __restrict__ mask, float clip,
                       const double* __restrict__ s_keep_d, const float* __restrict__ clip_mean, const float* __restrict__ clip_inv_std,
                       float* __restrict__ cmin_out, float* __restrict__ cmax_out,
                       ZdotSums* __restrict__ zs_out, KadaneState* __restrict__ kp_out,
                       KadaneState* __restrict__ kn_out, int seg_bytes, int rows) {
    extern __shared__ __align__(16) uint8_t stage_buf[];
    const uint64_t c0 = static_cast<uint64_t>(blockIdx.x) * kStageChans;
    const uint64_t c  = c0 + threadIdx.x;
    const uint64_t k  = blockIdx.y;
    const bool in     = c < d.nchans;
    const bool active = in && mask[c] != 0;
    ScanColAcc<ZDOT, KCHAN> acc{&d, loc, inv, clip_mean, clip_inv_std, s_keep_d, c, clip};
    const uint64_t t0   = k * d.chunk;
    const uint64_t t1   = (t0 + d.chunk < d.nsamps) ? t0 + d.chunk : d.nsamps;
    if (!ZDOT && !KCHAN && !block_has_unmeasured(d, inv, c, active, t0, t1)) {
        if (in)
            acc.store(k, cmin_out, cmax_out, zs_out, kp_out, kn_out);
        return;
    }
    const uint64_t off  = c0 * kBitsOf<D> / 8;
    const uint64_t left = d.row_bytes - off;
    const int copy      = static_cast<int>(left < static_cast<uint64_t>(seg_bytes) ? left : seg_bytes);
    stage::Stager st(stage_buf, raw + off, d.row_bytes, seg_bytes, copy, rows, t0, t1);
    if (active && t0 < t1)
        acc.begin(t0);
    st.start();
    for (int kb = 0; kb < st.nblk; ++kb) {
        st.wait(kb);
        const uint8_t* buf = st.buf(kb);
        const int nr       = st.rows_of(kb);
        const uint64_t tb  = st.t0(kb);
        if (active) {
            auto at = [&](int r) { return rd<D>(buf + r * seg_bytes, threadIdx.x); };
            int r   = 0;
#pragma unroll 1
            for (; r + 8 <= nr; r += 8)
                acc.template rows<8>([&](int j) { return at(r + j); }, tb + r);
#pragma unroll 1
            for (; r < nr; ++r)
                acc.template rows<1>([&](int) { return at(r); }, tb + r);
        }
        st.release(kb);
    }
    if (in)
        acc.store(k, cmin_out, cmax_out, zs_out, kp_out, kn_out);
}

// Per channel, in chunk order: the block min/max of unmeasured cells and the
// zdot sums (blockIdx.y 0), the combined Kadane-along-time states of u (1)
// and of -u (2), and of those the best run (lib/cpu/rfi_cpu.cpp:352-366,
// 413-466). A chain of up to 64 states a channel, bound by their loads'
// latency: a warp a CTA, one kind of state each, the next state read while
// one is combined. 1024 channels, 64 chunks: 31 us (209 with all three in one
// thread's turn).
__global__ void __launch_bounds__(32)
    k_combine_chunks(Dims d, int zdot, const float* __restrict__ cmin, const float* __restrict__ cmax,
                     const ZdotSums* __restrict__ zs, const KadaneState* __restrict__ kp,
                     const KadaneState* __restrict__ kn, float* __restrict__ lo_out, float* __restrict__ hi_out,
                     ZdotSums* __restrict__ zs_out, Run* __restrict__ kp_best, Run* __restrict__ kn_best) {
    const uint64_t c = blockIdx.x * 32ULL + threadIdx.x;
    if (c >= d.nchans)
        return;
    const uint64_t n = d.nchans;
    if (blockIdx.y != 0) {
        const KadaneState* in = blockIdx.y == 1 ? kp : kn;
        KadaneState sum = KadaneState::make(), next = in[c];
        for (uint64_t k = 0; k < d.nchunks; ++k) {
            const KadaneState now = next;
            if (k + 1 < d.nchunks)
                next = in[(k + 1) * n + c];
            sum = KadaneState::combine(sum, now);
        }
        (blockIdx.y == 1 ? kp_best : kn_best)[c] = sum.best;
        return;
    }
    float lo = FLT_MAX, hi = -FLT_MAX;
    ZdotSums s{0, 0, 0, 0, 0};
#pragma unroll 4
    for (uint64_t k = 0; k < d.nchunks; ++k) {
        lo = smin(lo, cmin[k * n + c]);
        hi = smax(hi, cmax[k * n + c]);
        if (zdot) {
            const ZdotSums& p = zs[k * n + c];
            s.n += p.n;
            s.sz += p.sz;
            s.ss += p.ss;
            s.sss += p.sss;
            s.szs += p.szs;
        }
    }
    lo_out[c] = lo;
    hi_out[c] = hi;
    if (zdot)
        zs_out[c] = s;
}

// ---- apply ------------------------------------------------------------------

__device__ __forceinline__ float level_of(const ApplyParams& p, float loc, float scale, float v) {
    return p.equalize ? p.eq_loc + (p.eq_scale * v) : loc + (scale * v);
}

// Unflagged rows (lib/cpu/rfi_cpu.cpp:537-624) in two kernels. Every
// measured cell of a row is clean when the row has no span across
// frequency, no cell past the clip (the row scan computed the same z of
// every measured cell from the same row, constants and clip; masks only
// grow after it, so a cell it did not clip is never clipped here) and no
// Kadane-along-time segment covering it. k_apply_clean writes those rows'
// clean values (no cell states, few registers) and lists
// the others; k_apply_unflagged classifies the listed rows' cells, writes
// their values and, where a cell needs one, the fills: a row's samples and
// cell states are staged in shared memory so neighbour draws read them
// without touching HBM again. Masked cells are not written: the normalized
// output zeroes them, so their fill values are never observed.
//
// k_apply_clean is bound by the latency of a row's loads (flags, constants,
// samples) over the loads in flight. A CTA takes a strip of whole rows, at
// least one and up to kStripCells groups of V channels; a thread asks for the
// samples of its kStrip groups, one load each, before the rows' flags are
// read. Without a transform the constants are not read at all: the cleaned
// value is the sample. With one, more groups a thread cost registers and so
// warps: measured over 1, 2 and 4 groups at 4 to 8 CTAs an SM, one group at 8
// is best for a per-row term (4096 uint8 channels x 262 144 rows: 1646 us;
// 2103 with four), two at 6 for a per-cell one (1024 float32 channels x
// 65 536 rows: 153 us; 165 with one, 176 with four). Against a CTA a row that
// always read the constants, and samples one by one for types other than
// uint8: 1620 -> 1646 and 228 -> 153 us; without a transform 1024 uint8
// channels x 65 536 rows 132 -> 75 us, 1536 2-bit channels x 40 001 rows
// 90 -> 80 us.

enum class CleanKind { kCopy, kLevel, kZdot }; // no transform; a per-row term; a per-cell one

// groups of V channels that a thread holds at a time, and CTAs an SM
template <CleanKind K> constexpr int kStrip    = K == CleanKind::kCopy ? 4 : K == CleanKind::kZdot ? 2 : 1;
template <CleanKind K> constexpr int kStripOcc = K == CleanKind::kCopy ? 5 : K == CleanKind::kZdot ? 6 : 8;
constexpr uint64_t kStripCells = 1024; // groups of V channels a CTA takes: whole rows, at least one
constexpr uint64_t kStripRows = 64;

__host__ __device__ inline uint64_t strip_rows(uint64_t nchans, int v) {
    const uint64_t r = kStripCells * static_cast<uint64_t>(v) / nchans;
    return r < 1 ? 1 : r < kStripRows ? r : kStripRows;
}

// V consecutive samples of a row as loaded: one load of 4 (from a multiple of
// 4 channels in a row of whole groups at a 16-byte aligned block) or one
// sample.
template <int D, int V> struct Cells {
    uint4 w;
    __device__ __forceinline__ void load(const uint8_t* __restrict__ in, uint32_t c) {
        if constexpr (V == 1) {
            w.x = __float_as_uint(rd<D>(in, c));
        } else if constexpr (kBitsOf<D> == 32) {
            w = *reinterpret_cast<const uint4*>(in + 4ULL * c);
        } else if constexpr (kBitsOf<D> == 16) {
            const uint2 a = *reinterpret_cast<const uint2*>(in + 2ULL * c);
            w.x = a.x;
            w.y = a.y;
        } else if constexpr (kBitsOf<D> == 8) {
            w.x = *reinterpret_cast<const uint32_t*>(in + c);
        } else if constexpr (kBitsOf<D> == 4) {
            w.x = *reinterpret_cast<const uint16_t*>(in + c / 2);
        } else if constexpr (kBitsOf<D> == 2) {
            w.x = in[c / 4];
        } else {
            w.x = static_cast<uint32_t>(in[c / 8]) >> (c % 8);
        }
    }
    __device__ __forceinline__ float at(int e) const {
        if constexpr (V == 1)
            return __uint_as_float(w.x);
        else if constexpr (D == FROST_FLOAT32)
            return __uint_as_float(e == 0 ? w.x : e == 1 ? w.y : e == 2 ? w.z : w.w);
        else if constexpr (kBitsOf<D> == 32)
            return static_cast<float>(e == 0 ? w.x : e == 1 ? w.y : e == 2 ? w.z : w.w);
        else if constexpr (kBitsOf<D> == 16)
            return static_cast<float>(((e < 2 ? w.x : w.y) >> (16 * (e & 1))) & 0xFFFFU);
        else
            return static_cast<float>((w.x >> (static_cast<int>(kBitsOf<D>) * e)) & ((1U << kBitsOf<D>) - 1U));
    }
};

template <int V> __device__ __forceinline__ void load_cells(const float* __restrict__ p, float (&v)[V]) {
    if constexpr (V == 4) {
        const float4 a = *reinterpret_cast<const float4*>(p);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    } else {
        v[0] = p[0];
    }
}

template <int V> __device__ __forceinline__ void load_cells(const uint8_t* __restrict__ p, uint8_t (&v)[V]) {
    if constexpr (V == 4) {
        const uchar4 a = *reinterpret_cast<const uchar4*>(p);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    } else {
        v[0] = p[0];
    }
}

template <int D, int V, CleanKind K>
__global__ void __launch_bounds__(256, kStripOcc<K>)
    k_apply_clean(Dims d, ApplyParams p, const uint8_t* __restrict__ raw, const float* __restrict__ loc,
                  const float* __restrict__ scale, const float* __restrict__ inv,
                  const uint8_t* __restrict__ mask, const uint8_t* __restrict__ time_flags,
                  const Span32* __restrict__ kspec_pos, const Span32* __restrict__ kspec_neg,
                  const float* __restrict__ s_keep_f, const float* __restrict__ zdot_a,
                  const float* __restrict__ zdot_b, const uint8_t* __restrict__ row_clip,
                  const uint8_t* __restrict__ row_kchan, float* __restrict__ work,
                  uint32_t* __restrict__ slow_rows, unsigned int* __restrict__ nslow) {
    constexpr int S = kStrip<K>;
    __shared__ float sh_term[kStripRows];
    __shared__ int sh_window[kStripRows]; // the row's window, or -1: not written here
    const uint64_t n    = d.nchans;
    const uint32_t n32  = static_cast<uint32_t>(n);
    const uint64_t t0   = blockIdx.x * strip_rows(n, V);
    const uint64_t left = d.nsamps - t0;
    const uint32_t rows = static_cast<uint32_t>(left < strip_rows(n, V) ? left : strip_rows(n, V));
    const uint32_t per  = n32 / V; // groups a row
    const uint32_t all  = rows * per;
    for (uint32_t base = 0; base < all; base += 256 * S) {
        Cells<D, V> x[S];
        uint32_t row[S], c[S];
#pragma unroll
        for (int k = 0; k < S; ++k) {
            const uint32_t i = base + static_cast<uint32_t>(k) * 256 + threadIdx.x;
            row[k]           = rows == 1 ? 0 : i / per;
            c[k]             = (i - row[k] * per) * V;
            if (i < all)
                x[k].load(raw + (t0 + row[k]) * d.row_bytes, c[k]);
        }
        if (base == 0) {
            if (threadIdx.x < rows) {
                const uint64_t t     = t0 + threadIdx.x;
                const bool row_kspec = p.kspec && (kspec_pos[t].lo >= 0 || kspec_neg[t].lo >= 0);
                const bool slow = row_kspec || (p.narrow_active && row_clip[t] != 0) || (p.kchan && row_kchan[t] != 0);
                int w = -1;
                if (time_flags[t] == 0) {
                    if (slow)
                        slow_rows[atomicAdd(nslow, 1U)] = static_cast<uint32_t>(t);
                    else
                        w = static_cast<int>(window_of(t, d.window, d.nwin));
                }
                sh_window[threadIdx.x] = w;
                // z less 0 is z
                sh_term[threadIdx.x] = K == CleanKind::kCopy || p.zero_dm == FROST_ZERO_DM_OFF ? 0.0F : s_keep_f[t];
            }
            __syncthreads();
        }
#pragma unroll
        for (int k = 0; k < S; ++k) {
            const uint32_t i = base + static_cast<uint32_t>(k) * 256 + threadIdx.x;
            const int w      = i < all ? sh_window[row[k]] : -1;
            if (w < 0)
                continue;
            float ls[V], ss[V] = {}, is[V], za[V], zb[V], outv[V];
            uint8_t ms[V];
            const uint64_t o = static_cast<uint64_t>(w) * n + c[k];
            load_cells<V>(mask + c[k], ms);
            if constexpr (K != CleanKind::kCopy) {
                load_cells<V>(loc + o, ls);
                load_cells<V>(inv + o, is);
                if (!p.equalize)
                    load_cells<V>(scale + o, ss);
            }
            if constexpr (K == CleanKind::kZdot) {
                load_cells<V>(zdot_a + c[k], za);
                load_cells<V>(zdot_b + c[k], zb);
            }
            const float sk = sh_term[row[k]];
#pragma unroll
            for (int e = 0; e < V; ++e) {
                const float xe = x[k].at(e);
                float v        = xe;
                if constexpr (K != CleanKind::kCopy) {
                    const float z    = (xe - ls[e]) * is[e];
                    const float term = K == CleanKind::kZdot ? (za[e] * sk) + zb[e] : sk;
                    if (is[e] != 0.0F)
                        v = level_of(p, ls[e], ss[e], z - term);
                }
                outv[e] = ms[e] == 0 ? 0.0F : v;
            }
            float* out = work + (t0 + row[k]) * n + c[k];
            if constexpr (V == 4)
                *reinterpret_cast<float4*>(out) = make_float4(outv[0], outv[1], outv[2], outv[3]);
            else
                out[0] = outv[0];
        }
    }
}

template <int D, int V>
__global__ void k_apply_unflagged(Dims d, ApplyParams p, const uint8_t* __restrict__ raw,
                                  const float* __restrict__ loc, const float* __restrict__ scale,
                                  const float* __restrict__ inv, const uint8_t* __restrict__ mask,
                                  const uint8_t* __restrict__ time_flags,
                                  const Span32* __restrict__ kspec_pos,
                                  const Span32* __restrict__ kspec_neg,
                                  const Segment* __restrict__ kchan_pos,
                                  const Segment* __restrict__ kchan_neg,
                                  const uint8_t* __restrict__ kchan_any,
                                  const float* __restrict__ s_keep_f,
                                  const float* __restrict__ zdot_a,
                                  const float* __restrict__ zdot_b, const uint32_t* __restrict__ slow_rows,
                                  const unsigned int* __restrict__ nslow, float* __restrict__ work,
                                  unsigned long long* __restrict__ counters) {
    extern __shared__ unsigned char smem[];
    const uint64_t n = d.nchans;
    float* sv        = reinterpret_cast<float*>(smem);           // v = z - zero-DM term
    uint8_t* state   = reinterpret_cast<uint8_t*>(sv + n);
    __shared__ unsigned long long cnt[kCountSlots];
    if (threadIdx.x < kCountSlots)
        cnt[threadIdx.x] = 0;
    unsigned long long narrow = 0, nks = 0, nkc = 0, fallbacks = 0;
    const unsigned int nrows = *nslow;
    for (unsigned int i = blockIdx.x; i < nrows; i += gridDim.x) {
        const uint64_t t = slow_rows[i];
        const uint64_t w  = window_of(t, d.window, d.nwin);
        const float* lw   = loc + w * n;
        const float* sw   = scale + w * n;
        const float* iw   = inv + w * n;
        const uint8_t* in = raw + t * d.row_bytes;
        float* out        = work + t * n;
        const float sk    = s_keep_f[t];
        const Span32 ksp  = p.kspec ? kspec_pos[t] : Span32{-1, -1};
        const Span32 ksn  = p.kspec ? kspec_neg[t] : Span32{-1, -1};
        // a row with no Kadane span across frequency (almost every row)
        // skips the per-cell span tests
        const bool row_kspec = ksp.lo >= 0 || ksn.lo >= 0;
        auto span_has     = [](const Span32& s, uint64_t c) {
            return s.lo >= 0 && static_cast<int32_t>(c) >= s.lo && static_cast<int32_t>(c) <= s.hi;
        };
        auto seg_has = [](const Segment& s, uint64_t tt) {
            const int64_t i = static_cast<int64_t>(tt);
            return i >= s.start && i <= s.end;
        };

        // V consecutive channels per thread (V = 4: 16-byte loads of the
        // per-window constants and stores of the row, when nchans % 4 == 0);
        // channel indices fit 32 bits (the launcher checks)
        const uint32_t n32 = static_cast<uint32_t>(n);
        // One pass over the thread's cells: classify each, then either write
        // the row's values (STATES false: every row) or the cell states and
        // zero-DM-corrected values the fills draw from (STATES true: only a
        // row with a cell to fill, recomputed the same way).
        auto cells = [&](auto states_tag) -> bool {
        constexpr bool STATES = decltype(states_tag)::value;
        bool dirty = false; // a cell of this thread's needs a fill
        for (uint32_t cb = threadIdx.x * V; cb < n32; cb += blockDim.x * V) {
            float xs[V], ls[V], ss[V], is[V], outv[V];
            uint8_t ms[V], ka[V];
            if constexpr (V == 4) {
                const float4 l4 = *reinterpret_cast<const float4*>(lw + cb);
                const float4 s4 = *reinterpret_cast<const float4*>(sw + cb);
                const float4 i4 = *reinterpret_cast<const float4*>(iw + cb);
                const uchar4 m4 = *reinterpret_cast<const uchar4*>(mask + cb);
                ls[0] = l4.x; ls[1] = l4.y; ls[2] = l4.z; ls[3] = l4.w;
                ss[0] = s4.x; ss[1] = s4.y; ss[2] = s4.z; ss[3] = s4.w;
                is[0] = i4.x; is[1] = i4.y; is[2] = i4.z; is[3] = i4.w;
                ms[0] = m4.x; ms[1] = m4.y; ms[2] = m4.z; ms[3] = m4.w;
                if (p.kchan) {
                    const uchar4 k4 = *reinterpret_cast<const uchar4*>(kchan_any + cb);
                    ka[0] = k4.x; ka[1] = k4.y; ka[2] = k4.z; ka[3] = k4.w;
                } else {
                    ka[0] = ka[1] = ka[2] = ka[3] = 0;
                }
                if constexpr (D == FROST_UINT8) {
                    const uchar4 x4 = *reinterpret_cast<const uchar4*>(in + cb);
                    xs[0] = static_cast<float>(x4.x); xs[1] = static_cast<float>(x4.y);
                    xs[2] = static_cast<float>(x4.z); xs[3] = static_cast<float>(x4.w);
                } else {
    #pragma unroll
                    for (int e = 0; e < V; ++e)
                        xs[e] = rd<D>(in, cb + e);
                }
            } else {
                ls[0] = lw[cb];
                ss[0] = sw[cb];
                is[0] = iw[cb];
                ms[0] = mask[cb];
                ka[0] = p.kchan ? kchan_any[cb] : 0;
                xs[0] = rd<D>(in, cb);
            }
    #pragma unroll
            for (int e = 0; e < V; ++e) {
                const uint32_t c = cb + e;
                const float x    = xs[e];
                uint8_t st;
                float v = 0.0F;
                outv[e] = 0.0F;
                if (ms[e] == 0) {
                    st = kMasked;
                } else if (is[e] == 0.0F) {
                    st      = kUnmeasured;
                    outv[e] = x;
                } else {
                    const float z = (x - ls[e]) * is[e];
                    if (p.narrow_active && fabsf(z) > p.clip) {
                        st = kNarrow;
                    } else if (row_kspec && (span_has(ksp, c) || span_has(ksn, c))) {
                        st = kKadaneSpectrum;
                    } else if (ka[e] != 0 && (seg_has(kchan_pos[c], t) || seg_has(kchan_neg[c], t))) {
                        st = kKadaneChannel;
                    } else {
                        st = kClean;
                        float term = 0.0F;
                        if (p.zero_dm == FROST_ZERO_DM_SUBTRACT)
                            term = sk;
                        else if (p.zero_dm == FROST_ZERO_DM_ZDOT)
                            term = (zdot_a[c] * sk) + zdot_b[c];
                        v       = z - term;
                        outv[e] = p.transform ? level_of(p, ls[e], ss[e], v) : x;
                    }
                }
                if constexpr (STATES) {
                    state[c] = st;
                    sv[c]    = v;
                }
                dirty = dirty || st == kNarrow || st == kKadaneSpectrum || st == kKadaneChannel;
            }
            // masked and flagged cells are (re)written below or never read
            if constexpr (!STATES) {
                if constexpr (V == 4)
                    *reinterpret_cast<float4*>(out + cb) = make_float4(outv[0], outv[1], outv[2], outv[3]);
                else
                    out[cb] = outv[0];
            }
        }
        return dirty;
        };
        // a row with no cell to fill (almost every row) is done
        if (!__syncthreads_or(cells(std::false_type{})))
            continue;
        cells(std::true_type{});
        __syncthreads(); // every cell state is written before the fills read them

        for (uint32_t c = threadIdx.x; c < n32; c += blockDim.x) {
            const uint8_t st = state[c];
            if (st == kClean || st == kUnmeasured || st == kMasked)
                continue;
            if (st == kNarrow)
                ++narrow;
            else if (st == kKadaneSpectrum)
                ++nks;
            else
                ++nkc;
            if (!p.neighbour) {
                const float v = p.noise ? normal_deviate(draw(p, kStreamNoise, t, c, 0)) : 0.0F;
                out[c]        = level_of(p, lw[c], sw[c], v);
                continue;
            }
            const uint64_t r  = p.chan_fill_radius;
            const uint64_t lo = c > r ? c - r : 0;
            const uint64_t hi = (c + r < n - 1) ? c + r : n - 1;
            float value       = 0.0F;
            bool found        = false;
            for (int a = 0; a < kMaxDraws && !found; ++a) {
                const uint64_t src = uniform_index(draw(p, kStreamCell, t, c, a), lo, hi);
                if (state[src] == kClean) {
                    value = sv[src];
                    found = true;
                }
            }
            fallbacks += found ? 0 : 1;
            out[c] = level_of(p, lw[c], sw[c], value);
        }
        __syncthreads(); // the fills read this row's states before the next row rewrites them
    }
    if (narrow | nks | nkc | fallbacks) {
        atomicAdd(&cnt[kCountNarrow], narrow);
        atomicAdd(&cnt[kCountKspec], nks);
        atomicAdd(&cnt[kCountKchan], nkc);
        atomicAdd(&cnt[kCountFallback], fallbacks);
    }
    __syncthreads();
    if (threadIdx.x < kCountSlots && cnt[threadIdx.x] != 0)
        atomicAdd(&counters[threadIdx.x], cnt[threadIdx.x]);
}

// Flagged rows (lib/cpu/rfi_cpu.cpp:626-715): each copies, per channel,
// from a random unflagged row within the time-fill radius (already final),
// or rebuilds the spectrum in noise units and removes its band mean when a
// zero-DM transform is on. The band-mean sum keeps channel order.
__device__ void apply_flagged_row(const Dims& d, const ApplyParams& p, uint64_t t, const float* __restrict__ loc,
                                  const float* __restrict__ scale, const float* __restrict__ inv,
                                  const uint8_t* __restrict__ mask, const uint8_t* __restrict__ time_flags,
                                  float* __restrict__ work, unsigned long long* __restrict__ counters,
                                  float* sv, uint8_t* contrib, float& s_mean, unsigned long long& s_fallbacks) {
    const uint64_t n = d.nchans;
    if (threadIdx.x == 0)
        s_fallbacks = 0;
    __syncthreads();
    const uint64_t w  = window_of(t, d.window, d.nwin);
    const uint64_t r  = p.time_fill_radius;
    const uint64_t lo = t > r ? t - r : 0;
    const uint64_t hi = (t + r < d.nsamps - 1) ? t + r : d.nsamps - 1;
    const bool rezero = p.zero_dm != FROST_ZERO_DM_OFF;
    float* out        = work + t * n;
    unsigned long long fallbacks = 0;

    for (uint64_t c = threadIdx.x; c < n; c += blockDim.x) {
        contrib[c] = 0;
        sv[c]      = 0.0F;
        if (mask[c] == 0)
            continue;
        float v = 0.0F;
        if (!p.neighbour) {
            v = p.noise ? normal_deviate(draw(p, kStreamNoise, t, c, 0)) : 0.0F;
        } else {
            bool found = false;
            for (int a = 0; a < kMaxDraws && !found; ++a) {
                const uint64_t src = uniform_index(draw(p, kStreamTime, t, c, a), lo, hi);
                if (time_flags[src] != 0)
                    continue;
                found = true;
                const float sval = work[src * n + c];
                if (rezero) {
                    const uint64_t ws = window_of(src, d.window, d.nwin);
                    v = p.equalize ? (sval - p.eq_loc) / p.eq_scale
                                   : (sval - loc[ws * n + c]) * inv[ws * n + c];
                } else {
                    out[c] = sval;
                }
            }
            if (!found)
                ++fallbacks;
            if (found && !rezero)
                continue;
        }
        sv[c] = v;
        if (rezero) {
            contrib[c] = inv[w * n + c] != 0.0F ? 1 : 0;
        } else {
            out[c] = level_of(p, loc[w * n + c], scale[w * n + c], v);
        }
    }
    if (fallbacks)
        atomicAdd(&s_fallbacks, fallbacks);
    __syncthreads();
    if (rezero) {
        if (threadIdx.x == 0) {
            double sum = 0.0, count = 0.0;
            for (uint64_t c = 0; c < n; ++c) {
                if (contrib[c]) {
                    sum += sv[c];
                    count += 1.0;
                }
            }
            s_mean = static_cast<float>(count > 0.0 ? sum / count : 0.0);
        }
        __syncthreads();
        // Float samples: quantisation is the identity, so the carried
        // rounding error of lib/cpu/rfi_cpu.cpp:704-713 stays +0.
        for (uint64_t c = threadIdx.x; c < n; c += blockDim.x) {
            if (mask[c] == 0)
                continue;
            out[c] = level_of(p, loc[w * n + c], scale[w * n + c], sv[c] - s_mean) + 0.0F;
        }
    }
    if (threadIdx.x == 0 && s_fallbacks)
        atomicAdd(&counters[kCountFallback], s_fallbacks);
    __syncthreads();
}

// The flagged rows listed in flagged[0 .. *count), a row per CTA at a time
// (the count is known only on the device).
__global__ void k_apply_flagged(Dims d, ApplyParams p, const uint64_t* __restrict__ flagged,
                                const unsigned long long* __restrict__ count, const float* __restrict__ loc,
                                const float* __restrict__ scale, const float* __restrict__ inv,
                                const uint8_t* __restrict__ mask, const uint8_t* __restrict__ time_flags,
                                float* __restrict__ work, unsigned long long* __restrict__ counters) {
    extern __shared__ unsigned char smem[];
    float* sv        = reinterpret_cast<float*>(smem);
    uint8_t* contrib = reinterpret_cast<uint8_t*>(sv + d.nchans);
    __shared__ float s_mean;
    __shared__ unsigned long long s_fallbacks;
    const unsigned long long rows = *count;
    for (unsigned long long i = blockIdx.x; i < rows; i += gridDim.x)
        apply_flagged_row(d, p, flagged[i], loc, scale, inv, mask, time_flags, work, counters, sv, contrib, s_mean,
                          s_fallbacks);
}

// ---- re-measure and normalise ---------------------------------------------

template <int D>
__global__ void k_unpack(Dims d, const uint8_t* __restrict__ raw, float* __restrict__ work) {
    const uint64_t i      = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
    const uint64_t total  = d.nsamps * d.nchans;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t j = i; j < total; j += stride) {
        const uint64_t t = j / d.nchans, c = j % d.nchans;
        work[j]          = rd<D>(raw + t * d.row_bytes, c);
    }
}

// Division in the Welford re-measure. The reference updates
// mean += (x - mean) / n in double. A dependent double division costs
// ~400 cycles on sm_100; the division by the count is instead
// q = RN(delta * y_hi + RN(delta * y_lo)) (one multiply, one fused
// multiply-add), with y_hi = RN(1/n) and y_lo = RN((1 - n y_hi) / n) from
// the host (1 - n y_hi is exact in double). y_hi + y_lo is within 2^-105 / n
// of 1/n and the product's rounding adds at most 2^-105 |delta| / n, so the
// value rounded is within 2^-104 relative of delta / n; delta / n is never a
// rounding midpoint (n delta-midpoint products need more than 53 bits) and
// lies at least 2^-54 / n relative from every midpoint, far more than
// 2^-104 for n < 2^40, so q is the correctly rounded quotient, as
// Markstein-style corrections argue (P. Markstein, IBM J. Res. Develop. 34,
// 1990; Muller et al., Handbook of Floating-Point Arithmetic, ch. 4).
//
// A nonzero delta is never so small that delta * y_lo loses bits, so the
// form needs no branch. Samples are floats: zero or at least 2^-149. Let m
// be the mean before a row n < 2^31. A row x != 0 leaves |mean| >= 2^-236
// or 0: with |m| <= 2^-183, |q| >= 2^-182 outweighs m; else m is a multiple
// of 2^-235, and q is either below 2^-184 or a multiple of 2^-236. Rows of
// zeros scale the mean by the product of (1 - 1/n), at least 2^-32 in all.
// So a nonzero mean stays above 2^-268 and is a multiple of 2^-320, as is
// x - mean: delta * y_lo is a normal number.

// The Welford statistics of the re-measure after a transform
// (lib/cpu/rfi_cpu.cpp:219-238): a lane per channel, a CTA per 32 channels
// of a window; a row's samples and its count's two-term reciprocal are
// streamed together (rfi_columns.cuh). Bound by the chain of four dependent
// FP64 operations a row (32 cycles) where groups are few, by issue where
// they are many. The mean never becomes -0 (it starts at +0 and a rounded
// sum is -0 only when both terms are), so a zero quotient (delta = +-0)
// leaves it unchanged without a select. var's increment is added a row late,
// in the chain's gaps. 1024 channels x 65 536 rows, 2 windows: 702 us (2276
// before: 126 cycles a row); 4096 channels, 8 windows: 1274 us (2979).
template <int U, int G> using WorkRing = cols::Ring<32, U, G == 1 ? 64 : 32, 4, true>;

template <int U, int G>
__global__ void __launch_bounds__(32 * (G + 1))
    k_welford(Dims d, const float* __restrict__ work, const double* __restrict__ recip, float* __restrict__ loc,
              float* __restrict__ scale) {
    using R = WorkRing<U, G>;
    extern __shared__ __align__(16) uint8_t rings[]; // [G][R::kBytes], the records
    const uint64_t first = static_cast<uint64_t>(blockIdx.x) * 32 * G;
    const uint64_t w     = blockIdx.y;
    const uint64_t n     = d.nchans;
    const uint64_t b = window_begin(w, d.window), e = window_end(w, d);
    auto ring = [&](int g) {
        const uint64_t c0 = first + 32 * static_cast<uint64_t>(g);
        // record r: the reciprocal of r + 1
        return R(rings + g * R::kBytes, reinterpret_cast<const uint8_t*>(work + b * n + c0), n * sizeof(float),
                 c0 < n ? (n - c0) * sizeof(float) : 0, e - b, rings + G * R::kBytes,
                 g == 0 ? reinterpret_cast<const double2*>(recip) + 1 : nullptr);
    };
    if (threadIdx.x < 32) {
        R::template feed<G>(ring);
        return;
    }
    const uint64_t c = first + threadIdx.x - 32;
    const R rows     = ring(static_cast<int>(threadIdx.x >> 5U) - 1);
    constexpr int A = cols::kAhead;
    double mean = 0.0, var = 0.0;
    double pd = 0.0, pr = 0.0; // the last row's delta and x - mean
    uint32_t raw[A];
    double x[2], yh[4], yl[4]; // widened 2 rows ahead, reciprocals read 4
    rows.walk(
        [&](uint32_t a) {
#pragma unroll
            for (int j = 0; j < A; ++j)
                raw[j] = rows.bits(a + j * R::kPitch, j);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                cols::pair(yh[j], yl[j], rows.record(j));
            cols::widen(x[0], __uint_as_float(raw[0]));
            cols::widen(x[1], __uint_as_float(raw[1]));
        },
        [&](int r, uint32_t a, uint32_t after) {
            const uint32_t ya = rows.record(r), yb = rows.record(r + cols::kBatch);
#pragma unroll
            for (int j = 0; j < cols::kBatch; ++j) {
                double delta, u, q, pv;
                const double xj = x[j & 1];
                cols::sub(delta, xj, mean);
                raw[j % A] = rows.bits(j + A < cols::kBatch ? a + (j + A) * R::kPitch
                                                            : after + (j + A - cols::kBatch) * R::kPitch, r + j + A);
                cols::mul(pv, pd, pr);
                cols::mul(u, delta, yl[j & 3]);
                cols::widen(x[j & 1], __uint_as_float(raw[(j + 2) % A]));
                cols::add(var, var, pv);
                cols::fma(q, delta, yh[j & 3], u);
                cols::pair(yh[j & 3], yl[j & 3], j + 4 < cols::kBatch ? ya + (j + 4) * 16
                                                                      : yb + (j + 4 - cols::kBatch) * 16);
                pd = delta;
                cols::add(mean, mean, q);
                cols::sub(pr, xj, mean);
            }
        },
        [&](int r, uint32_t a) {
            var += pd * pr;
            const double xj    = __uint_as_float(rows.bits(a, r));
            const double delta = xj - mean;
            double h, l;
            cols::pair(h, l, rows.record(r));
            mean += ::fma(delta, h, delta * l);
            pd = delta;
            pr = xj - mean;
        });
    var += pd * pr;
    if (c < d.nchans) {
        loc[w * d.nchans + c]   = static_cast<float>(mean);
        scale[w * d.nchans + c] = e > b ? static_cast<float>(sqrt(var / static_cast<double>(e - b))) : 0.0F;
    }
}

// Normalise + transpose (lib/cpu/rfi_cpu.cpp:242-255): out[c][t] =
// (work[t][c] - loc) * (scale > 0 ? 1 / scale : 1) per (window, channel),
// masked channels and rows past the valid ones zero, so that every float of
// out is written. A block covers 64 channels and kNormSpan samples in 64 x
// 64 tiles through shared memory; each thread keeps its channels' window
// constants and reloads them only when its rows cross into the next window.
// Bound by HBM (4 bytes in and out a cell); 16 bytes a load where the
// channels are a multiple of 4 (VL) and a store where the capacity is (VS),
// else one float a lane and 16 in flight a thread. 1536 channels x 40 001
// samples: 284 us with 32 x 32 tiles and four loads in flight, 133 us here; 4096 x
// 262 144: 1750 -> 1386 us.
constexpr int kNormSpan = 256;
constexpr int kNT       = 64;

template <bool VL, bool VS>
__global__ void __launch_bounds__(256)
    k_normalize(Dims d, const float* __restrict__ work, const float* __restrict__ loc,
                const float* __restrict__ scale, const uint8_t* __restrict__ mask, int flip,
                uint64_t capacity, float* __restrict__ out) {
    __shared__ float tile[kNT][kNT + 1]; // [channel][time]
    constexpr int E     = VL ? 4 : 1;            // channels a load
    constexpr int kRows = VL ? 16 : 4;           // rows the block loads at once
    const uint64_t n  = d.nchans;
    const uint64_t c0 = static_cast<uint64_t>(blockIdx.y) * kNT;
    const int q       = threadIdx.x % (kNT / E); // channels E q .. of the tile
    const int r       = threadIdx.x / (kNT / E);
    const uint64_t c  = c0 + E * q;
    bool on[E];
#pragma unroll
    for (int e = 0; e < E; ++e)
        on[e] = c + e < n && mask[c + e] != 0;
    uint64_t wend = 0;
    float l[E], is[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        l[e]  = 0.0F;
        is[e] = 1.0F;
    }
    const uint64_t span0 = static_cast<uint64_t>(blockIdx.x) * kNormSpan;
    for (uint64_t t0 = span0; t0 < span0 + kNormSpan && t0 < capacity; t0 += kNT) {
        float x[kNT / kRows][E];
#pragma unroll
        for (int pass = 0; pass < kNT / kRows; ++pass) {
            const uint64_t t = t0 + r + kRows * pass;
#pragma unroll
            for (int e = 0; e < E; ++e)
                x[pass][e] = 0.0F;
            if (t < d.nsamps && c < n) {
                if constexpr (VL) {
                    const float4 v = *reinterpret_cast<const float4*>(work + t * n + c);
                    x[pass][0] = v.x, x[pass][1] = v.y, x[pass][2] = v.z, x[pass][3] = v.w;
                } else {
                    x[pass][0] = work[t * n + c];
                }
            }
        }
#pragma unroll
        for (int pass = 0; pass < kNT / kRows; ++pass) {
            const int tl     = r + kRows * pass;
            const uint64_t t = t0 + tl;
            float v[E];
#pragma unroll
            for (int e = 0; e < E; ++e)
                v[e] = 0.0F;
            if (t < d.nsamps && c < n) {
                if (t >= wend) {
                    const uint64_t w = window_of(t, d.window, d.nwin);
                    wend             = window_end(w, d);
#pragma unroll
                    for (int e = 0; e < E; ++e) {
                        l[e]           = loc[w * n + c + e];
                        const float sc = scale[w * n + c + e];
                        is[e]          = sc > 0.0F ? 1.0F / sc : 1.0F;
                    }
                }
#pragma unroll
                for (int e = 0; e < E; ++e)
                    v[e] = on[e] ? (x[pass][e] - l[e]) * is[e] : 0.0F;
            }
#pragma unroll
            for (int e = 0; e < E; ++e)
                tile[E * q + e][tl] = v[e];
        }
        __syncthreads();
        if constexpr (VS) {
            const int tq     = threadIdx.x % 16;
            const uint64_t t = t0 + 4 * tq;
            if (t < capacity) {
#pragma unroll
                for (int pass = 0; pass < kNT / 16; ++pass) {
                    const int cl      = threadIdx.x / 16 + 16 * pass;
                    const uint64_t cc = c0 + cl;
                    if (cc < n) {
                        const uint64_t dst = flip ? n - 1 - cc : cc;
                        const float4 o = make_float4(tile[cl][4 * tq], tile[cl][4 * tq + 1], tile[cl][4 * tq + 2],
                                                     tile[cl][4 * tq + 3]);
                        *reinterpret_cast<float4*>(out + dst * capacity + t) = o;
                    }
                }
            }
        } else {
            const int tl     = threadIdx.x % kNT;
            const uint64_t t = t0 + tl;
            if (t < capacity) {
#pragma unroll
                for (int pass = 0; pass < kNT / 4; ++pass) {
                    const int cl      = threadIdx.x / kNT + 4 * pass;
                    const uint64_t cc = c0 + cl;
                    if (cc < n)
                        out[(flip ? n - 1 - cc : cc) * capacity + t] = tile[cl][tl];
                }
            }
        }
        __syncthreads();
    }
}

__global__ void k_normalize_short(Dims d, ApplyParams p, const float* __restrict__ work,
                                  const float* __restrict__ tl, const float* __restrict__ ts,
                                  const float* __restrict__ tol, const float* __restrict__ tos,
                                  const uint8_t* __restrict__ mask, const float* __restrict__ za,
                                  const float* __restrict__ zb, int flip, uint64_t capacity,
                                  float* __restrict__ out) {
    extern __shared__ unsigned char smem[];
    const uint64_t n = d.nchans;
    float* z         = reinterpret_cast<float*>(smem);
    __shared__ float band_mean;
    const uint64_t t = blockIdx.x;
    for (uint64_t c = threadIdx.x; c < n; c += blockDim.x)
        z[c] = (work[t * n + c] - tl[c]) * (ts[c] > 0.0F ? 1.0F / ts[c] : 1.0F);
    __syncthreads();
    if (threadIdx.x == 0) {
        double sum     = 0.0;
        uint64_t count = 0;
        for (uint64_t c = 0; c < n; ++c) {
            if (mask[c] && ts[c] > 0.0F && fabsf(z[c]) <= p.clip) {
                sum += z[c];
                ++count;
            }
        }
        band_mean = count ? static_cast<float>(sum / static_cast<double>(count)) : 0.0F;
    }
    __syncthreads();
    for (uint64_t c = threadIdx.x; c < n; c += blockDim.x) {
        if (!mask[c])
            continue;
        float term = 0.0F;
        if (p.zero_dm == FROST_ZERO_DM_SUBTRACT)
            term = band_mean;
        else if (p.zero_dm == FROST_ZERO_DM_ZDOT)
            term = za[c] * band_mean + zb[c];
        const float x = work[t * n + c];
        const float transformed = ts[c] <= 0.0F ? x
                                  : p.equalize  ? p.eq_loc + p.eq_scale * (z[c] - term)
                                  : p.transform ? tl[c] + ts[c] * (z[c] - term)
                                                : x;
        const float s      = tos[c] > 0.0F ? 1.0F / tos[c] : 1.0F;
        const uint64_t dst = flip ? n - 1 - c : c;
        out[dst * capacity + t] = (transformed - tol[c]) * s;
    }
}

unsigned grid1(uint64_t n, unsigned block) { return static_cast<unsigned>((n + block - 1) / block); }

std::atomic<uint64_t> g_launches{0};

} // namespace

#define FB_COUNT_LAUNCH()                                                                         \
    do {                                                                                          \
        FB_LAUNCH_CHECK();                                                                        \
        g_launches.fetch_add(1, std::memory_order_relaxed);                                       \
    } while (0)

uint64_t launch_counter() { return g_launches.load(std::memory_order_relaxed); }

// ---- launchers ----------------------------------------------------------------

static void set_smem(const void* fn, size_t bytes) {
    if (bytes > 48 * 1024)
        allow_large_smem(fn);
}

// f(copy bytes, groups a CTA) for a column kernel of `groups` 32-channel
// groups, one a CTA while they are no more than `per_sm` an SM.
template <int WIDE = 16, class F> static void on_groups(uint64_t groups, uint64_t per_sm, bool aligned, F&& f) {
    using One  = std::integral_constant<int, 1>;
    using Many = std::integral_constant<int, cols::kManyGroups>;
    const bool few = cols::few_groups(groups, per_sm);
    if (aligned && few)
        f(std::integral_constant<int, WIDE>{}, One{});
    else if (aligned)
        f(std::integral_constant<int, WIDE>{}, Many{});
    else if (few)
        f(std::integral_constant<int, 4>{}, One{});
    else
        f(std::integral_constant<int, 4>{}, Many{});
}

void launch_check_finite(const uint8_t* raw, uint64_t nwords, unsigned long long* first_bad,
                         cudaStream_t s) {
    if (nwords == 0)
        return;
    const uint64_t head   = std::min<uint64_t>(nwords, (16 - reinterpret_cast<uintptr_t>(raw) % 16) % 16 / 4);
    const unsigned blocks = static_cast<unsigned>(std::min<uint64_t>((nwords + 4095) / 4096, 8 * sm_count()));
    k_check_finite<<<blocks, 256, 0, s>>>(reinterpret_cast<const uint32_t*>(raw), nwords, head, first_bad);
    FB_COUNT_LAUNCH();
}

void launch_begin(const Dims& d, unsigned long long* counters, uint64_t nslots, uint32_t* unmeasured,
                  uint8_t* kchan_any, uint8_t* time_flags, uint8_t* row_kchan, unsigned int* nslow, cudaStream_t s) {
    const uint64_t most   = std::max({nslots, d.nchans, d.nsamps, uint64_t{1}});
    const unsigned blocks = static_cast<unsigned>(std::min<uint64_t>((most + 255) / 256, 4 * sm_count()));
    k_begin<<<blocks, 256, 0, s>>>(counters, nslots, unmeasured, kchan_any, d.nchans, time_flags, row_kchan, d.nsamps,
                                   nslow);
    FB_COUNT_LAUNCH();
}

void launch_keep_tail(uint64_t nchans, const float* loc, const float* scale, const float* out_loc,
                      const float* out_scale, float* tail_loc, float* tail_scale, float* tail_out_loc,
                      float* tail_out_scale, cudaStream_t s) {
    if (nchans == 0)
        return;
    k_keep_tail<<<grid1(nchans, 256), 256, 0, s>>>(nchans, loc, scale, out_loc, out_scale, tail_loc, tail_scale,
                                                   tail_out_loc, tail_out_scale);
    FB_COUNT_LAUNCH();
}

void launch_sample_rows(const Dims& d, const uint8_t* raw, float* samples, cudaStream_t s) {
    const dim3 grid(kMaxBandpassRows, static_cast<unsigned>(d.nwin));
    FB_DISPATCH(d.dtype, k_sample_rows<D><<<grid, 256, 0, s>>>(d, raw, samples));
    FB_COUNT_LAUNCH();
}

void launch_bandpass(const Dims& d, const float* samples, float* loc, float* scale, float* inv,
                     uint32_t* unmeasured, cudaStream_t s) {
    // level, flat flag and scale, then the clipped refinement
    const dim3 grid(grid1(d.nchans, 32), static_cast<unsigned>(d.nwin));
    k_remedian<<<grid, 32 * kRemedianWarps, 0, s>>>(d, samples, loc, scale, inv);
    FB_COUNT_LAUNCH();
    auto refine = [&](auto u, auto groups) {
        constexpr int U = decltype(u)::value, G = decltype(groups)::value;
        constexpr size_t smem = G * SampleRing<U, G>::kBytes;
        set_smem(reinterpret_cast<const void*>(&k_bandpass_refine<U, G>), smem);
        const dim3 g(grid1(d.nchans, 32 * G), static_cast<unsigned>(d.nwin));
        k_bandpass_refine<U, G><<<g, 32 * (G + 1), smem, s>>>(d, samples, loc, scale, inv, unmeasured);
    };
    on_groups(static_cast<uint64_t>(grid.x) * grid.y, cols::kBandpassFew,
              d.nchans % 4 == 0 && reinterpret_cast<uintptr_t>(samples) % 16 == 0, refine);
    FB_COUNT_LAUNCH();
}

// Staging geometry of a kStageChans-channel column segment: bytes per row
// and rows per stage (about kStageBytes per buffer), or seg_bytes = 0 when
// the layout cannot be staged with 16-byte copies.
constexpr int kStageBytes = 16 * 1024;

struct StageGeom {
    int seg_bytes = 0, rows = 0;
    size_t smem() const { return 2 * static_cast<size_t>(seg_bytes) * rows; }
};

bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

StageGeom stage_geom(const void* base, uint64_t row_bytes, int bits) {
    StageGeom g;
    const uint64_t full = static_cast<uint64_t>(kStageChans) * bits / 8;
    if (!aligned16(base) || row_bytes % 16 != 0 || full % 16 != 0)
        return g;
    // every segment starts on a 16-byte boundary; the last may be shorter
    g.seg_bytes = static_cast<int>(std::min<uint64_t>(full, row_bytes));
    g.rows      = std::max(8, std::min(256, kStageBytes / g.seg_bytes));
    return g;
}

void launch_moments(const Dims& d, const uint8_t* raw, const float* loc, const float* inv,
                    const uint8_t* static_mask, float clip, MomentSums* out, cudaStream_t s) {
    FB_DISPATCH(d.dtype, {
        constexpr int kWide = kBitsOf<D> >= 4 ? 16 : 4; // 32 narrower samples are no 16 bytes
        on_groups<kWide>(grid1(d.nchans, 32) * d.nwin, cols::kMomentsFew, aligned16(raw) && d.row_bytes % 16 == 0,
                         [&](auto u, auto groups) {
                             constexpr int U = decltype(u)::value, G = decltype(groups)::value;
                             constexpr size_t smem = G * MomentRing<D, U, G>::kBytes;
                             set_smem(reinterpret_cast<const void*>(&k_moments<D, U, G>), smem);
                             const dim3 g(grid1(d.nchans, 32 * G), static_cast<unsigned>(d.nwin));
                             k_moments<D, U, G><<<g, G == 1 ? 128 : 32 * (G + 1), smem, s>>>(
                                 d, raw, loc, inv, static_mask, clip, out);
                         });
    });
    FB_COUNT_LAUNCH();
}

void launch_scan_rows(const Dims& d, const uint8_t* raw, const float* loc, const float* inv,
                      const uint8_t* mask, float clip, const KspecParams& kp,
                      const uint64_t* good_prefix, float* s_det, double* s_keep_d, float* s_keep_f,
                      float* row_std, Span32* kspec_pos, Span32* kspec_neg, uint8_t* kspec_whole,
                      uint8_t* row_clip, cudaStream_t s) {
    if (d.nchans >= (uint64_t{1} << 31))
        throw Error(FROST_ERR_INVALID_ARGUMENT, "scan: too many channels for 32-bit channel indices");
    const unsigned grid = grid1(d.nsamps, kScanRows);
    const bool wide     = d.row_bytes % 16 == 0 && aligned16(raw);
    FB_DISPATCH(d.dtype, {
        auto go = [&](auto u, auto kspec) {
            constexpr int U       = decltype(u)::value;
            constexpr size_t smem = static_cast<size_t>(kRowTiles<D>) * kScanRows * kRowStride<U>;
            const auto k          = &k_scan_rows<D, U, decltype(kspec)::value>;
            set_smem(reinterpret_cast<const void*>(k), smem);
            k<<<grid, kScanRows, smem, s>>>(d, raw, loc, inv, mask, clip, kp, good_prefix, s_det, s_keep_d, s_keep_f,
                                            row_std, kspec_pos, kspec_neg, kspec_whole, row_clip);
        };
        auto with = [&](auto u) { kp.enabled ? go(u, std::true_type{}) : go(u, std::false_type{}); };
        wide ? with(std::integral_constant<int, 16>{}) : with(std::integral_constant<int, 4>{});
    });
    FB_COUNT_LAUNCH();
}

void launch_scan_cols(const Dims& d, const uint8_t* raw, const float* loc, const float* inv,
                      const uint8_t* mask, float clip, const double* s_keep_d, int zdot, int kchan,
                      const float* clip_mean, const float* clip_inv_std, float* chunk_min,
                      float* chunk_max, ZdotSums* chunk_zdot, KadaneState* chunk_kpos,
                      KadaneState* chunk_kneg, float* lo, float* hi, ZdotSums* zdot_sum,
                      Run* kpos_best, Run* kneg_best, cudaStream_t s) {
    if (d.nsamps >= (uint64_t{1} << 31))
        throw Error(FROST_ERR_INVALID_ARGUMENT, "scan: too many samples for 32-bit time indices");
    const StageGeom g = stage_geom(raw, d.row_bytes, bits_of(d.dtype));
    FB_DISPATCH(d.dtype, {
        auto go = [&](auto z, auto kc) {
            constexpr bool ZDOT = decltype(z)::value, KCHAN = decltype(kc)::value;
            if (g.seg_bytes == 0) {
                const dim3 grid(grid1(d.nchans, 64), static_cast<unsigned>(d.nchunks));
                k_scan_cols<D, ZDOT, KCHAN><<<grid, 64, 0, s>>>(d, raw, loc, inv, mask, clip, s_keep_d, clip_mean,
                                                                clip_inv_std, chunk_min, chunk_max, chunk_zdot,
                                                                chunk_kpos, chunk_kneg);
            } else {
                const dim3 grid(grid1(d.nchans, kStageChans), static_cast<unsigned>(d.nchunks));
                k_scan_cols_staged<D, ZDOT, KCHAN><<<grid, kStageChans, g.smem(), s>>>(
                    d, raw, loc, inv, mask, clip, s_keep_d, clip_mean, clip_inv_std, chunk_min, chunk_max, chunk_zdot,
                    chunk_kpos, chunk_kneg, g.seg_bytes, g.rows);
            }
        };
        if (zdot)
            kchan ? go(std::true_type{}, std::true_type{}) : go(std::true_type{}, std::false_type{});
        else
            kchan ? go(std::false_type{}, std::true_type{}) : go(std::false_type{}, std::false_type{});
    });
    FB_COUNT_LAUNCH();
    k_combine_chunks<<<dim3(grid1(d.nchans, 32), kchan ? 3 : 1), 32, 0, s>>>(
        d, zdot, chunk_min, chunk_max, chunk_zdot, chunk_kpos, chunk_kneg, lo, hi, zdot_sum, kpos_best, kneg_best);
    FB_COUNT_LAUNCH();
}


namespace {
// row_kchan[t] = 1 for the rows a channel's Kadane-along-time segment
// covers (the caller zeroes it): CTA 2c + k takes channel c's positive
// (k = 0) or negative segment.
__global__ void __launch_bounds__(256)
    k_kchan_rows(uint64_t nchans, uint64_t nsamps, const Segment* __restrict__ kchan_pos,
                 const Segment* __restrict__ kchan_neg, const uint8_t* __restrict__ kchan_any,
                 uint8_t* __restrict__ row_kchan) {
    const uint64_t c = blockIdx.x >> 1;
    if (c >= nchans || kchan_any[c] == 0)
        return;
    const Segment g  = (blockIdx.x & 1) == 0 ? kchan_pos[c] : kchan_neg[c];
    const int64_t lo = g.start < 0 ? 0 : g.start;
    const int64_t hi = g.end < static_cast<int64_t>(nsamps) ? g.end : static_cast<int64_t>(nsamps) - 1;
    for (int64_t t = lo + threadIdx.x; t <= hi; t += blockDim.x)
        row_kchan[t] = 1;
}
} // namespace

void launch_kchan_rows(const Dims& d, const Segment* kchan_pos, const Segment* kchan_neg,
                       const uint8_t* kchan_any, uint8_t* row_kchan, cudaStream_t s) {
    if (d.nsamps == 0 || d.nchans == 0)
        return;
    k_kchan_rows<<<static_cast<unsigned>(2 * d.nchans), 256, 0, s>>>(d.nchans, d.nsamps, kchan_pos, kchan_neg,
                                                                     kchan_any, row_kchan);
    FB_COUNT_LAUNCH();
}

void launch_apply_unflagged(const Dims& d, const ApplyParams& p, const uint8_t* raw,
                            const float* loc, const float* scale, const float* inv,
                            const uint8_t* mask, const uint8_t* time_flags, const Span32* kspec_pos,
                            const Span32* kspec_neg, const Segment* kchan_pos,
                            const Segment* kchan_neg, const uint8_t* kchan_any,
                            const float* s_keep_f, const float* zdot_a,
                            const float* zdot_b, const uint8_t* row_clip, const uint8_t* row_kchan,
                            uint32_t* slow_rows, unsigned int* nslow, float* work,
                            unsigned long long* counters, cudaStream_t s) {
    const size_t smem = d.nchans * (sizeof(float) + 1);
    if (d.nsamps == 0)
        return;
    if (d.nchans >= (uint64_t{1} << 31) || d.nsamps >= (uint64_t{1} << 31))
        throw Error(FROST_ERR_INVALID_ARGUMENT, "apply: too many channels or samples for one block");
    // 4-channel vectors need nchans % 4 == 0 and, for the loads of 4 samples of
    // the raw row, an aligned block (the cleaner's always is)
    const bool vec = d.nchans % 4 == 0 && aligned16(raw);
    const CleanKind kind = !p.transform                         ? CleanKind::kCopy
                           : p.zero_dm == FROST_ZERO_DM_ZDOT ? CleanKind::kZdot
                                                              : CleanKind::kLevel;
    // the listed rows: a few CTAs an SM loop over them (the count is read on the device)
    const unsigned slow_grid = static_cast<unsigned>(std::min<uint64_t>(d.nsamps, 4 * sm_count()));
    FB_DISPATCH(d.dtype, {
        auto clean = [&](auto vtag) {
            constexpr int V = decltype(vtag)::value;
            const auto k    = kind == CleanKind::kCopy    ? &k_apply_clean<D, V, CleanKind::kCopy>
                              : kind == CleanKind::kLevel ? &k_apply_clean<D, V, CleanKind::kLevel>
                                                          : &k_apply_clean<D, V, CleanKind::kZdot>;
            const uint64_t rows = strip_rows(d.nchans, V);
            k<<<static_cast<unsigned>((d.nsamps + rows - 1) / rows), 256, 0, s>>>(
                d, p, raw, loc, scale, inv, mask, time_flags, kspec_pos, kspec_neg, s_keep_f, zdot_a, zdot_b,
                row_clip, row_kchan, work, slow_rows, nslow);
        };
        if (vec) {
            clean(std::integral_constant<int, 4>{});
            set_smem(reinterpret_cast<const void*>(&k_apply_unflagged<D, 4>), smem);
            k_apply_unflagged<D, 4><<<slow_grid, 256, smem, s>>>(
                d, p, raw, loc, scale, inv, mask, time_flags, kspec_pos, kspec_neg, kchan_pos,
                kchan_neg, kchan_any, s_keep_f, zdot_a, zdot_b, slow_rows, nslow, work, counters);
        } else {
            clean(std::integral_constant<int, 1>{});
            set_smem(reinterpret_cast<const void*>(&k_apply_unflagged<D, 1>), smem);
            k_apply_unflagged<D, 1><<<slow_grid, 256, smem, s>>>(
                d, p, raw, loc, scale, inv, mask, time_flags, kspec_pos, kspec_neg, kchan_pos,
                kchan_neg, kchan_any, s_keep_f, zdot_a, zdot_b, slow_rows, nslow, work, counters);
        }
    });
    FB_COUNT_LAUNCH();
    FB_COUNT_LAUNCH();
}

void launch_apply_flagged(const Dims& d, const ApplyParams& p, const uint64_t* flagged,
                          const unsigned long long* nflagged, const float* loc, const float* scale,
                          const float* inv, const uint8_t* mask, const uint8_t* time_flags,
                          float* work, unsigned long long* counters, cudaStream_t s) {
    if (d.nsamps == 0)
        return;
    const size_t smem     = d.nchans * (sizeof(float) + 1);
    const unsigned blocks = static_cast<unsigned>(std::min<uint64_t>(d.nsamps, 8 * sm_count()));
    set_smem(reinterpret_cast<const void*>(&k_apply_flagged), smem);
    k_apply_flagged<<<blocks, 256, smem, s>>>(d, p, flagged, nflagged, loc, scale, inv, mask, time_flags, work,
                                              counters);
    FB_COUNT_LAUNCH();
}

void launch_unpack(const Dims& d, const uint8_t* raw, float* work, cudaStream_t s) {
    const uint64_t total = d.nsamps * d.nchans;
    if (total == 0)
        return;
    const unsigned blocks = static_cast<unsigned>(std::min<uint64_t>((total + 255) / 256, 32 * sm_count()));
    FB_DISPATCH(d.dtype, k_unpack<D><<<blocks, 256, 0, s>>>(d, raw, work));
    FB_COUNT_LAUNCH();
}

void launch_welford(const Dims& d, const float* work, const double* recip, float* loc, float* scale,
                    cudaStream_t s) {
    on_groups(grid1(d.nchans, 32) * d.nwin, cols::kWelfordFew, aligned16(work) && d.nchans % 4 == 0, [&](auto u, auto groups) {
        constexpr int U = decltype(u)::value, G = decltype(groups)::value;
        constexpr size_t smem = G * WorkRing<U, G>::kBytes + WorkRing<U, G>::kSideBytes;
        set_smem(reinterpret_cast<const void*>(&k_welford<U, G>), smem);
        const dim3 g(grid1(d.nchans, 32 * G), static_cast<unsigned>(d.nwin));
        k_welford<U, G><<<g, 32 * (G + 1), smem, s>>>(d, work, recip, loc, scale);
    });
    FB_COUNT_LAUNCH();
}

void launch_normalize(const Dims& d, const float* work, const float* loc, const float* scale,
                      const uint8_t* mask, int flip, uint64_t capacity, float* out, cudaStream_t s) {
    const dim3 grid(grid1(capacity, kNormSpan), grid1(d.nchans, kNT));
    const bool vl = d.nchans % 4 == 0, vs = capacity % 4 == 0;
    const auto k  = vl ? (vs ? &k_normalize<true, true> : &k_normalize<true, false>)
                       : (vs ? &k_normalize<false, true> : &k_normalize<false, false>);
    k<<<grid, 256, 0, s>>>(d, work, loc, scale, mask, flip, capacity, out);
    FB_COUNT_LAUNCH();
}

void launch_normalize_short(const Dims& d, const ApplyParams& p, const float* work,
                            const float* tail_loc, const float* tail_scale,
                            const float* tail_out_loc, const float* tail_out_scale,
                            const uint8_t* mask, const float* zdot_a, const float* zdot_b,
                            int flip, uint64_t capacity, float* out, cudaStream_t s) {
    if (d.nsamps == 0)
        return;
    const size_t smem = d.nchans * sizeof(float);
    set_smem(reinterpret_cast<const void*>(&k_normalize_short), smem);
    k_normalize_short<<<static_cast<unsigned>(d.nsamps), 256, smem, s>>>(
        d, p, work, tail_loc, tail_scale, tail_out_loc, tail_out_scale, mask, zdot_a, zdot_b, flip,
        capacity, out);
    FB_COUNT_LAUNCH();
}

} // namespace fb::rfi
