// Time-ordered streaming of 32 channel columns through shared memory, for
// the order-exact statistics: a lane per channel, whose double sums must
// follow the reference's order, so each is a chain of dependent FP64
// operations a row long (8 cycles an operation on sm_100).
//
// A CTA holds one 32-channel group, or four of them side by side. Warp 0
// copies rows ahead with cp.async (a ring of S stages of H rows a group); the
// other warps walk the rows, each with sums of its own, and meet it once a
// stage. A warp that has a scheduler to
// itself issues in order, so whatever stands between two operations of its
// chain, or is not there in time, is added to the chain: the walkers are
// written as software pipelines (loads 8 rows ahead, conversions 3) whose
// order the volatile asm of the operations below keeps. A warp by itself takes
// 9 - 10 cycles a row for one sum and 35 for the Welford update so, and 17 - 27
// and 48 for the same loops written plainly. In the kernels (at 1965 MHz, one
// group a CTA) a row takes 19 cycles in the bandpass sweeps, whose walker also
// widens, compares and selects, 25 in the moments with two or three sums a
// warp, and 40 in the Welford update.
//
// Copies are 16 bytes where the row pitch and the base are multiples of 16,
// else 4 bytes from the word a row's first sample lies in (rows of any byte
// pitch; a row's data then starts up to 3 bytes into its slot). No copy
// reads past the row's last sample.
#pragma once

#include <cstdint>

#include "common.hpp"
#include "rfi_stage.cuh"

namespace fb::rfi::cols {

// ---- operations in the order they are written -------------------------------

__device__ __forceinline__ void add(double& d, double a, double b) {
    asm volatile("add.rn.f64 %0, %1, %2;" : "=d"(d) : "d"(a), "d"(b));
}
__device__ __forceinline__ void sub(double& d, double a, double b) {
    asm volatile("sub.rn.f64 %0, %1, %2;" : "=d"(d) : "d"(a), "d"(b));
}
__device__ __forceinline__ void mul(double& d, double a, double b) {
    asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(d) : "d"(a), "d"(b));
}
__device__ __forceinline__ void fma(double& d, double a, double b, double c) {
    asm volatile("fma.rn.f64 %0, %1, %2, %3;" : "=d"(d) : "d"(a), "d"(b), "d"(c));
}
__device__ __forceinline__ void widen(double& d, float f) { asm volatile("cvt.f64.f32 %0, %1;" : "=d"(d) : "f"(f)); }
/** d = |v| <= cut ? v : 0, one = that it is. */
__device__ __forceinline__ void keep(double& d, uint32_t& one, double v, double cut) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .f64 a;\n\tabs.f64 a, %2;\n\tsetp.le.f64 p, a, %3;\n\t"
                 "selp.f64 %0, %2, 0d0000000000000000, p;\n\tselp.u32 %1, 1, 0, p;\n\t}"
                 : "=d"(d), "=r"(one)
                 : "d"(v), "d"(cut));
}
/** BITS-bit word(s) at a shared address as they are. */
template <int BITS> __device__ __forceinline__ uint32_t word(uint32_t a) {
    uint32_t v;
    if constexpr (BITS == 32)
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    else if constexpr (BITS == 16)
        asm volatile("{\n\t.reg .u16 h;\n\tld.shared.u16 h, [%1];\n\tcvt.u32.u16 %0, h;\n\t}" : "=r"(v) : "r"(a) : "memory");
    else
        asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void pair(double& x, double& y, uint32_t a) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x), "=d"(y) : "r"(a) : "memory");
}

// Copies n (1..4) bytes to a 4-byte shared word, the rest of it zero.
__device__ __forceinline__ void cp_async4(void* dst, const void* src, int n) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(stage::smem_u32(dst)), "l"(src), "r"(n)
                 : "memory");
}

// ---- the ring ----------------------------------------------------------------

constexpr int kBatch = 16; // rows a walker takes without a branch
constexpr int kAhead = 8;  // rows its loads run ahead

// Groups a CTA holds: one while the groups are no more than so many an SM, as
// a walker then has a scheduler to itself, and four from there on, as the
// warps of a CTA go to the schedulers in turn, so that one walker in every
// two-warp CTA leaves half of the schedulers to the feeders. Measured at
// windows of 31 250 rows on both sides of each line, one group : four, us, by
// groups an SM:
//   bandpass  2.2: 186 : 276, 3.9: 190 : 282, 5.2: 270 : 325 | 6.9: 369 : 333,
//             10.4: 526 : 400 (12.1: 613 : 670, four's second wave)
//   moments   uint8: 1.9: 612 : 659 | 2.2: 870 : 659, 3.9: 960 : 672, 6.9: 1756 : 1172;
//             float32: 1.9: 562 : 835 | 2.2: 775 : 839, 3.0: 844 : 842, 6.9: 1584 : 1317
//   Welford   1.9: 643 : 801, 3.9: 763 : 804 | 5.2: 1017 : 965, 6.9: 1550 : 971
constexpr int kManyGroups     = 4;
constexpr uint64_t kBandpassFew = 6, kMomentsFew = 2, kWelfordFew = 4;
inline bool few_groups(uint64_t groups, uint64_t per_sm) { return groups <= per_sm * sm_count(); }

/** Rows [0, n) of a 32-channel segment of BITS-bit samples, row r at
 * src + r * pitch. U: bytes a copy (16 or 4); S stages of H rows; SIDE: a
 * 16-byte record per row (the same for every lane) travels with it, from
 * side + r. */
template <int BITS, int U, int H, int S, bool SIDE = false> struct Ring {
    static constexpr int kSeg    = 32 * BITS / 8; // bytes of a whole segment's row
    static constexpr int kUnits  = U == 16 ? kSeg / 16 : kSeg / 4 + (BITS < 32 ? 1 : 0);
    static constexpr int kPitch  = kUnits * U; // shared bytes a row
    static constexpr int kRows   = S * H;
    static constexpr int kBytes  = kRows * kPitch;
    static constexpr int kSideBytes = SIDE ? kRows * 16 : 0;
    static constexpr bool kShift = U == 4 && BITS < 32; // rows may start inside their first word
    static constexpr bool kEven  = !kShift && 32 % kUnits == 0; // whole rows a warp copy
    static_assert(U == 4 || (U == 16 && kSeg % 16 == 0), "16-byte copies need whole 16-byte segments");
    static_assert((kRows & (kRows - 1)) == 0 && S >= 4 && H % kBatch == 0, "a power of two of rows");

    uint8_t* smem;    // kBytes, 16-byte aligned
    uint8_t* records; // kSideBytes (the groups of a CTA share them)
    const uint8_t* src;
    const double2* side; // null: another group's ring copies the records
    uint64_t pitch;
    int copy; // bytes of the segment that exist (the band's last one can be short)
    int n, lane;

    /** left: bytes of the row from the segment's start on (0: no such segment). */
    __device__ Ring(uint8_t* smem_, const uint8_t* src_, uint64_t pitch_, uint64_t left, uint64_t n_,
                    uint8_t* records_ = nullptr, const double2* side_ = nullptr)
        : smem(smem_), records(records_), src(src_), side(side_), pitch(pitch_),
          copy(static_cast<int>(left < static_cast<uint64_t>(kSeg) ? left : kSeg)), n(static_cast<int>(n_)),
          lane(static_cast<int>(threadIdx.x & 31U)) {}

    __device__ __forceinline__ int stages() const { return (n + H - 1) / H; }

    __device__ __forceinline__ void issue(int k) const {
        const int r0 = k * H;
        if (r0 < n) {
            const int nr     = n - r0 < H ? n - r0 : H;
            uint8_t* dst     = smem + (r0 & (kRows - 1)) * kPitch;
            const uint8_t* s = src + static_cast<uint64_t>(r0) * pitch;
            if constexpr (kEven) {
                constexpr int kPer = 32 / kUnits; // rows a warp copy
                const int r = lane / kUnits, u = lane % kUnits;
                const uint8_t* a    = s + static_cast<uint64_t>(r) * pitch + u * U;
                const uint64_t step = kPer * pitch;
                if (u * U < copy) {
                    auto put = [&](int j) {
                        if constexpr (U == 16)
                            stage::cp_async16(dst + (lane + 32 * j) * 16, a);
                        else
                            cp_async4(dst + (lane + 32 * j) * 4, a, 4);
                        a += step;
                    };
                    if (nr == H) { // a whole stage
#pragma unroll 16
                        for (int j = 0; j < H / kPer; ++j)
                            put(j);
                    } else {
                        for (int j = 0; r + j * kPer < nr; ++j)
                            put(j);
                    }
                }
            } else {
#pragma unroll 4
                for (int i = lane; i < H * kUnits; i += 32) {
                    const int r = i / kUnits, u = i - r * kUnits;
                    const uint8_t* a = s + static_cast<uint64_t>(r) * pitch;
                    const int m      = kShift ? static_cast<int>(reinterpret_cast<uintptr_t>(a) & 3U) : 0;
                    const int left   = m + copy - u * 4;
                    if (r < nr && left > 0)
                        cp_async4(dst + i * 4, a - m + u * 4, left < 4 ? left : 4);
                }
            }
            if constexpr (SIDE)
                if (side != nullptr)
                    for (int r = lane; r < nr; r += 32)
                        stage::cp_async16(records + ((r0 + r) & (kRows - 1)) * 16, side + r0 + r);
        }
    }

    /** Warp 0's part of a sweep over the rows of groups ring(0) ..
     * ring(G - 1); the walkers' is walk(). */
    template <int G, class GET> static __device__ __forceinline__ void feed(GET&& ring) {
        if constexpr (G == 1) {
            const Ring one = ring(0);
            feed_through(one.stages(), [&](int k) { one.issue(k); });
        } else {
            feed_through(ring(0).stages(), [&](int k) {
                for (int g = 0; g < G; ++g)
                    ring(g).issue(k);
            });
        }
    }
    template <class F> static __device__ __forceinline__ void feed_through(int nst, F&& issue_all) {
        for (int k = 0; k < S - 1; ++k) {
            issue_all(k);
            stage::commit();
        }
        for (int k = 0; k < nst; ++k) {
            stage::wait_pending<S - 3>(); // stages k and k + 1 have landed
            __syncthreads();              // and stage k - 1 has been read
            issue_all(k + S - 1);
            stage::commit();
        }
        stage::wait_pending<0>();
        __syncthreads();
    }

    /** A walker's part: start(a, b) once the first rows are there, batch(r,
     * a, b) for every kBatch rows from r on and one(r, a) for each row after
     * the last whole batch. a: the shared byte address of the rows' slots,
     * b: that of the kBatch rows after them, whose first kAhead a batch
     * reads ahead (past the last row: stale, to be dropped). */
    template <class ST, class BA, class ON>
    __device__ __forceinline__ void walk(ST&& start, BA&& batch, ON&& one) const {
        const uint32_t base = stage::smem_u32(smem);
        const int nst       = stages();
        for (int k = 0; k < nst; ++k) {
            __syncthreads();
            if (k == 0)
                start(base);
            const int e = n - k * H < H ? n : (k + 1) * H;
            int r       = k * H;
#pragma unroll 1
            for (; r + kBatch <= e; r += kBatch)
                batch(r, base + (r & (kRows - 1)) * kPitch, base + ((r + kBatch) & (kRows - 1)) * kPitch);
#pragma unroll 1
            for (; r < e; ++r)
                one(r, base + (r & (kRows - 1)) * kPitch);
        }
        __syncthreads();
    }

    /** This lane's offset in row r's slot. */
    __device__ __forceinline__ uint32_t at(int r) const {
        const uint32_t o = static_cast<uint32_t>(lane * BITS / 8);
        return kShift ? o + static_cast<uint32_t>(
                                (reinterpret_cast<uintptr_t>(src) + static_cast<uint64_t>(r) * (pitch & 3U)) & 3U)
                      : o;
    }
    /** This lane's sample of a row as the bits it is stored in. */
    __device__ __forceinline__ uint32_t bits(uint32_t slot, int r) const {
        const uint32_t v = word<BITS < 8 ? 8 : BITS>(slot + at(r));
        return BITS < 8 ? (v >> ((lane * BITS) & 7)) & ((1U << BITS) - 1U) : v;
    }
    __device__ __forceinline__ uint32_t record(int r) const {
        return stage::smem_u32(records) + (r & (kRows - 1)) * 16;
    }
};

} // namespace fb::rfi::cols
