// Time-ordered streaming of 32 channel columns through one warp's own
// shared memory.
//
// The order-exact statistics give every lane one channel, whose double sums
// must follow the reference's order: a chain of dependent FP64 operations a
// row long. What a kernel can do is to have nothing else on that chain: the
// rows are copied ahead with cp.async (S - 1 stages of ROWS rows in flight),
// read from shared memory B rows at a time into registers, and only then
// consumed. The ring belongs to one warp, so no block barrier ever holds a
// chain up, and few channels can be spread over many SMs.
//
// Copies are 16 bytes where the row pitch and the base are multiples of 16,
// else 4 bytes from the word a row's first sample lies in (rows of any byte
// pitch; a row's data then starts up to 3 bytes into its slot). No copy
// reads past the row's last sample.
#pragma once

#include <cstdint>
#include <type_traits>

#include "rfi_stage.cuh"

namespace fb::rfi::cols {

// Copies n (1..4) bytes to a 4-byte shared word, the rest of it zero.
__device__ __forceinline__ void cp_async4(void* dst, const void* src, int n) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(stage::smem_u32(dst)), "l"(src), "r"(n)
                 : "memory");
}

/** Rows [0, n) of a 32-channel segment of BITS-bit samples, row r at
 * src + r * pitch. U: bytes a copy (16 or 4); S (a power of two) stages of
 * ROWS rows; SIDE: a 16-byte record per row (the same for every lane)
 * travels with it, from side + r. */
template <int BITS, int U, int ROWS, int S, bool SIDE = false> struct Reader {
    static constexpr int kSeg   = 32 * BITS / 8; // bytes of a whole segment's row
    static constexpr int kUnits = U == 16 ? kSeg / 16 : kSeg / 4 + (BITS < 32 ? 1 : 0);
    static constexpr int kPitch = kUnits * U; // shared bytes a row
    static constexpr int kBytes = S * ROWS * kPitch;
    static constexpr bool kShift = U == 4 && BITS < 32; // rows may start inside their first word
    static constexpr bool kEven  = !kShift && kUnits <= 32 && 32 % kUnits == 0; // whole rows a warp copy
    static_assert(U == 4 || (U == 16 && kSeg % 16 == 0), "16-byte copies need whole 16-byte segments");
    static_assert((S & (S - 1)) == 0 && S >= 2, "a power of two of stages");
    static_assert(!SIDE || ROWS <= 32, "one side record a lane");

    uint8_t* smem;      // kBytes of this warp's own, 16-byte aligned
    double2* side_smem; // S * ROWS records (SIDE)
    const uint8_t* src;
    const double2* side;
    uint64_t pitch;
    int copy; // bytes of the segment that exist (the band's last one can be short)
    int n, lane;

    __device__ Reader(uint8_t* smem_, const uint8_t* src_, uint64_t pitch_, uint64_t left, uint64_t n_,
                      double2* side_smem_ = nullptr, const double2* side_ = nullptr)
        : smem(smem_), side_smem(side_smem_), src(src_), side(side_), pitch(pitch_),
          copy(static_cast<int>(left < static_cast<uint64_t>(kSeg) ? left : kSeg)), n(static_cast<int>(n_)),
          lane(static_cast<int>(threadIdx.x & 31U)) {}

    __device__ __forceinline__ int mis(const uint8_t* a) const {
        return kShift ? static_cast<int>(reinterpret_cast<uintptr_t>(a) & 3U) : 0;
    }

    __device__ __forceinline__ void issue(int k) const {
        const int r0 = k * ROWS;
        if (r0 < n) {
            const int nr     = n - r0 < ROWS ? n - r0 : ROWS;
            uint8_t* dst     = smem + (k & (S - 1)) * ROWS * kPitch;
            const uint8_t* s = src + static_cast<uint64_t>(r0) * pitch;
            if constexpr (kEven) {
                constexpr int kRows = 32 / kUnits; // rows a warp copy
                const int r = lane / kUnits, u = lane % kUnits;
                const uint8_t* a    = s + static_cast<uint64_t>(r) * pitch + u * U;
                const uint64_t step = kRows * pitch;
                if (u * U < copy) {
#pragma unroll
                    for (int j = 0; j < ROWS / kRows; ++j) {
                        if (r + j * kRows < nr) {
                            if constexpr (U == 16)
                                stage::cp_async16(dst + (lane + 32 * j) * 16, a);
                            else
                                cp_async4(dst + (lane + 32 * j) * 4, a, 4);
                        }
                        a += step;
                    }
                }
            } else {
#pragma unroll
                for (int j = 0; j < (ROWS * kUnits + 31) / 32; ++j) {
                    const int i = lane + 32 * j;
                    const int r = i / kUnits, u = i - r * kUnits;
                    const uint8_t* a = s + static_cast<uint64_t>(r) * pitch;
                    const int m      = mis(a);
                    const int left   = m + copy - u * 4;
                    if (r < nr && left > 0)
                        cp_async4(dst + i * 4, a - m + u * 4, left < 4 ? left : 4);
                }
            }
            if constexpr (SIDE)
                if (lane < nr)
                    stage::cp_async16(side_smem + (k & (S - 1)) * ROWS + lane, side + r0 + lane);
        }
        stage::commit();
    }

    /** f(nb, x, r0, y): nb (a compile-time count, B or 1) samples x[] of this
     * lane's column from row r0 on, y their side records. Every lane calls. */
    template <int B, class RD, class F> __device__ __forceinline__ void each(RD&& rd, F&& f) const {
        static_assert(ROWS % B == 0, "whole batches a stage");
        const int nblk = (n + ROWS - 1) / ROWS;
        for (int k = 0; k < S - 1; ++k)
            issue(k);
        for (int k = 0; k < nblk; ++k) {
            // into the slot of stage k - 1: every lane is done with it
            issue(k + S - 1);
            stage::wait_pending<S - 1>();
            __syncwarp();
            const int slot   = k & (S - 1);
            const uint8_t* p = smem + slot * ROWS * kPitch;
            const double2* y = SIDE ? side_smem + slot * ROWS : nullptr;
            const int r0     = k * ROWS;
            const int m0     = kShift ? mis(src + static_cast<uint64_t>(r0) * pitch) : 0;
            const int step   = kShift ? static_cast<int>(pitch & 3U) : 0;
            auto row         = [&](int r) { return p + r * kPitch + (kShift ? (m0 + r * step) & 3 : 0); };
            if (r0 + ROWS <= n) {
#pragma unroll
                for (int r = 0; r < ROWS; r += B) {
                    float x[B];
#pragma unroll
                    for (int j = 0; j < B; ++j)
                        x[j] = rd(row(r + j), lane);
                    f(std::integral_constant<int, B>{}, x, r0 + r, y + (SIDE ? r : 0));
                }
            } else {
                for (int r = 0; r < n - r0; ++r) {
                    const float x[1] = {rd(row(r), lane)};
                    f(std::integral_constant<int, 1>{}, x, r0 + r, y + (SIDE ? r : 0));
                }
            }
            __syncwarp();
        }
        // every copy has landed: the ring can be used again
        stage::wait_pending<0>();
        __syncwarp();
    }
};

} // namespace fb::rfi::cols
