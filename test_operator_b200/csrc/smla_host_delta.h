// Delta = rowsum(O * dO) of rows of SMLA_D_V bf16 columns, on the host.
//
// The sums in the order of the device's warp (32 lanes of sixteen columns, then a butterfly over the lanes), so that a Delta is the same
// bits wherever it is found: the product of two bf16 is exact in fp32 as long as it neither over- nor underflows, and so is what a fused
// add rounds.
#pragma once
#include <cstdint>
#include <cstring>

#include "../../include/smla_bwd.h"

// Eight lanes in a vector, compiled for several widths, where the compiler has GCC's vectors and the target is x86; a plain loop elsewhere.
#if defined(__x86_64__) && defined(__GNUC__) && !defined(__clang__) && !defined(SMLA_PLAIN_DELTA)
typedef uint16_t u16x8 __attribute__((vector_size(16)));
typedef uint32_t u32x8 __attribute__((vector_size(32)));
typedef int32_t i32x8 __attribute__((vector_size(32)));
typedef float f32x8 __attribute__((vector_size(32)));

__attribute__((target_clones("avx512f", "avx2", "default")))
static void delta_rows_host(const uint16_t* o, const uint16_t* g, float* out, int64_t rows) {
    constexpr i32x8 kLo = {0, 8, 1, 9, 4, 12, 5, 13}, kHi = {2, 10, 3, 11, 6, 14, 7, 15}, kEven = {0, 1, 8, 9, 4, 5, 12, 13},
                    kOdd = {2, 3, 10, 11, 6, 7, 14, 15}, kLower = {0, 1, 2, 3, 8, 9, 10, 11}, kUpper = {4, 5, 6, 7, 12, 13, 14, 15};
    for (int64_t r = 0; r < rows; ++r, o += SMLA_D_V, g += SMLA_D_V) {
        f32x8 acc[4] = {};                                   // lanes 8 i .. 8 i + 7
        for (int half = 0; half < 2; ++half) {
            for (int i = 0; i < 4; ++i) {
                f32x8 m[8];                                  // products of eight columns of a lane; then of a column of eight lanes
                for (int l = 0; l < 8; ++l) {
                    u16x8 a, b;
                    std::memcpy(&a, o + half * 256 + (8 * i + l) * 8, sizeof a);
                    std::memcpy(&b, g + half * 256 + (8 * i + l) * 8, sizeof b);
                    const u32x8 a32 = __builtin_convertvector(a, u32x8) << 16, b32 = __builtin_convertvector(b, u32x8) << 16;
                    f32x8 x, y;
                    std::memcpy(&x, &a32, sizeof x);
                    std::memcpy(&y, &b32, sizeof y);
                    m[l] = x * y;
                }
                f32x8 u[8], v[8];
                for (int l = 0; l < 4; ++l) {
                    u[2 * l] = __builtin_shuffle(m[2 * l], m[2 * l + 1], kLo);
                    u[2 * l + 1] = __builtin_shuffle(m[2 * l], m[2 * l + 1], kHi);
                }
                for (int l = 0; l < 2; ++l) {
                    for (int k = 0; k < 2; ++k) {
                        v[4 * l + 2 * k] = __builtin_shuffle(u[4 * l + k], u[4 * l + 2 + k], kEven);
                        v[4 * l + 2 * k + 1] = __builtin_shuffle(u[4 * l + k], u[4 * l + 2 + k], kOdd);
                    }
                }
                for (int k = 0; k < 4; ++k) acc[i] += __builtin_shuffle(v[k], v[4 + k], kLower);
                for (int k = 0; k < 4; ++k) acc[i] += __builtin_shuffle(v[k], v[4 + k], kUpper);
            }
        }
        float sum[8];
        const f32x8 all = (acc[0] + acc[2]) + (acc[1] + acc[3]);
        std::memcpy(sum, &all, sizeof sum);
        for (int n = 4; n; n >>= 1)
            for (int l = 0; l < n; ++l) sum[l] += sum[l + n];
        out[r] = sum[0];
    }
}
#else
static void delta_rows_host(const uint16_t* o, const uint16_t* g, float* out, int64_t rows) {
    const auto value = [](uint16_t bits) {
        const uint32_t wide = static_cast<uint32_t>(bits) << 16;
        float x;
        std::memcpy(&x, &wide, sizeof x);
        return x;
    };
    for (int64_t r = 0; r < rows; ++r, o += SMLA_D_V, g += SMLA_D_V) {
        float lane[32] = {};
        for (int half = 0; half < 2; ++half)
            for (int l = 0; l < 32; ++l)
                for (int k = 0; k < 8; ++k) lane[l] += value(o[half * 256 + l * 8 + k]) * value(g[half * 256 + l * 8 + k]);
        for (int n = 16; n; n >>= 1)
            for (int l = 0; l < n; ++l) lane[l] += lane[l + n];
        out[r] = lane[0];
    }
}
#endif
