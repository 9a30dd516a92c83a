// tq_tables.h -- host-side construction of a space's tables (tq_tables.cpp).
#pragma once

#include <cstddef>
#include <cstdint>
#include <cstring>
#include <vector>

namespace tq {

// x rounded to the nearest FP16 or BF16 value, ties to even (finite values within
// FP16's range), for tables that try many scales.
inline float round_fp16(float x) {
    uint32_t u;
    std::memcpy(&u, &x, 4);
    if ((u & 0x7FFFFFFFu) < 0x38800000u) return (x + 0.75f) - 0.75f;  // below 2^-14: steps of 2^-24
    u += 0xFFFu + ((u >> 13) & 1u);
    u &= ~0x1FFFu;
    std::memcpy(&x, &u, 4);
    return x;
}
inline float round_bf16(float x) {
    uint32_t u;
    std::memcpy(&u, &x, 4);
    u += 0x7FFFu + ((u >> 16) & 1u);
    u &= 0xFFFF0000u;
    std::memcpy(&x, &u, 4);
    return x;
}

// generateSigns (turbo_quant.h:74-86): splitmix64 draw i, bit 0 set -> +1.
std::vector<float> sign_vector(size_t d, uint64_t seed);

// computeLloydMax (space_turbo_quant.h:76-131) for 2^mse_bits levels:
// FP64 iteration, FP32 output, ascending boundaries.
void lloyd_max(int mse_bits, std::vector<float> &centroids, std::vector<float> &boundaries);

// Bucket table of the quantizer for many boundaries: bucket(z) =
// clamp(fma(z, s, c), 0, buckets-1) truncated; lo[j] = boundaries below every
// z of bucket j; at most k more boundaries lie inside a bucket.
struct QuantLut {
    float s = 0.0f, c = 0.0f;
    int buckets = 0, k = 0;
    std::vector<uint8_t> lo;
    std::vector<uint8_t> span;  // boundaries inside bucket j (0 .. k)
};
int quant_bucket(float z, float s, float c, int buckets);
bool build_quant_lut(const std::vector<float> &boundaries, int buckets, int max_k, QuantLut &lut);
// Largest shift (8 at most) for which 2^shift neighbouring buckets, from a
// multiple of 2^shift on, hold one of the nb boundaries at most (0: none).
int coarse_shift(const QuantLut &lut, int nb);

}  // namespace tq
