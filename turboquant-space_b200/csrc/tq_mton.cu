// tq_mton.cu -- the BF16 operand planes of the serving contraction.
//
// The asymmetric distance is a contraction of K = 2D once a code is decoded:
//
//   A[i] = [ q_rot_i | s_q_i ]     B[j] = [ sigma_j c[idx_j] / g_j | (+-1)_j ]
//
// with g_j = scale gamma_j, so that g_j (A B^T)[i, j] = ip_mse + correction of
// distSearch (space_turbo_quant.h:676-683) and
// d = max(0, r2_i + c2_j - 2 (C_ij r1_i) c1_j), r1 = |q|, r2 = |q|^2,
// c1 = g_j |x|, c2 = |x|^2.
//
// Both sides are hi/lo BF16 pairs, x = hi + lo with hi = bf16(x),
// lo = bf16(x - hi); the tcgen05 kernels (tq_tc.cu) form hi*hi + hi*lo +
// lo*hi.  The QJL half of B is exact in BF16 (its lo plane is zero and is not
// stored: the lo plane has asym_lo_width(D) columns) and needs two products
// there instead of three.  A code with g_j < 1e-20 (gamma = 0, e.g. a zero
// row) keeps B[j] = [ sigma_j c[idx_j] | 0 ] and c1 = |x|: its correction term
// is below 1e-18 of |q| |x| and is left out.
#include <cuda_bf16.h>

#include <algorithm>

#include "tq_internal.h"
#include "tq_mton.h"

namespace tq {
namespace {

__device__ __forceinline__ unsigned unit_at(const uint8_t *code, int p, int nibble) {
    if (nibble) {
        const unsigned b = code[p >> 1];
        return (p & 1) ? (b >> 4) : (b & 15u);
    }
    return code[p];
}

// Value v at position k of row r: hi at plane0[r K + k], lo at plane1[r ldl + k]
// (k < ldl; beyond ldl lo is zero by construction and not stored).
__device__ __forceinline__ void put(void *plane0, void *plane1, size_t r, int K, int ldl, int k,
                                    float v) {
    const __nv_bfloat16 hi = __float2bfloat16_rn(v);
    static_cast<__nv_bfloat16 *>(plane0)[r * K + k] = hi;
    if (k < ldl)
        static_cast<__nv_bfloat16 *>(plane1)[r * ldl + k] =
            __float2bfloat16_rn(v - __bfloat162float(hi));
}

// One thread per (row, 4 consecutive positions).  Rows in [rows, rows_pad)
// are zero so that padded tiles contribute nothing.
__global__ void __launch_bounds__(256) planes_from_codes_kernel(
    const uint8_t *__restrict__ codes, size_t rows, size_t rows_pad, Params P, DevTables T,
    int ldl, void *plane0, void *plane1, float *__restrict__ s1, float *__restrict__ s2) {
    const int K = 2 * P.D;
    const size_t quads_per_row = (size_t)(K / 4);
    const size_t total = rows_pad * quads_per_row;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        const size_t r = t / quads_per_row;
        const int k0 = (int)(t - r * quads_per_row) * 4;
        if (r >= rows) {
            for (int q = 0; q < 4; ++q) put(plane0, plane1, r, K, ldl, k0 + q, 0.0f);
            if (k0 == 0) {
                s1[r] = 0.0f;
                s2[r] = 0.0f;
            }
            continue;
        }
        const uint8_t *code = codes + r * (size_t)P.cs;
        float meta[3];
        for (int q = 0; q < 3; ++q) {
            uint32_t w = 0;
            for (int b = 0; b < 4; ++b) w |= (uint32_t)code[P.pb + 4 * q + b] << (8 * b);
            meta[q] = __uint_as_float(w);
        }
        const float norm = meta[0], gamma = meta[1], sigma = meta[2];
        const float sg = __fmul_rn(P.scale, gamma);
        // exact-sign form (see the file header); !(g >= 1e-20f) also catches a NaN trailer
        const bool ratio = sg >= 1e-20f && sg <= 3.0e38f;
        for (int q = 0; q < 4; ++q) {
            const int k = k0 + q;
            float v;
            if (k < P.D) {
                v = __fmul_rn(sigma, T.centroids[unit_at(code, k, P.nibble) >> 1]);
                if (ratio) v = __fdiv_rn(v, sg);
            } else {
                const bool pos = unit_at(code, k - P.D, P.nibble) & 1u;
                v = !ratio ? 0.0f : pos ? 1.0f : -1.0f;
            }
            put(plane0, plane1, r, K, ldl, k, v);
        }
        if (k0 == 0) {
            s1[r] = ratio ? __fmul_rn(sg, norm) : norm;
            s2[r] = __fmul_rn(norm, norm);
        }
    }
}

// Scalars of the decoded-B kernels (launch_dec_factors): the same per-code
// quantities as the planes' s1 / s2 and exact-sign ratio, with the ratio as a
// chunk factor instead of a division of every value.
__global__ void __launch_bounds__(256) dec_factors_kernel(const uint8_t *__restrict__ codes,
                                                          size_t rows, size_t rows_pad, Params P,
                                                          float *__restrict__ c1,
                                                          float *__restrict__ c2,
                                                          float *__restrict__ fc,
                                                          float *__restrict__ fs) {
    for (size_t r = (size_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows_pad;
         r += (size_t)gridDim.x * blockDim.x) {
        float a = 0.0f, b = 0.0f, f = 0.0f, g1 = 0.0f;
        if (r < rows) {
            const uint8_t *t = codes + r * (size_t)P.cs + P.pb;
            float meta[3];
            for (int q = 0; q < 3; ++q) {
                uint32_t w = 0;
                for (int k = 0; k < 4; ++k) w |= (uint32_t)t[4 * q + k] << (8 * k);
                meta[q] = __uint_as_float(w);
            }
            const float norm = meta[0], gamma = meta[1], sigma = meta[2];
            b = __fmul_rn(norm, norm);
            const float sg = __fmul_rn(P.scale, gamma);
            const bool ratio = sg >= 1e-20f && sg <= 3.0e38f;  // as the exact-sign planes
            a = ratio ? __fmul_rn(sg, norm) : norm;
            f = ratio ? __fdiv_rn(sigma, sg) : sigma;
            g1 = ratio ? 1.0f : 0.0f;
        }
        c1[r] = a;
        c2[r] = b;
        fc[r] = f;
        fs[r] = g1;
    }
}

__global__ void __launch_bounds__(256) planes_from_prepared_kernel(
    const float *__restrict__ q_rot, const float *__restrict__ s_q, const float *__restrict__ norms,
    size_t rows, size_t rows_pad, int D, void *plane0, void *plane1,
    float *__restrict__ r1, float *__restrict__ r2) {
    const int K = 2 * D;
    const size_t total = rows_pad * (size_t)K;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        const size_t r = t / K;
        const int k = (int)(t - r * K);
        float v = 0.0f;
        if (r < rows) v = (k < D) ? q_rot[r * D + k] : s_q[r * D + (k - D)];
        put(plane0, plane1, r, K, K, k, v);
        if (k == 0) {
            r1[r] = (r < rows) ? norms[2 * r + 1] : 0.0f;
            r2[r] = (r < rows) ? norms[2 * r] : 0.0f;
        }
    }
}

unsigned grid_for(size_t work, int threads) {
    size_t b = (work + threads - 1) / threads;
    const size_t cap = (size_t)148 * 32;
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (unsigned)b;
}

}  // namespace

cudaError_t launch_planes_from_codes(const Params &P, const DevTables &T, const uint8_t *codes,
                                     size_t rows, size_t rows_pad, void *plane0, void *plane1,
                                     float *s1, float *s2, cudaStream_t st) {
    if (rows_pad == 0) return cudaSuccess;
    planes_from_codes_kernel<<<grid_for(rows_pad * (P.D / 2), 256), 256, 0, st>>>(
        codes, rows, rows_pad, P, T, asym_lo_width(P.D), plane0, plane1, s1, s2);
    return cudaGetLastError();
}

cudaError_t launch_dec_factors(const Params &P, const uint8_t *codes, size_t rows, size_t rows_pad,
                               float *c1, float *c2, float *fc, float *fs, cudaStream_t st) {
    if (rows_pad == 0) return cudaSuccess;
    const size_t blocks = std::min<size_t>((rows_pad + 255) / 256, 148 * 16);
    dec_factors_kernel<<<(unsigned)blocks, 256, 0, st>>>(codes, rows, rows_pad, P, c1, c2, fc, fs);
    return cudaGetLastError();
}

cudaError_t launch_planes_from_prepared(const float *q_rot, const float *s_q, const float *norms,
                                        size_t rows, size_t rows_pad, int D, void *plane0,
                                        void *plane1, float *r1, float *r2, cudaStream_t st) {
    if (rows_pad == 0) return cudaSuccess;
    planes_from_prepared_kernel<<<grid_for(rows_pad * 2 * D, 256), 256, 0, st>>>(
        q_rot, s_q, norms, rows, rows_pad, D, plane0, plane1, r1, r2);
    return cudaGetLastError();
}

}  // namespace tq
