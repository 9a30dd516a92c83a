// tq_encode.cu -- encode of many rows at padded dims 256, 512 and 1024, rows
// held in registers.
//
// The computation is encode2_kernel's (tq_kernels.cu), every rounding in the
// same place and order: the codes are the same bytes.  Lane k of a group of 8
// holds the elements k + 8 m of its row, which is how the 8-lane reduction
// trees read a row; at D = 1024 a row has two groups, one for each half, so
// that a lane holds 64 elements at most and 16 warps fit a multiprocessor.
//   - The three reductions run on registers (the second half's lanes continue
//     the first half's sums).
//   - FWHT strides 1, 2, 4 (and D / 2 with two groups) are lane shuffles,
//     x * (+-1) + y as one FMA: the product is exact, so the sum is the
//     butterfly's one rounding.  The other strides are register pairs.  The row
//     never goes back to shared memory.
//   - The quantizer's bucket table holds {boundary, centroid row} per bucket,
//     coarse enough for one boundary a bucket (256 buckets at b = 8), in 16
//     copies: lanes l and l + 16 read copy l & 15, one bank pair each, so a
//     lookup has no bank conflicts.  The centroids have 32 copies.
//   - A group's rows arrive by cp.async while the previous group is encoded;
//     its codes leave as one bulk store.
//
// What bounds it: no pipe alone.  Shared memory takes about 526 wavefronts a row at
// D = 1024, 256 of them shuffles (encode2: 694), instruction issue 2024 a row (2334);
// both are 64% busy, with instruction fetch of the straight-line code (64 elements a
// lane) and the packed-FP32 pipe among the stalls.  300k rows, encode2 -> this kernel:
// 256-d 4-bit 289 -> 174 us, 384-d 4-bit 510 -> 372, 500-d 8-bit 492 -> 391, 768-d
// 4-bit 992 -> 897, 768-d 8-bit 918 -> 866.  Eight lanes a row at D = 1024 leave 8
// warps of 255 registers: 920 us.
#include "tq_internal.h"
#include "tq_async.cuh"
#include "tq_rht.cuh"

namespace tq {
namespace {

__device__ __forceinline__ u64 ffma2(u64 a, u64 b, u64 c) {
    u64 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// The tail of the sum-of-squares tree (chain_sq_reduce): the eight lanes'
// accumulators of a group -> their sum; t0 .. t3 as the leftovers need them.
__device__ __forceinline__ float tree8(float acc, float (&t)[4]) {
    const float hi = __shfl_down_sync(kFull, acc, 4, 8);
    const float s = __fadd_rn(acc, hi);
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = __shfl_sync(kFull, s, i, 8);
    return __fadd_rn(__fadd_rn(t[0], t[2]), __fadd_rn(t[1], t[3]));
}

// acc continued over a lane's elements.  AGAIN: the squares as x * x + (-0), the
// same values, so that the compiler does not keep the first pass's in registers.
template <bool AGAIN, int NP>
__device__ __forceinline__ float chain_part(float acc, const u64 (&p)[NP]) {
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        float a, b;
        un2(AGAIN ? ffma2(p[i], p[i], 0x8000000080000000ull) : fmul2(p[i], p[i]), a, b);
        acc = __fadd_rn(__fadd_rn(acc, a), b);
    }
    return acc;
}

// |row|^2 over all of a row's registers.  Sixteen lanes a row: the upper eight
// hold the second half of each chain and continue the lower eight's sums.
template <int LPR, int NP>
__device__ __forceinline__ float chain_regs(const u64 (&p)[NP], int lane) {
    float t[4], acc = chain_part<false>(0.0f, p);
    if constexpr (LPR == 16) {
        acc = chain_part<true>(__shfl_sync(kFull, acc, lane & 7, 16), p);
        acc = __shfl_sync(kFull, acc, lane | 8, 16);
    }
    return tree8(acc, t);
}

// Buffer offset of element e of a row: with 16 lanes a row the second half lies
// 8 floats further, so that its lanes read other banks than the first half's.
template <int D, int LPR>
__device__ __forceinline__ int at(int e) {
    return LPR == 16 && e >= D / 2 ? e + 8 : e;
}

// |row|^2 of the first n elements of a row in shared memory (n not a multiple
// of 8: the leftovers join by FMAs).
template <int D, int LPR>
__device__ __noinline__ float chain_row(const float *row, int n, int lane) {
    const int n8 = n & ~7;
    float acc = 0.0f, t[4];
#pragma unroll 8
    for (int i = lane & 7; i < n8; i += 8) {
        const float x = row[at<D, LPR>(i)];
        acc = __fadd_rn(acc, __fmul_rn(x, x));
    }
    float s = tree8(acc, t);
    row += at<D, LPR>(n8);  // the leftovers: one block of 8
    int b = 0, r = n - n8;
    if (r >= 4) {
#pragma unroll
        for (int i = 0; i < 4; ++i) t[i] = __fmaf_rn(row[i], row[i], t[i]);
        s = __fadd_rn(__fadd_rn(t[0], t[2]), __fadd_rn(t[1], t[3]));
        b = 4;
    }
    for (; b < r; ++b) s = __fmaf_rn(row[b], row[b], s);
    return s;
}

// Butterflies of pair stride PS (element stride 16 PS) and up.
template <int NP, int PS>
__device__ __forceinline__ void pair_stages(u64 (&p)[NP]) {
    if constexpr (PS < NP) {
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            if (!(i & PS)) {
                const u64 a = p[i], b = p[i + PS];
                p[i] = fadd2(a, b);
                p[i + PS] = fsub2(a, b);
            }
        }
        pair_stages<NP, 2 * PS>(p);
    }
}

// One stride across lanes, lane bit B: the low lane takes y + x, the high lane
// y - x (y: the other lane's value).
template <int B, int NP>
__device__ __forceinline__ void lane_stage(u64 (&p)[NP], int lane) {
    const float s = (lane >> B) & 1 ? -1.0f : 1.0f;
    const u64 s2 = mk2(s, s);
#pragma unroll
    for (int i = 0; i < NP; ++i) p[i] = ffma2(p[i], s2, __shfl_xor_sync(kFull, p[i], 1 << B));
}

// Row pitch of the input buffer in floats: the padding moves each 8-lane group
// of a warp to other banks.
template <int D, int LPR>
__host__ __device__ constexpr int row_pitch() { return D + LPR; }

// Shared bytes: sign masks, bucket table (buckets + 1 entries x 16 copies x 8
// bytes), centroids (levels x 32 copies), then per warp four rows and four codes.
__host__ __device__ __forceinline__ int encode_regs_table_bytes(const Params &P) {
    return 2 * 128 + ((kQlutBuckets >> P.qshift) + 1) * 128 + P.levels * 128;
}
template <int D, int LPR>
__host__ __device__ __forceinline__ int encode_regs_warp_bytes(const Params &P) {
    const int idx = 32 / LPR * D, codes = (32 / LPR * P.cs + 15) & ~15;
    return (32 / LPR) * 4 * row_pitch<D, LPR>() + (idx > codes ? idx : codes);
}

template <int LOG_D, bool NIBBLE, int LPR, int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 1)
    encode_regs_kernel(const float *__restrict__ X, size_t n, uint8_t *__restrict__ out, Params P, DevTables T) {
    constexpr int D = 1 << LOG_D;
    constexpr int RPW = 32 / LPR, NM = D / LPR, NP = NM / 2;  // rows a warp; a lane's elements, and pairs of them
    constexpr int PITCH = row_pitch<D, LPR>();
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t *signs = reinterpret_cast<uint32_t *>(smem);  // [2][32]: rotation, QJL
    const int nbk = kQlutBuckets >> P.qshift;
    unsigned char *table = smem + 256;                            // [nbk + 1][16]
    float *crep = reinterpret_cast<float *>(table + (nbk + 1) * 128);  // [levels][32]
    unsigned char *wbase = reinterpret_cast<unsigned char *>(crep + P.levels * 32) +
                           (threadIdx.x >> 5) * encode_regs_warp_bytes<D, LPR>(P);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int g = lane / LPR, k = lane & 7, h = LPR == 16 ? (lane >> 3) & 1 : 0;
    const int cs = P.cs;
    float *buf = reinterpret_cast<float *>(wbase);
    uint8_t *stage = wbase + RPW * 4 * PITCH;
    uint32_t *idxw = reinterpret_cast<uint32_t *>(stage);  // [NM / 4][32]: idx << 1 in each byte

    // The tables: a warp reads 32 entries with one chain of loads and hands them
    // round, since every entry has many copies.  Entry nbk is the last bucket's
    // again: a saturated coordinate of 1 reads it.
    for (int i = threadIdx.x; i < D / 32; i += blockDim.x) {
        signs[i] = T.rot_mask[i];
        signs[32 + i] = T.qjl_mask[i];
    }
    for (int e0 = 32 * warp; e0 <= nbk; e0 += 32 * nwarps) {
        const uint32_t lo = T.qlut[min(e0 + lane, nbk - 1) << P.qshift];
        const float bnd = T.boundaries[lo];
        for (int e = lane >> 4; e < 32; e += 2) {
            const uint2 v = make_uint2(__float_as_uint(__shfl_sync(kFull, bnd, e)), __shfl_sync(kFull, lo, e) * 128u);
            if (e0 + e <= nbk) reinterpret_cast<uint2 *>(table)[(e0 + e) * 16 + (lane & 15)] = v;
        }
    }
    for (int e0 = 32 * warp; e0 < P.levels; e0 += 32 * nwarps) {
        const float c = T.centroids[min(e0 + lane, P.levels - 1)];
        for (int e = 0; e < 32; ++e) {
            const float v = __shfl_sync(kFull, c, e);
            if (e0 + e < P.levels) crep[(e0 + e) * 32 + lane] = v;
        }
    }
    __syncthreads();

    // bucket(z) = floor(fma(z, s, c) clamped to [0, 2048)) >> qshift.  s and c
    // over 2048 give the same value over 2048, exactly; adding 2^23 / nbk
    // toward zero leaves its floor times nbk in the low bits.
    const float qs = P.qlut_s * (1.0f / kQlutBuckets), qc = P.qlut_c * (1.0f / kQlutBuckets);
    const float magic = 8388608.0f / (float)nbk;
    const uint32_t entry0 = smem_u32(table) + (lane & 15) * 8 - (__float_as_uint(magic) << 7);
    const uint32_t cent0 = smem_u32(crep) + lane * 4;
    const bool vec4 = ((P.dim & 3) == 0) && ((reinterpret_cast<uintptr_t>(X) & 15) == 0);
    const bool whole8 = (P.dim & 7) == 0;
    const size_t ngroups = (n + RPW - 1) / RPW, step = (size_t)gridDim.x * nwarps;
    const size_t first = (size_t)blockIdx.x * nwarps + warp;

    // the padding past dim stays zero
    for (int v = 0; v < RPW; ++v)
        for (int i = P.dim + lane; i < D; i += 32) buf[v * PITCH + at<D, LPR>(i)] = 0.0f;
    auto fetch = [&](size_t q) {  // rows of group q, asynchronously
        const int nv = n - RPW * q < RPW ? (int)(n - RPW * q) : RPW, d4 = P.dim >> 2;
        for (int v = 0; v < nv; ++v) {
            const float *src = X + (RPW * q + v) * (size_t)P.dim;
            for (int i = lane; i < d4; i += 32)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(buf + v * PITCH + at<D, LPR>(4 * i))),
                             "l"(src + 4 * i) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (vec4 && first < ngroups) fetch(first);

    for (size_t q = first; q < ngroups; q += step) {
        const size_t row0 = RPW * q;
        const int nv = n - row0 < RPW ? (int)(n - row0) : RPW;
        if (vec4) {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        } else {
            for (int v = 0; v < nv; ++v) {
                const float *src = X + (row0 + v) * (size_t)P.dim;
#pragma unroll 1
                for (int i = lane; i < P.dim; i += 32) buf[v * PITCH + at<D, LPR>(i)] = __ldcs(src + i);
            }
        }
        __syncwarp();
        // A group's rows to registers (rows past the last repeat old ones: their
        // codes are not written)
        const float *row = buf + g * PITCH, *mine = row + k + h * (D / 2 + 8);
        u64 p[NP];
#pragma unroll
        for (int i = 0; i < NP; ++i) p[i] = mk2(mine[16 * i], mine[16 * i + 8]);
        // norm: zeros past dim leave the chains as they are
        const float nsq = whole8 ? chain_regs<LPR>(p, lane) : chain_row<D, LPR>(row, P.dim, lane);
        __syncwarp();
        if (vec4 && q + step < ngroups) fetch(q + step);
        // the previous group's codes have left the stage: it holds this group's
        // indices until the units are packed
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
        const float norm = __fsqrt_rn(nsq);
        float pre = (nsq > f32_bits(kNormSqFloorBits)) ? __fdiv_rn(1.0f, norm) : 0.0f;
        float sigma = 0.0f, gamma = 0.0f;

        // pass 0: rotation, sigma, quantize, gamma; pass 1: QJL transform of the
        // residual (one copy of the transform's code)
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass) {
            const uint32_t *sg = signs + 32 * pass + h * (NM / 4);
            const u64 pre2 = mk2(pre, pre), post2 = mk2(P.wht_scale, P.wht_scale);
#pragma unroll
            for (int w = 0; w < NM / 4; ++w) {
                // bit k + 8 j of word w: element k + 8 (4 w + j) keeps its sign
                const uint32_t m = ~sg[w] << (7 - k);
                const u64 f0 = ((u64)((m << 16) & 0x80000000u) << 32) | ((m << 24) & 0x80000000u);
                const u64 f1 = ((u64)(m & 0x80000000u) << 32) | ((m << 8) & 0x80000000u);
                p[2 * w] = fmul2(p[2 * w], pre2) ^ f0;
                p[2 * w + 1] = fmul2(p[2 * w + 1], pre2) ^ f1;
            }
            lane_stage<0>(p, lane);
            lane_stage<1>(p, lane);
            lane_stage<2>(p, lane);
#pragma unroll
            for (int i = 0; i < NP; ++i) {
                float a, b;
                un2(p[i], a, b);
                p[i] = mk2(__fadd_rn(a, b), __fsub_rn(a, b));
            }
            pair_stages<NP, 1>(p);
            if constexpr (LPR == 16) lane_stage<3>(p, lane);  // stride D / 2
#pragma unroll
            for (int i = 0; i < NP; ++i) p[i] = fmul2(p[i], post2);
            if (pass) break;

            sigma = __fsqrt_rn(__fdiv_rn(chain_regs<LPR>(p, lane), (float)D));
            float isg;
            if (f32_bits(kSigmaFloorBits) > sigma) {
                sigma = f32_bits(kSigmaFloorBits);
                isg = f32_bits(kInvSigmaFloorBits);
            } else {
                isg = __fdiv_rn(1.0f, sigma);
            }
#pragma unroll
            for (int w = 0; w < NM / 4; ++w) {
                float x[4];
                un2(p[2 * w], x[0], x[1]);
                un2(p[2 * w + 1], x[2], x[3]);
                uint32_t word = 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float z = __fmul_rn(x[j], isg);
                    float y;
                    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(z), "f"(qs), "f"(qc));
                    const uint32_t u = __float_as_uint(__fadd_rz(y, magic));
                    uint32_t bnd, off;
                    asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(bnd), "=r"(off) : "r"((u << 7) + entry0));
                    if (z > __uint_as_float(bnd)) off += 128;
                    float c;
                    asm("ld.shared.f32 %0, [%1];" : "=f"(c) : "r"(off + cent0));
                    x[j] = __fmaf_rn(-c, sigma, x[j]);
                    word += j == 0 ? off >> 6 : off << (8 * j - 6);  // idx << 1 in byte j
                }
                idxw[32 * w + lane] = word;
                p[2 * w] = mk2(x[0], x[1]);
                p[2 * w + 1] = mk2(x[2], x[3]);
            }
            gamma = __fsqrt_rn(chain_regs<LPR>(p, lane));
            pre = 1.0f;
        }

        // units, trailer
        uint32_t wq[NM / 4];
#pragma unroll
        for (int w = 0; w < NM / 4; ++w) wq[w] = idxw[32 * w + lane];
        __syncwarp();
        uint8_t *code = stage + g * cs;
        constexpr int EB = NIBBLE ? 2 : 1;  // elements a byte
        uint8_t *st0 = code + (k + h * (D / 2 + 8)) / EB, *st1 = code + (k + h * (D / 2 - 8)) / EB;
#pragma unroll
        for (int w = 0; w < NM / 4; ++w) {
            float x[4];
            un2(p[2 * w], x[0], x[1]);
            un2(p[2 * w + 1], x[2], x[3]);
            uint32_t word = wq[w];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (x[j] >= 0.0f) word |= 1u << (8 * j);
            // byte j of a word is element k + 8 (4 w + j): the upper half's lanes
            // store 1, 0, 3, 2, to other banks than the lower half's
            if constexpr (LPR == 16) word = h ? __byte_perm(word, 0, 0x2301) : word;
            if constexpr (NIBBLE) {
                word |= __shfl_down_sync(kFull, word, 1) << 4;
                if (!(k & 1)) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) (j & 1 ? st1 : st0)[4 * (4 * w + j)] = (uint8_t)(word >> (8 * j));
                }
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j) (j & 1 ? st1 : st0)[8 * (4 * w + j)] = (uint8_t)(word >> (8 * j));
            }
        }
        if (k == 0 && h == 0) {
            uint8_t *t = code + P.pb;
            const uint32_t w[3] = {__float_as_uint(norm), __float_as_uint(gamma), __float_as_uint(sigma)};
#pragma unroll
            for (int i = 0; i < 12; ++i) t[i] = (uint8_t)(w[i >> 2] >> (8 * (i & 3)));
        }
        uint8_t *dst = out + row0 * (size_t)cs;
        const int len = nv * cs;
        if (((reinterpret_cast<uintptr_t>(dst) & 15) == 0) && ((len & 15) == 0)) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                             "r"(smem_u32(stage)), "r"(len) : "memory");
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
        } else {
            __syncwarp();
            if (((reinterpret_cast<uintptr_t>(dst) & 3) == 0) && ((len & 3) == 0)) {
                const uint32_t *s1 = reinterpret_cast<const uint32_t *>(stage);
                uint32_t *d1 = reinterpret_cast<uint32_t *>(dst);
#pragma unroll 1
                for (int i = lane; i < (len >> 2); i += 32) __stcs(d1 + i, s1[i]);
            } else {
#pragma unroll 1
                for (int i = lane; i < len; i += 32) dst[i] = stage[i];
            }
        }
    }
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

constexpr int kSmemMax = 227 * 1024;

template <int LOG_D, bool NIBBLE, int LPR, int WARPS>
cudaError_t run(const Params &P, const DevTables &T, const float *X, size_t n, uint8_t *out, int sms,
                cudaStream_t st) {
    constexpr int D = 1 << LOG_D, RPW = 32 / LPR;
    const size_t groups = (n + RPW - 1) / RPW;
    int warps = (kSmemMax - encode_regs_table_bytes(P)) / encode_regs_warp_bytes<D, LPR>(P);
    if (warps > WARPS) warps = WARPS;
    if (warps < 1) return cudaErrorInvalidConfiguration;
    // few rounds: no more warps than they need, so that the last round is as full
    // as the others (20k rows of 384: 35 -> 30 us).  More rounds run into one
    // another, and all warps are better (20k rows of 768, 5 rounds: 70, not 76 us).
    const size_t spread = (groups + sms - 1) / sms;
    const size_t rounds = (spread + warps - 1) / warps;
    if (rounds <= 3) warps = (int)((spread + rounds - 1) / rounds);
    const size_t smem = (size_t)encode_regs_table_bytes(P) + (size_t)warps * encode_regs_warp_bytes<D, LPR>(P);
    auto kern = encode_regs_kernel<LOG_D, NIBBLE, LPR, WARPS>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
    if (e != cudaSuccess) return e;
    size_t blocks = (groups + warps - 1) / warps;
    if (blocks > (size_t)sms) blocks = sms;
    kern<<<(unsigned)blocks, 32 * warps, smem, st>>>(X, n, out, P, T);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_encode_regs(const Params &P, const DevTables &T, const float *X, size_t n, uint8_t *out,
                               int sms, cudaStream_t st) {
    switch (P.log2D) {
        case 8: return P.nibble ? run<8, true, 8, 20>(P, T, X, n, out, sms, st) : run<8, false, 8, 20>(P, T, X, n, out, sms, st);
        case 9: return P.nibble ? run<9, true, 8, 16>(P, T, X, n, out, sms, st) : run<9, false, 8, 16>(P, T, X, n, out, sms, st);
        default: return P.nibble ? run<10, true, 16, 16>(P, T, X, n, out, sms, st) : run<10, false, 16, 16>(P, T, X, n, out, sms, st);
    }
}

}  // namespace tq
