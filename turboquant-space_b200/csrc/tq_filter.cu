// tq_filter.cu -- the filter pass of the serving top-k (variant 6): for each
// query row the kc codes of smallest approximate distance, which the exact
// stage (tq_exact.cu) rescores and certifies against the pass's error bound.
//
// One FP16 product per term instead of a hi/lo pair's two or three: the pass
// only has to leave out codes that cannot be among the top-k, and its error
// bound can be stated from the roundings themselves.  With q~ = fp16(q_rot),
// s~ = fp16(s_q), c~ = fp16(alpha c) / alpha and rho~ = fp16(alpha g / sigma) /
// alpha (g = scale gamma, the QJL factor of a code; b = its +-1 signs) the pass
// forms S = <q~, c~> + rho~ <s~, b> in one accumulator and takes
// sigma |x| |q| S for |x| |q| (sigma <q_rot, c> + g <s_q, b>).  By
// Cauchy-Schwarz the difference is at most |q| times
//     |dq| M0 + |q| M1 + |ds| M2 + |s~| M3          (2-norms; dq = q_rot - q~ ...)
//   + (mmas + 1) 2^-20 (|q~| M0 + |s~| (M2 + M3))   (accumulation, see rescore)
//   + sums (M0 + M1 + M2)                           (FP32 sums on both sides: filter_sums)
// with the index-wide maxima
//   M0 = sigma |x| |c~|, M1 = sigma |x| |c - c~|, M2 = g |x| sqrt(D),
//   M3 = |g - sigma rho~| |x| sqrt(D).
// At 384-d 4-bit that is 0.5 times the bound of the hi/lo pairs' pass (which
// bounds every term by its own largest value), for two fifths of the MMAs and
// no operand planes of the corpus.
//
// The kc smallest come from thresholds, not from lists kept per thread:
//   1. the distances of kFilterSample codes are written out, one code from each
//      of as many equal runs of the corpus, at a hashed place in it: whatever the
//      order that the corpus is stored in (by cluster, by time, round robin), a
//      group of codes has about its share of the sample.  The kc-th smallest of a
//      row is a threshold that at least kc codes meet;
//   2. a larger spread sample, about sqrt(kFilterSample n) codes, lists the
//      codes that meet it, and the kc-th smallest of the list is a closer one
//      (larger corpora only);
//   3. every code that meets it is listed, about kc sqrt(n / kFilterSample) of
//      them a row (kc n / kFilterSample without step 2), and the kc smallest of the list are the candidates.
// A row whose list overflows, holds fewer than kc codes or whose scalings are
// out of range is marked bad and stays uncertified.
//
// Kernel: as cgemm_kernel (tq_cgemm.cu) on CTA pairs: 256 codes by up to 256
// rows a tile, code words through a cp.async ring, decoded in shared memory.
// A K block of centroids and one of signs come from the same words, decoded by
// four warps each.  22 warps:
//   0 TMA producer, 1 MMA issuer, 2..5 code loaders, 6..9 centroid decoders,
//   10..13 sign decoders, 14..21 epilogue.
// A block's MMAs take 512 clocks; its shared-memory traffic per CTA is 68 KB
// (16 KB row tile, 16 KB decoded codes, 32 KB operand reads), 133 B/clk.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "tq_filter.h"
#include "tq_tables.h"
#include "tq_tc.cuh"

namespace tq {
namespace {

constexpr int FL_BM = 128, FL_BK = 64, FL_ROWS = 256;
constexpr int FL_A_BYTES = FL_BM * 128;
constexpr int FL_THREADS = 22 * 32;
constexpr int FL_MAX_STAGES = 8, FL_MAX_RING = 8;
constexpr int FL_BAR_BYTES = 512;
constexpr int FL_UV_BYTES = 8 * 1024;       // each epilogue warp's copy of its columns' constants
constexpr int FL_QUEUE = 64;               // hits an epilogue warp holds back
constexpr int FL_HIT_BYTES = 8 * FL_QUEUE * 20;
constexpr int FL_FIXED = 1024 + FL_BAR_BYTES + FL_UV_BYTES + FL_HIT_BYTES;
constexpr int FL_TAB_BYTES = 128 * 128;    // byte codes: 128 entries x 32 lanes, 4 bytes
constexpr int FL_SMEM_MAX = 227 * 1024;
constexpr float kRowScale = 16384.0f;
constexpr int kErrFull = 1, kErrEmpty = 2, kErrTmemFull = 3, kErrTmemEmpty = 4;
constexpr unsigned kAll = 0xffffffffu;

// Passes: the distances of a spread sample; the codes of a larger one that meet the
// thresholds; all codes that do.
enum { kSample = 0, kCollect = 1, kCollectAll = 2 };

struct FlArgs {
    const uint8_t *codes;
    size_t n;
    int cs, pb, levels;
    const float *centroids;
    float alpha, undo;     // S = undo x accumulator
    const uint32_t *rho;
    int KBm;               // 64-value blocks of each part
    int box, stages, ring;
    unsigned nt;           // code tiles of this launch
    unsigned long long step;  // codes per position of them, 32.32 fixed point (code_at)
    const int *m_dev;
    const float2 *uv, *r12;
    const float *thr;
    float *samp;
    int *cnt;
    float *list_d;
    int *list_i;
    int *err;
};

// 8 units (a word of nibbles) -> 8 FP16 centroids by byte tables of entries 0..7.
__device__ __forceinline__ uint4 nib_cent1(uint32_t x, const uint32_t (&l)[2], const uint32_t (&h)[2]) {
    const uint32_t s0 = (x >> 1) & 0x77777777u, s1 = s0 >> 16;
    uint32_t a = __byte_perm(l[0], l[1], s0), b = __byte_perm(h[0], h[1], s0);
    uint4 r;
    r.x = __byte_perm(a, b, 0x5140u);
    r.y = __byte_perm(a, b, 0x7362u);
    a = __byte_perm(l[0], l[1], s1), b = __byte_perm(h[0], h[1], s1);
    r.z = __byte_perm(a, b, 0x5140u);
    r.w = __byte_perm(a, b, 0x7362u);
    return r;
}
// The QJL bits of 8 units -> +-rho (`rho` a pair of non-negative FP16, `pm`
// the high bytes of -rho and rho): a PRMT picks four coordinates' high bytes
// by their bits, two more put rho's low byte beside each.
__device__ __forceinline__ uint32_t sign_bytes(uint32_t rho) {
    return ((rho >> 8) & 0xFFu) * 0x0101u | 0x80u;
}
__device__ __forceinline__ uint4 nib_sign1(uint32_t x, uint32_t rho, uint32_t pm) {
    const uint32_t s = x & 0x11111111u;
    const uint32_t a = __byte_perm(pm, 0u, s), b = __byte_perm(pm, 0u, s >> 16);
    return make_uint4(__byte_perm(a, rho, 0x1404u), __byte_perm(a, rho, 0x3424u), __byte_perm(b, rho, 0x1404u),
                      __byte_perm(b, rho, 0x3424u));
}
// The same for units of a byte each.
__device__ __forceinline__ uint4 byte_sign1(uint32_t x0, uint32_t x1, uint32_t rho, uint32_t pm) {
    return make_uint4(__byte_perm(rho, pm, ((x0 << 4) & 0x1010u) | 0x4040u),
                      __byte_perm(rho, pm, ((x0 >> 12) & 0x1010u) | 0x4040u),
                      __byte_perm(rho, pm, ((x1 << 4) & 0x1010u) | 0x4040u),
                      __byte_perm(rho, pm, ((x1 >> 12) & 0x1010u) | 0x4040u));
}

__device__ __forceinline__ unsigned long long pack2f(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
// Two independent IEEE FMAs on a register pair.
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// Position `lin` of a pass over one code in step / 2^32 -> code: a hashed place in the
// position's run of the corpus, [lin, lin + 1) step / 2^32.  (step = 2^32: every code.)
__device__ __forceinline__ size_t code_at(unsigned long long step, uint32_t lin) {
    uint32_t h = lin * 0x9E3779B1u;
    h = (h ^ (h >> 15)) * 0x85EBCA6Bu;
    h ^= h >> 13;
    return (size_t)((lin * step + __umul64hi(step, (unsigned long long)h << 32)) >> 32);
}

// The approximate distance of one pair: S the unscaled accumulator, c1 = sigma
// |x| undo, c2 = |x|^2, r = (|q|, |q|^2).
__device__ __forceinline__ float fl_dist(float S, float c1, float c2, float2 r) {
    return fmaxf(__fmaf_rn(-2.0f, __fmul_rn(__fmul_rn(S, r.x), c1), __fadd_rn(r.y, c2)), 0.0f);
}

template <bool NIB, int MODE>
__global__ void __launch_bounds__(FL_THREADS, 1) filter_kernel(const __grid_constant__ CUtensorMap map,
                                                               const FlArgs p) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    constexpr int WPI = NIB ? 1 : 2;
    constexpr int RING_BYTES = FL_BM * 32 * WPI;
    const uint32_t rank = cluster_rank();
    const int b_bytes = p.box * 128;
    const int stage_bytes = FL_A_BYTES + b_bytes;
    const uint32_t tiles0 = smem_u32(smem);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + p.stages * stage_bytes);
    // full[8], empty[8], pfull[8], cfull[8], cempty[8], xfull[2], xempty[2], drain; the TMEM slot
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 64, pfull0 = empty0 + 64, cfull0 = pfull0 + 64;
    const uint32_t cempty0 = cfull0 + 64, xfull0 = cempty0 + 64, xempty0 = xfull0 + 16, drain = xempty0 + 16;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 45);
    float4 *s_uv = reinterpret_cast<float4 *>(reinterpret_cast<unsigned char *>(bars) + FL_BAR_BYTES);
    float *s_hits = reinterpret_cast<float *>(reinterpret_cast<unsigned char *>(s_uv) + FL_UV_BYTES);
    unsigned char *ring = reinterpret_cast<unsigned char *>(s_hits) + FL_HIT_BYTES;
    const uint32_t ring0 = smem_u32(ring);
    uint32_t *btab = reinterpret_cast<uint32_t *>(ring + p.ring * RING_BYTES);
    const int warp = __shfl_sync(kAll, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(full0 + 8 * s, 1 + 4);  // the producer and four decoder warps
            mbar_init(empty0 + 8 * s, 1);
            mbar_init(pfull0 + 8 * s, 1);
        }
        for (int k = 0; k < p.ring; ++k) {
            mbar_init(cfull0 + 8 * k, 128);  // every loader thread
            mbar_init(cempty0 + 8 * k, 8);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(xfull0 + 8 * b, 1);
            mbar_init(xempty0 + 8 * b, 16);  // eight epilogue warps of each CTA
        }
        mbar_init(drain, 1);
        mbar_init_fence();
    }
    if (warp == 1) tmem_alloc512<true>(smem_u32(tmem_slot));
    if constexpr (!NIB) {
        for (int i = threadIdx.x; i < 128 * 32; i += FL_THREADS) {
            const int v = i >> 5;
            btab[i] = v < p.levels ? __half_as_ushort(__float2half_rn(p.centroids[v] * p.alpha)) : 0u;
        }
    }
    tc_fence_before();
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int m = *p.m_dev, KBm = p.KBm, KB = 2 * KBm;
    // rows per MMA: all 256, or a small batch's own count
    const int N = m >= FL_ROWS ? FL_ROWS : ((m + 31) & ~31);
    const unsigned mbs = (unsigned)((m + FL_ROWS - 1) / FL_ROWS);
    const unsigned tiles = m > 0 ? mbs * p.nt : 0u, grid = gridDim.x >> 1, t0 = blockIdx.x >> 1;
    // code of row r of this CTA's half of tile t
    auto code_of = [&](unsigned t, int r) -> size_t {
        const uint32_t lin = (t % p.nt) * (unsigned)kFilterTile + rank * FL_BM + r;
        return MODE == kCollectAll ? lin : code_at(p.step, lin);
    };

    if (warp == 0) {
        // ---------------- TMA producer: the rows' K blocks ----------------
        if (lane == 0) {
            uint32_t s = 0, ph = 1, it = 0;
            bool ok = true;
            for (unsigned t = t0; t < tiles && ok; t += grid) {
                const int row = (int)((t / p.nt) * FL_ROWS + rank * (N / 2));
                for (int kb = 0; kb < KB; ++kb, ++it) {
                    if (!mbar_wait(empty0 + 8 * s, ph, p.err, kErrEmpty)) { ok = false; break; }
                    const uint32_t fb = full0 + 8 * s;
                    mbar_expect_tx(fb, b_bytes);
                    tma_load_2d(tiles0 + s * stage_bytes + FL_A_BYTES, &map,
                                ((kb >> 1) + (kb & 1) * KBm) * FL_BK, row, fb);
                    if (++s == (uint32_t)p.stages) { s = 0; ph ^= 1u; }
                }
            }
            for (uint32_t k = 0; k < (uint32_t)p.stages && k < it; ++k) {
                const uint32_t j = it - 1 - k;
                mbar_drain(full0 + 8 * (j % p.stages), (j / p.stages) & 1u);
            }
        }
    } else if (warp == 1 && rank != 0) {
        // ---------------- rank 1: reports each full stage to rank 0 ----------------
        uint32_t s = 0, ph = 0;
        bool ok = true;
        for (unsigned t = t0; t < tiles && ok; t += grid) {
            for (int kb = 0; kb < KB; ++kb) {
                if (!mbar_wait_warp(full0 + 8 * s, ph, p.err, kErrFull)) { ok = false; break; }
                if (lane == 0) mbar_arrive_cluster(rank0_addr(pfull0 + 8 * s));
                if (++s == (uint32_t)p.stages) { s = 0; ph ^= 1u; }
            }
        }
        // the pair's last commit: nothing of rank 0's is under way to this CTA's barriers
        if (lane == 0) mbar_drain(drain, 0);
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer (uniform warp, one elected lane) ----------------
        const bool lead = elect_one();
        const uint32_t idesc = (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(2 * FL_BM >> 4) << 24);
        uint32_t s = 0, ph = 0, gc = 0;
        bool ok = true;
        for (unsigned t = t0; t < tiles && ok; t += grid, ++gc) {
            const uint32_t b = gc & 1u, xph = (gc >> 1) & 1u;
            if (!mbar_wait_cluster_warp(xempty0 + 8 * b, xph ^ 1u, p.err, kErrTmemEmpty)) { ok = false; break; }
            tc_fence_after();
            const uint32_t d = tmem_base + b * 256u;
            for (int kb = 0; kb < KB; ++kb) {
                if (!mbar_wait_warp(full0 + 8 * s, ph, p.err, kErrFull)) { ok = false; break; }
                if (!mbar_wait_cluster_warp(pfull0 + 8 * s, ph, p.err, kErrFull)) { ok = false; break; }
                tc_fence_after();
                const uint32_t a = sw128_desc_lo(tiles0 + s * stage_bytes), bd = a + (FL_A_BYTES >> 4);
                if (lead) {
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        umma_f16<true>(d, a + 2 * kk, bd + 2 * kk, idesc, (kb | kk) ? 1u : 0u);
                    umma_commit_pair(empty0 + 8 * s);
                }
                if (++s == (uint32_t)p.stages) { s = 0; ph ^= 1u; }
            }
            if (ok && lead) umma_commit_pair(xfull0 + 8 * b);
        }
        // every MMA issued must be complete before the tensor memory is freed
        if (lead) {
            umma_commit_pair(drain);
            mbar_drain(drain, 0);
        }
        __syncwarp();
    } else if (warp < 6) {
        // ---------------- code loaders ----------------
        const int r0 = (warp - 2) * 32 + (lane >> 3), c = lane & 7;
        uint32_t cs = 0, cph = 1;
        bool ok = true;
        for (unsigned t = t0; t < tiles && ok; t += grid) {
            // rows past n repeat the last code; a tile half's codes span at most a
            // 64th of the corpus where it is sampled, so 32 bits hold their offsets
            const size_t j0 = min(code_of(t, 0), p.n - 1);
            const uint8_t *base = p.codes + j0 * (size_t)p.cs + 4 * c;
            uint32_t ro[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                ro[i] = (uint32_t)(min(code_of(t, r0 + 4 * i), p.n - 1) - j0) * (uint32_t)p.cs;
            for (int q = 0; q < KBm; ++q) {
                if (!mbar_wait_warp(cempty0 + 8 * cs, cph, p.err, kErrEmpty)) { ok = false; break; }
                const uint32_t dst = ring0 + cs * RING_BYTES + r0 * (32 * WPI) + 4 * c;
                const int o = q * (32 * WPI);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
#pragma unroll
                    for (int w = 0; w < WPI; ++w)  // zero beyond the packed bytes (D < 64)
                        cp_async4(dst + 4 * i * (32 * WPI) + 32 * w, base + ro[i] + o + 32 * w,
                                  o + 32 * w + 4 * c < p.pb ? 4u : 0u);
                }
                cp_async_arrive(cfull0 + 8 * cs);
                if (++cs == (uint32_t)p.ring) { cs = 0; cph ^= 1u; }
            }
        }
        cp_async_wait_all();
    } else if (warp < 14) {
        // ---------------- decoders: warps 6..9 centroids, 10..13 signs ----------------
        const bool cent = warp < 10;
        const int r0 = ((warp - 6) & 3) * 32 + (lane >> 3), c = lane & 7;
        const int sw = (c ^ (r0 & 7)) << 4;  // the chunk's place in a row; rows 4 apart flip bit 6
        uint32_t tl[2] = {0u, 0u}, th[2] = {0u, 0u};
        if (NIB && cent) {
#pragma unroll
            for (int v = 0; v < 8; ++v) {
                const uint32_t h =
                    v < p.levels ? __half_as_ushort(__float2half_rn(p.centroids[v] * p.alpha)) : 0u;
                tl[v >> 2] |= (h & 0xFFu) << (8 * (v & 3));
                th[v >> 2] |= (h >> 8) << (8 * (v & 3));
            }
        }
        const uint32_t *tb = btab + lane;
        // stage s of this group's next block: every other one
        uint32_t s = cent ? 0u : 1u, ph = 1, cs = 0, cph = 0;
        bool ok = true;
        for (unsigned t = t0; t < tiles && ok; t += grid) {
            uint32_t rho[8], pm[8];
            if (!cent) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const size_t j = code_of(t, r0 + 4 * i);
                    rho[i] = j < p.n ? __ldg(p.rho + j) : 0u;
                    pm[i] = sign_bytes(rho[i]);
                }
            }
            for (int q = 0; q < KBm; ++q) {
                if (!mbar_wait_warp(cfull0 + 8 * cs, cph, p.err, kErrFull)) { ok = false; break; }
                uint32_t w[8][WPI];
                const unsigned char *rb = ring + cs * RING_BYTES;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if constexpr (NIB) {
                        w[i][0] = *reinterpret_cast<const uint32_t *>(rb + (r0 + 4 * i) * 32 + 4 * c);
                    } else {
                        const uint2 v = *reinterpret_cast<const uint2 *>(rb + (r0 + 4 * i) * 64 + 8 * c);
                        w[i][0] = v.x;
                        w[i][WPI - 1] = v.y;
                    }
                }
                if (!mbar_wait_warp(empty0 + 8 * s, ph, p.err, kErrEmpty)) { ok = false; break; }
                unsigned char *dst = smem + s * stage_bytes + r0 * 128;
                if (cent) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        uint4 v;
                        if constexpr (NIB) {
                            v = nib_cent1(w[i][0], tl, th);
                        } else {
                            uint32_t e[8];
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                                e[k] = tb[((w[i][k >> 2] >> (8 * (k & 3) + 1)) & 0x7Fu) * 32];
                            v = make_uint4(__byte_perm(e[0], e[1], 0x5410u), __byte_perm(e[2], e[3], 0x5410u),
                                           __byte_perm(e[4], e[5], 0x5410u), __byte_perm(e[6], e[7], 0x5410u));
                        }
                        *reinterpret_cast<uint4 *>(dst + 512 * i + (sw ^ ((i & 1) << 6))) = v;
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        uint4 v;
                        if constexpr (NIB) v = nib_sign1(w[i][0], rho[i], pm[i]);
                        else v = byte_sign1(w[i][0], w[i][WPI - 1], rho[i], pm[i]);
                        *reinterpret_cast<uint4 *>(dst + 512 * i + (sw ^ ((i & 1) << 6))) = v;
                    }
                }
                fence_proxy_async_smem();  // the generic stores before the MMAs' async reads
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(full0 + 8 * s);
                    mbar_arrive(cempty0 + 8 * cs);
                }
                s += 2;
                if (s >= (uint32_t)p.stages) { s -= p.stages; ph ^= 1u; }
                if (++cs == (uint32_t)p.ring) { cs = 0; cph ^= 1u; }
            }
        }
    } else {
        // ---------------- epilogue: one code per thread, half of the rows ----------------
        const int quad = warp & 3, half = (warp - 14) >> 2, cpt = N >> 1;
        const uint32_t lanes = tmem_base + ((uint32_t)(32 * quad) << 16) + (uint32_t)(half * cpt);
        float4 *uv = s_uv + (warp - 14) * 64;  // (u, u, v, v) of two columns each
        // Hits wait in the warp's queue, so that up to 64 of them share the latency
        // of the list counters' atomics.
        float *hq = s_hits + (warp - 14) * (5 * FL_QUEUE);
        int nq = 0;
        auto flush = [&]() {
            __syncwarp();
            for (int i = lane; i < nq; i += 32) {
                const int row = __float_as_int(hq[3 * FL_QUEUE + i]);
                const float d = fl_dist(hq[i], hq[FL_QUEUE + i], hq[2 * FL_QUEUE + i], __ldg(p.r12 + row));
                if (!(d > __ldg(p.thr + row))) {
                    const int at = atomicAdd(p.cnt + row, 1);
                    if (at < kFilterCap) {
                        p.list_d[(size_t)row * kFilterCap + at] = d;
                        p.list_i[(size_t)row * kFilterCap + at] = __float_as_int(hq[4 * FL_QUEUE + i]);
                    }
                }
            }
            __syncwarp();
            nq = 0;
        };
        uint32_t gc = 0;
        bool ok = true;
        unsigned mb_have = 0xffffffffu;
        for (unsigned t = t0; t < tiles && ok; t += grid, ++gc) {
            const unsigned mb = t / p.nt;
            const int row0 = (int)(mb * FL_ROWS) + half * cpt;  // this warp's rows row0 .. row0 + cpt - 1
            if (MODE != kSample && mb != mb_have) {
                __syncwarp();
                for (int i = lane; i < (cpt >> 1); i += 32) {
                    // rows past m never pass
                    const int r = row0 + 2 * i;
                    const float2 a = r < m ? __ldg(p.uv + r) : make_float2(INFINITY, 0.0f);
                    const float2 c = r + 1 < m ? __ldg(p.uv + r + 1) : make_float2(INFINITY, 0.0f);
                    uv[i] = make_float4(a.x, c.x, a.y, c.y);
                }
                __syncwarp();
                mb_have = mb;
            }
            const size_t code = code_of(t, 32 * quad + lane);
            const bool live = code < p.n;
            float norm = 0.0f, sigma = 0.0f;
            if (live) {
                const float *meta = reinterpret_cast<const float *>(p.codes + code * (size_t)p.cs + p.pb);
                norm = __ldg(meta);
                sigma = __ldg(meta + 2);
            }
            const float c1 = __fmul_rn(__fmul_rn(sigma, norm), p.undo);
            // a code past the end never passes
            const float c2 = live ? __fmul_rn(norm, norm) : INFINITY;
            const uint32_t b = gc & 1u, xph = (gc >> 1) & 1u;
            if (!mbar_wait_warp(xfull0 + 8 * b, xph, p.err, kErrTmemFull)) { ok = false; break; }
            tc_fence_after();
            const uint32_t X = lanes + b * 256u;
            uint32_t xa[16], xb[16];
            __syncwarp();
            tmem_ld16_nw(X, xa);
            auto piece = [&](const uint32_t (&x)[16], int k0) {
                if constexpr (MODE == kSample) {
                    float *o = p.samp + (size_t)(row0 + k0) * kFilterSample + (t % p.nt) * kFilterTile +
                               rank * FL_BM + 32 * quad + lane;
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (row0 + k0 + j < m)
                            o[(size_t)j * kFilterSample] =
                                live ? fl_dist(__uint_as_float(x[j]), c1, c2, __ldg(p.r12 + row0 + k0 + j)) : INFINITY;
                    }
                } else {
                    // a column may pass where u + v |x|^2 - S sigma |x| is negative
                    const unsigned long long c2c2 = pack2f(c2, c2), c1n = pack2f(-c1, -c1);
                    uint32_t g[16], any = 0u;
#pragma unroll
                    for (int j = 0; j < 16; j += 2) {
                        const float4 w = uv[(k0 + j) >> 1];
                        const unsigned long long lim = fma2(c2c2, pack2f(w.z, w.w), pack2f(w.x, w.y));
                        const unsigned long long gap =
                            fma2(pack2f(__uint_as_float(x[j]), __uint_as_float(x[j + 1])), c1n, lim);
                        g[j] = (uint32_t)gap;
                        g[j + 1] = (uint32_t)(gap >> 32);
                        any |= g[j] | g[j + 1];
                    }
                    if (__any_sync(kAll, (int)any < 0)) {
                        uint32_t mine = 0u;
#pragma unroll
                        for (int j = 0; j < 16; ++j) mine |= (g[j] >> 31) << j;
                        do {  // up to two hits a lane a round
                            const uint32_t rest = mine & (mine - 1u), take = mine & ~(rest & (rest - 1u));
                            const unsigned b1 = __ballot_sync(kAll, mine != 0u), b2 = __ballot_sync(kAll, rest != 0u);
                            if (nq + __popc(b1) + __popc(b2) > FL_QUEUE) flush();
                            const unsigned lt = (1u << lane) - 1u;
                            int at = nq + __popc(b1 & lt) + __popc(b2 & lt);
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                if ((take >> j) & 1u) {
                                    hq[at] = __uint_as_float(x[j]);
                                    hq[FL_QUEUE + at] = c1;
                                    hq[2 * FL_QUEUE + at] = c2;
                                    hq[3 * FL_QUEUE + at] = __int_as_float(row0 + k0 + j);  // below m
                                    hq[4 * FL_QUEUE + at] = __int_as_float((int)code);
                                    ++at;
                                }
                            }
                            nq += __popc(b1) + __popc(b2);
                            mine &= ~take;
                        } while (__any_sync(kAll, mine != 0u));
                    }
                }
            };
            // pieces of 16 columns, the next one's load in flight
            for (int k0 = 0; k0 < cpt; k0 += 32) {
                tmem_wait_ld();
                if (k0 + 16 < cpt) tmem_ld16_nw(X + k0 + 16, xb);
                piece(xa, k0);
                if (k0 + 16 < cpt) {
                    __syncwarp();
                    tmem_wait_ld();
                    if (k0 + 32 < cpt) tmem_ld16_nw(X + k0 + 32, xa);
                    piece(xb, k0 + 16);
                }
                __syncwarp();
            }
            tc_fence_before();
            if (lane == 0) mbar_arrive_cluster(rank0_addr(xempty0 + 8 * b));
        }
        if (MODE != kSample && ok) flush();
    }
    tc_fence_before();
    cluster_sync();  // no CTA leaves while the other may still arrive on its barriers or read its memory
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc512<true>(tmem_base);
    }
}

// Prepared queries -> FP16 planes (rows of 2 x 64 KBm values, zero past D in each
// part), the bound's 2-norms and |q|, |q|^2.  One warp per row.
__global__ void __launch_bounds__(256) filter_rows_kernel(const float *__restrict__ q_rot,
                                                          const float *__restrict__ s_q,
                                                          const float *__restrict__ norms,
                                                          const int *__restrict__ m_dev, int D, int KBm,
                                                          __half *__restrict__ planes,
                                                          float4 *__restrict__ rowq,
                                                          float2 *__restrict__ r12) {
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= *m_dev) return;
    const int half = KBm * FL_BK;
    float e2[2] = {0.0f, 0.0f}, n2[2] = {0.0f, 0.0f};
#pragma unroll
    for (int part = 0; part < 2; ++part) {
        const float *src = (part ? s_q : q_rot) + (size_t)row * D;
        __half *dst = planes + (size_t)row * 2 * half + part * half;
        for (int k = 2 * lane; k < half; k += 64) {
            const float a = k < D ? src[k] : 0.0f, b = k + 1 < D ? src[k + 1] : 0.0f;
            const __half ha = __float2half_rn(a * kRowScale), hb = __float2half_rn(b * kRowScale);
            *reinterpret_cast<__half2 *>(dst + k) = __halves2half2(ha, hb);
            const float ra = __half2float(ha) * (1.0f / kRowScale), rb = __half2float(hb) * (1.0f / kRowScale);
            e2[part] += (a - ra) * (a - ra) + (b - rb) * (b - rb);
            n2[part] += ra * ra + rb * rb;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
        for (int part = 0; part < 2; ++part) {
            e2[part] += __shfl_xor_sync(kAll, e2[part], off);
            n2[part] += __shfl_xor_sync(kAll, n2[part], off);
        }
    }
    if (lane == 0) {
        // 1.0001: the FP32 sums' own rounding
        rowq[row] = make_float4(1.0001f * sqrtf(e2[0]), 1.0001f * sqrtf(e2[1]), 1.0001f * sqrtf(n2[0]),
                                1.0001f * sqrtf(n2[1]));
        r12[row] = make_float2(norms[2 * row + 1], norms[2 * row]);
    }
}

// The kc-th smallest of up to V x 256 non-negative values held V a thread as bit
// patterns (+inf when there are fewer): a four-way search over the patterns,
// one barrier a step.
template <int V>
__device__ __forceinline__ uint32_t kth_smallest(const uint32_t (&v)[V], int kc) {
    __shared__ int2 s_c[2][8];
    uint32_t lo = 0u, hi = 0x7f800000u;
    for (int step = 0; lo < hi; ++step) {
        const uint32_t w = hi - lo, q = w >> 2;
        const uint32_t p0 = lo + q, p1 = lo + (w >> 1), p2 = lo + (w >> 1) + q;  // below hi
        int c01 = 0, c2 = 0;
#pragma unroll
        for (int i = 0; i < V; ++i) {
            c01 += (v[i] <= p0 ? 1 : 0) + (v[i] <= p1 ? 0x10000 : 0);
            c2 += v[i] <= p2 ? 1 : 0;
        }
        c01 = __reduce_add_sync(kAll, c01);
        c2 = __reduce_add_sync(kAll, c2);
        int2 *s = s_c[step & 1];
        if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = make_int2(c01, c2);
        __syncthreads();
        c01 = c2 = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            c01 += s[k].x;
            c2 += s[k].y;
        }
        if ((c01 & 0xFFFF) >= kc) hi = p0;
        else if ((c01 >> 16) >= kc) { lo = p0 + 1; hi = p1; }
        else if (c2 >= kc) { lo = p1 + 1; hi = p2; }
        else lo = p2 + 1;
    }
    __syncthreads();  // the counts' memory may be used again
    return hi;
}

// A row's threshold from its sample (DENSE) or its list, and the test's
// constants: with k = 1 / (2 |q|), u = k (|q|^2 - T'), v = k, a code may
// pass where u + v |x|^2 - S sigma |x| < 0, that is where its distance is below
// T'; T' = T relaxed by the test's own rounding (the listing compares with T
// itself).  A NaN does not pass: its corpus or row is never certified.  A
// row of |q| = 0 has S = 0 and takes k = 1.  Empties the row's list.
template <bool DENSE>
__global__ void __launch_bounds__(256) filter_threshold_kernel(const int *__restrict__ m_dev, int kc,
                                                               int ns, const float *__restrict__ samp,
                                                               const float *__restrict__ list_d,
                                                               int *__restrict__ cnt,
                                                               const float2 *__restrict__ r12,
                                                               float2 *__restrict__ uv,
                                                               float *__restrict__ thr) {
    const int row = blockIdx.x;
    if (row >= *m_dev) return;
    constexpr int V = (DENSE ? kFilterSample : kFilterCap) / 256;
    const int have = DENSE ? ns : min(cnt[row], kFilterCap);
    const float *src = DENSE ? samp + (size_t)row * kFilterSample : list_d + (size_t)row * kFilterCap;
    uint32_t v[V];
#pragma unroll
    for (int i = 0; i < V; ++i) {
        const int k = threadIdx.x + 256 * i;
        v[i] = k < have ? __float_as_uint(src[k]) : 0x7f800000u;
    }
    float T = __uint_as_float(kth_smallest<V>(v, kc));
    if (threadIdx.x == 0) {
        if (!DENSE) T = fminf(T, thr[row]);  // a list that overflowed or fell short keeps the earlier one
        const float2 r = r12[row];
        const float k = r.x > 0.0f ? 0.5f / r.x : 1.0f;
        const float Tr = T + 8e-6f * (T + r.y) + 1e-30f;
        uv[row] = make_float2(k * (r.y - Tr), k);
        thr[row] = T;
        cnt[row] = 0;
    }
}

// A row's kc smallest listed codes, ascending by (distance, index).
__global__ void __launch_bounds__(256) filter_select_kernel(const int *__restrict__ m_dev, int kc, size_t n,
                                                            const int *__restrict__ cnt,
                                                            const float *__restrict__ list_d,
                                                            const int *__restrict__ list_i,
                                                            const float2 *__restrict__ r12,
                                                            float *__restrict__ cand_d,
                                                            long long *__restrict__ cand_i,
                                                            int *__restrict__ bad) {
    __shared__ float s_d[32];
    __shared__ int s_i[32], s_n;
    const int row = blockIdx.x;
    if (row >= *m_dev) return;
    const int total = cnt[row], have = min(total, kFilterCap);
    const float *ld = list_d + (size_t)row * kFilterCap;
    const int *li = list_i + (size_t)row * kFilterCap;
    uint32_t v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int k = threadIdx.x + 256 * i;
        v[i] = k < have ? __float_as_uint(ld[k]) : 0xffffffffu;
    }
    const uint32_t t = kth_smallest<16>(v, kc);
    if (threadIdx.x == 0) s_n = 0;
    if (threadIdx.x < 32) {
        s_d[threadIdx.x] = INFINITY;
        s_i[threadIdx.x] = 0x7fffffff;
    }
    __syncthreads();
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {  // below the kc-th value, then equal to it
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (pass == 0 ? v[i] < t : v[i] == t) {
                const int at = atomicAdd(&s_n, 1);
                if (at < kc) {
                    s_d[at] = __uint_as_float(v[i]);
                    s_i[at] = li[threadIdx.x + 256 * i];
                }
            }
        }
        __syncthreads();
    }
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    float d = s_d[lane];
    int ix = s_i[lane];
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            const float od = __shfl_xor_sync(kAll, d, stride);
            const int ox = __shfl_xor_sync(kAll, ix, stride);
            const bool mine_first = d < od || (d == od && ix < ox);
            const bool keep_min = ((lane & size) == 0) == ((lane & stride) == 0);
            if (keep_min != mine_first) {
                d = od;
                ix = ox;
            }
        }
    }
    if (lane < kc) {
        cand_d[(size_t)row * kc + lane] = d;
        cand_i[(size_t)row * kc + lane] = ix == 0x7fffffff ? -1 : (long long)ix;
    }
    if (lane == 0) {
        const float q = r12[row].x;  // the test's constants are out of range beyond this
        const bool range = q == 0.0f || (q > 1e-15f && q < 1e15f);
        bad[row] = (total > kFilterCap || (size_t)total < min((size_t)kc, n) || !range) ? 1 : 0;
    }
}

// rho and the index-wide maxima: one warp per code.
__global__ void __launch_bounds__(256) filter_index_kernel(Params P, DevTables T,
                                                           const uint8_t *__restrict__ codes, size_t n,
                                                           float alpha, uint32_t *__restrict__ rho,
                                                           float *__restrict__ bound) {
    __shared__ float s_c2[256], s_e2[256];  // (c~)^2 and (c - c~)^2 per entry
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        const float c = i < P.levels ? T.centroids[i] : 0.0f;
        const float r = __half2float(__float2half_rn(c * alpha)) / alpha;
        s_c2[i] = r * r;
        s_e2[i] = (c - r) * (c - r);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    float M[kFilterBound] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (size_t j = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5); j < n; j += (size_t)gridDim.x * 8) {
        const uint8_t *code = codes + j * (size_t)P.cs;
        float c2 = 0.0f, e2 = 0.0f;
        for (int b = lane; b < P.pb; b += 32) {
            const unsigned u = code[b];
            if (P.nibble) {
                const int i0 = (u & 15u) >> 1, i1 = u >> 5;
                c2 += s_c2[i0] + s_c2[i1];
                e2 += s_e2[i0] + s_e2[i1];
            } else {
                c2 += s_c2[u >> 1];
                e2 += s_e2[u >> 1];
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            c2 += __shfl_xor_sync(kAll, c2, off);
            e2 += __shfl_xor_sync(kAll, e2, off);
        }
        const float *meta = reinterpret_cast<const float *>(code + P.pb);
        const float xn = fabsf(meta[0]), g = P.scale * meta[1], sig = meta[2];
        // FP16 alpha g / sigma, clamped to the largest finite value (a clamped or
        // negative one shows in M3)
        float r = sig != 0.0f ? g / sig * alpha : 0.0f;
        r = fminf(fmaxf(r, 0.0f), 65000.0f);
        const __half h = __float2half_rn(r);
        if (lane == 0) rho[j] = (uint32_t)__half_as_ushort(h) * 0x10001u;
        const float rd = sqrtf((float)P.D) * 1.0001f, sx = fabsf(sig) * xn * 1.0001f;
        const float w[kFilterBound] = {sx * sqrtf(c2), sx * sqrtf(e2), fabsf(g) * xn * rd,
                                       (fabsf(g - sig * (__half2float(h) / alpha)) + 1e-6f * fabsf(g)) * xn * rd};
#pragma unroll
        for (int i = 0; i < kFilterBound; ++i)
            M[i] = (w[i] != w[i]) ? INFINITY : fmaxf(M[i], w[i]);
    }
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < kFilterBound; ++i) atomicMax(reinterpret_cast<int *>(bound) + i, __float_as_int(M[i]));
    }
}

cudaError_t launch_pass(const Params &P, const FlArgs &base, const CUtensorMap &map, int mode, size_t tiles_all,
                        size_t want, cudaStream_t st) {
    FlArgs a = base;
    // the codes of `want` tiles spread evenly over the corpus, or all of them
    const size_t total = want * kFilterTile;
    a.nt = (unsigned)std::min(tiles_all, want);
    a.step = total < a.n ? ((unsigned long long)a.n << 32) / total : 1ull << 32;
    const int stage_bytes = FL_A_BYTES + a.box * 128, ring_bytes = FL_BM * (P.nibble ? 32 : 64);
    const int tab = P.nibble ? 0 : FL_TAB_BYTES, avail = FL_SMEM_MAX - FL_FIXED - tab;
    a.stages = std::min(FL_MAX_STAGES, (avail - 4 * ring_bytes) / stage_bytes) & ~1;  // the decoder groups alternate
    a.ring = std::min(FL_MAX_RING, (avail - a.stages * stage_bytes) / ring_bytes);
    const size_t smem = (size_t)a.stages * stage_bytes + (size_t)a.ring * ring_bytes + FL_FIXED + tab;
    auto pick = [&](auto nib) {
        constexpr bool N = decltype(nib)::value;
        return mode == kSample ? filter_kernel<N, kSample> : mode == kCollect ? filter_kernel<N, kCollect>
                                                                              : filter_kernel<N, kCollectAll>;
    };
    auto kern = P.nibble ? pick(std::true_type{}) : pick(std::false_type{});
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * sm_grid(1 << 30, 2));
    cfg.blockDim = dim3(FL_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, map, a);
}

}  // namespace

size_t filter_k(const Params &P) { return 2 * (((size_t)P.D + FL_BK - 1) / FL_BK * FL_BK); }
int filter_mmas(const Params &P) { return (int)(filter_k(P) / 16); }
// Roundings of 2^-24 on the way of a term, as a share of sum |terms|.  The exact
// stage's running sums (tq_exact.cu) are 32 over the bytes of nibble codes, D / 64
// adds each, and 8 over byte codes, D / 8 FMAs each; what joins them (a tree of 5,
// or 16 bytes in a row at D < 64) and both sides' scalar factors are at most 24 more.
float filter_sums(const Params &P) {
    return (float)((P.nibble ? P.D / 64 : P.D / 8) + 24) * (1.0f / 16777216.0f);
}

float filter_alpha(const float *centroids, int levels) {
    // the levels below zero (the others are their negatives): value, and the density
    // of N(0,1) at it
    const int half = std::min(levels / 2, 128);
    std::vector<double> w(half);
    for (int v = 0; v < half; ++v) w[v] = std::exp(-0.5 * (double)centroids[v] * centroids[v]);
    float best = 2048.0f;
    double best_e = INFINITY;
    for (int t = 0; t < 1024; ++t) {
        const float alpha = 1024.0f + (float)t;
        const double ia = 1.0 / alpha;
        double e = 0.0;
        for (int v = 0; v < half; ++v) {
            const double x = (double)round_fp16(centroids[v] * alpha) * ia - centroids[v];
            e += x * x * w[v];
        }
        if (e < best_e) {
            best_e = e;
            best = alpha;
        }
    }
    return best;
}

cudaError_t launch_filter_index(const Params &P, const DevTables &T, const FilterIndex &ix, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(ix.bound, 0, kFilterBound * sizeof(float), st);
    if (e != cudaSuccess || ix.n == 0) return e;
    const unsigned blocks = (unsigned)std::min<size_t>((ix.n + 7) / 8, 148 * 8);
    filter_index_kernel<<<blocks, 256, 0, st>>>(P, T, ix.codes, ix.n, ix.alpha, ix.rho, ix.bound);
    return cudaGetLastError();
}

cudaError_t launch_filter(const Params &P, const DevTables &T, const FilterIndex &ix, const float *q_rot,
                          const float *s_q, const float *norms, const int *m_dev, int rows, int kc,
                          const FilterBuffers &b, float *cand_d, long long *cand_i, int *err,
                          cudaStream_t st) {
    if (rows < 128 || rows % 128 || kc < 1 || kc > 32 || ix.n == 0) return cudaErrorInvalidValue;
    if (P.cs % 4 || !aligned16({b.planes, b.samp, b.rowq})) return cudaErrorMisalignedAddress;
    FlArgs a{};
    a.codes = ix.codes;
    a.n = ix.n;
    a.cs = P.cs;
    a.pb = P.pb;
    a.levels = P.levels;
    a.centroids = T.centroids;
    a.alpha = ix.alpha;
    a.undo = 1.0f / (ix.alpha * kRowScale);
    a.rho = ix.rho;
    a.KBm = (P.D + FL_BK - 1) / FL_BK;
    a.box = rows >= FL_ROWS ? FL_ROWS / 2 : rows / 2;
    a.m_dev = m_dev;
    a.uv = b.uv;
    a.r12 = b.r12;
    a.thr = b.thr;
    a.samp = b.samp;
    a.cnt = b.cnt;
    a.list_d = b.list_d;
    a.list_i = b.list_i;
    a.err = err;
    const size_t tiles = (ix.n + kFilterTile - 1) / kFilterTile;
    if (tiles * (size_t)((rows + FL_ROWS - 1) / FL_ROWS) > 0x7FFFFFFFull) return cudaErrorInvalidValue;
    alignas(64) CUtensorMap map;
    if (!make_map(&map, b.planes, (int)filter_k(P), (size_t)rows, a.box)) return cudaErrorInvalidValue;
    filter_rows_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(
        q_rot, s_q, norms, m_dev, P.D, a.KBm, static_cast<__half *>(b.planes), b.rowq, b.r12);
    cudaError_t e = cudaGetLastError();
    const size_t s1 = std::min<size_t>(kFilterSample / kFilterTile, tiles);
    if (e == cudaSuccess) e = launch_pass(P, a, map, kSample, tiles, s1, st);
    if (e != cudaSuccess) return e;
    filter_threshold_kernel<true><<<(unsigned)rows, 256, 0, st>>>(m_dev, kc, (int)s1 * kFilterTile, b.samp,
                                                                  b.list_d, b.cnt, b.r12, b.uv, b.thr);
    e = cudaGetLastError();
    // The second threshold where the first would list too many codes a row
    // (kc n / kFilterSample of them).  One row block of few columns is faster
    // without it: 5 rows of 300,000 codes, 40 us of 258.
    if (e == cudaSuccess && (size_t)kc * tiles > (size_t)(kFilterCap / 4) * s1) {
        const size_t s2 = (size_t)std::sqrt((double)s1 * (double)tiles);
        e = launch_pass(P, a, map, kCollect, tiles, s2, st);
        if (e != cudaSuccess) return e;
        filter_threshold_kernel<false><<<(unsigned)rows, 256, 0, st>>>(m_dev, kc, 0, b.samp, b.list_d, b.cnt,
                                                                       b.r12, b.uv, b.thr);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = launch_pass(P, a, map, kCollectAll, tiles, tiles, st);
    if (e != cudaSuccess) return e;
    filter_select_kernel<<<(unsigned)rows, 256, 0, st>>>(m_dev, kc, ix.n, b.cnt, b.list_d, b.list_i, b.r12,
                                                         cand_d, cand_i, b.bad);
    return cudaGetLastError();
}

}  // namespace tq
