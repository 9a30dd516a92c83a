// tq_cgemm.cu -- the M x N distances as tensor-core contractions whose code
// tiles are decoded inside the kernel (distanceBatchMToN and
// distanceBatchMToNSymmetric, space_turbo_quant.h:588-615; the light
// QJL-corrected form, :634-647, 902-945).
//
//   asymmetric  C_ij = sigma_j <q_rot_i, c[idx_j]> + scale gamma_j <s_q_i, (+-1)_j>
//   symmetric   C_ij = <c[idx_i], c[idx_j]>
//   light       the symmetric C, plus clamp(p gamma_i gamma_j <(+-1)_i, (+-1)_j>)
//   d_ij = max(0, r2_i + c2_j - 2 (C_ij r1_i) c1_j)
//
// Codes are the M side of the MMA (128 codes a tile, one tensor-memory lane
// each) and the rows (queries, or row codes) the N side (NT <= 256 columns).
// So one code's scalars are one epilogue thread's registers, a warp's stores
// of one row are 128 consecutive bytes, and a batch of few rows costs a narrow
// MMA instead of a padded 128-row tile.
//
// Operands are pairs x = hi + lo of 16-bit values, C = hi hi + hi lo + lo hi:
//   FP16 (TQ_PRECISION_FP32): both sides scaled by powers of two into FP16's
//     normal range, so a pair holds 22-23 significant bits and the dropped
//     lo lo product is below 2^-24 of a term; the pair is about as exact as
//     the FP32 value, and the sums below are more exact than one FP32 chain;
//   BF16 (TQ_PRECISION_SPLIT_BF16): 16-17 bits.
// The +-1 signs are exact and need two products (one against +-1 rows).
//
// The code side needs no planes in device memory: four or eight decoder warps turn a
// tile's packed units into the 128-byte-swizzled hi / lo tiles of one K block
// (64 coordinates) in shared memory.  Nibble codes (at most 8 centroids) are
// looked up in registers: a unit's three index bits are a PRMT selector, so
// one PRMT gives one byte of four coordinates' values.  Byte codes go through
// a lane-replicated shared table (no bank conflicts).
//
// Accumulation: the MMAs of a chunk of K blocks accumulate from zero in one of
// two tensor-memory buffers (the tensor core's FP32 accumulation truncates
// toward zero, about 2^-24 of the running sum an MMA); the epilogue warps add
// each finished chunk into FP32 registers with IEEE adds while the other
// buffer fills.
//
// Persistent, one CTA per SM, 16 warps:
//   warp 0       TMA producer of the row operand's K blocks
//   warp 1       allocates tensor memory; one thread issues the MMAs
//   warps 4..    DW decoder warps
//   the rest     epilogue warps (two per lane quadrant, or one for NT <= 64)
// Every mbarrier wait is bounded and ends in a status code (tq_async.cuh).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "tq_cgemm.h"
#include "tq_tc.cuh"

namespace tq {
namespace {

constexpr int CG_BM = 128;                 // codes per tile
constexpr int CG_BK = 64;                  // values per K block (128 bytes)
constexpr int CG_A_BYTES = CG_BM * 128;    // one 16-bit code tile of a K block
constexpr int CG_THREADS = 512;
constexpr int CG_MAX_STAGES = 6;
constexpr int CG_TAB_BYTES = 128 * 128;    // byte codes: 128 entries x 32 lanes x (hi | lo << 16)
constexpr int CG_SMEM_MAX = 227 * 1024;
constexpr int CG_FIXED = 1024 /* alignment */ + 256 /* barriers */;
constexpr int kErrFull = 1, kErrEmpty = 2, kErrTmemFull = 3, kErrTmemEmpty = 4;

// FP16 scalings: |q_rot|, |s_q| <= 1 and |c| < 5 (Lloyd-Max of N(0,1), at most
// 9 bits), so hi stays below 65504 and lo of any value that matters is normal.
constexpr float kRowScale = 16384.0f, kCentScale = 2048.0f;

__device__ __forceinline__ void split16(float v, int fmt, uint32_t &h, uint32_t &l) {
    if (fmt == kCgFP16) {
        const __half hh = __float2half_rn(v);
        h = __half_as_ushort(hh);
        l = __half_as_ushort(__float2half_rn(__fsub_rn(v, __half2float(hh))));
    } else {
        const __nv_bfloat16 hh = __float2bfloat16_rn(v);
        h = __bfloat16_as_ushort(hh);
        l = __bfloat16_as_ushort(__float2bfloat16_rn(__fsub_rn(v, __bfloat162float(hh))));
    }
}

struct CgArgs {
    const uint8_t *codes;
    size_t n;
    int cs, pb, nibble, levels;
    const float *centroids;
    int fmt, form;
    int KBm, KB;         // K blocks of the centroid part, of all
    int chm, chs;        // K blocks per accumulation chunk: centroid part, sign part
    int NT, stages;      // row columns per tile, pipeline stages
    unsigned num_nt, num_tiles;
    size_t m;
    const float4 *rs;    // per row: r1, r2, s1, s2
    float scale;         // sqrt(pi / 2D)
    float undo_c, undo_s;  // undo the operand scalings of the two parts
    float *out;
    size_t ldo;
    int *err;
};

__device__ __forceinline__ void umma16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                       uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ int cg_chunk_end(const CgArgs &p, int c0) {
    return c0 < p.KBm ? min(c0 + p.chm, p.KBm) : min(c0 + p.chs, p.KB);
}

// One of the registers' byte tables of a nibble decoder: entries 0..7, the low
// and high bytes of the hi and lo halves.
struct NibTab {
    uint32_t hl[2], hh[2], ll[2], lh[2];
};

// 8 units (a word of nibbles) -> 8 hi and 8 lo values.
__device__ __forceinline__ void nib_cent(uint32_t x, const NibTab &t, uint4 &hi, uint4 &lo) {
    const uint32_t s0 = (x >> 1) & 0x77777777u, s1 = s0 >> 16;
    uint32_t a = __byte_perm(t.hl[0], t.hl[1], s0), b = __byte_perm(t.hh[0], t.hh[1], s0);
    hi.x = __byte_perm(a, b, 0x5140u);
    hi.y = __byte_perm(a, b, 0x7362u);
    a = __byte_perm(t.hl[0], t.hl[1], s1), b = __byte_perm(t.hh[0], t.hh[1], s1);
    hi.z = __byte_perm(a, b, 0x5140u);
    hi.w = __byte_perm(a, b, 0x7362u);
    a = __byte_perm(t.ll[0], t.ll[1], s0), b = __byte_perm(t.lh[0], t.lh[1], s0);
    lo.x = __byte_perm(a, b, 0x5140u);
    lo.y = __byte_perm(a, b, 0x7362u);
    a = __byte_perm(t.ll[0], t.ll[1], s1), b = __byte_perm(t.lh[0], t.lh[1], s1);
    lo.z = __byte_perm(a, b, 0x5140u);
    lo.w = __byte_perm(a, b, 0x7362u);
}

// The QJL bits of 8 units -> 8 values +-1 (`one` = a pair of +1).
__device__ __forceinline__ uint4 nib_sign(uint32_t x, uint32_t one) {
    const uint32_t y = ~x;
    uint4 r;
    r.x = one | ((y << 15) & 0x8000u) | ((y << 27) & 0x80000000u);
    r.y = one | ((y << 7) & 0x8000u) | ((y << 19) & 0x80000000u);
    r.z = one | ((y >> 1) & 0x8000u) | ((y << 11) & 0x80000000u);
    r.w = one | ((y >> 9) & 0x8000u) | ((y << 3) & 0x80000000u);
    return r;
}
__device__ __forceinline__ uint4 byte_sign(uint32_t x0, uint32_t x1, uint32_t one) {
    const uint32_t y0 = ~x0, y1 = ~x1;
    uint4 r;
    r.x = one | ((y0 << 15) & 0x8000u) | ((y0 << 23) & 0x80000000u);
    r.y = one | ((y0 >> 1) & 0x8000u) | ((y0 << 7) & 0x80000000u);
    r.z = one | ((y1 << 15) & 0x8000u) | ((y1 << 23) & 0x80000000u);
    r.w = one | ((y1 >> 1) & 0x8000u) | ((y1 << 7) & 0x80000000u);
    return r;
}

// DW: decoder warps (warps 4 .. 4 + DW - 1); the other 12 - DW warps are the
// epilogue: two column halves of 128 (DW = 4), or one of 64 (DW = 8).  Batches
// of few rows are bound by the decoders, wide ones by the MMAs.
template <int DW, bool NIB>
__global__ void __launch_bounds__(CG_THREADS, 1) cgemm_kernel(const __grid_constant__ CUtensorMap map_h,
                                                              const __grid_constant__ CUtensorMap map_l,
                                                              const CgArgs p) {
    constexpr int EW = 12 - DW;          // epilogue warps
    constexpr int HALVES = EW / 4;       // column parts of a tile
    constexpr int CPT = DW == 4 ? 128 : 64;  // columns per epilogue thread, at most
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int stage_bytes = 2 * CG_A_BYTES + 2 * p.NT * 128;
    const uint32_t tiles0 = smem_u32(smem);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + p.stages * stage_bytes);
    // bars: full[6], empty[6], xfull[2], xempty[2], drain; then the TMEM slot
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * CG_MAX_STAGES;
    const uint32_t xfull0 = empty0 + 8 * CG_MAX_STAGES, xempty0 = xfull0 + 16, drain = xempty0 + 16;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * CG_MAX_STAGES + 5);
    uint32_t *btab = reinterpret_cast<uint32_t *>(smem + p.stages * stage_bytes + 256);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(full0 + 8 * s, 1 + DW);  // the producer and one lane of each decoder warp
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(xfull0 + 8 * b, 1);
            mbar_init(xempty0 + 8 * b, EW);
        }
        mbar_init(drain, 1);
        mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if constexpr (!NIB) {
        // entry v of lane l at btab[32 v + l]: hi | lo << 16
        for (int i = threadIdx.x; i < 128 * 32; i += CG_THREADS) {
            const int v = i >> 5;
            uint32_t h, l;
            const float c = v < p.levels ? p.centroids[v] : 0.0f;
            split16(p.fmt == kCgFP16 ? c * kCentScale : c, p.fmt, h, l);
            btab[i] = h | (l << 16);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int KB = p.KB, KBm = p.KBm;
    const unsigned grid = gridDim.x;

    // Register shares (DW = 4): 48 + 96 + 2 x 184 = 4 x 128, the launch's total.
    if (warp < 4) {
        if constexpr (DW == 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
        if (warp == 0) {
            // ---------------- TMA producer: the rows' K blocks ----------------
            if (lane == 0) {
                uint32_t s = 0, ph = 1;
                uint32_t it = 0;
                bool ok = true;
                const uint32_t bytes = 2u * (uint32_t)p.NT * 128u;
                for (unsigned t = blockIdx.x; t < p.num_tiles && ok; t += grid) {
                    const int mb = (int)(t / p.num_nt);
                    for (int kb = 0; kb < KB; ++kb, ++it) {
                        if (!mbar_wait(empty0 + 8 * s, ph, p.err, kErrEmpty)) { ok = false; break; }
                        const uint32_t b = tiles0 + s * stage_bytes + 2 * CG_A_BYTES, fb = full0 + 8 * s;
                        mbar_expect_tx(fb, bytes);
                        tma_load_2d(b, &map_h, kb * CG_BK, mb * p.NT, fb);
                        tma_load_2d(b + p.NT * 128, &map_l, kb * CG_BK, mb * p.NT, fb);
                        if (++s == (uint32_t)p.stages) { s = 0; ph ^= 1u; }
                    }
                }
                // every stage issued must have landed before the CTA exits
                for (uint32_t k = 0; k < (uint32_t)p.stages && k < it; ++k) {
                    const uint32_t j = it - 1 - k;
                    mbar_drain(full0 + 8 * (j % p.stages), (j / p.stages) & 1u);
                }
            }
        } else if (warp == 1) {
            // ---------------- MMA issuer ----------------
            if (lane == 0) {
                const uint32_t f = p.fmt == kCgFP16 ? 0u : 1u;
                const uint32_t idesc = (1u << 4) | (f << 7) | (f << 10) | ((uint32_t)(p.NT >> 3) << 17) |
                                       ((uint32_t)(CG_BM >> 4) << 24);
                const bool one_sign = p.form == kCgLight;  // +-1 rows: their lo is zero
                uint32_t s = 0, ph = 0, gc = 0;
                bool ok = true;
                for (unsigned t = blockIdx.x; t < p.num_tiles && ok; t += grid) {
                    for (int c0 = 0, c1 = 0; c0 < KB && ok; c0 = c1, ++gc) {
                        c1 = cg_chunk_end(p, c0);
                        const uint32_t b = gc & 1u, xph = (gc >> 1) & 1u;
                        if (!mbar_wait(xempty0 + 8 * b, xph ^ 1u, p.err, kErrTmemEmpty)) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t d = tmem_base + b * 256u;
                        uint32_t acc = 0u;
                        for (int kb = c0; kb < c1; ++kb) {
                            if (!mbar_wait(full0 + 8 * s, ph, p.err, kErrFull)) { ok = false; break; }
                            tc_fence_after();
                            const uint32_t ah = tiles0 + s * stage_bytes, al = ah + CG_A_BYTES;
                            const uint32_t bh = al + CG_A_BYTES, bl = bh + p.NT * 128;
                            const bool cent = kb < KBm;
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk) {
                                const uint32_t ko = kk * 32;  // one MMA's K: 32 bytes
                                // the small products first, while the sum is smaller
                                if (cent) {
                                    umma16(d, sw128_desc(al + ko), sw128_desc(bh + ko), idesc, acc);
                                    acc = 1u;
                                }
                                if (cent || !one_sign) {
                                    umma16(d, sw128_desc(ah + ko), sw128_desc(bl + ko), idesc, acc);
                                    acc = 1u;
                                }
                                umma16(d, sw128_desc(ah + ko), sw128_desc(bh + ko), idesc, acc);
                                acc = 1u;
                            }
                            umma_commit(empty0 + 8 * s);
                            if (++s == (uint32_t)p.stages) { s = 0; ph ^= 1u; }
                        }
                        if (ok) umma_commit(xfull0 + 8 * b);
                    }
                }
                // every MMA issued must be complete before the tensor memory is freed
                umma_commit(drain);
                mbar_drain(drain, 0);
            }
        }
    } else if (warp < 4 + DW) {
        // ---------------- decoders ----------------
        // Warp w decodes rows RPW w ..: lane l takes 16-byte chunk l & 7 (8
        // coordinates) of rows 4 i + (l >> 3), so eight lanes read a row's
        // consecutive words and write its 128 bytes without bank conflicts.
        if constexpr (DW == 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 96;");
        constexpr int RPW = CG_BM / DW, ITEMS = RPW / 4, WPI = NIB ? 1 : 2;
        const int r0 = (warp - 4) * RPW + (lane >> 3), c = lane & 7;
        NibTab tab{};
        if constexpr (NIB) {
#pragma unroll
            for (int v = 0; v < 8; ++v) {
                uint32_t h, l;
                const float cv = v < p.levels ? p.centroids[v] : 0.0f;
                split16(p.fmt == kCgFP16 ? cv * kCentScale : cv, p.fmt, h, l);
                const int sh = 8 * (v & 3);
                tab.hl[v >> 2] |= (h & 0xFFu) << sh;
                tab.hh[v >> 2] |= (h >> 8) << sh;
                tab.ll[v >> 2] |= (l & 0xFFu) << sh;
                tab.lh[v >> 2] |= (l >> 8) << sh;
            }
        }
        const uint32_t one = p.fmt == kCgFP16 ? 0x3C003C00u : 0x3F803F80u;
        const uint32_t *tl = btab + lane;
        // the words of K block kb of tile t (zero beyond the packed bytes: D < 64)
        auto load = [&](uint32_t (&w)[ITEMS][WPI], unsigned t, int kb) {
            const size_t j0 = (size_t)(t % p.num_nt) * CG_BM;
            const int o = ((kb < KBm ? kb : kb - KBm) * 8 + c) * 4 * WPI;
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) {
                size_t row = j0 + r0 + 4 * i;
                if (row >= p.n) row = p.n - 1;
                const uint8_t *src = p.codes + row * (size_t)p.cs + o;
#pragma unroll
                for (int q = 0; q < WPI; ++q)
                    w[i][q] = o + 4 * q < p.pb ? __ldg(reinterpret_cast<const uint32_t *>(src) + q) : 0u;
            }
        };
        uint32_t s = 0, ph = 1;
        bool ok = true;
        uint32_t w[ITEMS][WPI], nw[ITEMS][WPI];
        if (blockIdx.x < p.num_tiles) load(w, blockIdx.x, 0);
        for (unsigned t = blockIdx.x; t < p.num_tiles && ok; t += grid) {
            for (int kb = 0; kb < KB; ++kb) {
                // the next block's words are in flight while this one is decoded
                if (kb + 1 < KB) load(nw, t, kb + 1);
                else if (t + grid < p.num_tiles) load(nw, t + grid, 0);
                if (!mbar_wait(empty0 + 8 * s, ph, p.err, kErrEmpty)) { ok = false; break; }
                unsigned char *base = smem + s * stage_bytes;
                const bool cent = kb < KBm;
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) {
                    const int r = r0 + 4 * i;
                    unsigned char *dst = base + r * 128 + ((c ^ (r & 7)) << 4);
                    if (cent) {
                        uint4 hi, lo;
                        if constexpr (NIB) {
                            nib_cent(w[i][0], tab, hi, lo);
                        } else {
                            uint32_t e[8];
#pragma unroll
                            for (int q = 0; q < 8; ++q)
                                e[q] = tl[((w[i][q >> 2] >> (8 * (q & 3) + 1)) & 0x7Fu) * 32];
                            hi = make_uint4(__byte_perm(e[0], e[1], 0x5410u), __byte_perm(e[2], e[3], 0x5410u),
                                            __byte_perm(e[4], e[5], 0x5410u), __byte_perm(e[6], e[7], 0x5410u));
                            lo = make_uint4(__byte_perm(e[0], e[1], 0x7632u), __byte_perm(e[2], e[3], 0x7632u),
                                            __byte_perm(e[4], e[5], 0x7632u), __byte_perm(e[6], e[7], 0x7632u));
                        }
                        *reinterpret_cast<uint4 *>(dst) = hi;
                        *reinterpret_cast<uint4 *>(dst + CG_A_BYTES) = lo;
                    } else {
                        uint4 v;
                        if constexpr (NIB) v = nib_sign(w[i][0], one);
                        else v = byte_sign(w[i][0], w[i][WPI - 1], one);
                        *reinterpret_cast<uint4 *>(dst) = v;
                    }
                }
                fence_proxy_async_smem();  // the generic stores before the MMAs' async reads
                __syncwarp();
                if (lane == 0) mbar_arrive(full0 + 8 * s);
                if (++s == (uint32_t)p.stages) { s = 0; ph ^= 1u; }
#pragma unroll
                for (int i = 0; i < ITEMS; ++i)
#pragma unroll
                    for (int q = 0; q < WPI; ++q) w[i][q] = nw[i][q];
            }
        }
    } else {
        // ---------------- epilogue ----------------
        if constexpr (DW == 4) asm volatile("setmaxnreg.inc.sync.aligned.u32 184;");
        const int quad = warp & 3, half = (warp - 4 - DW) >> 2;
        const int cpt = p.NT / HALVES;  // this thread's columns
        const uint32_t lanes = tmem_base + ((uint32_t)(32 * quad) << 16) + (uint32_t)(half * cpt);
        float y[CPT];
        uint32_t gc = 0;
        bool ok = true;
        for (unsigned t = blockIdx.x; t < p.num_tiles && ok; t += grid) {
            const size_t row = (size_t)(t % p.num_nt) * CG_BM + 32 * quad + lane;
            const size_t col0 = (size_t)(t / p.num_nt) * p.NT + half * cpt;
            // the code's trailer [norm, gamma, sigma]
            float norm = 0.0f, gamma = 0.0f, sigma = 0.0f;
            if (row < p.n) {
                const float *meta = reinterpret_cast<const float *>(p.codes + row * (size_t)p.cs + p.pb);
                norm = __ldg(meta);
                gamma = __ldg(meta + 1);
                sigma = __ldg(meta + 2);
            }
            for (int c0 = 0, c1 = 0; c0 < KB; c0 = c1, ++gc) {
                c1 = cg_chunk_end(p, c0);
                const uint32_t b = gc & 1u, xph = (gc >> 1) & 1u;
                if (!mbar_wait(xfull0 + 8 * b, xph, p.err, kErrTmemFull)) { ok = false; break; }
                tc_fence_after();
                const uint32_t X = lanes + b * 256u;
                // how a chunk joins the running sum: centroid chunks are added;
                // a sign chunk as fma(x, scale gamma, y), y first scaled by
                // sigma (asymmetric); the light form's one sign chunk is its
                // clamped correction
                const bool cent = c0 < KBm;
                const float fy = (!cent && c0 == KBm) ? __fmul_rn(sigma, p.undo_c) : 1.0f;
                const float fx = __fmul_rn(__fmul_rn(p.scale, gamma), p.undo_s);
#pragma unroll
                for (int pc = 0; pc < CPT / 16; ++pc) {
                    if (16 * pc >= cpt) break;
                    uint32_t x[16];
                    __syncwarp();
                    tmem_ld16_nw(X + 16 * pc, x);
                    tmem_wait_ld();
                    if (cent) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const float a = __uint_as_float(x[j]);
                            y[16 * pc + j] = c0 == 0 ? a : __fadd_rn(y[16 * pc + j], a);
                        }
                    } else if (p.form == kCgAsym) {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            y[16 * pc + j] = __fmaf_rn(__uint_as_float(x[j]), fx, __fmul_rn(y[16 * pc + j], fy));
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const size_t col = col0 + 16 * pc + j < p.m ? col0 + 16 * pc + j : p.m - 1;
                            const float4 r = __ldg(p.rs + col);
                            const float ip = __fmul_rn(__fmul_rn(__fmul_rn(y[16 * pc + j], p.undo_c), r.z), sigma);
                            const float corr = __fmul_rn(__fmul_rn(__uint_as_float(x[j]), r.w), gamma);
                            const float lim = fabsf(ip);
                            y[16 * pc + j] = __fadd_rn(ip, fmaxf(-lim, fminf(lim, corr)));
                        }
                    }
                }
                __syncwarp();
                tc_fence_before();
                if (lane == 0) mbar_arrive(xempty0 + 8 * b);
            }
            if (!ok) break;
            if (row >= p.n) continue;
            // d = max(0, r2 + c2 - 2 (C r1) c1)
            const float c2 = __fmul_rn(norm, norm);
            const float c1 = p.form == kCgSym ? __fmul_rn(sigma, norm) : norm;
            const float un = p.form == kCgSym ? p.undo_c : 1.0f;
            float *o = p.out + col0 * p.ldo + row;
#pragma unroll
            for (int pc = 0; pc < CPT / 16; ++pc) {
                if (16 * pc >= cpt) break;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const size_t col = col0 + 16 * pc + j;
                    if (col < p.m) {
                        const float2 r = __ldg(reinterpret_cast<const float2 *>(p.rs + col));
                        const float ipt = __fmul_rn(__fmul_rn(__fmul_rn(y[16 * pc + j], un), r.x), c1);
                        const float d = __fsub_rn(__fadd_rn(r.y, c2), __fmul_rn(2.0f, ipt));
                        __stcs(o, d > 0.0f ? d : 0.0f);
                    }
                    o += p.ldo;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512)
                     : "memory");
    }
}

// ---- row planes -----------------------------------------------------------
// hi / lo planes [m][K], K = 64 KBm (symmetric) or 2 x 64 KBm, zero past D in
// each part, and the per-row scalars.  One thread per 4 positions.
__device__ __forceinline__ void put4(const float (&v)[4], int fmt, __nv_bfloat16 *ph, __nv_bfloat16 *pl) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) split16(v[q], fmt, h[q], l[q]);
    *reinterpret_cast<uint2 *>(ph) = make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
    *reinterpret_cast<uint2 *>(pl) = make_uint2(l[0] | (l[1] << 16), l[2] | (l[3] << 16));
}

__global__ void __launch_bounds__(256) cg_rows_prepared_kernel(
    const float *__restrict__ q_rot, const float *__restrict__ s_q, const float *__restrict__ norms,
    size_t m, int D, int KBm, int fmt, __nv_bfloat16 *__restrict__ ph, __nv_bfloat16 *__restrict__ pl,
    float4 *__restrict__ rs) {
    const int half = KBm * CG_BK, K = 2 * half, quads = K / 4;
    const size_t total = m * (size_t)quads;
    const float f = fmt == kCgFP16 ? kRowScale : 1.0f;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        const size_t r = t / quads;
        const int k = (int)(t - r * quads) * 4;
        const float *src = (k < half ? q_rot : s_q) + r * D;
        const int k0 = k < half ? k : k - half;
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = k0 + q < D ? src[k0 + q] * f : 0.0f;
        put4(v, fmt, ph + r * K + k, pl + r * K + k);
        if (k == 0) rs[r] = make_float4(norms[2 * r + 1], norms[2 * r], 0.0f, 0.0f);
    }
}

// Row codes: centroid values, for the light form followed by the +-1 signs.
// rs: symmetric (sigma n, n^2, -, -); light (n, n^2, sigma, (pi / 2D) gamma).
__global__ void __launch_bounds__(256) cg_rows_codes_kernel(const uint8_t *__restrict__ codes, size_t m,
                                                            Params P, DevTables T, int KBm, int form,
                                                            int fmt, __nv_bfloat16 *__restrict__ ph,
                                                            __nv_bfloat16 *__restrict__ pl,
                                                            float4 *__restrict__ rs) {
    const int half = KBm * CG_BK, K = form == kCgLight ? 2 * half : half, quads = K / 4;
    const size_t total = m * (size_t)quads;
    const float f = fmt == kCgFP16 ? kCentScale : 1.0f;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (size_t)gridDim.x * blockDim.x) {
        const size_t r = t / quads;
        const int k = (int)(t - r * quads) * 4;
        const int k0 = k < half ? k : k - half;
        const uint8_t *code = codes + r * (size_t)P.cs;
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            v[q] = 0.0f;
            if (k0 + q < P.D) {
                const unsigned b = P.nibble ? code[(k0 + q) >> 1] : code[k0 + q];
                const unsigned u = P.nibble ? (((k0 + q) & 1) ? b >> 4 : b & 15u) : b;
                v[q] = k < half ? T.centroids[u >> 1] * f : ((u & 1u) ? 1.0f : -1.0f);
            }
        }
        put4(v, fmt, ph + r * K + k, pl + r * K + k);
        if (k == 0) {
            const float *meta = reinterpret_cast<const float *>(code + P.pb);
            const float norm = meta[0], gamma = meta[1], sigma = meta[2];
            const float n2 = __fmul_rn(norm, norm);
            rs[r] = form == kCgLight
                        ? make_float4(norm, n2, sigma,
                                      __fmul_rn((float)(3.14159265358979323846 / (2.0 * P.D)), gamma))
                        : make_float4(__fmul_rn(sigma, norm), n2, 0.0f, 0.0f);
        }
    }
}

unsigned rows_grid(size_t work) {
    return (unsigned)std::min<size_t>(std::max<size_t>(1, (work + 255) / 256), (size_t)148 * 16);
}

}  // namespace

size_t cg_row_k(const Params &P, int form) {
    const size_t half = ((size_t)P.D + CG_BK - 1) / CG_BK * CG_BK;
    return form == kCgSym ? half : 2 * half;
}

cudaError_t launch_cg_rows_prepared(const Params &P, const float *q_rot, const float *s_q,
                                    const float *norms, size_t m, int fmt, const CgRows &r,
                                    cudaStream_t st) {
    const int KBm = (P.D + CG_BK - 1) / CG_BK;
    cg_rows_prepared_kernel<<<rows_grid(m * (size_t)KBm * 32), 256, 0, st>>>(
        q_rot, s_q, norms, m, P.D, KBm, fmt, static_cast<__nv_bfloat16 *>(r.hi),
        static_cast<__nv_bfloat16 *>(r.lo), r.rs);
    return cudaGetLastError();
}

cudaError_t launch_cg_rows_codes(const Params &P, const DevTables &T, const uint8_t *codes, size_t m,
                                 int form, int fmt, const CgRows &r, cudaStream_t st) {
    const int KBm = (P.D + CG_BK - 1) / CG_BK;
    cg_rows_codes_kernel<<<rows_grid(m * (size_t)KBm * 32), 256, 0, st>>>(
        codes, m, P, T, KBm, form, fmt, static_cast<__nv_bfloat16 *>(r.hi),
        static_cast<__nv_bfloat16 *>(r.lo), r.rs);
    return cudaGetLastError();
}

cudaError_t launch_cgemm(const Params &P, const DevTables &T, int form, int fmt, const CgRows &rows,
                         size_t m, const uint8_t *codes, size_t n, float *out, size_t ldo, int *err,
                         cudaStream_t st) {
    if (m == 0 || n == 0) return cudaSuccess;
    if (P.cs % 4 || (reinterpret_cast<uintptr_t>(codes) & 3)) return cudaErrorMisalignedAddress;
    if (!aligned16({rows.hi, rows.lo, rows.rs})) return cudaErrorMisalignedAddress;
    CgArgs a{};
    a.codes = codes;
    a.n = n;
    a.cs = P.cs;
    a.pb = P.pb;
    a.nibble = P.nibble;
    a.levels = P.levels;
    a.centroids = T.centroids;
    a.fmt = fmt;
    a.form = form;
    a.KBm = (P.D + CG_BK - 1) / CG_BK;
    a.KB = form == kCgSym ? a.KBm : 2 * a.KBm;
    // Chunk lengths (K blocks).  FP16: 2, so that the truncation of one chunk
    // (24 MMAs) stays below the rounding of an FP32 chain; BF16: 8 for queries
    // and 4 for codes against codes, whose terms share a sign more often.
    a.chm = fmt == kCgFP16 ? 2 : form == kCgAsym ? 8 : 4;
    a.chs = form == kCgLight ? a.KBm : 16;  // +-1 by +-1 sums are exact integers
    a.m = m;
    a.rs = rows.rs;
    a.scale = P.scale;
    a.undo_s = fmt == kCgFP16 && form == kCgAsym ? 1.0f / kRowScale : 1.0f;
    a.undo_c = fmt == kCgFP16
                   ? 1.0f / (kCentScale * (form == kCgAsym ? kRowScale : kCentScale))
                   : 1.0f;
    a.out = out;
    a.ldo = ldo;
    a.err = err;
    const size_t nt = (n + CG_BM - 1) / CG_BM;
    // Columns per tile: the width that takes the least time by a rough count
    // of clocks: waves of 148 CTAs times a tile's K blocks, each the slower of
    // its MMAs (11 per block on average over both parts, NT / 2 clocks each)
    // and its decode (~650 clocks), plus the tile's epilogue.
    int best = 256;
    double best_t = 0.0;
    for (int NT = 256; NT >= 16; NT >>= 1) {
        const size_t tiles = nt * ((m + NT - 1) / NT);
        const double waves = (double)((tiles + 147) / 148);
        const double mma = 5.5 * NT, dec = NT <= 64 ? 400.0 : 650.0;
        const double tt = waves * (a.KB * std::max(mma, dec) + 2.0 * NT + 1000.0);
        if (NT == 256 || tt < best_t) {
            best = NT;
            best_t = tt;
        }
    }
    a.NT = best;
    const int stage_bytes = 2 * CG_A_BYTES + 2 * a.NT * 128;
    const int tab = P.nibble ? 0 : CG_TAB_BYTES;
    a.stages = std::min(CG_MAX_STAGES, (CG_SMEM_MAX - CG_FIXED - tab) / stage_bytes);
    const size_t smem = (size_t)a.stages * stage_bytes + CG_FIXED + tab;
    const size_t tiles = nt * ((m + a.NT - 1) / a.NT);
    if (tiles > 0x7FFFFFFFull || nt > 0x7FFFFFFFull) return cudaErrorInvalidValue;
    a.num_nt = (unsigned)nt;
    a.num_tiles = (unsigned)tiles;
    alignas(64) CUtensorMap mh, ml;
    const int K = a.KB * CG_BK;
    if (!make_map(&mh, rows.hi, K, m, a.NT) || !make_map(&ml, rows.lo, K, m, a.NT))
        return cudaErrorInvalidValue;
    const bool narrow = a.NT <= 64;
    auto kern = P.nibble ? (narrow ? cgemm_kernel<8, true> : cgemm_kernel<4, true>)
                         : (narrow ? cgemm_kernel<8, false> : cgemm_kernel<4, false>);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<sm_grid(tiles), CG_THREADS, smem, st>>>(mh, ml, a);
    return cudaGetLastError();
}

}  // namespace tq
