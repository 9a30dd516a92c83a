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
// two (four with split quarters) tensor-memory buffers (the tensor core's FP32 accumulation truncates
// toward zero, about 2^-24 of the running sum an MMA; a block's small products
// run before its hi hi ones, while the sum is small); the epilogue warps add
// each finished chunk into FP32 registers with IEEE adds while the other
// buffer fills.  Calls of fewer than 32 rows at FP16 go further: each quarter of a
// K block (one MMA's 16 values) has accumulators of its own, added in FP32, so that
// no sum is truncated at its full size more than once a K block; narrow tiles leave
// the tensor pipe and the columns idle that this takes.
//
// CTA pairs: wide tiles (NT > 64) run on clusters of two CTAs, 256 codes by NT
// rows, tcgen05.mma.cta_group::2: each CTA decodes its 128 codes and loads half
// of the rows' tile, so a K block's shared-memory traffic per CTA (MMA operand
// reads + copies + decode) is 162 KB in 1536 clocks, under the 128 B/clk that
// one CTA alone (243 KB) exceeded.
//
// Persistent, one CTA per SM, 16 warps:
//   warp 0       TMA producer of the row operand's K blocks
//   warp 1       allocates tensor memory; one thread issues the MMAs (in the
//                other CTA of a pair it reports that CTA's stages)
//   warps 2, 3   load the tiles' code words into a small ring (cp.async)
//   warps 4..    DW decoder warps
//   the rest     epilogue warps (two per lane quadrant, or one for NT <= 64)
// Every mbarrier wait is bounded and ends in a status code (tq_async.cuh).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "tq_cgemm.h"
#include "tq_tables.h"
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
constexpr int CG_MAX_RING = 8;             // K blocks of code words in flight
constexpr int CG_BAR_BYTES = 384;
constexpr int CG_FIXED = 1024 /* alignment */ + CG_BAR_BYTES;
constexpr int kErrFull = 1, kErrEmpty = 2, kErrTmemFull = 3, kErrTmemEmpty = 4;

// FP16 scalings: |q_rot|, |s_q| <= 1 and |c| < 5 (Lloyd-Max of N(0,1), at most
// 9 bits), so hi stays below 65504 and lo of any value that matters is normal.
// The centroids' scale is P.cent_scale: few distinct values, whose rounding
// errors do not average out over a row (40 x 20k symmetric distances of clustered
// 384-d rows, error against FP64 with the FP32 chain / scale 2048 / chosen scale:
// 3-bit 8.5 / 4.5 / 3.6e-8, 8-bit 3.5 / 3.7 / 3.4e-8; near pairs at BF16, largest
// error with no scale / the chosen one: 2-bit 4.4 / 2.0e-6, 8-bit 3.7 / 1.9e-6).
constexpr float kRowScale = 16384.0f;

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
    int fmt, form, post;
    int KBm, KB;         // K blocks of the centroid part, of all
    int chm, chs;        // K blocks per accumulation chunk: centroid part, sign part
    int NT, stages, ring;  // row columns per tile, pipeline stages, code-word ring slots
    unsigned num_nt, num_tiles;
    size_t m;
    const float4 *rs;    // per row: r1, r2, s1, s2
    float scale;         // sqrt(pi / 2D)
    float cent;          // the centroids' FP16 scale
    float undo_c, undo_s;  // undo the operand scalings of the two parts
    float *out;
    size_t ldo;
    int *err, *status;   // the call's error word, and the space's (may be null)
};

// The K blocks of a tile in the order they run: the asymmetric form's sign part
// first, so that its one long chunk covers the previous tile's output; the
// light form's last, since its sums are not added to the centroid part's.
template <bool LIGHT>
struct CgOrder {
    int KBm, KB, ns;  // ns: sign blocks that run first
    __device__ explicit CgOrder(const CgArgs &p) : KBm(p.KBm), KB(p.KB), ns(LIGHT ? 0 : p.KB - p.KBm) {}
    __device__ bool cent(int kb) const { return LIGHT ? kb < KBm : kb >= ns; }
    // block index within its part, and in the row planes (centroid part first)
    __device__ int part(int kb) const { return LIGHT ? (kb < KBm ? kb : kb - KBm) : (kb < ns ? kb : kb - ns); }
    __device__ int plane(int kb) const { return LIGHT ? kb : (kb < ns ? KBm + kb : kb - ns); }
    // end of the accumulation chunk that starts at c0
    __device__ int chunk_end(const CgArgs &p, int c0) const {
        if (cent(c0)) return min(c0 + p.chm, LIGHT ? KBm : KB);
        return min(c0 + p.chs, LIGHT ? KB : ns);
    }
};

template <bool PAIR>
__device__ __forceinline__ void commit(uint32_t bar) {
    if constexpr (PAIR) umma_commit_pair(bar);
    else umma_commit(bar);
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

// The QJL bits of 8 units -> 8 values +-1 (`one` = a pair of +1, `pm` the high
// bytes of -1 and +1): a PRMT picks four coordinates' high bytes by their
// bits, two more put the low byte beside each.
__device__ __forceinline__ uint4 nib_sign(uint32_t x, uint32_t one, uint32_t pm) {
    const uint32_t s = x & 0x11111111u;
    const uint32_t a = __byte_perm(pm, 0u, s), b = __byte_perm(pm, 0u, s >> 16);
    return make_uint4(__byte_perm(a, one, 0x1404u), __byte_perm(a, one, 0x3424u), __byte_perm(b, one, 0x1404u),
                      __byte_perm(b, one, 0x3424u));
}
// The same for units of a byte each.
__device__ __forceinline__ uint4 byte_sign(uint32_t x0, uint32_t x1, uint32_t one, uint32_t pm) {
    return make_uint4(__byte_perm(one, pm, ((x0 << 4) & 0x1010u) | 0x4040u),
                      __byte_perm(one, pm, ((x0 >> 12) & 0x1010u) | 0x4040u),
                      __byte_perm(one, pm, ((x1 << 4) & 0x1010u) | 0x4040u),
                      __byte_perm(one, pm, ((x1 >> 12) & 0x1010u) | 0x4040u));
}

// f(k, x) for at least the first `cols` of CPT columns of a chunk buffer, in
// pieces of 32, or of 16 where f needs the registers (a piece past `cols` holds
// values that are not used).
template <int CPT, bool HALF, class F>
__device__ __forceinline__ void chunk_pieces(uint32_t X, int cols, F f) {
    constexpr int W = HALF ? 16 : 32;
#pragma unroll
    for (int pc = 0; pc < CPT / W; ++pc) {
        if (W * pc >= cols) break;
        uint32_t x[W];
        __syncwarp();
        if constexpr (HALF) {
            tmem_ld16_nw(X + W * pc, x);
            tmem_wait_ld();
        } else {
            tmem_ld32(X + W * pc, x);
        }
#pragma unroll
        for (int j = 0; j < W; ++j) f(W * pc + j, __uint_as_float(x[j]));
    }
}

// The same for a chunk whose K-block quarters have accumulators of their own,
// NT (16 or 32) columns each: f(k, their sum).
template <class F>
__device__ __forceinline__ void chunk_quarters(uint32_t X, int NT, F f) {
#pragma unroll
    for (int c0 = 0; c0 < 32; c0 += 16) {
        if (c0 >= NT) break;
        uint32_t x[4][16];
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 4; ++q) tmem_ld16_nw(X + q * NT + c0, x[q]);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j)
            f(c0 + j, __fadd_rn(__fadd_rn(__uint_as_float(x[0][j]), __uint_as_float(x[1][j])),
                                __fadd_rn(__uint_as_float(x[2][j]), __uint_as_float(x[3][j]))));
    }
}

// DW: decoder warps (warps 4 .. 4 + DW - 1); the other 12 - DW warps are the
// epilogue: two column halves of 128 (DW = 4), or one of 64 (DW = 8).  Batches
// of few rows are bound by the decoders, wide ones by the MMAs.
// SPLIT: tiles of at most 32 columns, whose K-block quarters accumulate apart.
template <int DW, bool NIB, bool LIGHT, bool PAIR, bool FULL, bool SPLIT>
__global__ void __launch_bounds__(CG_THREADS, 1) cgemm_kernel(const __grid_constant__ CUtensorMap map_h,
                                                              const __grid_constant__ CUtensorMap map_l,
                                                              const CgArgs p) {
    constexpr int EW = 12 - DW;          // epilogue warps
    constexpr uint32_t NB = SPLIT ? 4 : 2, BUF = 512 / NB;  // chunk buffers in tensor memory, columns of each
    constexpr int HALVES = EW / 4;       // column parts of a tile
    constexpr int CPT = SPLIT ? 32 : DW == 4 ? 128 : 64;  // columns per epilogue thread, at most
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t rank = PAIR ? cluster_rank() : 0u;
    const int bt_bytes = p.NT * (PAIR ? 64 : 128);  // this CTA's rows of one B tile
    const int stage_bytes = 2 * CG_A_BYTES + 2 * bt_bytes;
    const uint32_t tiles0 = smem_u32(smem);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + p.stages * stage_bytes);
    // bars: full[6], empty[6], xfull[4], xempty[4], drain, cfull[8], cempty[8], pfull[6]; then the TMEM slot
    const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * CG_MAX_STAGES;
    const uint32_t xfull0 = empty0 + 8 * CG_MAX_STAGES, xempty0 = xfull0 + 32, drain = xempty0 + 32;
    const uint32_t cfull0 = drain + 8, cempty0 = cfull0 + 8 * CG_MAX_RING;
    const uint32_t pfull0 = cempty0 + 8 * CG_MAX_RING;  // PAIR, rank 0: the other CTA's stage is full
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 3 * CG_MAX_STAGES + 9 + 2 * CG_MAX_RING);
    // the ring of code words, then the byte codes' table
    constexpr int WPI = NIB ? 1 : 2;                 // words of 8 coordinates
    constexpr int RING_BYTES = CG_BM * 32 * WPI;     // one K block's words
    unsigned char *ring = smem + p.stages * stage_bytes + CG_BAR_BYTES;
    const uint32_t ring0 = smem_u32(ring);
    uint32_t *btab = reinterpret_cast<uint32_t *>(ring + p.ring * RING_BYTES);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(full0 + 8 * s, 1 + 4);  // the producer and the block's four decoder warps
            mbar_init(empty0 + 8 * s, 1);
            mbar_init(pfull0 + 8 * s, 1);
        }
        for (uint32_t b = 0; b < NB; ++b) {
            mbar_init(xfull0 + 8 * b, 1);
            mbar_init(xempty0 + 8 * b, PAIR ? 2 * EW : EW);  // PAIR: rank 0's counts both CTAs'
        }
        for (int k = 0; k < p.ring; ++k) {
            mbar_init(cfull0 + 8 * k, 64);  // every loader thread
            mbar_init(cempty0 + 8 * k, 4);
        }
        mbar_init(drain, 1);
        mbar_init_fence();
    }
    if (warp == 1) tmem_alloc512<PAIR>(smem_u32(tmem_slot));
    if constexpr (!NIB) {
        // entry v of lane l at btab[32 v + l]: hi | lo << 16
        for (int i = threadIdx.x; i < 128 * 32; i += CG_THREADS) {
            const int v = i >> 5;
            uint32_t h, l;
            const float c = v < p.levels ? p.centroids[v] : 0.0f;
            split16(c * p.cent, p.fmt, h, l);
            btab[i] = h | (l << 16);
        }
    }
    tc_fence_before();
    if constexpr (PAIR) cluster_sync();  // the other CTA's barriers and tensor memory too
    else __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int KB = p.KB;
    const CgOrder<LIGHT> ord(p);
    bool ok = true;  // no wait of this thread's has given up
    // tiles of this CTA (or pair): t0, t0 + grid, ...; this CTA's first code of tile t
    const unsigned grid = PAIR ? gridDim.x >> 1 : gridDim.x, t0 = PAIR ? blockIdx.x >> 1 : blockIdx.x;
    auto first_code = [&](unsigned t) {
        return (size_t)(t % p.num_nt) * (PAIR ? 2 * CG_BM : CG_BM) + rank * CG_BM;
    };

    // Register shares (DW = 4): 64 + 80 + 2 x 184 = 4 x 128, the launch's total.
    if (warp < 4) {
        if constexpr (DW == 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        if (warp == 0) {
            // ---------------- TMA producer: the rows' K blocks ----------------
            if (lane == 0) {
                uint32_t s = 0, ph = 1;
                uint32_t it = 0;
                for (unsigned t = t0; t < p.num_tiles && ok; t += grid) {
                    const int row = (int)((t / p.num_nt) * p.NT + rank * (p.NT / 2));
                    for (int kb = 0; kb < KB; ++kb, ++it) {
                        if (!mbar_wait(empty0 + 8 * s, ph, p.err, kErrEmpty)) { ok = false; break; }
                        const uint32_t b = tiles0 + s * stage_bytes + 2 * CG_A_BYTES, fb = full0 + 8 * s;
                        mbar_expect_tx(fb, 2u * bt_bytes);
                        tma_load_2d(b, &map_h, ord.plane(kb) * CG_BK, row, fb);
                        tma_load_2d(b + bt_bytes, &map_l, ord.plane(kb) * CG_BK, row, fb);
                        if (++s == (uint32_t)p.stages) { s = 0; ph ^= 1u; }
                    }
                }
                // every stage issued must have landed before the CTA exits
                for (uint32_t k = 0; k < (uint32_t)p.stages && k < it; ++k) {
                    const uint32_t j = it - 1 - k;
                    mbar_drain(full0 + 8 * (j % p.stages), (j / p.stages) & 1u);
                }
            }
        } else if (warp == 1 && rank != 0) {
            // ---------------- PAIR, rank 1: reports each full stage to rank 0 ----------------
            uint32_t s = 0, ph = 0;
            for (unsigned t = t0; t < p.num_tiles && ok; t += grid) {
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
            // ---------------- MMA issuer ----------------
            // The whole warp runs the loop, so that descriptors stay in uniform
            // registers; one elected lane issues.
            const bool lead = elect_one();
            const uint32_t f = p.fmt == kCgFP16 ? 0u : 1u;
            const uint32_t idesc = (1u << 4) | (f << 7) | (f << 10) | ((uint32_t)(p.NT >> 3) << 17) |
                                   ((uint32_t)((PAIR ? 2 * CG_BM : CG_BM) >> 4) << 24);
            constexpr bool one_sign = LIGHT;  // +-1 rows: their lo is zero
            const uint32_t dk = SPLIT ? (uint32_t)p.NT : 0u;  // quarter kk's accumulator: d + kk dk
            const uint32_t ab = CG_A_BYTES >> 4, bb = (uint32_t)bt_bytes >> 4;
            uint32_t s = 0, ph = 0, gc = 0;
            for (unsigned t = t0; t < p.num_tiles && ok; t += grid) {
                for (int c0 = 0, c1 = 0; c0 < KB && ok; c0 = c1, ++gc) {
                    c1 = ord.chunk_end(p, c0);
                    const uint32_t b = gc % NB, xph = (gc / NB) & 1u;
                    if (!(PAIR ? mbar_wait_cluster_warp(xempty0 + 8 * b, xph ^ 1u, p.err, kErrTmemEmpty)
                               : mbar_wait_warp(xempty0 + 8 * b, xph ^ 1u, p.err, kErrTmemEmpty))) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t d = tmem_base + b * BUF;
                    uint32_t acc = 0u;
                    for (int kb = c0; kb < c1; ++kb) {
                        if (!mbar_wait_warp(full0 + 8 * s, ph, p.err, kErrFull)) { ok = false; break; }
                        if (PAIR && !mbar_wait_cluster_warp(pfull0 + 8 * s, ph, p.err, kErrFull)) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t ah = sw128_desc_lo(tiles0 + s * stage_bytes), al = ah + ab;
                        const uint32_t bh = al + ab, bl = bh + bb;
                        if (lead) {
                            // one MMA's K: 32 bytes.  The block's small products first: each
                            // MMA truncates the sum, and it is small until hi hi joins.
                            auto acc0 = [&](int kk) { return kk == 0 || dk ? acc : 1u; };
                            bool fresh = true;  // no product of this block is in yet
                            if (ord.cent(kb)) {
#pragma unroll
                                for (int kk = 0; kk < 4; ++kk)
                                    umma_f16<PAIR>(d + kk * dk, al + 2 * kk, bh + 2 * kk, idesc, acc0(kk));
#pragma unroll
                                for (int kk = 0; kk < 4; ++kk)
                                    umma_f16<PAIR>(d + kk * dk, ah + 2 * kk, bl + 2 * kk, idesc, 1u);
                                fresh = false;
                            } else if (!one_sign) {
#pragma unroll
                                for (int kk = 0; kk < 4; ++kk)
                                    umma_f16<PAIR>(d + kk * dk, ah + 2 * kk, bl + 2 * kk, idesc, acc0(kk));
                                fresh = false;
                            }
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                umma_f16<PAIR>(d + kk * dk, ah + 2 * kk, bh + 2 * kk, idesc, fresh ? acc0(kk) : 1u);
                            commit<PAIR>(empty0 + 8 * s);
                        }
                        acc = 1u;
                        if (++s == (uint32_t)p.stages) { s = 0; ph ^= 1u; }
                    }
                    if (ok && lead) commit<PAIR>(xfull0 + 8 * b);
                }
            }
            // every MMA issued must be complete before the tensor memory is freed
            if (lead) {
                commit<PAIR>(drain);
                mbar_drain(drain, 0);
            }
            __syncwarp();
        } else {
            // ---------------- code loaders (warps 2, 3) ----------------
            // The words of each K block go to a small ring by 4-byte cp.async (a
            // code is only 4-byte aligned): lane l takes word l & 7 of rows
            // 4 i + (l >> 3).  They are warps of their own because a decoder's
            // proxy fence waits for its own loads in flight.
            const int r0 = (warp - 2) * 64 + (lane >> 3), c = lane & 7;
            uint32_t cs = 0, cph = 1;
            for (unsigned t = t0; t < p.num_tiles && ok; t += grid) {
                const size_t j0 = min(first_code(t), p.n - 1);
                const uint8_t *base = p.codes + j0 * (size_t)p.cs;
                const int last = (int)min((size_t)(CG_BM - 1), p.n - 1 - j0);  // rows past n repeat the last code
                for (int kb = 0; kb < KB; ++kb) {
                    if (!mbar_wait_warp(cempty0 + 8 * cs, cph, p.err, kErrEmpty)) { ok = false; break; }
                    const uint32_t dst = ring0 + cs * RING_BYTES;
                    const int o = ord.part(kb) * (32 * WPI) + 4 * c;
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const int r = r0 + 4 * i;
                        const uint8_t *src = base + min(r, last) * p.cs + o;
#pragma unroll
                        for (int q = 0; q < WPI; ++q)  // zero beyond the packed bytes (D < 64)
                            cp_async4(dst + r * (32 * WPI) + 32 * q + 4 * c, src + 32 * q,
                                      o + 32 * q < p.pb ? 4u : 0u);
                    }
                    cp_async_arrive(cfull0 + 8 * cs);
                    if (++cs == (uint32_t)p.ring) { cs = 0; cph ^= 1u; }
                }
            }
            cp_async_wait_all();
        }
    } else if (warp < 4 + DW) {
        // ---------------- decoders ----------------
        // Four warps decode a K block, 32 rows each: lane l takes 16-byte chunk
        // l & 7 (8 coordinates) of rows 4 i + (l >> 3), so eight lanes read a
        // row's consecutive words and write its 128 bytes without bank
        // conflicts.  Eight warps are two groups that take every other block:
        // a block's waits, loads and fence are latencies in series, which the
        // groups overlap (8 x 200k, 768-d 8-bit: 255 -> 242 us; 384-d 4-bit: 100 ->
        // 95 us; 40 x 50k, 1536-d 4-bit: 129 -> 118 us).
        if constexpr (DW == 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
        constexpr int GROUPS = DW / 4, ITEMS = 8;
        const int r0 = ((warp - 4) & 3) * 32 + (lane >> 3), c = lane & 7;
        NibTab tab{};
        if constexpr (NIB) {
#pragma unroll
            for (int v = 0; v < 8; ++v) {
                uint32_t h, l;
                const float cv = v < p.levels ? p.centroids[v] : 0.0f;
                split16(cv * p.cent, p.fmt, h, l);
                const int sh = 8 * (v & 3);
                tab.hl[v >> 2] |= (h & 0xFFu) << sh;
                tab.hh[v >> 2] |= (h >> 8) << sh;
                tab.ll[v >> 2] |= (l & 0xFFu) << sh;
                tab.lh[v >> 2] |= (l >> 8) << sh;
            }
        }
        const uint32_t one = p.fmt == kCgFP16 ? 0x3C003C00u : 0x3F803F80u;
        const uint32_t pm = p.fmt == kCgFP16 ? 0x3CBCu : 0x3FBFu;
        const uint32_t *tl = btab + lane;
        // block `it` of the CTA: stage it % stages and ring slot it % ring (both
        // counts are 2 or more)
        const uint32_t group = GROUPS == 2 ? (uint32_t)(warp - 4) >> 2 : 0u;
        uint32_t s = group, ph = 1, cs = group, cph = 0, it = 0;
        for (unsigned t = t0; t < p.num_tiles && ok; t += grid) {
            for (int kb = 0; kb < KB; ++kb, ++it) {
                if (GROUPS == 2 && (it & 1u) != group) continue;
                if (!mbar_wait_warp(cfull0 + 8 * cs, cph, p.err, kErrFull)) { ok = false; break; }
                uint32_t w[ITEMS][WPI];
                const unsigned char *rb = ring + cs * RING_BYTES;
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) {
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
                const int sw = (c ^ (r0 & 7)) << 4;  // the chunk's place in a row; rows 4 apart flip bit 6
                if (ord.cent(kb)) {
#pragma unroll
                    for (int i = 0; i < ITEMS; ++i) {
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
                        unsigned char *d = dst + 512 * i + (sw ^ ((i & 1) << 6));
                        *reinterpret_cast<uint4 *>(d) = hi;
                        *reinterpret_cast<uint4 *>(d + CG_A_BYTES) = lo;
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < ITEMS; ++i) {
                        uint4 v;
                        if constexpr (NIB) v = nib_sign(w[i][0], one, pm);
                        else v = byte_sign(w[i][0], w[i][WPI - 1], one, pm);
                        *reinterpret_cast<uint4 *>(dst + 512 * i + (sw ^ ((i & 1) << 6))) = v;
                    }
                }
                fence_proxy_async_smem();  // the generic stores before the MMAs' async reads
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(full0 + 8 * s);
                    mbar_arrive(cempty0 + 8 * cs);
                }
                s += GROUPS;
                if (s >= (uint32_t)p.stages) { s -= p.stages; ph ^= 1u; }
                cs += GROUPS;
                if (cs >= (uint32_t)p.ring) { cs -= p.ring; cph ^= 1u; }
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
        for (unsigned t = t0; t < p.num_tiles && ok; t += grid) {
            const size_t row = first_code(t) + 32 * quad + lane;
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
                c1 = ord.chunk_end(p, c0);
                const uint32_t b = gc % NB, xph = (gc / NB) & 1u;
                if (!mbar_wait_warp(xfull0 + 8 * b, xph, p.err, kErrTmemFull)) { ok = false; break; }
                tc_fence_after();
                const uint32_t X = lanes + b * BUF;
                auto pieces = [&](auto f, auto small) {
                    if constexpr (SPLIT) chunk_quarters(X, p.NT, f);
                    else chunk_pieces<CPT, decltype(small)::value>(X, cpt, f);
                };
                constexpr std::false_type wide{};
                // How a chunk joins the running sum.  Symmetric and light: centroid
                // chunks are added (the light form's last chunk is its clamped
                // correction).  Asymmetric: fma(x, f, y) with f = scale gamma for
                // the sign part and sigma for the centroid part.
                if (LIGHT || p.form == kCgSym) {
                    if (c0 == 0) pieces([&](int k, float x) { y[k] = x; }, wide);
                    else if (!LIGHT || ord.cent(c0)) pieces([&](int k, float x) { y[k] = __fadd_rn(y[k], x); }, wide);
                }
                if constexpr (!LIGHT) {
                    if (p.form == kCgAsym) {
                        const float fx = ord.cent(c0) ? __fmul_rn(sigma, p.undo_c)
                                                      : __fmul_rn(__fmul_rn(p.scale, gamma), p.undo_s);
                        if (c0 == 0) pieces([&](int k, float x) { y[k] = __fmul_rn(x, fx); }, wide);
                        else pieces([&](int k, float x) { y[k] = __fmaf_rn(x, fx, y[k]); }, wide);
                    }
                } else if (!ord.cent(c0)) {
                    const CgCols cols(col0, cpt, p.m);
                    const float4 *rs = p.rs + cols.base;
                    pieces([&](int k, float x) {
                        const float2 r = __ldg(reinterpret_cast<const float2 *>(rs + cols.offset(k)) + 1);
                        const float ip = __fmul_rn(__fmul_rn(__fmul_rn(y[k], p.undo_c), r.x), sigma);
                        const float corr = __fmul_rn(__fmul_rn(x, r.y), gamma);
                        const float lim = fabsf(ip);
                        y[k] = __fadd_rn(ip, fmaxf(-lim, fminf(lim, corr)));
                    }, std::true_type{});
                }
                __syncwarp();
                tc_fence_before();
                if (lane == 0) {
                    if (PAIR) mbar_arrive_cluster(rank0_addr(xempty0 + 8 * b));
                    else mbar_arrive(xempty0 + 8 * b);
                }
            }
            if (!ok) break;
            if (row >= p.n) continue;
            // d = max(0, r2 + c2 - 2 (C r1) c1); a NaN gives 0
            const float c2 = __fmul_rn(norm, norm);
            const float c1 = p.form == kCgSym ? __fmul_rn(__fmul_rn(sigma, norm), p.undo_c) : norm;
            float *o = p.out + col0 * p.ldo + row;
            const CgCols cols(col0, cpt, p.m);
            const float4 *rs = p.rs + cols.base;
            const int live = cols.live;
            if constexpr (FULL) {
                // products, or distances with another pass's products clamped in (all
                // loads of 16 columns in flight at once).  The norms join last: an
                // infinite one times a sum of two signs gives what it does in the
                // reference, where products that held it could cancel to a NaN.
                const bool add = p.post == kCgClampedSum;
#pragma unroll
                for (int k0 = 0; k0 < CPT; k0 += 16) {
                    if (k0 >= live) break;
                    float other[16];
#pragma unroll
                    for (int k = 0; k < 16; ++k) other[k] = add && k0 + k < live ? __ldcs(o + k * p.ldo) : 0.0f;
#pragma unroll
                    for (int k = k0; k < k0 + 16; ++k) {
                        if (k < live) {
                            const float4 r = __ldg(rs + k);
                            float v = __fmul_rn(y[k], r.x);
                            if (add) {
                                const float ip = __fmul_rn(__fmul_rn(__fmul_rn(y[k], p.undo_c), r.z), sigma);
                                const float lim = fabsf(ip);
                                const float sum = __fadd_rn(ip, fmaxf(-lim, fminf(lim, other[k - k0])));
                                v = fmaxf(__fmaf_rn(-2.0f, __fmul_rn(__fmul_rn(sum, r.w), norm), __fadd_rn(r.y, c2)), 0.0f);
                            }
                            __stcs(o, v);
                        }
                        o += p.ldo;
                    }
                }
            } else {
#pragma unroll
                for (int k = 0; k < CPT; ++k) {
                    if (k % 16 == 0 && k >= live) break;
                    if (k < live) {
                        const float2 r = __ldg(reinterpret_cast<const float2 *>(rs + k));
                        const float ipt = __fmul_rn(__fmul_rn(y[k], r.x), c1);
                        __stcs(o, fmaxf(__fmaf_rn(-2.0f, ipt, __fadd_rn(r.y, c2)), 0.0f));
                    }
                    o += p.ldo;
                }
            }
        }
    }
    if (!ok) report_wait(p.err, p.status);
    tc_fence_before();
    // PAIR: no CTA leaves while the other may still arrive on its barriers or
    // read its shared memory
    if constexpr (PAIR) cluster_sync();
    else __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc512<PAIR>(tmem_base);
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
    float4 *__restrict__ rs, int *__restrict__ err) {
    if (err && blockIdx.x == 0 && threadIdx.x == 0) *err = 0;
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
// rs: symmetric (sigma n, n^2, sigma, n); light (n, n^2, sigma, (pi / 2D) gamma).
__global__ void __launch_bounds__(256) cg_rows_codes_kernel(const uint8_t *__restrict__ codes, size_t m,
                                                            Params P, DevTables T, int KBm, int form,
                                                            int fmt, __nv_bfloat16 *__restrict__ ph,
                                                            __nv_bfloat16 *__restrict__ pl,
                                                            float4 *__restrict__ rs, int *__restrict__ err) {
    if (err && blockIdx.x == 0 && threadIdx.x == 0) *err = 0;
    const int half = KBm * CG_BK, K = form == kCgLight ? 2 * half : half, quads = K / 4;
    const size_t total = m * (size_t)quads;
    const float f = P.cent_scale[fmt];
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
                        : make_float4(__fmul_rn(sigma, norm), n2, sigma, norm);
        }
    }
}

unsigned rows_grid(size_t work) {
    return (unsigned)std::min<size_t>(std::max<size_t>(1, (work + 255) / 256), (size_t)148 * 16);
}

}  // namespace

// What the truncation of the chunks takes off a sum of terms of one sign, which a
// scale may give back.  FP16: near rows of 32 to 2048 values at 2 to 8 bits, 1.6e-8
// to 5e-8.  BF16: half an ulp, 0.72 2^-24 of the sum so far on average, an MMA, over
// 12 MMAs a block: 44.5 of the whole sum in chunks of 8 blocks (queries), whose sum
// grows evenly, 20.5 in chunks of 4 (codes against codes).
constexpr double kTruncBias[2][2] = {{0.0, 3e-8}, {1.9e-6, 8.8e-7}};  // [fmt][rows are codes]
float cg_cent_scale(const float *centroids, int levels, int fmt) {
    const bool h16 = fmt == kCgFP16;
    const float top = h16 ? 2048.0f : 2.0f, step = h16 ? 4.0f : 1.0f / 256, rows = h16 ? kRowScale : 1.0f;
    const double t1 = kTruncBias[fmt][0], t2 = kTruncBias[fmt][1];
    // the positive levels (the others are their negatives): value, 1 / c, and c^2 times
    // about its share
    struct Level {
        float c;
        double inv, w;
    };
    std::vector<Level> lv;
    double sw = 0.0;
    for (int v = levels / 2; v < levels; ++v) {
        const double c = centroids[v];
        lv.push_back({centroids[v], 1.0 / c, c * c * std::exp(-c * c / 3.0)});
        sw += lv.back().w;
    }
    float best = top;
    double best_err = 1e300;
    for (int i = 0; i < 256; ++i) {
        const float a = top - step * (float)i;
        const double ia = 1.0 / a;
        double d1 = 0.0, d2 = 0.0, l2 = 0.0;
        for (const Level &e : lv) {
            const float x = e.c * a, h = h16 ? round_fp16(x) : round_bf16(x);
            const float l = h16 ? round_fp16(x - h) : round_bf16(x - h);
            const double s = e.inv * ia, d = ((double)h + l) * s - 1.0, r = l * s;
            d1 += e.w * d;
            d2 += e.w * d * d;
            l2 += e.w * r * r;
        }
        // a product of two values is off by d + d' - r r', and the undoing factor by
        // its rounding.  Over near rows, whose values agree, that is a bias, to which
        // the tensor core's truncation of the chunks adds; over others it averages out.
        const double u2 = (double)(1.0f / (a * a)) * a * a - 1.0;
        const double u1 = (double)(1.0f / (a * rows)) * a * rows - 1.0;
        const double b2 = (2.0 * d1 - l2) / sw + u2 - t2, b1 = d1 / sw + u1 - t1;
        const double err = b2 * b2 + b1 * b1 + (2.0 * d2 + l2 * l2 / sw) / sw / 64.0;
        if (err < best_err) {
            best = a;
            best_err = err;
        }
    }
    return best;
}

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
        static_cast<__nv_bfloat16 *>(r.lo), r.rs, r.err);
    return cudaGetLastError();
}

cudaError_t launch_cg_rows_codes(const Params &P, const DevTables &T, const uint8_t *codes, size_t m,
                                 int form, int fmt, const CgRows &r, cudaStream_t st) {
    const int KBm = (P.D + CG_BK - 1) / CG_BK;
    cg_rows_codes_kernel<<<rows_grid(m * (size_t)KBm * 32), 256, 0, st>>>(
        codes, m, P, T, KBm, form, fmt, static_cast<__nv_bfloat16 *>(r.hi),
        static_cast<__nv_bfloat16 *>(r.lo), r.rs, r.err);
    return cudaGetLastError();
}

// The tiles of the code side: 256 codes over a CTA pair for wide ones, 128 otherwise.
static size_t code_tiles(size_t n, int NT) { return NT > 64 ? (n + 255) / 256 : (n + 127) / 128; }

// Columns per tile: the width that takes the least time by a rough count of
// clocks: waves of 148 CTAs times a tile's K blocks, each the slower of its
// MMAs (10 per block on average over both parts, NT / 2 clocks each) and its
// decode, plus the tile's epilogue.  Wide tiles (128, 256) run on CTA pairs.
int cg_tile_cols(const Params &P, int form, size_t m, size_t n) {
    const int KBm = (P.D + CG_BK - 1) / CG_BK, KB = form == kCgSym ? KBm : 2 * KBm;
    int best = 256;
    double best_t = 0.0;
    for (int NT = 256; NT >= 16; NT >>= 1) {
        const size_t tiles = code_tiles(n, NT) * ((m + NT - 1) / NT), slots = NT > 64 ? 74 : 148;
        const double waves = (double)((tiles + slots - 1) / slots);
        const double mma = 5.0 * NT, dec = NT <= 64 ? 600.0 : 1000.0;
        const double t = waves * (KB * std::max(mma, dec) + 8.0 * NT + 1000.0);
        if (NT == 256 || t < best_t) {
            best = NT;
            best_t = t;
        }
    }
    return best;
}

cudaError_t launch_cgemm(const Params &P, const DevTables &T, int form, int fmt, const CgRows &rows,
                         size_t m, const uint8_t *codes, size_t n, float *out, size_t ldo, int *status,
                         cudaStream_t st, int post) {
    if (m == 0 || n == 0) return cudaSuccess;
    if (P.cs % 4 || (reinterpret_cast<uintptr_t>(codes) & 3)) return cudaErrorMisalignedAddress;
    if (!aligned16({rows.hi, rows.lo, rows.rs}) || !rows.err) return cudaErrorMisalignedAddress;
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
    a.post = post;
    a.KBm = (P.D + CG_BK - 1) / CG_BK;
    a.KB = form == kCgSym ? a.KBm : 2 * a.KBm;
    // Chunk lengths (K blocks), so that what truncation takes off a chunk stays below
    // the rounding of an FP32 sum.  FP16: 2 (1 where the whole part is 4 blocks or
    // fewer).  BF16: 8 for queries and 4 for codes against codes, whose terms share a
    // sign more often.  The sign part: +-1 by +-1 sums (light) are exact integers;
    // otherwise FP16 takes 8, since its hi products are nearly exact in FP32 and its
    // share of a near pair's sum is a third at most (near pairs of 1536-d 2-bit, mean
    // error with 16 / 8 / 2 blocks 3.4 / 2.0 / 1.1e-7, and 2000 x 100k of 768-d 1.40 /
    // 1.44 / 1.49 ms; an FP32 chain's largest error there is 3e-6, this one's 1.1e-6),
    // and BF16 16 (8 change its near pairs' mean error by 1e-7 of 0.7e-6; under the
    // power cap 4096 x 500k of 768-d take 15.9 ms with 8 and 15.3 with 16).
    // Fewer than 32 rows, where the scan kernel's short FP32 chains stand for
    // comparison: chunks of 1 and 4 blocks with the quarters apart, an error like the
    // scan's (near pairs of 2-bit codes, 8 rows, largest 5.5e-7 -> 3.3e-7 against the
    // scan's 2.9e-7) for 97 -> 102 us at 8 x 200k of 384-d, 245 -> 250 of 768-d 8-bit,
    // 93 -> 100 at 24 x 200k.
    a.chm = fmt == kCgFP16 ? (a.KBm <= 4 || m < 32 ? 1 : 2) : form == kCgAsym ? 8 : 4;
    a.chs = form == kCgLight ? a.KBm : fmt != kCgFP16 ? 16 : m < 32 ? 4 : 8;
    a.m = m;
    a.rs = rows.rs;
    a.scale = P.scale;
    a.cent = P.cent_scale[fmt];
    a.undo_s = fmt == kCgFP16 && form == kCgAsym ? 1.0f / kRowScale : 1.0f;
    a.undo_c = 1.0f / (a.cent * (form != kCgAsym ? a.cent : fmt == kCgFP16 ? kRowScale : 1.0f));
    a.out = out;
    a.ldo = ldo;
    a.err = rows.err;
    a.status = status;
    a.NT = cg_tile_cols(P, form, m, n);
    const bool split = fmt == kCgFP16 && m < 32 && a.NT <= 32;
    const bool pair = a.NT > 64;
    const int stage_bytes = 2 * CG_A_BYTES + 2 * a.NT * (pair ? 64 : 128);
    const int tab = P.nibble ? 0 : CG_TAB_BYTES, ring_bytes = CG_BM * (P.nibble ? 32 : 64);
    const int avail = CG_SMEM_MAX - CG_FIXED - tab;
    a.stages = std::min(CG_MAX_STAGES, (avail - 2 * ring_bytes) / stage_bytes);
    a.ring = std::min(CG_MAX_RING, (avail - a.stages * stage_bytes) / ring_bytes);
    const size_t smem = (size_t)a.stages * stage_bytes + a.ring * ring_bytes + CG_FIXED + tab;
    const size_t nt = code_tiles(n, a.NT), tiles = nt * ((m + a.NT - 1) / a.NT);
    if (tiles > 0x7FFFFFFFull || nt > 0x7FFFFFFFull) return cudaErrorInvalidValue;
    a.num_nt = (unsigned)nt;
    a.num_tiles = (unsigned)tiles;
    alignas(64) CUtensorMap mh, ml;
    const int K = a.KB * CG_BK, box = pair ? a.NT / 2 : a.NT;
    if (!make_map(&mh, rows.hi, K, m, box) || !make_map(&ml, rows.lo, K, m, box)) return cudaErrorInvalidValue;
    const bool light = form == kCgLight;
    // wide tiles, narrow ones, and narrow ones with split accumulators
    auto pick = [&](auto nib, auto form_light, auto form_full) {
        constexpr bool N = decltype(nib)::value, L = decltype(form_light)::value, F = decltype(form_full)::value;
        return pair    ? cgemm_kernel<4, N, L, true, F, false>
               : split ? cgemm_kernel<8, N, L, false, F, true>
                       : cgemm_kernel<8, N, L, false, F, false>;
    };
    using T_ = std::true_type;
    using F_ = std::false_type;
    auto by_form = [&](auto nib) {
        return post != kCgDist ? pick(nib, F_{}, T_{}) : light ? pick(nib, T_{}, F_{}) : pick(nib, F_{}, F_{});
    };
    auto kern = P.nibble ? by_form(T_{}) : by_form(F_{});
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(pair ? 2 * sm_grid(tiles, 2) : sm_grid(tiles));
    cfg.blockDim = dim3(CG_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = pair ? 2 : 1;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, mh, ml, a);
}

}  // namespace tq
