// tq_cgemm.h -- the M x N distances with in-kernel decoded code tiles (tq_cgemm.cu).
#pragma once

#include "tq_internal.h"

namespace tq {

enum CgForm { kCgAsym = 0, kCgSym = 1, kCgLight = 2 };  // queries / codes / codes + light QJL term
// What the epilogue does with the products: distances; the products ip themselves,
// times the row's first scalar but neither norm (kCgAsym); or distances with out's
// own values, such products of another pass, added to ip after clamping them to
// +-|ip| (kCgSym: the full QJL form's correction).
enum CgPost { kCgDist = 0, kCgProducts = 1, kCgClampedSum = 2 };
enum CgFmt { kCgFP16 = 0, kCgBF16 = 1 };                // 16-bit type of the hi / lo pairs

// The row operand: hi and lo planes of m x cg_row_k 16-bit values and four
// scalars a row, all 16-byte aligned, and the error word of the call that they
// belong to: a word of its own, since a wait gives up as soon as it sees a set one.
struct CgRows {
    void *hi = nullptr, *lo = nullptr;
    float4 *rs = nullptr;
    int *err = nullptr;
};
size_t cg_row_k(const Params &P, int form);

// The rows behind the columns [col0, col0 + cpt) of one part of a tile: `live` of
// them (0 where the part lies past row m - 1, as the second half of a tile does
// whose rows end in the first), and the row whose scalars column k may read: its
// own, or for columns past the live ones, whose values are not used, one that exists.
struct CgCols {
    size_t base;
    int live, last;
    __host__ __device__ CgCols(size_t col0, int cpt, size_t m)
        : base(col0 < m ? col0 : m - 1),
          live(col0 >= m ? 0 : m - col0 < (size_t)cpt ? (int)(m - col0) : cpt),
          last(live > 0 ? live - 1 : 0) {}
    // column k reads row base + offset(k)
    __host__ __device__ int offset(int k) const { return k < last ? k : last; }
};
// Columns per tile of a call, and the parts a tile's columns are split in.
int cg_tile_cols(const Params &P, int form, size_t m, size_t n);
inline int cg_tile_parts(int cols) { return cols > 64 ? 2 : 1; }

// P.cent_scale[fmt]: the scale in (1024, 2048] (FP16) or (1, 2] (BF16) at which
// products of the centroids' pairs (without lo lo) have the least bias and error.
float cg_cent_scale(const float *centroids, int levels, int fmt);

// Prepared queries (kCgAsym) or codes (kCgSym, kCgLight) -> row operand; *r.err = 0
// (r.err null: left alone).
cudaError_t launch_cg_rows_prepared(const Params &P, const float *q_rot, const float *s_q,
                                    const float *norms, size_t m, int fmt, const CgRows &r,
                                    cudaStream_t st);
cudaError_t launch_cg_rows_codes(const Params &P, const DevTables &T, const uint8_t *codes, size_t m,
                                 int form, int fmt, const CgRows &r, cudaStream_t st);

// out[i * ldo + j] = distance of row i to code j.  Codes 4-byte aligned, the
// code size a multiple of 4 (every padded dim but 4).  *rows.err is set non-zero if
// a bounded wait in the kernel gave up, and *status (device int, may be null) with it.
cudaError_t launch_cgemm(const Params &P, const DevTables &T, int form, int fmt, const CgRows &rows,
                         size_t m, const uint8_t *codes, size_t n, float *out, size_t ldo, int *status,
                         cudaStream_t st, int post = kCgDist);

}  // namespace tq
