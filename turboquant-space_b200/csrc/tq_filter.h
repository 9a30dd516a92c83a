// tq_filter.h -- the serving top-k's filter pass (tq_filter.cu): every code
// whose approximate distance can be among a row's kc smallest, from one FP16
// product per term on the tensor cores, with a rigorous per-row error bound.
#pragma once

#include "tq_internal.h"

namespace tq {

constexpr int kFilterBound = 4;      // index-wide maxima of the bound (see tq_filter.cu)
constexpr int kFilterTile = 256;     // codes per tile (a CTA pair)
constexpr int kFilterSample = 8192;  // codes of the first threshold's sample
constexpr int kFilterCap = 4096;     // codes listed per row and level

// What the filter keeps of a corpus, beside its codes.
struct FilterIndex {
    const uint8_t *codes = nullptr;  // 4-byte aligned
    size_t n = 0;
    uint32_t *rho = nullptr;   // [n rounded up to kFilterTile]: a pair of FP16 alpha g / sigma
    float *bound = nullptr;    // [kFilterBound]
    float alpha = 0.0f;        // scale of the FP16 centroids
};
// The scale in [1024, 2048) whose FP16 centroids have the least rounding error.
float filter_alpha(const float *centroids, int levels);
// rho and bound of ix.codes; ix.alpha set.
cudaError_t launch_filter_index(const Params &P, const DevTables &T, const FilterIndex &ix, cudaStream_t st);

// Per-batch buffers for up to `rows` query rows.
struct FilterBuffers {
    void *planes = nullptr;      // rows x filter_k(P) FP16
    float4 *rowq = nullptr;      // rows: |dq|, |ds|, |q~|, |s~| (2-norms, see the bound)
    float2 *r12 = nullptr;       // rows: |q|, |q|^2
    float2 *uv = nullptr;        // rows: the threshold test's constants
    float *thr = nullptr;        // rows: the threshold itself
    float *samp = nullptr;       // rows x kFilterSample
    int *cnt = nullptr;          // rows: listed codes (may exceed kFilterCap)
    float *list_d = nullptr;     // rows x kFilterCap
    int *list_i = nullptr;       // rows x kFilterCap
    int *bad = nullptr;          // rows: 1 where the candidates are not the kc smallest
};
size_t filter_k(const Params &P);  // values per query row: two parts of whole 64-value blocks

// MMAs into one accumulator (the bound's accumulation term).
int filter_mmas(const Params &P);
// The bound's term for the FP32 sums of both sides, a share of sum |terms|.
float filter_sums(const Params &P);

// Prepared queries -> the kc smallest approximate distances of each row,
// ascending, cand_d / cand_i [rows][kc] (index -1 past the corpus), and bad.
// The row count is read from m_dev (at most rows); every launch may be
// captured.  `err` as in launch_cgemm.
cudaError_t launch_filter(const Params &P, const DevTables &T, const FilterIndex &ix,
                          const float *q_rot, const float *s_q, const float *norms, const int *m_dev,
                          int rows, int kc, const FilterBuffers &b, float *cand_d, long long *cand_i,
                          int *err, cudaStream_t st);

}  // namespace tq
