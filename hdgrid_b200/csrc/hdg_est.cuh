// Tensor-core estimates of query-row distances and the pass that keeps what they cannot exclude.
//
// A row x (a decoded PQ vector or a base vector) and a query q are rounded to BF16; the product
// S = bf16(q) . bf16(x) accumulates in FP32 on the tensor cores.  With rq = |q - bf16(q)| and
// rx = |x - bf16(x)|,
//     |q . x - S| <= rq |x| + |bf16(q)| rx + g |q| |x|,
// g covering the FP32 accumulation, so |q - x|^2 is at least
//     |q|^2 + |x|^2 - 2 S - 2 (rq |x| + |bf16(q)| rx + g |q| |x|).
// A row whose bound exceeds a query's threshold t cannot have a distance at or below t; every
// other row is handed on to the exact FP32 arithmetic, which alone decides the results.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "hdg_index.h"

namespace hdg {

constexpr int kEstM = 128;   // rows per tile (TMEM lanes)
constexpr int kEstN = 128;   // queries per tile (TMEM columns)
// slack on every norm (the FP32 rounding of norms, bounds and of the exact sums) and the
// accumulation term per dimension
constexpr float kEstSlack = 1e-5f;
constexpr float kEstAcc = 2.4e-7f;

// Per row: {|x|^2 (1 - slack), |x|, rx, 0}
// Per query: {2 (rq + g |q|), 2 |bf16(q)|, |q|^2 (1 - slack) - t, 0}; -FLT_MAX third: no threshold
struct EstArgs {
    const float4* rowc;
    const float4* qc;
    const uint16_t* qb;        // bf16 queries, row stride ldq elements (a multiple of 8)
    uint64_t ldq;
    uint32_t n_rows;
    uint32_t tiles;            // row tiles
    // candidate ranges (k_est<true>): the (query, range) entries of every row tile
    const uint32_t* ent_off;   // [tiles + 1]
    const uint32_t* nt_off;    // [tiles + 1] prefix of the entries' query tiles
    const uint4* ent;          // {query, first row | last row + 1 << 16 in the tile, position - pool row, 0}
    const uint64_t* qoff;      // row of each query in dist / spos
    uint32_t* drow;            // kept pool rows
    uint32_t* prow;            // and their candidate positions
    // every query against every row (k_est<false>), label boxes tested on the way
    uint32_t nq;
    uint32_t row0, row_step;   // base row of row r: row0 + r * row_step
    const float* labels;       // [base rows x l]
    const float* boxes;        // [nq x 2 l]
    int l;
    uint32_t* list;            // [nq x cap] kept base rows
    uint32_t cap;              // a query's count may pass it: the entries past it are not stored
    uint32_t* cnt;             // kept rows of each query
};

// rows: bf16 [n_rows x ld] (ld a multiple of 8, d <= ld); RANGES as in EstArgs.  err: set when a
// wait expired.
void est_ranges(const EstArgs& a, const void* rows_bf16, int ld, int* err, cudaStream_t st);
void est_all(const EstArgs& a, const void* rows_bf16, int ld, int* err, cudaStream_t st);

}  // namespace hdg
