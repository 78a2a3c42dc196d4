// Tensor-core estimates of query-row distances and the pass that keeps what they cannot exclude.
//
// A row x (a decoded PQ vector or a base vector) and a query q are rounded to FP16; the product
// S = h(q) . h(x) accumulates in FP32 on the tensor cores.  With rq = |q - h(q)| and
// rx = |x - h(x)|,
//     |q . x - S| <= rq |x| + |h(q)| rx + g |q| |x|,
// g covering the FP32 accumulation, so |q - x|^2 is at least
//     |q|^2 + |x|^2 - 2 S - 2 (rq |x| + |h(q)| rx + g |q| |x|)
// (FP16 rather than BF16: its bounds are eight times tighter, and values it cannot hold make the
// residuals, and so the bounds, infinite).
// A row whose bound exceeds a query's threshold t cannot have a distance at or below t and is
// dropped.  Of every other row k_est reports the bound's depth below the threshold in steps of one
// byte; what the bounds leave open is decided by the exact FP32 arithmetic.
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
// Per query: {2 (rq + g |q|), 2 |h(q)|, z = |q|^2 (1 - slack) - t, steps per unit of distance};
// z = -FLT_MAX: no threshold
struct EstArgs {
    const float4* rowc;
    const float4* qc;
    const uint16_t* qb;        // FP16 queries, row stride ldq elements (a multiple of 8)
    uint64_t ldq;
    uint32_t n_rows;
    uint32_t tiles;            // row tiles
    // candidate ranges (k_est<true>): the (query, range) entries of every row tile
    const uint32_t* ent_off;   // [tiles + 1]
    const uint32_t* nt_off;    // [tiles + 1] prefix of the entries' query tiles
    const uint4* ent;          // {query, first row | last row + 1 << 16 in the tile, position - pool row, 0}
    const uint64_t* qoff;      // row of each query in prow
    uint32_t* prow;            // kept rows: candidate position (below 2^24) | step << 24, the step
                               // 1 + (t - bound) * steps per unit, rounded, at most 255
                               // (one word: with the steps as bytes beside the positions the
                               // 10,000 x 227,000-candidate batch took 11.6 ms, 11.1 so)
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

// rows: FP16 [n_rows x ld] (ld a multiple of 8, d <= ld); RANGES as in EstArgs.  err: set when a
// wait expired.
void est_ranges(const EstArgs& a, const void* rows_f16, int ld, int* err, cudaStream_t st);
void est_all(const EstArgs& a, const void* rows_f16, int ld, int* err, cudaStream_t st);

}  // namespace hdg
