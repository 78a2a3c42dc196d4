// The filtered query path: super_grid::index::query
// (src/index/2-level_index/Super-Grid-IVF_PQ.cu:985-1249) as B200 kernels.
//
//   k_prologue   per query: filter recovery (preprocessing.cu:3-32) -> f32 box, cell box
//                (:930-961), label-rank box, Morton corners (:903-928, zorder.cu:3-15), per-list filtered
//                counts by 2^d-corner inclusion-exclusion over the dense prefix counts
//                (:693-765) and per-cluster sums (:767-790).
//   k_coarse     per query: exact f32 L2 to the non-empty clusters, top n_list
//                (::refine, :1034-1042); their non-empty lists, exact L2 to the list
//                centroids, top sub_lists (select_sub_clusters, :849-901); Morton interval
//                [lower_bound(zlo), lower_bound(zhi+1)) inside every probed list (zorder.cu:656-685).
//   k_batch      candidate offsets, work items and the batch sums of the post-filter budget
//                beta (:1198-1222).
//   k_pre_scan   predicate-first queries: label-rank boxes, then the label predicate
//                (filter.cu:30-64), survivors listed for the ADC (prefiltering.cu:36-51).
//   k_lut        per query PQ lookup table (build_pq_lut_kernel, product-quantization.cu:4-35).
//   k_scan       persistent streaming ADC over the contiguous Z-ordered candidate ranges
//                (compute_batched_L2_distance_kernel, :37-77) with the LUT in shared memory,
//                optional fused label predicate (filter.cu:30-64); one f32 per candidate.
//   k_select     per query: the K smallest (distance, position) pairs (RAFT select_k in the
//                reference) by a two-pass histogram select.
//   k_refine     per query: label predicate on the ADC top-n_cand (post-filter, :1227-1236),
//                exact f32 re-rank and top-k (refine.cu:36-120).
// There is no dense [q x max_row_len] candidate table and one host round trip per batch
// (the candidate total and the batch-wide budget).
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <type_traits>

#include "hdg_device.cuh"
#include "hdg_est.cuh"
#include "hdg_internal.h"

namespace hdg {

constexpr int kThreads = 256;
constexpr uint32_t kInvalid = 0xffffffffu;
constexpr uint32_t kChunk = 32768;  // default most candidates per scan work item (SCAN_CHUNK)
constexpr uint32_t kChunkMin = 1024;
constexpr int kBins = 4096;         // select histogram
constexpr int kBCap = 4096;         // boundary-bin buffer of the select
constexpr uint32_t kPreChunk = 16384, kPreChunkMin = 1024;  // candidates per work item of the predicate pass

struct Workspace {
    float* box;              // [q x 2l]
    int* cells;              // [q x 2l]
    uint32_t* rank_box;      // [q x 4] rank box (low ranks, high ranks | guard bits), inner box (same)
    uint64_t* zrange;        // [q x 2]
    uint32_t* list_counts;   // [q x L]
    uint32_t* cluster_counts;// [q x C]
    uint32_t* probe_clusters;// [q x Pc]
    uint32_t* probe_lists;   // [q x Ps]
    uint32_t* range_start;   // [q x Ps]
    uint32_t* range_len;     // [q x Ps]
    uint32_t* range_pre;     // [q x (Ps + 1)] exclusive prefix of range_len (last: the candidate total)
    uint32_t* qstat;         // [q x 4]: cand_total, exact_total, n_lists, n_clusters
    uint32_t* qtiles;        // [q] row tiles (kEstM pool rows) that the query's candidate ranges touch
    uint64_t* scal;          // [8]: cand sum, exact sum, max cand, items, beta (f32 bits),
                             //      queries dropped by a capacity, kept candidates, selected sum;
                             //      then (in its padding) the GEMM status word and the row-tile sum
    uint64_t* qoff;          // [q + 1] candidate offsets into dist
    uint32_t* item_off;      // [q + 1] work-item offsets of the ADC scan
    uint32_t* pitem_off;     // [q + 1] work-item offsets of the predicate pass (predicate-first queries)
    uint32_t* mm;            // [q x 2] min / max finite distance key
    uint32_t* nfin;          // [q] finite distances (predicate passed)
    uint32_t* lab_read;      // [q] candidates of the predicate pass whose labels were read
    uint32_t* rank_read;     // [q] candidates of the predicate pass whose label ranks were read
    uint32_t* counter;       // [8] work counters: ADC scan, refine, predicate pass; [3] candidates per scan item,
                             //     [4] per predicate item
    float* lut;              // [q x G x 256 x 32] f32, or __half when lut16
    int lut16;               // LUT stored in FP16 (LUT_FP16=1); the scan sums in FP32
    uint32_t* qbud;          // [q] candidate budget n_cand of each query (k_batch)
    uint64_t* soff;          // [q + 1] offsets of the queries' selections in cand_pool
    uint32_t* cand_pool;     // [soff[q]] selected candidates: min(n_cand, candidates) per query
    uint32_t* cand_count;    // [q]
    uint64_t sel_cap;        // cand_pool capacity in entries
    uint32_t* ritem_off;     // [q + 1] refine work-item offsets (k_refine_plan)
    uint32_t* rdone;         // [q] refine items finished per query
    uint32_t* rsurv;         // [q] rows re-ranked exactly per query (predicate survivors of the selection)
    uint32_t* rlab;          // [q] selected entries whose labels the re-rank read (the ranks left them open)
    uint64_t* rpart;         // [refine items x k_max] best keys of each refine item
    int surv_list;           // 1: the predicate pass lists each predicate-first query's survivors
    float* dist;             // [sum of candidates]
    uint32_t* spos;          // [sum of candidates] candidate position of each entry of a compact row
    // the estimate pass of post-filter queries (nullptr: not run)
    uint32_t* prq;           // [q] 1: the ADC runs on the candidates that the estimates leave open only
    float4* est_qc;          // [q] constants of the estimate test
    int* est_w;              // [q] steps by which an ADC distance can differ from its bound
    uint32_t* est_in;        // [q] candidates sure to be selected (at the start of the query's selection)
    uint32_t* est_row;       // [q] entries of the row before the open candidates
    float* S;                // [q x (C + L)] tensor-core dot products (nullptr: exact path only)
    uint64_t ldS;
    float* qnorm;            // [q] squared query norms
    void* qbf;               // [q x d] bf16 queries of the coarse GEMM, then FP16 ones of the estimate pass
    int* gemm_err;           // tensor-core wait expiry flag
    float* feats;            // [q x 48] learned-schedule features
    uint32_t* lq_ps;         // [q] lists to probe predicted by the learned schedule
    uint8_t* lq_sched;       // [q] predicate-first flag predicted by the learned schedule
    // per-query parameters (nullptr: the batch-wide value)
    const uint32_t* qk;      // [q] k of each query (<= k_max)
    const uint32_t* qps;     // [q] lists probed (<= sub_lists)
    const uint8_t* qsched;   // [q] 0 = the index's reference schedule, 1 = predicate-first + re-rank
    uint32_t k_max;          // output row stride
    int mode;                // batch schedule: 0 pre-filter (exps0 <= 1), 1 post-filter, 2 single dim
    uint32_t exps0;
    uint32_t chunk;          // most candidates per scan work item (SCAN_CHUNK)
    uint32_t scan_items;     // work items k_batch aims at when it sets the items' size
    int is_split;            // IS_SPLIT: trimmed Morton sub-ranges per probed list
    int nsplit;              // sub-ranges per probed list (n_split when is_split, else 1)
    uint64_t cap;            // distance-buffer capacity in candidates
};

constexpr uint64_t kChainQueries = 4096;

enum ScanMode { kPre = 0, kPost = 1, kL1 = 2 };

// The kernels that launch_next may launch as programmatic dependents begin with this: the next kernel
// of the stream may be brought up (its blocks resident and waiting at the same point), and this one
// waits until the kernel before it has ended.  The others (k_pre_scan, k_scan_plan, the estimate
// pass's) are always launched without the attribute and start after the kernel before them; with
// it they would race.
__device__ __forceinline__ void chain_start() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ uint32_t q_k(const Workspace& w, uint64_t qi) {
    return w.qk ? max(1u, min(w.qk[qi], w.k_max)) : w.k_max;
}
__device__ __forceinline__ int q_sched(const Workspace& w, uint64_t qi) { return w.qsched ? (int)w.qsched[qi] : 0; }
// true when query qi evaluates the label predicate inside the scan
__device__ __forceinline__ bool q_prefilter(const Workspace& w, uint64_t qi) {
    return w.mode == kPre || q_sched(w, qi) == 1;
}
// true when query qi's row is compact: the predicate pass lists its survivors (position and
// pool row), the ADC scan replaces each pool row by the survivor's distance
__device__ __forceinline__ bool compacts(const Workspace& w, uint64_t qi) { return w.surv_list && q_prefilter(w, qi); }
// true when the ADC of query qi runs only on the candidates that its estimates leave open (positions
// and pool rows, as a compacting query's survivors, est_row entries into the row)
__device__ __forceinline__ bool pruned(const Workspace& w, uint64_t qi) { return w.prq && w.prq[qi] == 1; }
__device__ __forceinline__ uint64_t row_of(const Workspace& w, uint64_t qi) {
    return w.qoff[qi] + (pruned(w, qi) ? w.est_row[qi] : 0u);
}
// Candidate budget n_cand of query qi given the batch's beta and max_row_len: the query's k for
// the reference pre-filter schedule (exps0 <= 1), exps0 * k for the single-dim schedule and the
// predicate-first schedule, and the reference's min(exps0 * k * beta, max_row_len) for the
// post-filter schedule (Super-Grid-IVF_PQ.cu:1219-1222), with no further cap.  Here k is the
// call's k (the width of the output rows): the reference has one topk per batch, so a batch
// whose queries ask for different k runs as a batch of the largest k whose rows are cut to
// each query's k.  k_batch evaluates it once per query into w.qbud.
__device__ __forceinline__ uint64_t budget_of(const Workspace& w, uint64_t qi, float beta, uint64_t max_row) {
    if (w.mode == kPre) return q_k(w, qi);
    const uint32_t k = w.k_max;
    uint64_t K;
    if (w.mode == kL1 || q_sched(w, qi) == 1) {
        K = (uint64_t)w.exps0 * k;
    } else if (!(beta < INFINITY)) {
        K = max_row;
    } else {
        const float want = (float)((uint64_t)w.exps0 * k) * beta;
        K = want >= 1.8e19f ? ~0ull : (uint64_t)want;
        K = min(K, max_row);
    }
    return max((uint64_t)1, min(K, (uint64_t)0xffffffffu));
}
__device__ __forceinline__ uint32_t q_budget(const Workspace& w, uint64_t qi) { return w.qbud[qi]; }
// A compact row (predicate survivors) that its budget takes whole: the selection is the row
// itself -- its distance slots still hold the survivors' pool rows, as the ADC scan leaves such
// a row alone -- so the select skips it and the re-rank reads the row in place.  (nfin: the
// row's survivors, which the select does not change, unlike cand_count.)
__device__ __forceinline__ bool takes_row(const Workspace& w, uint64_t qi) {
    return compacts(w, qi) && w.nfin[qi] <= q_budget(w, qi);
}
// Candidates per scan work item (k_batch sets the word)
__device__ __forceinline__ uint32_t scan_chunk(const Workspace& w) { return w.counter[3]; }
__device__ __forceinline__ uint32_t pre_chunk(const Workspace& w) { return w.counter[4]; }
// The selected candidates (pool rows) of query qi: its row of the selection buffer, or its
// distance row when it takes the row whole
__device__ __forceinline__ uint32_t* sel_row(const Workspace& w, uint64_t qi) {
    return takes_row(w, qi) ? reinterpret_cast<uint32_t*>(w.dist + w.qoff[qi]) : w.cand_pool + w.soff[qi];
}

// Warp-wide sum / maximum of a u64 (every lane gets it)
__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = max(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}

// Slot of this lane among the lanes of its warp where f holds, taken from the counter *ctr
// with one atomic per warp (~0u where f is false).  Every lane of the warp must call it.
__device__ __forceinline__ uint32_t warp_reserve(bool f, uint32_t* ctr) {
    const unsigned bal = __ballot_sync(0xffffffffu, f);
    if (!bal) return ~0u;
    const int lane = threadIdx.x & 31, leader = __ffs(bal) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(ctr, (uint32_t)__popc(bal));
    base = __shfl_sync(0xffffffffu, base, leader);
    return f ? base + __popc(bal & ((1u << lane) - 1u)) : ~0u;
}

// Appends v at the next free slot of dst (counter *ctr) where f holds; every lane calls it.
__device__ __forceinline__ void warp_append(bool f, uint32_t v, uint32_t* ctr, uint32_t* dst) {
    const uint32_t slot = warp_reserve(f, ctr);
    if (f) dst[slot] = v;
}

// Inclusive sum of x over the block (blockDim.x a multiple of 32, <= 1024); s_w: 32 words of
// shared scratch that no other thread touches until the following barrier.
__device__ __forceinline__ unsigned long long block_inclusive_sum(unsigned long long x, unsigned long long* s_w,
                                                                  unsigned long long* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_w[warp] = x;
    __syncthreads();
    if (warp == 0) {
        unsigned long long y = lane < nw ? s_w[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long z = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) y += z;
        }
        s_w[lane] = y;
    }
    __syncthreads();
    *total = s_w[nw - 1];
    return x + (warp ? s_w[warp - 1] : 0);
}

// ------------------------------------------------------------------------------------
// k_prologue
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) k_prologue(IndexDev D, GridMeta g, FilterDev f,
                                                       const float* __restrict__ qlabels,
                                                       int label_cols, Workspace w) {
    chain_start();
    extern __shared__ uint32_t s_counts[];  // [L]
    __shared__ float s_box[2 * kMaxDims];
    __shared__ int s_cells[2 * kMaxDims];
    __shared__ uint64_t s_corner[1 << kMaxDims];
    __shared__ int s_sign[1 << kMaxDims];
    __shared__ uint32_t s_rank[4];
    __shared__ uint32_t s_count[kMaxDims][3];
    const uint64_t qi = blockIdx.x;
    const int t = threadIdx.x;
    const int l = g.l;
    const uint32_t L = D.n_lists;
    if (qi == 0 && t == 0) *w.gemm_err = 0;
    if (t < 4) s_rank[t] = 0;
    if (t < l) {
        float lo, hi;
        recover_dim(f, qlabels + qi * label_cols, t, &lo, &hi);
        s_box[2 * t] = lo;
        s_box[2 * t + 1] = hi;
        w.box[qi * 2 * l + 2 * t] = lo;
        w.box[qi * 2 * l + 2 * t + 1] = hi;
    }
    __syncthreads();
    // The threshold counts behind the rank boxes, one binary search per thread: thresholds <= lo,
    // <= hi and < lo of every dim (one after another they were 36 dependent loads on 12-bit ranks)
    if (D.rankpack && t >= 32 && t < 32 + 3 * l) {
        const int i = (t - 32) / 3, what = (t - 32) % 3;
        const float x = s_box[2 * i + (what == 1 ? 1 : 0)];
        const float* thr = D.rank_thr + (uint64_t)i * D.rank_stride;
        uint32_t a = 0, b = isnan(x) ? 0u : D.rank_n[i];
        while (a < b) {
            const uint32_t m = (a + b) >> 1;
            if (what != 2 ? thr[m] <= x : thr[m] < x) a = m + 1;
            else b = m;
        }
        s_count[i][what] = a;
    }
    if (t < l) {
        const int od = g.shuffle[t];
        int lo, hi;
        cell_range(s_box[2 * od], s_box[2 * od + 1], g.left[t], g.span[t], g.grid_dims[t], &lo, &hi);
        s_cells[2 * t] = lo;
        s_cells[2 * t + 1] = hi;
        w.cells[qi * 2 * l + 2 * t] = lo;
        w.cells[qi * 2 * l + 2 * t + 1] = hi;
    }
    __syncthreads();
    if (t < l && D.rankpack) {
        // The rank box of label dim t: a rank below that of lo holds labels below a threshold
        // <= lo, a rank above that of hi labels at or above a threshold > hi.  The inner box:
        // ranks whose labels all lie in [lo, hi] -- above the rank of the largest threshold
        // below lo (or every rank when the dim's smallest label is >= lo), and below the rank
        // of hi (or every rank when its largest label is <= hi).  NaN bounds reject nothing.
        const float blo = s_box[2 * t], bhi = s_box[2 * t + 1];
        const uint32_t n = D.rank_n[t];
        const uint32_t rlo = isnan(blo) ? 0u : s_count[t][0], rhi = isnan(bhi) ? n : s_count[t][1];
        const int ilo = isnan(blo) || D.rank_min[t] >= blo ? 0 : (int)s_count[t][2] + 1;
        const int ihi = isnan(bhi) || D.rank_max[t] <= bhi ? (int)n : (int)rhi - 1;
        const bool empty = ilo > ihi;  // no rank is sure to pass: the field's box [1, 0]
        const int off = t * (int)(D.rank_bits + 1);
        if (rlo) atomicOr(&s_rank[0], rlo << off);
        atomicOr(&s_rank[1], rhi << off);
        if (empty || ilo) atomicOr(&s_rank[2], (empty ? 1u : (uint32_t)ilo) << off);
        if (!empty && ihi) atomicOr(&s_rank[3], (uint32_t)ihi << off);
    }
    __syncthreads();
    if (t == 0) {
        int clo[kMaxDims], chi[kMaxDims];
        for (int i = 0; i < l; i++) {
            clo[i] = s_cells[2 * i];
            chi[i] = s_cells[2 * i + 1];
        }
        w.zrange[qi * 2] = morton_encode(clo, g.morton_dims, g.morton_max_bits, g.morton_valid_map);
        w.zrange[qi * 2 + 1] = morton_encode(chi, g.morton_dims, g.morton_max_bits, g.morton_valid_map);
        w.rank_box[qi * 4] = s_rank[0];
        w.rank_box[qi * 4 + 1] = s_rank[1] | D.rank_guard;
        w.rank_box[qi * 4 + 2] = s_rank[2];
        w.rank_box[qi * 4 + 3] = s_rank[3] | D.rank_guard;
    }
    // corners of the cell box over the valid (unmasked) dims (get_prefix_sum_device :693-724)
    const int dv = __popc(g.morton_valid_map);
    const int n_corner = 1 << dv;
    for (int mask = t; mask < n_corner; mask += blockDim.x) {
        int sign = 1, vi = 0;
        bool zero = false;
        uint64_t flat = 0;
        for (int i = 0; i < l; i++) {
            int c = 0;
            if ((g.morton_valid_map >> i) & 1) {
                if ((mask >> vi) & 1) {
                    c = s_cells[2 * i] - 1;
                    sign = -sign;
                    if (c < 0) zero = true;
                } else {
                    c = s_cells[2 * i + 1];
                }
                vi++;
            }
            flat += (uint64_t)(c < 0 ? 0 : c) * g.cell_stride[i];
        }
        s_corner[mask] = flat;
        s_sign[mask] = zero ? 0 : sign;
    }
    __syncthreads();
    if (D.prefix16) {  // dense in 16 bits: eight lists per 16-byte load when L allows, else two per 4 bytes
        if ((L & 7) == 0) {
            for (uint32_t jo = t; 8 * jo < L; jo += blockDim.x) {
                long long a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                for (int m = 0; m < n_corner; m++) {
                    const int sg = s_sign[m];
                    if (!sg) continue;
                    const uint4 v = reinterpret_cast<const uint4*>(D.prefix16 + s_corner[m] * L)[jo];
                    const uint32_t wv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int h = 0; h < 4; h++) {
                        a[2 * h] += (long long)sg * (long long)(wv[h] & 0xffffu);
                        a[2 * h + 1] += (long long)sg * (long long)(wv[h] >> 16);
                    }
                }
#pragma unroll
                for (int h = 0; h < 8; h++) s_counts[8 * jo + h] = (uint32_t)a[h];
                uint4* lc = reinterpret_cast<uint4*>(w.list_counts + qi * L + 8 * jo);
                lc[0] = make_uint4((uint32_t)a[0], (uint32_t)a[1], (uint32_t)a[2], (uint32_t)a[3]);
                lc[1] = make_uint4((uint32_t)a[4], (uint32_t)a[5], (uint32_t)a[6], (uint32_t)a[7]);
            }
        } else if ((L & 1) == 0) {
            for (uint32_t jp = t; 2 * jp < L; jp += blockDim.x) {
                long long a0 = 0, a1 = 0;
                for (int m = 0; m < n_corner; m++) {
                    const int sg = s_sign[m];
                    if (!sg) continue;
                    const uint32_t v = reinterpret_cast<const uint32_t*>(D.prefix16 + s_corner[m] * L)[jp];
                    a0 += (long long)sg * (long long)(v & 0xffffu);
                    a1 += (long long)sg * (long long)(v >> 16);
                }
                s_counts[2 * jp] = (uint32_t)a0;
                s_counts[2 * jp + 1] = (uint32_t)a1;
                w.list_counts[qi * L + 2 * jp] = (uint32_t)a0;
                w.list_counts[qi * L + 2 * jp + 1] = (uint32_t)a1;
            }
        } else {
            for (uint32_t j = t; j < L; j += blockDim.x) {
                long long acc = 0;
                for (int m = 0; m < n_corner; m++) {
                    const int sg = s_sign[m];
                    if (sg) acc += (long long)sg * (long long)D.prefix16[s_corner[m] * L + j];
                }
                s_counts[j] = (uint32_t)acc;
                w.list_counts[qi * L + j] = (uint32_t)acc;
            }
        }
    } else if (D.prefix) {  // dense: one coalesced row of L counts per corner
        for (uint32_t j = t; j < L; j += blockDim.x) {
            long long acc = 0;
            for (int m = 0; m < n_corner; m++) {
                const int sg = s_sign[m];
                if (sg) acc += (long long)sg * (long long)D.prefix[s_corner[m] * L + j];
            }
            s_counts[j] = (uint32_t)acc;
            w.list_counts[qi * L + j] = (uint32_t)acc;
        }
    } else {
        // compressed rows (query_compressed_sum_device, Super-Grid-IVF_PQ.cu:648-691): the corner
        // at flat cell t * Dd + z reads list j's row t, the last change point at or before z
        const uint32_t Dd = (uint32_t)g.grid_dims[g.diff_dim];
        for (uint32_t j = t; j < L; j += blockDim.x) {
            long long acc = 0;
            for (int m = 0; m < n_corner; m++) {
                const int sg = s_sign[m];
                if (!sg) continue;
                const uint64_t r = (s_corner[m] / Dd) * L + j;
                const uint32_t z = (uint32_t)(s_corner[m] % Dd);
                const uint64_t b0 = D.prefix_off[r];
                uint64_t lo = b0, hi = D.prefix_off[r + 1];
                while (lo < hi) {  // first change point past z
                    const uint64_t mid = (lo + hi) >> 1;
                    if ((uint32_t)(D.prefix_rows[mid] >> 32) <= z) lo = mid + 1;
                    else hi = mid;
                }
                if (lo > b0) acc += (long long)sg * (long long)(uint32_t)D.prefix_rows[lo - 1];
            }
            s_counts[j] = (uint32_t)acc;
            w.list_counts[qi * L + j] = (uint32_t)acc;
        }
    }
    __syncthreads();
    for (uint32_t c = t; c < D.C; c += blockDim.x) {
        uint32_t s = 0;
        for (uint32_t j = D.cluster_off[c]; j < D.cluster_off[c + 1]; j++) s += s_counts[j];
        w.cluster_counts[qi * D.C + c] = s;
    }
}

// ------------------------------------------------------------------------------------
// k_coarse
// ------------------------------------------------------------------------------------
__device__ __forceinline__ float seq_l2_v4(const float* __restrict__ q, const float* __restrict__ c,
                                           int d) {
    // sequential f32 sum in dimension order, 16-byte loads of the centroid row
    float s = 0.f;
    const float4* c4 = reinterpret_cast<const float4*>(c);
    for (int i = 0; i < d / 4; i++) {
        const float4 v = __ldg(c4 + i);
        float t0 = __fsub_rn(q[4 * i], v.x);
        s = __fadd_rn(s, __fmul_rn(t0, t0));
        t0 = __fsub_rn(q[4 * i + 1], v.y);
        s = __fadd_rn(s, __fmul_rn(t0, t0));
        t0 = __fsub_rn(q[4 * i + 2], v.z);
        s = __fadd_rn(s, __fmul_rn(t0, t0));
        t0 = __fsub_rn(q[4 * i + 3], v.w);
        s = __fadd_rn(s, __fmul_rn(t0, t0));
    }
    for (int i = d & ~3; i < d; i++) {
        const float t0 = __fsub_rn(q[i], c[i]);
        s = __fadd_rn(s, __fmul_rn(t0, t0));
    }
    return s;
}

__device__ __forceinline__ uint32_t lower_bound_u64(const uint64_t* __restrict__ a, uint32_t n,
                                                    uint64_t key) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a[mid] < key)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// N lower_bounds (key k[i] in the sorted a[i][0, n[i])) with their searches interleaved so the
// dependent loads overlap; each result equals lower_bound_u64's
template <int N>
__device__ __forceinline__ void lower_bound_u64_multi(const uint64_t* const (&a)[N], const uint32_t (&n)[N],
                                                      const uint64_t (&k)[N], uint32_t (&r)[N]) {
    uint32_t lo[N], hi[N];
#pragma unroll
    for (int i = 0; i < N; i++) {
        lo[i] = 0;
        hi[i] = n[i];
    }
    for (;;) {
        bool any = false;
        uint64_t v[N];
        uint32_t m[N];
#pragma unroll
        for (int i = 0; i < N; i++) {
            m[i] = (lo[i] + hi[i]) >> 1;
            v[i] = lo[i] < hi[i] ? a[i][m[i]] : 0;
        }
#pragma unroll
        for (int i = 0; i < N; i++) {
            if (lo[i] < hi[i]) {
                if (v[i] < k[i]) lo[i] = m[i] + 1;
                else hi[i] = m[i];
            }
            any |= lo[i] < hi[i];
        }
        if (!any) break;
    }
#pragma unroll
    for (int i = 0; i < N; i++) r[i] = lo[i];
}

// One sub-range of a probed list's Morton interval [lo, hi) when is_split = 1.
// get_query_end_points_kernel (zorder.cu:596-654) cuts the interval into
// min(len, n_split) near-equal parts; zorder_range_query_kernel (:474-594) then moves each
// part's start forward by up to three next-in-box jumps and drops the part when a jump fails
// or lands past the part's last code.  (The reference reads the probed list as
// candidates[c] instead of candidates[q * n + c], :500; the list of this query is used.)
// Empty parts get start kInvalid.
__device__ void split_subrange(const uint64_t* __restrict__ z, uint32_t off, uint32_t lo, uint32_t hi, int s,
                               int ns, const int* box, const GridMeta& g, uint32_t* start, uint32_t* len) {
    const uint32_t n = hi - lo;
    const uint32_t nsp = min(n, (uint32_t)ns);
    if (n == 0 || (uint32_t)s >= nsp) {
        *start = kInvalid;
        *len = 0;
        return;
    }
    const uint32_t qn = n / nsp, r = n % nsp;
    uint32_t a = off + lo + (uint32_t)s * qn + min((uint32_t)s, r);
    const uint32_t b = a + qn + ((uint32_t)s < r ? 1u : 0u);
    const uint64_t zmax = z[b - 1];
    uint64_t cur = z[a];
    bool valid = true;
    for (int jump = 0; jump < 3; jump++) {
        const uint32_t idx = a + lower_bound_u64(z + a, b - a, cur);
        if (idx >= b) break;
        a = idx;
        int c[kMaxDims];
        morton_decode(z[idx], c, g.morton_dims, g.morton_max_bits, g.morton_valid_map);
        if (cells_in_box(c, box, g.morton_dims)) break;
        uint64_t nz = 0;
        if (!next_code_in_box(z[idx], box, g.morton_dims, g.morton_max_bits, g.morton_valid_map, &nz) || nz >= zmax) {
            valid = false;
            break;
        }
        cur = nz;
    }
    *start = a;
    *len = valid ? b - a : 0;
}


// Band [lo, hi] around the exact f32 distance of query qi to centroid col (clusters first,
// then lists) from the tensor-core dot product S: |(|q|^2 + |c|^2 - 2 q.c) - exact| is below
// 2 * 2^-8 |q||c| for BF16-rounded inputs, plus f32 rounding of the norms and sums; the band
// doubles both terms.
__device__ __forceinline__ void approx_band(const IndexDev& D, const Workspace& w, uint64_t qi, uint32_t col,
                                            float* lo, float* hi) {
    coarse_band(w.qnorm[qi], D.cnorm[col], w.S[qi * w.ldS + col], lo, hi);
}

// One block of kCoarseThreads per query: the query's phases are serial (selections, searches),
// so smaller blocks keep more queries in flight per SM
constexpr int kCoarseThreads = 128;
__global__ void __launch_bounds__(kCoarseThreads) k_coarse(IndexDev D, GridMeta g, const float* __restrict__ queries,
                                                     int Pc, int Ps, int sort_n1, int sort_n2,
                                                     Workspace w) {
    chain_start();
    extern __shared__ uint64_t s_keys[];  // [max(sort_n1, sort_n2)], then the bands' lows, the query vector
    float* s_lo = reinterpret_cast<float*>(s_keys + max(sort_n1, sort_n2));
    float* s_q = s_lo + max(sort_n1, sort_n2);
    __shared__ uint32_t s_chosen[1024];
    __shared__ uint32_t s_red[3];
    __shared__ uint32_t s_wc[32];
    __shared__ unsigned long long s_scan[32];
    __shared__ uint32_t s_hist[256];
    __shared__ unsigned long long s_sel[4];
    __shared__ int s_nvalid;
    __shared__ float s_bound;
    const uint64_t qi = blockIdx.x;
    const int t = threadIdx.x;
    const int d = D.d;
    const bool est = w.S != nullptr;  // tensor-core estimates of the centroid distances
    for (int i = t; i < d; i += blockDim.x) s_q[i] = queries[qi * d + i];
    if (t == 0) {
        s_nvalid = 0;
        s_red[0] = s_red[1] = s_red[2] = 0;
    }
    __syncthreads();
    // One pass over the clusters: those with a non-zero filtered count (filter_none_zero_data
    // :1027-1028) get a key -- the upper end of their estimate band and the cluster -- and the
    // band's lower end; the others ~0.  When all of them fit in n_list the ranking cannot change
    // the chosen set: no distances needed.
    {
        uint32_t nz = 0;
        for (int c = t; c < sort_n1; c += blockDim.x) {
            uint64_t key = ~0ull;
            if (c < (int)D.C && w.cluster_counts[qi * D.C + c] > 0) {
                float lo = 0.f, hi = 0.f;
                if (est) approx_band(D, w, qi, c, &lo, &hi);
                key = ((uint64_t)float_key(hi) << 32) | (uint32_t)c;
                s_lo[c] = lo;
                nz++;
            }
            s_keys[c] = key;
        }
        nz = __reduce_add_sync(0xffffffffu, nz);  // one shared atomic per warp
        if ((t & 31) == 0 && nz) atomicAdd(&s_nvalid, (int)nz);
    }
    __syncthreads();
    const bool all_c = s_nvalid <= Pc;
    // With the tensor-core estimates, only clusters whose lower bound is below the n_list-th
    // smallest upper bound can be in the exact top n_list; only those get exact distances.
    const bool prune_c = !all_c && est;
    if (prune_c) {
        const uint64_t kth = block_select_smallest(s_keys, sort_n1, Pc, s_hist, s_wc, s_sel, false);
        if (t == 0) s_bound = key_float((uint32_t)(kth >> 32));
        __syncthreads();
    }
    for (int c = t; c < sort_n1; c += blockDim.x) {
        uint64_t key = s_keys[c];
        if (key != ~0ull) {
            if (all_c) key = (uint32_t)key;
            else if (prune_c && s_lo[c] > s_bound) key = ~0ull;
            else key = ((uint64_t)float_key(seq_l2_v4(s_q, D.centers + (uint64_t)c * d, d)) << 32) | (uint32_t)c;
        }
        s_keys[c] = key;
    }
    __syncthreads();
    // with every non-empty cluster taken the keys hold no distance: cluster order, compacted;
    // otherwise the n_list smallest (distance, cluster) keys, a set in no particular order
    if (all_c) block_compact_keys(s_keys, sort_n1, s_wc);
    else block_select_smallest(s_keys, sort_n1, Pc, s_hist, s_wc, s_sel);
    const int npc = min(Pc, s_nvalid);
    for (int i = t; i < Pc; i += blockDim.x) {
        const uint32_t c = i < npc ? (uint32_t)s_keys[i] : kInvalid;
        w.probe_clusters[qi * Pc + i] = c;
        if (i < 1024) s_chosen[i] = c;
    }
    __syncthreads();
    if (t == 0) s_nvalid = 0;
    __syncthreads();
    // the same for the non-empty lists of the chosen clusters
    const uint32_t Smax = D.S_max;
    // list slot e = chosen cluster e / Smax, its list e % Smax (shifts when Smax is a power of two)
    const bool sm_pow2 = (Smax & (Smax - 1)) == 0;
    const int sm_shift = __ffs((int)Smax) - 1;
    {
        uint32_t nzl = 0;
        for (int e = t; e < sort_n2; e += blockDim.x) {
            uint64_t key = ~0ull;
            const int i = sm_pow2 ? (e >> sm_shift) : e / (int)Smax, jj = sm_pow2 ? (e & (int)(Smax - 1)) : e % (int)Smax;
            if (i < npc) {
                const uint32_t c = s_chosen[i], j = D.cluster_off[c] + jj;
                if (j < D.cluster_off[c + 1] && w.list_counts[qi * D.n_lists + j] > 0) {
                    float lo = 0.f, hi = 0.f;
                    if (est) approx_band(D, w, qi, D.C + j, &lo, &hi);
                    key = ((uint64_t)float_key(hi) << 32) | j;
                    s_lo[e] = lo;
                    nzl++;
                }
            }
            s_keys[e] = key;
        }
        nzl = __reduce_add_sync(0xffffffffu, nzl);
        if ((t & 31) == 0 && nzl) atomicAdd(&s_nvalid, (int)nzl);
    }
    __syncthreads();
    // lists probed by this query: sub_lists, or the query's own n_probe when given
    const int Psq = w.qps ? max(1, min(Ps, (int)w.qps[qi])) : Ps;
    const bool all_l = s_nvalid <= Psq;
    const bool prune_l = !all_l && est;
    if (prune_l) {
        const uint64_t kth = block_select_smallest(s_keys, sort_n2, Psq, s_hist, s_wc, s_sel, false);
        if (t == 0) s_bound = key_float((uint32_t)(kth >> 32));
        __syncthreads();
    }
    for (int e = t; e < sort_n2; e += blockDim.x) {
        uint64_t key = s_keys[e];
        if (key != ~0ull) {
            const uint32_t j = (uint32_t)key;
            if (all_l) key = j;
            else if (prune_l && s_lo[e] > s_bound) key = ~0ull;
            else key = ((uint64_t)float_key(seq_l2_v4(s_q, D.sub_centers + (uint64_t)j * d, d)) << 32) | j;
        }
        s_keys[e] = key;
    }
    __syncthreads();
    // every list taken: the keys carry no distance, compacted (in list-id order when the chosen
    // clusters are in cluster order too); otherwise the sub_lists smallest (distance, list) keys
    if (all_l) block_compact_keys(s_keys, sort_n2, s_wc);
    else block_select_smallest(s_keys, sort_n2, Psq, s_hist, s_wc, s_sel);
    const int nps = min(Psq, s_nvalid);
    // the probed lists in list-id (= pool) order, so candidate positions follow pool order:
    // marked in a bitmap over the lists (s_chosen is free again), then emitted word by word
    if (!(all_l && all_c)) {
        if (D.n_lists <= 32u * 1024u) {
            const int W = (int)((D.n_lists + 31) / 32);
            for (int i = t; i < W; i += blockDim.x) s_chosen[i] = 0;
            __syncthreads();
            for (int i = t; i < nps; i += blockDim.x) {
                const uint32_t j = (uint32_t)s_keys[i];
                atomicOr(&s_chosen[j >> 5], 1u << (j & 31));
            }
            __syncthreads();
            unsigned long long run = 0;
            for (int b0 = 0; b0 < W; b0 += blockDim.x) {
                const int i = b0 + t;
                const uint32_t word = i < W ? s_chosen[i] : 0u;
                const unsigned long long x = (unsigned long long)__popc(word);
                unsigned long long tot = 0;
                uint32_t at = (uint32_t)(run + block_inclusive_sum(x, s_scan, &tot) - x);
                for (uint32_t m = word; m; m &= m - 1) s_keys[at++] = (uint32_t)(32 * i + __ffs((int)m) - 1);
                run += tot;
                __syncthreads();  // s_scan is reused by the next chunk
            }
        } else {
            const int sort_n3 = (int)next_pow2_dev((uint32_t)max(nps, 2));
            for (int i = t; i < sort_n3; i += blockDim.x)
                s_keys[i] = i < nps ? (uint64_t)(uint32_t)s_keys[i] : ~0ull;
            __syncthreads();
            block_bitonic_sort(s_keys, sort_n3);
        }
    }
    const uint64_t zlo = w.zrange[qi * 2], zhi = w.zrange[qi * 2 + 1];
    uint32_t my_cand = 0, my_exact = 0, my_tiles = 0;
    auto tiles_of = [](uint32_t start, uint32_t len) {
        return len ? (start + len - 1) / (uint32_t)kEstM - start / (uint32_t)kEstM + 1u : 0u;
    };
    const int ns = w.nsplit;
    int box[2 * kMaxDims];
    if (w.is_split)
        for (int i = 0; i < 2 * g.l; i++) box[i] = w.cells[qi * 2 * g.l + i];
    // two probed lists per thread and step: their four Morton bound searches interleaved
    for (int i0 = t; i0 < Ps; i0 += 2 * blockDim.x) {
        const uint64_t* arr[4];
        uint32_t nn[4], rr[4], list[2], off[2];
        uint64_t kk[4];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int i = i0 + u * (int)blockDim.x;
            uint32_t size = 0;
            list[u] = kInvalid;
            off[u] = 0;
            if (i < nps) {
                list[u] = (uint32_t)s_keys[i];
                off[u] = D.list_off[list[u]];
                size = D.list_off[list[u] + 1] - off[u];
            }
            arr[2 * u] = arr[2 * u + 1] = D.zcodes + off[u];
            nn[2 * u] = nn[2 * u + 1] = size;
            kk[2 * u] = zlo;
            kk[2 * u + 1] = zhi + 1;
        }
        lower_bound_u64_multi<4>(arr, nn, kk, rr);
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int i = i0 + u * (int)blockDim.x;
            if (i >= Ps) break;
            const uint32_t lo = rr[2 * u], hi = rr[2 * u + 1];
            uint32_t start = 0, len = 0;
            if (i < nps) {
                start = off[u] + lo;
                len = hi - lo;
                my_exact += w.list_counts[qi * D.n_lists + list[u]];
            }
            w.probe_lists[qi * Ps + i] = list[u];
            const uint64_t r0 = (qi * Ps + i) * (uint64_t)ns;
            if (!w.is_split) {
                w.range_start[r0] = start;
                w.range_len[r0] = len;
                my_cand += len;
                my_tiles += tiles_of(start, len);
            } else {
                for (int sp = 0; sp < ns; sp++) {
                    uint32_t st = kInvalid, ln = 0;
                    if (i < nps) split_subrange(D.zcodes, off[u], lo, hi, sp, ns, box, g, &st, &ln);
                    w.range_start[r0 + sp] = st;
                    w.range_len[r0 + sp] = ln;
                    my_cand += ln;
                    my_tiles += tiles_of(st, ln);
                }
            }
        }
    }
    my_cand = __reduce_add_sync(0xffffffffu, my_cand);
    my_exact = __reduce_add_sync(0xffffffffu, my_exact);
    my_tiles = __reduce_add_sync(0xffffffffu, my_tiles);
    if ((t & 31) == 0) {
        atomicAdd(&s_red[0], my_cand);
        atomicAdd(&s_red[1], my_exact);
        atomicAdd(&s_red[2], my_tiles);
    }
    __syncthreads();
    // the exclusive prefix of the ranges' lengths (its last entry the candidate total): the
    // predicate pass, the scan and the select find a position's range by searching it
    {
        // (the ranges past the probed lists' are empty: their prefix is the total)
        const int Rq = Ps * ns, Rn = nps * ns;
        const uint32_t* len = w.range_len + qi * Rq;
        uint32_t* pre = w.range_pre + qi * (Rq + 1);
        unsigned long long run = 0;
        for (int b0 = 0; b0 < Rn; b0 += blockDim.x) {
            const int i = b0 + t;
            const unsigned long long x = i < Rn ? len[i] : 0;
            unsigned long long tot = 0;
            const unsigned long long inc = block_inclusive_sum(x, s_scan, &tot);
            if (i < Rn) pre[i] = (uint32_t)(run + inc - x);
            run += tot;
            __syncthreads();  // s_scan is reused by the next chunk
        }
        for (int i = Rn + t; i <= Rq; i += blockDim.x) pre[i] = (uint32_t)run;
    }
    if (t == 0) {
        w.qstat[qi * 4 + 0] = s_red[0];
        w.qstat[qi * 4 + 1] = s_red[1];
        w.qstat[qi * 4 + 2] = nps;
        w.qstat[qi * 4 + 3] = npc;
        w.qtiles[qi] = s_red[2];
    }
}


// ------------------------------------------------------------------------------------
// k_batch: per-query candidate offsets and work items, batch sums (one block)
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) k_batch(uint64_t q, Workspace w) {
    chain_start();
    __shared__ unsigned long long s_tot[32], s_items[32], s_pitems[32], s_sel[32];
    __shared__ unsigned long long s_red[4], s_drop[2];
    __shared__ float s_beta;
    __shared__ uint32_t s_chunk;
    const int t = threadIdx.x;
    if (t == 0) s_red[0] = s_red[1] = s_red[2] = s_red[3] = s_drop[0] = s_drop[1] = 0;
    __syncthreads();
    const uint64_t per = (q + blockDim.x - 1) / blockDim.x;
    const uint64_t b = t * per, e = min(q, b + per);
    // a predicate-first query of the predicate pass has predicate items over its candidates
    // (its ADC items follow from its survivors, k_scan_plan); any other query has ADC items
    // Candidates per scan item: the smallest power of two from kChunkMin to SCAN_CHUNK (which the
    // autotuner takes from one batch, and which bounds every other one's items only) that leaves at
    // most scan_items items.  A small batch then fills the SMs (37 queries of
    // 73,000 candidates ran as 111 items of up to 32,768 in 325 us, in 125 us this way); a large one keeps long
    // items, since each loads its query's LUT.
    // Predicate items likewise, for 64 times as many items (a warp each, 16 per resident warp): an
    // item costs some 4 us of searches before its first word, a long one leaves a tail.  Predicate
    // stage, us, at items of 16,384 / 8,192 / 4,096 / 2,048: 2 G candidates 1,307 / 1,405 / 1,649 /
    // 2,183; 1 G 1,263 / 1,262 / 1,364 / 1,648; 161 M 265 / 199 / 186 / 211; 3 M (1,024) 38, as items of
    // 8,192 188.
    __shared__ uint32_t s_pchunk;
    {
        unsigned long long c = 0, all = 0;
        for (uint64_t i = b; i < e; i++) c += w.qstat[i * 4];
        block_inclusive_sum(c, s_tot, &all);
        if (t == 0) {
            uint32_t ch = kChunkMin, pc = kPreChunkMin;
            while (ch < w.chunk && (unsigned long long)ch * w.scan_items < all) ch *= 2;
            while (pc < kPreChunk && (unsigned long long)pc * w.scan_items * 64u < all) pc *= 2;
            s_chunk = ch;
            s_pchunk = pc;
        }
        __syncthreads();
    }
    const uint32_t chunk = s_chunk, pchunk = s_pchunk;
    auto n_items = [&](uint64_t i, uint32_t c) { return compacts(w, i) ? 0u : (c + chunk - 1) / chunk; };
    auto n_pitems = [&](uint64_t i, uint32_t c) { return compacts(w, i) ? (c + pchunk - 1) / pchunk : 0u; };
    unsigned long long cand = 0, items = 0, pitems = 0, exact = 0, mx = 0, rtiles = 0;
    for (uint64_t i = b; i < e; i++) {
        rtiles += w.qtiles[i];
        const uint32_t c = w.qstat[i * 4];
        cand += c;
        items += n_items(i, c);
        pitems += n_pitems(i, c);
        exact += w.qstat[i * 4 + 1];
        mx = max(mx, (unsigned long long)c);
    }
    unsigned long long tot_c = 0, tot_i = 0, tot_p = 0;
    unsigned long long rc = block_inclusive_sum(cand, s_tot, &tot_c) - cand;
    unsigned long long ri = block_inclusive_sum(items, s_items, &tot_i) - items;
    unsigned long long rp = block_inclusive_sum(pitems, s_pitems, &tot_p) - pitems;
    unsigned long long dropped = 0, kept = 0;
    for (uint64_t i = b; i < e; i++) {
        const uint32_t c = w.qstat[i * 4];
        w.qoff[i] = rc;
        w.item_off[i] = (uint32_t)ri;
        w.pitem_off[i] = (uint32_t)rp;
        // queries past the distance capacity (a prefix cut: offsets grow with i) get no
        // candidates; the batch's beta and max_row above still count them
        if (rc + c > w.cap) {
            if (c) {
                w.qstat[i * 4] = 0;
                dropped++;
            }
        } else {
            kept += c;
        }
        ri += n_items(i, c);
        rp += n_pitems(i, c);
        rc += c;
        w.mm[2 * i] = 0xffffffffu;
        w.mm[2 * i + 1] = 0u;
        w.nfin[i] = 0;
        w.lab_read[i] = 0;
        w.rank_read[i] = 0;
        w.cand_count[i] = 0;
    }
    if (e == q && b < e) {
        w.qoff[q] = rc;
        w.item_off[q] = (uint32_t)ri;
        w.pitem_off[q] = (uint32_t)rp;
    }
    // one shared atomic per warp (1,024 threads on one word would serialise)
    cand = warp_sum_u64(cand);
    exact = warp_sum_u64(exact);
    mx = warp_max_u64(mx);
    rtiles = warp_sum_u64(rtiles);
    if ((t & 31) == 0) {
        atomicAdd(&s_red[3], rtiles);
        atomicAdd(&s_red[0], cand);
        atomicAdd(&s_red[1], exact);
        atomicMax(&s_red[2], mx);
    }
    __syncthreads();
    if (t == 0) {
        w.scal[0] = s_red[0];
        w.scal[1] = s_red[1];
        w.scal[2] = s_red[2];
        w.scal[3] = tot_i + tot_p;
        w.scal[9] = s_red[3];
        // beta = coarse / real as the reference computes it (Super-Grid-IVF_PQ.cu:1219)
        const float beta = s_red[1] == 0 ? INFINITY : __fdiv_rn((float)s_red[0], (float)s_red[1]);
        w.scal[4] = __float_as_uint(beta);
        s_beta = beta;
        w.counter[0] = 0;
        w.counter[2] = 0;
        w.counter[3] = chunk;
        w.counter[4] = pchunk;
    }
    __syncthreads();
    // each query's budget n_cand, now that the batch's beta and max_row are known, and the
    // offset of its selection (min(n_cand, candidates) entries) in cand_pool
    const float beta = s_beta;
    const uint64_t max_row = s_red[2];
    unsigned long long sel = 0;
    for (uint64_t i = b; i < e; i++) {
        const uint64_t K = budget_of(w, i, beta, max_row);
        w.qbud[i] = (uint32_t)K;
        sel += min(K, (uint64_t)w.qstat[i * 4]);
    }
    unsigned long long tot_s = 0;
    unsigned long long rs = block_inclusive_sum(sel, s_sel, &tot_s) - sel;
    for (uint64_t i = b; i < e; i++) {
        const uint32_t c = w.qstat[i * 4];
        const uint64_t si = min((uint64_t)w.qbud[i], (uint64_t)c);
        w.soff[i] = rs;
        if (rs + si > w.sel_cap && c) {  // past the selection capacity: no candidates either
            w.qstat[i * 4] = 0;
            dropped++;
            kept -= c;
        }
        rs += si;
    }
    if (e == q && b < e) w.soff[q] = rs;
    dropped = warp_sum_u64(dropped);
    kept = warp_sum_u64(kept);
    if ((t & 31) == 0) {
        atomicAdd(&s_drop[0], dropped);
        atomicAdd(&s_drop[1], kept);
    }
    __syncthreads();
    if (t == 0) {
        w.scal[5] = s_drop[0];
        w.scal[6] = s_drop[1];
        w.scal[7] = tot_s;
    }
}

// ------------------------------------------------------------------------------------
// k_lut: LUT[q][g][c][j] = sum_t (C[m][c][t] - x[q][m*pq_len + t])^2, m = 32g + j
// (build_pq_lut_kernel, product-quantization.cu:4-35; the reference's `ans += (c-q)*(c-q)`
// is an FMA under nvcc's default contraction), zero for m >= M.
// ------------------------------------------------------------------------------------
constexpr int kLutQ = 64;          // queries per k_lut block
constexpr int kLutMaxPqLen = 6;    // staged codebook group fits shared memory up to this pq_len

// one LUT entry, FP32 or rounded to FP16 (round to nearest even)
__device__ __forceinline__ void store_lut(float* lut, int f16, uint64_t i, float v) {
    if (f16)
        reinterpret_cast<__half*>(lut)[i] = __float2half_rn(v);
    else
        lut[i] = v;
}

// Block = (64 queries, one group of 32 subspaces, a slice of the codewords).  The slice's codebook
// rows are staged once in shared memory as [c*pq_len + t][33] (conflict-free stores from coalesced
// global reads and conflict-free lane reads); lane = subspace column j, so a warp stores one
// contiguous 128-byte LUT row per codeword.  The warps share out (query, part of the slice) pairs,
// as many parts as it takes to give every warp one.  Bound: the LUT's writes.
// The slice: the largest that still gives four blocks per SM (lut_slices); with the whole codebook
// per block 1,000 queries ran on 16 blocks and one query on one warp.  Sliced, the stage went
// 32 -> 8 us (1 query), 100 -> 27 us (1,000) and 192 -> 131 us (10,000, M = 32).
__global__ void __launch_bounds__(512) k_lut(IndexDev D, const float* __restrict__ queries, uint64_t q, int G,
                                             float* __restrict__ lut, int f16, const uint32_t* __restrict__ item_off) {
    chain_start();
    extern __shared__ float smem_lut[];
    // a block none of whose queries has ADC work stages nothing
    {
        const uint64_t qt = (uint64_t)blockIdx.x * kLutQ + threadIdx.x;
        const bool need = threadIdx.x < kLutQ && qt < q && item_off[qt + 1] != item_off[qt];
        if (!__syncthreads_or(need)) return;
    }
    const int g = blockIdx.y, pq_len = D.pq_len, d = D.d, M = D.M;
    const int nc = kCodes / (int)gridDim.z, c0 = (int)blockIdx.z * nc;  // this slice's codewords
    float* s_cb = smem_lut;                          // [((c - c0) * pq_len + t) * 33 + j]
    const int n1 = nc * pq_len;                      // words per subspace
    const float* src = D.pq_centers + (uint64_t)(32 * g) * kCodes * pq_len + (uint64_t)c0 * pq_len;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int j = warp; j < 32; j += nw) {
        const bool real_j = 32 * g + j < M;
        for (int r = lane; r < n1; r += 32)
            s_cb[r * 33 + j] = real_j ? __ldg(src + (uint64_t)j * kCodes * pq_len + r) : 0.f;
    }
    __syncthreads();
    const int m = 32 * g + lane;
    const bool real = m < M;
    const int nq = (int)min((uint64_t)kLutQ, q - (uint64_t)blockIdx.x * kLutQ);
    int parts = 1;  // parts of the slice per query (a power of two dividing nc)
    while (parts < nc && parts * nq < nw) parts *= 2;
    const int pc = nc / parts;
    for (int u = warp; u < nq * parts; u += nw) {
        const uint64_t qi = (uint64_t)blockIdx.x * kLutQ + u / parts;
        if (item_off[qi + 1] == item_off[qi]) continue;  // no ADC work: no LUT
        // lane j keeps the query's slice of subspace 32g+j in registers
        float qv[kLutMaxPqLen];
#pragma unroll
        for (int t = 0; t < kLutMaxPqLen; t++)
            qv[t] = (real && t < pq_len) ? queries[qi * d + (uint64_t)m * pq_len + t] : 0.f;
        const uint64_t row0 = (qi * G + g) * (kCodes * 32);
        const int cb = u % parts * pc;
        for (int c = cb; c < cb + pc; c++) {
            float s = 0.f;
#pragma unroll
            for (int t = 0; t < kLutMaxPqLen; t++) {
                if (t < pq_len) {
                    const float df = __fsub_rn(s_cb[(c * pq_len + t) * 33 + lane], qv[t]);
                    s = fmaf(df, df, s);
                }
            }
            store_lut(lut, f16, row0 + (uint64_t)(c0 + c) * 32 + lane, real ? s : 0.f);
        }
    }
}

// Codeword slices of k_lut: the fewest (at most 16) that give four blocks per SM
static int lut_slices(uint64_t q, int G, int sms) {
    const uint64_t blocks = (q + kLutQ - 1) / kLutQ * (uint64_t)G;
    int s = 1;
    while (s < 16 && blocks * s < 4ull * sms) s *= 2;
    return s;
}

// Fallback for long subspaces: one query per block, thread = codeword, transposed store.
__global__ void __launch_bounds__(256) k_lut_plain(IndexDev D, const float* __restrict__ queries, int G,
                                                   float* __restrict__ lut, int f16,
                                                   const uint32_t* __restrict__ item_off) {
    chain_start();
    extern __shared__ float s_q[];     // [d]
    __shared__ float s_t[kCodes][33];  // [c][j]
    const uint64_t qi = blockIdx.x;
    if (item_off[qi + 1] == item_off[qi]) return;  // no ADC work: no LUT (block-uniform)
    const int g = blockIdx.y, d = D.d, pq_len = D.pq_len, c = threadIdx.x;
    for (int i = threadIdx.x; i < d; i += blockDim.x) s_q[i] = queries[qi * d + i];
    __syncthreads();
    for (int j = 0; j < 32; j++) {
        const int m = g * 32 + j;
        float s = 0.f;
        if (m < (int)D.M) {
            const float* cw = D.pq_centers + ((uint64_t)m * kCodes + c) * pq_len;
            for (int tt = 0; tt < pq_len; tt++) {
                const float df = __fsub_rn(__ldg(cw + tt), s_q[m * pq_len + tt]);
                s = fmaf(df, df, s);
            }
        }
        s_t[c][j] = s;
    }
    __syncthreads();
    const uint64_t row0 = (qi * G + g) * (kCodes * 32);
    for (int e = threadIdx.x; e < kCodes * 32; e += blockDim.x) store_lut(lut, f16, row0 + e, s_t[e >> 5][e & 31]);
}

// ------------------------------------------------------------------------------------
// k_scan: persistent ADC stream
// ------------------------------------------------------------------------------------
// Shared-memory LUT layout (fast path): for each group g of 32 subspaces a [256][64] f32
// table whose columns 32..63 repeat 0..31.  Lane r rotates its candidate's 32 code bytes of
// the group left by r, so at step s it looks up subspace (r + s) mod 32 at column r + s:
// the 32 lanes of a warp read 32 different banks, the column offset 4*s is an immediate,
// and no wrap-around arithmetic is needed.

// (a0, a1) += (b0, b1) as one packed FP32x2 add (round to nearest, like two FADDs)
__device__ __forceinline__ void add_f32x2(float& a0, float& a1, float b0, float b1) {
    asm("{\n\t.reg .b64 ra, rb;\n\tmov.b64 ra, {%0, %1};\n\tmov.b64 rb, {%2, %3};\n\t"
        "add.rn.f32x2 ra, ra, rb;\n\tmov.b64 {%0, %1}, ra;\n\t}"
        : "+f"(a0), "+f"(a1)
        : "f"(b0), "f"(b1));
}

// rotate 8 words left by R words (out[i] = in[(i + R) & 7]) with selects only
__device__ __forceinline__ void rotate_words(uint32_t (&w)[8], uint32_t R) {
    uint32_t t[8];
#pragma unroll
    for (int i = 0; i < 8; i++) t[i] = (R & 1) ? w[(i + 1) & 7] : w[i];
#pragma unroll
    for (int i = 0; i < 8; i++) w[i] = (R & 2) ? t[(i + 2) & 7] : t[i];
#pragma unroll
    for (int i = 0; i < 8; i++) t[i] = (R & 4) ? w[(i + 4) & 7] : w[i];
#pragma unroll
    for (int i = 0; i < 8; i++) w[i] = t[i];
}

struct ScanShared {
    int item, query;
};

// ADC of one candidate's 32-subspace group g in the fast path's lane-rotated order (the
// same loads, rotation and lookups as the interleaved loop of k_scan_fast)
__device__ __forceinline__ void adc_group1(const uint4* cp, uint64_t n_pts, int g, uint32_t R, uint32_t sh,
                                           uint32_t lane4, const float* s_lut, float& s0, float& s1) {
    const uint4 a = __ldg(cp + (2 * g) * n_pts), b = __ldg(cp + (2 * g + 1) * n_pts);
    uint32_t wv[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    rotate_words(wv, R);
    uint32_t x[8];
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = __funnelshift_r(wv[i], wv[(i + 1) & 7], sh);
    const char* L = reinterpret_cast<const char*>(s_lut + g * (kCodes * 64));
#pragma unroll
    for (int st = 0; st < 32; st += 2) {
        const uint32_t a0 = __byte_perm(x[st >> 2], lane4, 0x5504u | ((st & 3) << 4));
        const uint32_t a1 = __byte_perm(x[st >> 2], lane4, 0x5504u | (((st + 1) & 3) << 4));
        add_f32x2(s0, s1, reinterpret_cast<const float*>(L + a0)[st], reinterpret_cast<const float*>(L + a1)[st + 1]);
    }
}

// Loads the query's range table (prefix of the range lengths and range starts) into shared
// memory.  All threads; ends with a barrier.
__device__ __forceinline__ void scan_load_query(const Workspace& w, int Ps, int qq, uint32_t* s_pre,
                                                uint32_t* s_start) {
    const uint32_t* pre = w.range_pre + (uint64_t)qq * (Ps + 1);
    for (int i = threadIdx.x; i <= Ps; i += blockDim.x) s_pre[i] = pre[i];
    for (int i = threadIdx.x; i < Ps; i += blockDim.x) s_start[i] = w.range_start[(uint64_t)qq * Ps + i];
    __syncthreads();
}

// ------------------------------------------------------------------------------------
// k_pre_scan: the label predicate of the predicate-first queries, ahead of their ADC
// ------------------------------------------------------------------------------------
// A predicate-first query (query_prefilter, prefiltering.cu:36-51; the learned schedule's
// predicate-first flag) keeps only its candidates that pass the label predicate
// (filter.cu:30-64), and only those need an ADC distance.  This pass runs before the ADC scan:
// one warp per work item (pre_chunk consecutive candidate positions of one query), no
// shared-memory LUT.  A lane takes words of 32 pool rows and tests their label ranks by bit planes,
// the two at the ends of every constrained dim's box ANDed:
//   1. against the query's rank box: a rank outside it proves that the label test fails;
//   2. against its inner box: a rank inside proves that the test passes (a survivor);
//   3. only the rows between the two have their labels read, up to 128 per batch from a per-warp
//      queue, so that a batch's label loads are all useful;
//   4. the survivors are staged per warp and appended to the query's row -- the candidate position
//      into spos and the pool row into the distance slot, which the ADC scan then overwrites with
//      the survivor's distance.
// Bound: latency of the plane words (ncu, 161 M candidates of 2,000 queries: issue slots 39 % busy, a third
// of the stalls on loads; DRAM 1.8 B per candidate on 10 M points, 2.7 TB/s).  One packed rank word per
// candidate took 2,505 us for 1.9 G candidates of 10,000 queries (issue and L2 latency), planes with
// the labels of every row inside the outer box 1,305, the inner box as well 1,790 -> 1,263 on 1 G
// candidates of which a third pass; survivors pushed a bit per word and lane, out of row order, cost the
// ADC scan 2,558 against 2,017.  Slower on 10 M points (1,308): the inner box's words of every lane, open
// rows or not (1,398), five blocks per SM with spills (1,438), items of up to 32,768 (1,321).
// The row's order depends on timing; the distance of each survivor does not (the ADC order
// follows its position) and the select orders ties by position.
constexpr int kPreThreads = 256;
// shared words per warp: labels, queue, survivors, ranges, planes
constexpr int kPreRingWords = 4 * 128 + 2 * 256 + 2 * 128 + 4 * 32 + 2 * 4 * kMaxDims;

// Largest i in [0, n) with a[i] <= key (a nondecreasing, a[0] <= key), by 32-way rounds.
// Every lane of the warp calls it and gets the answer.
__device__ __forceinline__ int warp_find_le(const uint32_t* a, int n, uint32_t key) {
    const int lane = threadIdx.x & 31;
    int lo = 0, len = n;
    while (len > 1) {
        const int step = (len + 31) >> 5;
        const int off = lane * step;
        const bool ok = off < len && a[lo + off] <= key;
        const unsigned b = __ballot_sync(0xffffffffu, ok);  // bit 0 set: a[lo] <= key
        const int j = 31 - __clz(b);
        lo += j * step;
        len = min(step, len - j * step);
    }
    return lo;
}

// Per-warp rings in shared memory: word i of entry s at ring[i * size + s], head h and tail t
// warp-uniform and free-running (entries t - h).

// Appends (a, b) of the lanes where f holds at the ring's tail.  All lanes.
template <uint32_t SIZE>
__device__ __forceinline__ void ring_push(uint32_t* ring, uint32_t& t, bool f, uint32_t a, uint32_t b) {
    const unsigned bal = __ballot_sync(0xffffffffu, f);
    if (f) {
        const uint32_t s = (t + __popc(bal & ((1u << (threadIdx.x & 31)) - 1u))) & (SIZE - 1);
        ring[s] = a;
        ring[SIZE + s] = b;
    }
    t += __popc(bal);
}

// Appends the rows of every lane's word m (first row p32, position - row delta; n of them in the
// warp) in row order.  All lanes.
template <uint32_t SIZE>
__device__ __forceinline__ void push_own(uint32_t* ring, uint32_t& t, uint32_t m, uint32_t n, uint32_t p32, uint32_t delta) {
    const int lane = threadIdx.x & 31;
    uint32_t at = __popc(m);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, at, o);
        if (lane >= o) at += y;
    }
    at += t - __popc(m);
    for (; m; m &= m - 1u, at++) {
        const uint32_t p = p32 + (uint32_t)__ffs((int)m) - 1u, s = at & (SIZE - 1);
        ring[s] = p + delta;
        ring[SIZE + s] = p;
    }
    __syncwarp();
    t += n;
}

// 16-byte asynchronous global -> shared copy (cp.async, cached in L2 only) and its groups
__device__ __forceinline__ void cp16_async(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// m (<= 32) entries from a ring's head to the query's row: position into spos, pool row into the
// distance slot.  All lanes.
__device__ __forceinline__ void pre_flush(const uint32_t* ring, uint32_t size, uint32_t h, int m, uint32_t* ctr,
                                          uint32_t* drow, uint32_t* prow) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(ctr, (uint32_t)m);
    at = __shfl_sync(0xffffffffu, at, 0);
    if (lane < m) {
        const uint32_t s = (h + lane) & (size - 1);
        prow[at + lane] = ring[s];
        drow[at + lane] = ring[size + s];
    }
    __syncwarp();
}

// the label predicate (a NaN label passes, as in the reference); bx_s: the query's box in shared memory
__device__ __forceinline__ bool pre_box4(const float* bx_s, const float4& v) {
    const float4 b0 = reinterpret_cast<const float4*>(bx_s)[0], b1 = reinterpret_cast<const float4*>(bx_s)[1];
    return !(v.x < b0.x || v.x > b0.y) && !(v.y < b0.z || v.y > b0.w) && !(v.z < b1.x || v.z > b1.y) &&
           !(v.w < b1.z || v.w > b1.w);
}
template <bool LAB4>
__device__ __forceinline__ bool pre_label_ok(const IndexDev& D, int lbl, const float* bx_s, uint32_t p) {
    if (LAB4) return pre_box4(bx_s, __ldg(reinterpret_cast<const float4*>(D.labels) + p));
    bool ok = true;
    const float* lab = D.labels + (uint64_t)p * lbl;
    for (int i = 0; i < lbl; i++) {
        const float v = __ldg(lab + i);
        if (v < bx_s[2 * i] || v > bx_s[2 * i + 1]) ok = false;
    }
    return ok;
}

// The planes of one rank box: first words p[0 .. n), those from n_hi on to be inverted.
struct PreBox {
    const uint32_t* const* p;
    int n_hi, n;
};
__device__ __forceinline__ uint32_t pre_word(const PreBox& x, uint32_t w) {
    uint32_t m = 0xffffffffu;
    for (int k = 0; k < x.n; k += 4) {
        uint32_t v[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
            v[i] = k + i < x.n ? __ldg(x.p[k + i] + w) ^ (k + i < x.n_hi ? 0u : 0xffffffffu) : 0xffffffffu;
        m &= v[0] & v[1] & v[2] & v[3];
    }
    return m;
}

// One predicate-pass work item by the ranks' bit planes: positions [e0, e1) of one query (R ranges,
// prefix pre, starts start; r0 the range of e0), outer / inner: its rank boxes (has_inner: some rank
// passes for sure).  LAB4: four 16-byte-aligned label dims.  qr: [2][256] ring of candidates whose
// labels decide, sr: [2][128] survivor ring, lst: [128] staged labels (LAB4), rt: [32] ranges.
// n_read: candidates whose labels were read.
template <bool LAB4>
__device__ __forceinline__ void pre_bits(const IndexDev& D, int lbl, const float* bx_s, const PreBox& outer,
                                         const PreBox& inner, bool has_inner, const uint32_t* pre, const uint32_t* start, int R, int r0, uint32_t e0,
                                         uint32_t e1, uint32_t* qr, uint32_t* sr, float4* lst, uint4* rt, uint32_t* ctr,
                                         uint32_t* drow, uint32_t* prow, uint32_t& n_read) {
    constexpr uint32_t QS = 256, SS = 128, LB = 128;
    const int lane = threadIdx.x & 31;
    const float4* lab4 = reinterpret_cast<const float4*>(D.labels);
    uint32_t sh = 0, st = 0;
    auto stage_surv = [&](bool f, uint32_t e, uint32_t p) {
        ring_push<SS>(sr, st, f, e, p);
        if (st - sh >= 32) {
            pre_flush(sr, SS, sh, 32, ctr, drow, prow);
            sh += 32;
        }
    };
    // qr holds [qh, qi) whose labels are on their way into lst, then [qi, qt) queued.  issue() starts
    // a batch's 16-byte label copies (cp.async: no registers held while they fly), consume() tests a
    // batch once its copies have landed.
    uint32_t qh = 0, qi = 0, qt = 0;
    auto issue = [&]() {
        const uint32_t m = qt - qi;  // at most LB
        __syncwarp();                // the pushes of every lane are visible
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint32_t k = lane + 32u * u;
            if (LAB4 && k < m) cp16_async(lst + k, lab4 + qr[QS + ((qi + k) & (QS - 1))]);
        }
        if (LAB4) cp_commit();
        qi = qt;
    };
    auto consume = [&]() {
        const uint32_t m = qi - qh;
        if (LAB4) cp_wait<0>();
        __syncwarp();  // every lane's copies have landed
#pragma unroll 1
        for (uint32_t k0 = 0; k0 < m; k0 += 32) {
            const uint32_t k = k0 + lane;
            const bool v = k < m;
            const uint32_t s = (qh + k) & (QS - 1);
            const uint32_t e = v ? qr[s] : 0u, p = v ? qr[QS + s] : 0u;
            bool ok = false;
            if (v) ok = LAB4 ? pre_box4(bx_s, lst[k]) : pre_label_ok<LAB4>(D, lbl, bx_s, p);
            stage_surv(ok, e, p);
        }
        qh = qi;
        __syncwarp();  // lst and the consumed ring slots are free again
    };
    // Ranges come 32 at a time, the non-empty ones of them as rt[j] = {first word - words before, first
    // row, end row, position - row}; lane j keeps the words before range j (first).  A step is 32 of
    // their words, one per lane.
    int rnext = r0;
    uint32_t first = 0xffffffffu, total = 0, t0 = 0, done = 0;  // done: ranges that begin before word t0
    uint32_t m = 0, p32 = 0, delta = 0;                         // the lane's word: open rows, its first row
    for (bool more = true;;) {
        while (qt - qi <= LB - 64u) {
            // the open rows in row order (so that the survivors' codes are read in order): a lane's own
            // rows one after another while they are few, else word by word with a lane per row
            const uint32_t open = __reduce_add_sync(0xffffffffu, __popc(m));
            if (open > 64) {
                unsigned nz = __ballot_sync(0xffffffffu, m != 0);
                while (nz && qt - qi <= LB - 32u) {
                    const int j = __ffs((int)nz) - 1;
                    const uint32_t mj = __shfl_sync(0xffffffffu, m, j), pj = __shfl_sync(0xffffffffu, p32, j) + lane;
                    const uint32_t dj = __shfl_sync(0xffffffffu, delta, j);
                    if (mj >> lane & 1u) {
                        const uint32_t s = (qt + __popc(mj & ((1u << lane) - 1u))) & (QS - 1);
                        qr[s] = pj + dj;
                        qr[QS + s] = pj;
                    }
                    qt += __popc(mj);
                    if (lane == j) m = 0;
                    nz &= nz - 1;
                }
                continue;
            }
            if (open) {
                push_own<QS>(qr, qt, m, open, p32, delta);
                m = 0;
                continue;
            }
            if (t0 >= total) {
                if (rnext >= R || pre[rnext] >= e1) {
                    more = false;
                    break;
                }
                const int r = rnext + lane;
                uint32_t nw = 0, w0 = 0, p0 = 0, p1 = 0, dl = 0;
                if (r < R) {
                    const uint32_t f = pre[r], a = max(f, e0), b = min(pre[r + 1], e1);
                    if (a < b) {
                        dl = f - start[r];
                        p0 = a - dl;
                        p1 = b - dl;
                        w0 = p0 >> 5;
                        nw = ((p1 - 1u) >> 5) - w0 + 1u;
                    }
                }
                uint32_t inc = nw;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o) inc += y;
                }
                const unsigned some = __ballot_sync(0xffffffffu, nw != 0);
                __syncwarp();  // the last step's reads of rt are done
                if (nw) rt[__popc(some & ((1u << lane) - 1u))] = make_uint4(w0 - (inc - nw), p0, p1, dl);
                total = __shfl_sync(0xffffffffu, inc, 31);
                first = nw ? inc - nw : 0xffffffffu;
                __syncwarp();
                t0 = done = 0;
                rnext += 32;
                if (!total) continue;
            }
            const uint32_t starts = __reduce_or_sync(0xffffffffu, first - t0 < 32u ? 1u << (first - t0) : 0u);
            const uint32_t u = t0 + lane;
            uint32_t sure = 0;
            if (u < total) {
                const uint4 g = rt[done + __popc(starts & (0xffffffffu >> (31 - lane))) - 1u];
                const uint32_t w = g.x + u;
                p32 = w << 5;
                delta = g.w;
                m = 0xffffffffu;
                if (g.y > p32) m <<= g.y - p32;
                if (g.z - p32 < 32u) m &= (1u << (g.z - p32)) - 1u;
                m &= pre_word(outer, w);
                if (has_inner && m) {
                    sure = m & pre_word(inner, w);
                    m &= ~sure;
                }
            }
            const uint32_t n_sure = __reduce_add_sync(0xffffffffu, __popc(sure));
            if (n_sure > 64) {  // straight to the query's row, word by word with a lane per row
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(ctr, n_sure);
                at = __shfl_sync(0xffffffffu, at, 0);
                for (unsigned nz = __ballot_sync(0xffffffffu, sure != 0); nz; nz &= nz - 1) {
                    const int j = __ffs((int)nz) - 1;
                    const uint32_t mj = __shfl_sync(0xffffffffu, sure, j), pj = __shfl_sync(0xffffffffu, p32, j) + lane;
                    const uint32_t dj = __shfl_sync(0xffffffffu, delta, j);
                    if (mj >> lane & 1u) {
                        const uint32_t s = at + __popc(mj & ((1u << lane) - 1u));
                        prow[s] = pj + dj;
                        drow[s] = pj;
                    }
                    at += __popc(mj);
                }
            } else if (n_sure) {
                push_own<SS>(sr, st, sure, n_sure, p32, delta);
                while (st - sh >= 32) {
                    pre_flush(sr, SS, sh, 32, ctr, drow, prow);
                    sh += 32;
                }
            }
            done += __popc(starts);
            t0 += 32;
        }
        if (qi != qh) consume();
        if (qt != qi) issue();
        else if (!more) break;
    }
    n_read += qt;  // every queued candidate had its labels read
    if (st != sh) pre_flush(sr, SS, sh, (int)(st - sh), ctr, drow, prow);
}

// The same position by position, where there are no bit planes: with RANKS (no memory for the planes)
// the packed ranks are tested against the outer and the inner box (rb: rank_box, high words with the
// guard bits gd) before labels are read; without (NaN labels: a NaN passes the label test) every
// candidate's labels are.  qr: [2][256] ring of survivors.  Returns the candidates whose labels were
// read.
template <bool LAB4, bool RANKS>
__device__ __forceinline__ uint32_t pre_labels(const IndexDev& D, int lbl, const float* bx_s, uint4 rb, const uint32_t* pre,
                                               const uint32_t* start, int R, int r0, uint32_t e0, uint32_t e1, uint32_t* qr,
                                               uint32_t* ctr, uint32_t* drow, uint32_t* prow) {
    constexpr int J = 4;  // windows of 32 positions in one step: as many label loads in flight
    constexpr uint32_t QS = 256;
    const int lane = threadIdx.x & 31;
    const float4* lab4 = reinterpret_cast<const float4*>(D.labels);
    // Position -> pool row (warp-uniform state): the current range rc holds positions up to
    // nb1 (pool row = bc + position), the next non-empty range from nb1 up to nb2 (bn).  A window
    // with two or more range starts walks per lane.
    int rc = r0, rn = r0;
    uint32_t nb1 = pre[r0 + 1], bc = start[r0] - pre[r0], nb2 = 0xffffffffu, bn = 0;
    const uint32_t total = pre[R];
    auto find_next = [&]() {  // the first non-empty range after rc (none past the last position)
        int r = nb1 < total ? rc + 1 : R;
        while (r < R && pre[r + 1] == nb1) r++;
        rn = r;
        nb2 = r < R ? pre[r + 1] : 0xffffffffu;
        bn = r < R ? start[r] - nb1 : 0u;
    };
    find_next();
    auto advance_to = [&](uint32_t p) {  // the state at the range of position p
        while (nb1 <= p && nb1 < e1) {
            rc = rn;
            nb1 = nb2;
            bc = bn;
            find_next();
        }
    };
    const uint32_t gd = D.rank_guard;
    uint32_t qh = 0, qt = 0, n_read = 0;
    for (uint32_t eb = e0; eb < e1; eb += 32u * J) {
        uint32_t pp[J];
        bool pv[J];
#pragma unroll
        for (int j = 0; j < J; j++) {
            const uint32_t p = eb + 32u * j, e = p + lane;  // the window [p, p + 32)
            pv[j] = e < e1;
            uint32_t base;
            if (p + 31u < nb2) {
                base = e < nb1 ? bc : bn;
            } else {  // two or more ranges start inside the window
                int r = rc;
                if (pv[j])
                    while (pre[r + 1] <= e) r++;
                base = start[r] - pre[r];
            }
            pp[j] = pv[j] ? base + e : 0u;
            advance_to(p + 32u);
        }
        bool sure[J];  // pass without a look at their labels; pv: the labels decide
#pragma unroll
        for (int j = 0; j < J; j++) sure[j] = false;
        if (RANKS) {
            uint32_t c[J];
#pragma unroll
            for (int j = 0; j < J; j++) c[j] = pv[j] ? __ldg(D.rankpack + pp[j]) : 0u;
#pragma unroll
            for (int j = 0; j < J; j++) {
                // every field at or above its low bound and at or below its high bound: the guard bit
                // above a field survives both subtractions exactly then
                auto inside = [&](uint32_t lo, uint32_t hi) { return ((((c[j] | gd) - lo) & (hi - c[j])) & gd) == gd; };
                sure[j] = pv[j] && inside(rb.z, rb.w);
                pv[j] = pv[j] && !sure[j] && inside(rb.x, rb.y);
            }
        }
#pragma unroll
        for (int j = 0; j < J; j++) n_read += __popc(__ballot_sync(0xffffffffu, pv[j]));
        if (LAB4) {
            float4 v[J];
#pragma unroll
            for (int j = 0; j < J; j++) v[j] = pv[j] ? __ldg(lab4 + pp[j]) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int j = 0; j < J; j++)
                ring_push<QS>(qr, qt, sure[j] || (pv[j] && pre_box4(bx_s, v[j])), eb + 32u * j + lane, pp[j]);
        } else {
#pragma unroll
            for (int j = 0; j < J; j++)
                ring_push<QS>(qr, qt, sure[j] || (pv[j] && pre_label_ok<LAB4>(D, lbl, bx_s, pp[j])), eb + 32u * j + lane,
                              pp[j]);
        }
        while (qt - qh >= 32) {
            pre_flush(qr, QS, qh, 32, ctr, drow, prow);
            qh += 32;
        }
    }
    if (qt != qh) pre_flush(qr, QS, qh, (int)(qt - qh), ctr, drow, prow);
    return n_read;
}

// What a candidate is tested by before its labels: bit planes, packed ranks, nothing.  Kernels of their
// own: the planes' loop is compact in the instruction cache (with the others called out of line beside
// it 5,431 us for the 10 M point batch of the learned schedule, 5,351 so).
enum PreTest { kPlaneTest, kRankTest, kLabelTest };
template <bool LAB4, int TEST>
__global__ void __launch_bounds__(kPreThreads, 4) k_pre_scan(IndexDev D, int R, int lbl, uint64_t q, Workspace w) {
    constexpr int NW = kPreThreads / 32;
    extern __shared__ __align__(16) uint32_t s_rings[];  // per warp: staged labels, ranges, planes, queue ring, survivor ring
    __shared__ __align__(16) float s_bx[NW][2 * kMaxDims];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const uint32_t n_items = w.pitem_off[q], chunk = pre_chunk(w);
    for (;;) {
        __syncwarp();  // the previous item's reads of the warp's tables are done
        uint32_t item = 0;
        if (lane == 0) item = atomicAdd(&w.counter[2], 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= n_items) break;
        const int qq = warp_find_le(w.pitem_off, (int)q, item);
        const uint32_t total = w.qstat[(uint64_t)qq * 4];
        const uint32_t e0 = (item - w.pitem_off[qq]) * chunk;
        if (e0 >= total) continue;  // a query cut by a capacity
        const uint32_t e1 = min(total, e0 + chunk);
        if (lane < 2 * lbl) s_bx[wp][lane] = w.box[(uint64_t)qq * 2 * lbl + lane];
        float4* lst = reinterpret_cast<float4*>(s_rings + (size_t)wp * kPreRingWords);
        uint4* rt = reinterpret_cast<uint4*>(lst + 128);
        const uint32_t** pl = reinterpret_cast<const uint32_t**>(rt + 32);
        uint32_t* qr = reinterpret_cast<uint32_t*>(pl + 4 * kMaxDims);
        uint32_t* sr = qr + 2 * 256;
        // lane i: the planes of dim i's bounds, absent where a bound excludes no (shifted) rank
        auto planes_of = [&](uint32_t a, uint32_t b, const uint32_t** out) {
            bool hi = false, lo = false;
            const uint32_t *ph = nullptr, *plo = nullptr;
            if (lane < lbl) {
                hi = b < D.rank_n[lane] >> D.plane_shift;
                lo = a > 0;
                ph = D.rank_planes + ((uint64_t)D.plane_off[lane] + b) * D.plane_words;
                plo = D.rank_planes + ((uint64_t)D.plane_off[lane] + a - 1u) * D.plane_words;
            }
            const unsigned bh = __ballot_sync(0xffffffffu, hi), bl = __ballot_sync(0xffffffffu, lo);
            const unsigned below = (1u << lane) - 1u;
            const int n_hi = __popc(bh);
            if (hi) out[__popc(bh & below)] = ph;
            if (lo) out[n_hi + __popc(bl & below)] = plo;
            return PreBox{out, n_hi, n_hi + __popc(bl)};
        };
        PreBox outer{}, inner{};
        bool has_inner = false;
        if (TEST == kPlaneTest) {
            const uint32_t sft = D.plane_shift, mask = (1u << D.rank_bits) - 1u;
            const uint32_t off = lane < lbl ? lane * (D.rank_bits + 1) : 0u, top = lane < lbl ? D.rank_n[lane] : 0u;
            auto field = [&](int k) { return (w.rank_box[4 * qq + k] >> off) & mask; };
            outer = planes_of(field(0) >> sft, field(1) >> sft, pl);
            // the inner box in shifted ranks: those whose every rank lies in it
            const uint32_t il = field(2), ih = field(3), a = (il + (1u << sft) - 1u) >> sft;
            const uint32_t b1 = ih >= top ? (top >> sft) + 1u : (ih + 1u) >> sft;  // one past the last
            has_inner = __all_sync(0xffffffffu, lane >= lbl || (il <= ih && a < b1));
            if (has_inner) inner = planes_of(a, b1 - 1u, pl + 2 * kMaxDims);
        }
        __syncwarp();  // s_bx and pl are written
        const uint32_t* pre = w.range_pre + (uint64_t)qq * (R + 1);
        const uint32_t* start = w.range_start + (uint64_t)qq * R;
        const int r0 = warp_find_le(pre, R, e0);
        uint32_t* ctr = &w.cand_count[qq];
        uint32_t* drow = reinterpret_cast<uint32_t*>(w.dist + w.qoff[qq]);
        uint32_t* prow = w.spos + w.qoff[qq];
        uint32_t n_read = 0, n_chk = 0;
        const float* bxs = s_bx[wp];
        if constexpr (TEST == kPlaneTest) {
            pre_bits<LAB4>(D, lbl, bxs, outer, inner, has_inner, pre, start, R, r0, e0, e1, qr, sr, lst, rt, ctr, drow, prow, n_read);
        } else {
            const uint4 rb = make_uint4(w.rank_box[4 * qq], w.rank_box[4 * qq + 1], w.rank_box[4 * qq + 2], w.rank_box[4 * qq + 3]);
            n_read = pre_labels<LAB4, TEST == kRankTest>(D, lbl, bxs, rb, pre, start, R, r0, e0, e1, qr, ctr, drow, prow);
        }
        if (TEST != kLabelTest) n_chk = e1 - e0;
        if (lane == 0 && n_read) atomicAdd(&w.lab_read[qq], n_read);
        if (lane == 0 && n_chk) atomicAdd(&w.rank_read[qq], n_chk);
    }
}

// ADC work items once the predicate pass has listed the survivors: a compact row has
// cand_count entries, any other row one per candidate position.  One block.
__global__ void __launch_bounds__(1024) k_scan_plan(uint64_t q, Workspace w) {
    __shared__ unsigned long long s_w[32];
    const int t = threadIdx.x;
    const uint64_t per = (q + blockDim.x - 1) / blockDim.x;
    const uint64_t b = t * per, e = min(q, b + per);
    const uint32_t chunk = scan_chunk(w);
    auto n_items = [&](uint64_t i) {
        uint32_t c = compacts(w, i) || pruned(w, i) ? w.cand_count[i] : w.qstat[i * 4];
        // a compact row that its budget takes whole needs no ADC distance (the select takes
        // every survivor and the re-rank orders them), unless the distances are the output
        // (the reference's pre-filter schedule)
        if (compacts(w, i) && w.mode != kPre && c <= w.qbud[i]) c = 0;
        return (c + chunk - 1) / chunk;
    };
    // such a row's survivors all count as passed (the ADC scan counts them for the others)
    for (uint64_t i = b; i < e; i++)
        if (compacts(w, i) && w.mode != kPre && w.cand_count[i] <= w.qbud[i]) w.nfin[i] = w.cand_count[i];
    unsigned long long items = 0;
    for (uint64_t i = b; i < e; i++) items += n_items(i);
    unsigned long long tot = 0;
    unsigned long long r = block_inclusive_sum(items, s_w, &tot) - items;
    for (uint64_t i = b; i < e; i++) {
        w.item_off[i] = (uint32_t)r;
        r += n_items(i);
    }
    if (e == q && b < e) w.item_off[q] = (uint32_t)r;
    if (t == 0) w.counter[0] = 0;
}

// Fast path (M a multiple of 32).  The CTA computes the query's LUT straight into shared
// memory when it switches query (codeword-major loads, one subspace per lane), then streams
// candidates; CPT candidates per thread are interleaved step by step so every thread keeps
// CPT independent load->add chains in flight.  A candidate at position e sums from subspace
// (e mod 32) of each group: for a full row that is the lane, for a compact row (the predicate
// pass's survivors) it comes from the survivor's recorded position.
template <int G, int NT, int CPT>
__global__ void __launch_bounds__(NT, (G == 1 && CPT == 1) ? 2 : 1) k_scan_fast(IndexDev D, int Ps, uint64_t q,
                                                                                 Workspace w) {
    chain_start();
    extern __shared__ __align__(16) float s_lut[];  // [G][256][64]
    uint32_t* s_pre = reinterpret_cast<uint32_t*>(s_lut + G * kCodes * 64);  // [Ps + 1]
    uint32_t* s_start = s_pre + Ps + 1;                                       // [Ps]
    __shared__ ScanShared s;
    const int t = threadIdx.x, lane = t & 31;
    const uint32_t n_items = w.item_off[q], chunk = scan_chunk(w);
    int cur = -1;
    for (;;) {
        if (t < 32) {  // the item's query: the last one with item_off <= item, by 32-way rounds
            int item = 0;
            if (t == 0) item = (int)atomicAdd(w.counter, 1u);
            item = __shfl_sync(0xffffffffu, item, 0);
            const int qf = item < (int)n_items ? warp_find_le(w.item_off, (int)q, (uint32_t)item) : 0;
            if (t == 0) {
                s.item = item;
                s.query = qf;
            }
        }
        __syncthreads();
        const int item = s.item;
        if (item >= (int)n_items) break;
        const int qq = s.query;
        const bool compact = compacts(w, qq) || pruned(w, qq);
        const uint32_t total = compact ? w.cand_count[qq] : w.qstat[(uint64_t)qq * 4];
        const uint32_t e0 = (uint32_t)(item - w.item_off[qq]) * chunk;
        if (e0 >= total) {  // a query cut by the distance capacity
            __syncthreads();
            continue;
        }
        if (qq != cur) {
            if (w.lut16) {  // FP16 entries widened to FP32 in shared memory
                const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const __half*>(w.lut) +
                                                                  (uint64_t)qq * G * kCodes * 32);
                for (int e = t; e < G * kCodes * 4; e += NT) {
                    const uint4 v = __ldg(src + e);
                    const int row = e >> 2, col = (e & 3) * 8;
                    const __half2* h = reinterpret_cast<const __half2*>(&v);
                    const float2 f0 = __half22float2(h[0]), f1 = __half22float2(h[1]);
                    const float2 f2 = __half22float2(h[2]), f3 = __half22float2(h[3]);
                    float4* dstl = reinterpret_cast<float4*>(s_lut + row * 64 + col);
                    dstl[0] = make_float4(f0.x, f0.y, f1.x, f1.y);
                    dstl[1] = make_float4(f2.x, f2.y, f3.x, f3.y);
                    dstl[8] = dstl[0];
                    dstl[9] = dstl[1];
                }
            } else {
                const float4* src = reinterpret_cast<const float4*>(w.lut + (uint64_t)qq * G * kCodes * 32);
                for (int e = t; e < G * kCodes * 8; e += NT) {
                    const float4 v = __ldg(src + e);
                    const int row = e >> 3, col = (e & 7) * 4;  // row = g*256 + c
                    float4* dstl = reinterpret_cast<float4*>(s_lut + row * 64 + col);
                    dstl[0] = v;
                    dstl[8] = v;  // columns 32..63 repeat 0..31
                }
            }
            // a query's rows are all compact or all full: a compact query needs no range table
            if (!compact) scan_load_query(w, Ps, qq, s_pre, s_start);  // ends with a barrier
            else __syncthreads();
            cur = qq;
        }
        const uint32_t e1 = min(total, e0 + chunk);
        float* dst = w.dist + row_of(w, qq);
        const uint32_t* srow = reinterpret_cast<const uint32_t*>(dst);  // compact: the survivors' pool rows
        const uint32_t* sp = w.spos + row_of(w, qq);
        uint32_t kmin = 0xffffffffu, kmax = 0u, nf = 0;
        // each warp takes a contiguous span of the item (a multiple of 32 * CPT entries, so in
        // a full row position mod 32 stays the lane), so a lane's walk to its candidate's range
        // crosses few range boundaries per step
        constexpr uint32_t kStep = 32u * CPT;
        const uint32_t span = ((e1 - e0 + NT / 32 - 1) / (NT / 32) + kStep - 1) / kStep * kStep;
        const uint32_t wb = e0 + (uint32_t)(t >> 5) * span;
        const uint32_t we = min(e1, wb + span);
        int r[CPT];
#pragma unroll
        for (int u = 0; u < CPT; u++) {
            r[u] = 0;
            if (compact) continue;
            const uint32_t e = wb + lane + u * 32;
            int lo = 0, hi = Ps - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (s_pre[mid] <= e) lo = mid;
                else hi = mid - 1;
            }
            r[u] = lo;
        }
        const uint4* planes = reinterpret_cast<const uint4*>(D.codes);
        const uint64_t n_pts = D.n;
        for (uint32_t eb = wb + lane; eb < we; eb += kStep) {
            const uint4* cp[CPT];
            bool live[CPT];
            uint32_t rot[CPT];
            float sum[CPT], sum1[CPT];  // even / odd steps, added at the end
#pragma unroll
            for (int u = 0; u < CPT; u++) {
                const uint32_t e = eb + u * 32;
                live[u] = e < we;
                sum[u] = sum1[u] = 0.f;
                uint32_t row = 0;  // a dead lane reads row 0 (in bounds), result discarded
                rot[u] = (uint32_t)lane;
                if (live[u]) {
                    if (compact) {
                        row = srow[e];
                        rot[u] = sp[e] & 31u;
                    } else {
                        while (s_pre[r[u] + 1] <= e) r[u]++;
                        row = s_start[r[u]] + (e - s_pre[r[u]]);
                    }
                }
                cp[u] = planes + row;  // chunk j of this point at cp[u][j * n_pts]
            }
#pragma unroll
            for (int g = 0; g < G; g++) {
                uint32_t x[CPT][8];
#pragma unroll
                for (int u = 0; u < CPT; u++) {
                    const uint4 a = __ldg(cp[u] + (2 * g) * n_pts), b = __ldg(cp[u] + (2 * g + 1) * n_pts);
                    uint32_t wv[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                    rotate_words(wv, rot[u] >> 2);
                    const uint32_t sh = 8u * (rot[u] & 3u);
#pragma unroll
                    for (int i = 0; i < 8; i++) x[u][i] = __funnelshift_r(wv[i], wv[(i + 1) & 7], sh);
                }
                const char* L = reinterpret_cast<const char*>(s_lut + g * (kCodes * 64));
#pragma unroll
                for (int st = 0; st < 32; st += 2) {
#pragma unroll
                    for (int u = 0; u < CPT; u++) {
                        // one PRMT builds the byte offset c*256 + rot*4 (code byte -> byte 1,
                        // the column byte -> byte 0); the step's column is the immediate
                        const uint32_t c4 = 4u * rot[u];
                        const uint32_t a0 = __byte_perm(x[u][st >> 2], c4, 0x5504u | ((st & 3) << 4));
                        const uint32_t a1 = __byte_perm(x[u][st >> 2], c4, 0x5504u | (((st + 1) & 3) << 4));
                        add_f32x2(sum[u], sum1[u], reinterpret_cast<const float*>(L + a0)[st],
                                  reinterpret_cast<const float*>(L + a1)[st + 1]);
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < CPT; u++) {
                sum[u] += sum1[u];
                if (!live[u]) continue;
                const uint32_t e = eb + u * 32;
                if (sum[u] < INFINITY) {
                    const uint32_t key = float_key(sum[u]);
                    kmin = min(kmin, key);
                    kmax = max(kmax, key);
                    nf++;
                }
                dst[e] = sum[u];
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            kmin = min(kmin, __shfl_xor_sync(0xffffffffu, kmin, o));
            kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
            nf += __shfl_xor_sync(0xffffffffu, nf, o);
        }
        if (lane == 0 && nf) {
            atomicMin(&w.mm[2 * qq], kmin);
            atomicMax(&w.mm[2 * qq + 1], kmax);
            atomicAdd(&w.nfin[qq], nf);
        }
        __syncthreads();
    }
}
// Generic ADC (any M): natural subspace order.  The LUT sits in shared memory by subspace, entry c
// of subspace m at m * 256 + (c ^ (m & 31)): the lanes of a warp read one subspace at a time, and
// their codes spread over the banks (codeword-major rows put every lane on the subspace's one
// bank); the XOR keeps the staging writes free of conflicts.  Each warp takes a contiguous span of
// the item and walks the ranges.  2.7 M candidates x 25 subspaces: 125 -> 66 us.
__global__ void __launch_bounds__(512) k_scan_generic(IndexDev D, int G, int Ps, int pre, int lbl, uint64_t q,
                                                      Workspace w) {
    chain_start();
    extern __shared__ __align__(16) float s_lut[];  // [32 G][256], swizzled
    uint32_t* s_pre = reinterpret_cast<uint32_t*>(s_lut + G * kCodes * 32);
    uint32_t* s_start = s_pre + Ps + 1;
    __shared__ ScanShared s;
    __shared__ float s_box[2 * kMaxDims];
    const int t = threadIdx.x, lane = t & 31;
    const uint32_t n_items = w.item_off[q], chunk = scan_chunk(w);
    const int M = D.M;
    // shared-memory place of entry e of the global LUT ([G][256][32])
    auto lut_at = [](int e) {
        const int m = (e >> 13) * 32 + (e & 31), c = (e >> 5) & (kCodes - 1);
        return m * kCodes + (c ^ (m & 31));
    };
    int cur = -1;
    for (;;) {
        if (t < 32) {  // the item's query: the last one with item_off <= item, by 32-way rounds
            int item = 0;
            if (t == 0) item = (int)atomicAdd(w.counter, 1u);
            item = __shfl_sync(0xffffffffu, item, 0);
            const int qf = item < (int)n_items ? warp_find_le(w.item_off, (int)q, (uint32_t)item) : 0;
            if (t == 0) {
                s.item = item;
                s.query = qf;
            }
        }
        __syncthreads();
        const int item = s.item;
        if (item >= (int)n_items) break;
        const int qq = s.query;
        const uint32_t total = w.qstat[(uint64_t)qq * 4];
        const uint32_t e0 = (uint32_t)(item - w.item_off[qq]) * chunk;
        if (e0 >= total) {  // a query cut by the distance capacity
            __syncthreads();
            continue;
        }
        if (qq != cur) {
            const uint64_t src0 = (uint64_t)qq * G * kCodes * 32;
            if (w.lut16) {
                const __half* src = reinterpret_cast<const __half*>(w.lut) + src0;
                for (int e = t; e < G * kCodes * 32; e += blockDim.x) s_lut[lut_at(e)] = __half2float(src[e]);
            } else {
                const float* src = w.lut + src0;
                for (int e = t; e < G * kCodes * 32; e += blockDim.x) s_lut[lut_at(e)] = src[e];
            }
            if (t < 2 * lbl) s_box[t] = w.box[(uint64_t)qq * 2 * lbl + t];
            scan_load_query(w, Ps, qq, s_pre, s_start);  // ends with a barrier
            cur = qq;
        }
        const uint32_t e1 = min(total, e0 + chunk);
        float* dst = w.dist + w.qoff[qq];
        const bool preq = pre || q_prefilter(w, qq);
        uint32_t kmin = 0xffffffffu, kmax = 0u, nf = 0;
        const uint32_t nw = blockDim.x >> 5, span = ((e1 - e0 + nw - 1) / nw + 31) / 32 * 32;
        const uint32_t wb = e0 + (uint32_t)(t >> 5) * span, we = min(e1, wb + span);
        int rg = 0;
        {
            int hi = Ps - 1;
            while (rg < hi) {
                const int mid = (rg + hi + 1) >> 1;
                if (s_pre[mid] <= wb + lane) rg = mid;
                else hi = mid - 1;
            }
        }
        for (uint32_t e = wb + lane; e < we; e += 32) {
            while (s_pre[rg + 1] <= e) rg++;
            const uint32_t pool = s_start[rg] + (e - s_pre[rg]);
            bool pass = true;
            if (preq) {
                const float* lab = D.labels + (uint64_t)pool * lbl;
                for (int i = 0; i < lbl; i++) {
                    const float v = lab[i];
                    if (v < s_box[2 * i] || v > s_box[2 * i + 1]) pass = false;
                }
            }
            float sum = INFINITY;
            if (pass) {
                sum = 0.f;
                const uint4* cp = reinterpret_cast<const uint4*>(D.codes) + pool;
                for (int j = 0; j * 16 < M; j++) {
                    const uint4 v = __ldg(cp + (uint64_t)j * D.n);
                    const uint32_t wv[4] = {v.x, v.y, v.z, v.w};
                    const int nb = M - 16 * j;
                    float x[16];
#pragma unroll
                    for (int b = 0; b < 16; b++) {
                        const int m = j * 16 + b;
                        const uint32_t c = (wv[b >> 2] >> (8 * (b & 3))) & 0xffu;
                        x[b] = b < nb ? s_lut[m * kCodes + (int)(c ^ (uint32_t)(m & 31))] : 0.f;
                    }
#pragma unroll
                    for (int b = 0; b < 16; b++)
                        if (b < nb) sum += x[b];
                }
                const uint32_t key = float_key(sum);
                kmin = min(kmin, key);
                kmax = max(kmax, key);
                nf++;
            }
            dst[e] = sum;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            kmin = min(kmin, __shfl_xor_sync(0xffffffffu, kmin, o));
            kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
            nf += __shfl_xor_sync(0xffffffffu, nf, o);
        }
        if (lane == 0 && nf) {
            atomicMin(&w.mm[2 * qq], kmin);
            atomicMax(&w.mm[2 * qq + 1], kmax);
            atomicAdd(&w.nfin[qq], nf);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------
// k_select: the K smallest (distance, position) pairs of one query
// ------------------------------------------------------------------------------------
// Pass 1 histograms the finite distances over kBins linear bins between the query's
// min and max; pass 2 emits every candidate below the bin that holds the K-th and gathers
// that boundary bin, which is sorted by (distance key, position).  A boundary bin larger
// than kBCap is split again over its own min/max (at most kMaxLevels levels); a bin whose
// entries all share one distance is resolved by position order.
constexpr int kMaxLevels = 4;
// 512 threads and four loads in flight each; fewer queries than SMs (one block each) take 1,024
// threads and eight loads (37 queries of 73,000 candidates: 88 -> 51 us)
constexpr int kSelThreads = 512, kSelThreadsFew = 1024;

struct SelLevel {
    float lo, inv;
    int bin;
};

__device__ __forceinline__ int sel_bin(float d, float lo, float inv) {
    const int b = (int)__fmul_rn(__fsub_rn(d, lo), inv);
    return b < 0 ? 0 : (b >= kBins ? kBins - 1 : b);
}

__device__ __forceinline__ uint32_t pos_to_pool(const uint32_t* s_pre, const uint32_t* s_start, int Ps,
                                                uint32_t e) {
    int lo = 0, hi = Ps - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (s_pre[mid] <= e) lo = mid;
        else hi = mid - 1;
    }
    return s_start[lo] + (e - s_pre[lo]);
}

template <int NT, int U>
__global__ void __launch_bounds__(NT) k_select(IndexDev D, int Ps, int Kcap, int sorted_out, Workspace w,
                                                        float* __restrict__ out_dist,
                                                        uint64_t* __restrict__ out_ids, int k_out) {
    chain_start();
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t* s_hist = reinterpret_cast<uint32_t*>(smem);                   // [kBins]
    uint64_t* s_bbuf = reinterpret_cast<uint64_t*>(s_hist + kBins);         // [kBCap]
    uint64_t* s_sel = s_bbuf + kBCap;                                        // [sel_cap] (sorted mode)
    const int sel_cap = sorted_out ? (int)next_pow2_dev((uint32_t)max(Kcap, 2)) : 0;
    // this query's budget: its k for the sorted pre-filter output, else the candidate budget
    const int K = (sorted_out ? (int)q_k(w, blockIdx.x) : (int)q_budget(w, blockIdx.x)) -
                  (pruned(w, blockIdx.x) ? (int)w.est_in[blockIdx.x] : 0);
    uint32_t* s_pre = reinterpret_cast<uint32_t*>(s_sel + sel_cap);        // [Ps + 1]
    uint32_t* s_start = s_pre + Ps + 1;                                      // [Ps]
    __shared__ uint32_t s_warp[32];
    __shared__ SelLevel s_lv[kMaxLevels];
    __shared__ int s_bin;
    __shared__ uint32_t s_below, s_cntb, s_out, s_nb, s_bmin, s_bmax, s_need;
    const uint64_t qi = blockIdx.x;
    const int t = threadIdx.x;
    // A predicate-first query of the predicate pass has a compact row: its survivors' distances
    // in arrival order with their candidate positions beside them (cand_count entries); any
    // other query's row holds one distance per candidate position.
    // A query of the estimate pass has a compact row too: the candidates that its estimates leave
    // open; the sure ones are selected already.
    const bool prn = pruned(w, qi), compact = compacts(w, qi) || prn;
    const uint32_t sure = prn ? w.est_in[qi] : 0u;
    if (!sorted_out && takes_row(w, qi)) return;  // the selection is the row (cand_count entries)
    const uint32_t total = compact ? w.cand_count[qi] : w.qstat[qi * 4];
    const float* dist = w.dist + row_of(w, qi);
    const uint32_t* prow = compact ? w.spos + row_of(w, qi) : nullptr;
    {
        const uint32_t* rpre = w.range_pre + qi * (Ps + 1);
        for (int i = t; i <= Ps; i += blockDim.x) s_pre[i] = rpre[i];
        for (int i = t; i < Ps; i += blockDim.x) s_start[i] = w.range_start[qi * Ps + i];
    }
    if (t == 0) s_out = 0;
    __syncthreads();
    const uint32_t nfin = w.nfin[qi];
    const uint32_t need0 = min((uint32_t)K, nfin);
    uint32_t* sel_dst = sorted_out ? nullptr : w.cand_pool + w.soff[qi] + sure;
    // candidate position of row entry e (e < total)
    auto posof = [&](uint32_t e) { return prow ? prow[e] : e; };
    // Selected entries are recorded by candidate position; positions become pool slots once the
    // selection is complete, in one divergence-free loop over the K entries (converting at
    // emit time made nearly every warp of the pass run the range search for one lane).  Ties in
    // distance are broken by the lower position.
    auto emit = [&](uint32_t pos, float d) {
        const uint32_t at = atomicAdd(&s_out, 1u);
        if (sorted_out)
            s_sel[at] = ((uint64_t)float_key(d) << 32) | pos;
        else
            sel_dst[at] = pos;
    };
    auto inside = [&](float d, int nlv) {
        for (int l = 0; l < nlv; l++)
            if (sel_bin(d, s_lv[l].lo, s_lv[l].inv) != s_lv[l].bin) return false;
        return true;
    };
    // First bin of s_hist whose cumulative count reaches need: s_bin (-1: none), s_below (count
    // before it) and s_cntb (its count).  Warp 0 scans 128 bins per step (one 16-byte read per
    // lane) and stops at the bin; the caller synchronises.  (32 bins per step took up to 4 us; a
    // scan by the whole block costs its barriers at every level and reads every bin.)
    auto find_bin = [&](uint32_t need) {
        if (t < 32) {
            uint32_t run = 0;
            bool found = false;
            for (int base = 0; base < kBins && !found; base += 128) {
                const uint4 v = reinterpret_cast<const uint4*>(s_hist + base)[t];
                const uint32_t sum = v.x + v.y + v.z + v.w;
                uint32_t x = sum;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                    if (t >= o) x += y;
                }
                const unsigned hit = __ballot_sync(0xffffffffu, run + x >= need);
                if (hit) {
                    found = true;
                    if (t == __ffs(hit) - 1) {
                        const uint32_t c[4] = {v.x, v.y, v.z, v.w};
                        uint32_t below = run + x - sum;
                        int i = 0;
                        while (i < 3 && below + c[i] < need) below += c[i++];
                        s_bin = base + 4 * t + i;
                        s_below = below;
                        s_cntb = c[i];
                    }
                }
                run += __shfl_sync(0xffffffffu, x, 31);
            }
            if (t == 0 && !found) {
                s_bin = -1;
                s_below = 0;
                s_cntb = 0;
            }
        }
    };
    if (need0 > 0 && nfin <= (uint32_t)K) {
        // every finite candidate is selected (the loop bound is block-uniform so that every
        // lane reaches the warp appends)
        for (uint32_t base = 0; base < total; base += blockDim.x) {
            const uint32_t e = base + t;
            const float d = e < total ? dist[e] : INFINITY;
            const bool f = d < INFINITY;
            const uint32_t p = f ? posof(e) : 0u;
            if (sorted_out) {
                if (f) emit(p, d);
            } else {
                warp_append(f, p, &s_out, sel_dst);
            }
        }
        __syncthreads();
    } else if (need0 > 0) {
        float lo = key_float(w.mm[2 * qi]), hi = key_float(w.mm[2 * qi + 1]);
        uint32_t need = need0;
        for (int level = 0; level < kMaxLevels; level++) {
            const float inv = hi > lo ? (float)kBins / (hi - lo) : 0.f;
            for (int i = t; i < kBins; i += blockDim.x) s_hist[i] = 0;
            if (t == 0) {
                s_bmin = 0xffffffffu;
                s_bmax = 0u;
                s_nb = 0;
            }
            __syncthreads();
            for (uint32_t e0 = t; e0 < total; e0 += U * blockDim.x) {
                float dv[U];
#pragma unroll
                for (int u = 0; u < U; u++) {  // U independent loads in flight per thread
                    const uint32_t e = e0 + u * blockDim.x;
                    dv[u] = e < total ? __ldg(dist + e) : INFINITY;
                }
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (dv[u] < INFINITY && inside(dv[u], level)) atomicAdd(&s_hist[sel_bin(dv[u], lo, inv)], 1u);
            }
            __syncthreads();
            find_bin(need);
            __syncthreads();
            const int b = s_bin;
            const bool fits = s_cntb <= (uint32_t)kBCap;
            for (uint32_t e0 = 0; e0 < total; e0 += U * blockDim.x) {  // block-uniform bound
                float dv[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const uint32_t e = e0 + t + u * blockDim.x;
                    dv[u] = e < total ? __ldg(dist + e) : INFINITY;
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const float d = dv[u];
                    const uint32_t e = e0 + t + u * blockDim.x;
                    const bool in = d < INFINITY && inside(d, level);
                    const int bb = in ? sel_bin(d, lo, inv) : kBins;
                    const uint32_t p = bb <= b ? posof(e) : 0u;
                    if (!sorted_out) warp_append(bb < b, p, &s_out, sel_dst);
                    if (!in) continue;
                    if (bb < b) {
                        if (sorted_out) emit(p, d);
                    } else if (bb == b) {
                        if (fits) {
                            const uint32_t at = atomicAdd(&s_nb, 1u);
                            s_bbuf[at] = ((uint64_t)float_key(d) << 32) | p;
                        } else {
                            atomicMin(&s_bmin, float_key(d));
                            atomicMax(&s_bmax, float_key(d));
                        }
                    }
                }
            }
            __syncthreads();
            need -= s_below;
            if (fits) {
                // the boundary bin, sorted by (distance, position)
                const int nb = (int)s_nb;
                const int n2 = (int)next_pow2_dev((uint32_t)max(nb, 2));
                for (int i = nb + t; i < n2; i += blockDim.x) s_bbuf[i] = ~0ull;
                __syncthreads();
                block_bitonic_sort(s_bbuf, n2);
                for (uint32_t i = t; i < need; i += blockDim.x) {
                    const uint64_t key = s_bbuf[i];
                    emit((uint32_t)key, key_float((uint32_t)(key >> 32)));
                }
                __syncthreads();
                break;
            }
            if (s_bmin == s_bmax || level == kMaxLevels - 1) {
                // one distance value (or no levels left): the boundary bin's entries (of that
                // one distance) are taken in position order
                const uint32_t tie_key = s_bmin;
                const bool one = s_bmin == s_bmax;
                const int nlv = level;
                auto tie = [&](float d) {
                    return d < INFINITY && inside(d, nlv) && sel_bin(d, lo, inv) == b && (!one || float_key(d) == tie_key);
                };
                if (t == 0) s_need = need;
                __syncthreads();
                if (!compact) {
                    // row order is position order: the first s_need tie entries of the row
                    for (uint32_t base = 0; base < total && s_need > 0; base += blockDim.x) {
                        const uint32_t e = base + t;
                        bool f = false;
                        float d = 0.f;
                        if (e < total) {
                            d = dist[e];
                            f = tie(d);
                        }
                        const unsigned bal = __ballot_sync(0xffffffffu, f);
                        if ((t & 31) == 0) s_warp[t >> 5] = __popc(bal);
                        __syncthreads();
                        uint32_t before = 0;
                        for (int i = 0; i < (t >> 5); i++) before += s_warp[i];
                        const uint32_t rank = before + __popc(bal & ((1u << (t & 31)) - 1));
                        if (f && rank < s_need) emit(e, d);
                        __syncthreads();
                        if (t == 0) {
                            uint32_t tot = 0;
                            for (int i = 0; i < (int)(blockDim.x >> 5); i++) tot += s_warp[i];
                            s_need = s_need > tot ? s_need - tot : 0;
                        }
                        __syncthreads();
                    }
                } else {
                    // a compact row is in arrival order: the s_need smallest positions among
                    // the tie entries, by a radix select over positions (kBins bins per level;
                    // positions are unique, so a one-position bin holds one entry)
                    uint32_t plo = 0, phi = w.qstat[qi * 4];
                    for (;;) {
                        const uint32_t binw = max(1u, (phi - plo + kBins - 1) / kBins);
                        for (int i = t; i < kBins; i += blockDim.x) s_hist[i] = 0;
                        __syncthreads();
                        for (uint32_t e = t; e < total; e += blockDim.x) {
                            const float d = dist[e];
                            const uint32_t p = prow[e];
                            if (tie(d) && p >= plo && p < phi) atomicAdd(&s_hist[(p - plo) / binw], 1u);
                        }
                        __syncthreads();
                        find_bin(s_need);
                        __syncthreads();
                        const int pb = s_bin;
                        const bool last = binw == 1;
                        for (uint32_t e = t; e < total; e += blockDim.x) {
                            const float d = dist[e];
                            const uint32_t p = prow[e];
                            if (!tie(d) || p < plo || p >= phi) continue;
                            const int bin = (int)((p - plo) / binw);
                            if (bin < pb || (last && bin == pb)) emit(p, d);
                        }
                        __syncthreads();
                        if (last || pb < 0) break;
                        if (t == 0) s_need -= s_below;
                        plo += (uint32_t)pb * binw;
                        phi = min(phi, plo + binw);
                        __syncthreads();
                    }
                }
                break;
            }
            if (t == 0) {
                s_lv[level].lo = lo;
                s_lv[level].inv = inv;
                s_lv[level].bin = b;
            }
            lo = key_float(s_bmin);
            hi = key_float(s_bmax);
            __syncthreads();
        }
    }
    __syncthreads();
    const uint32_t nsel = s_out;
    if (!sorted_out) {
        for (uint32_t i = t; i < nsel; i += blockDim.x) sel_dst[i] = pos_to_pool(s_pre, s_start, Ps, sel_dst[i]);
        if (t == 0) w.cand_count[qi] = sure + nsel;
        return;
    }
    const int n2 = (int)next_pow2_dev((uint32_t)max((int)nsel, 2));
    for (int i = nsel + t; i < n2; i += blockDim.x) s_sel[i] = ~0ull;
    __syncthreads();
    block_bitonic_sort(s_sel, n2);
    for (int i = t; i < k_out; i += blockDim.x) {
        if (i < (int)nsel) {
            const uint64_t key = s_sel[i];
            out_dist[qi * k_out + i] = key_float((uint32_t)(key >> 32));
            out_ids[qi * k_out + i] = D.ids[pos_to_pool(s_pre, s_start, Ps, (uint32_t)key)];
        } else {
            out_dist[qi * k_out + i] = INFINITY;
            out_ids[qi * k_out + i] = ~0ull;
        }
    }
}

// ------------------------------------------------------------------------------------
// k_refine: post-filter predicate, exact f32 L2, top-k
// ------------------------------------------------------------------------------------
// A query's selection (min(n_cand, candidates) entries, which the reference's uncapped
// budget can put in the hundreds of thousands) is cut into work items of kRefChunk entries;
// k_refine_plan lays them out and a persistent k_refine takes them from a counter.  An item
// compacts its predicate survivors, computes their exact distances and keeps its best k;
// a query with one item writes its output row directly, otherwise every item leaves its
// best k in the partial buffer and the last item of the query to finish merges them.
constexpr uint32_t kRefChunk = 4096;


__global__ void __launch_bounds__(1024) k_refine_plan(uint64_t q, Workspace w) {
    chain_start();
    __shared__ unsigned long long s_w[32];
    const int t = threadIdx.x;
    const uint64_t per = (q + blockDim.x - 1) / blockDim.x;
    const uint64_t b = t * per, e = min(q, b + per);
    unsigned long long items = 0;
    for (uint64_t i = b; i < e; i++) items += max(1u, (w.cand_count[i] + kRefChunk - 1) / kRefChunk);
    unsigned long long tot = 0;
    unsigned long long r = block_inclusive_sum(items, s_w, &tot) - items;
    for (uint64_t i = b; i < e; i++) {
        w.ritem_off[i] = (uint32_t)r;
        r += max(1u, (w.cand_count[i] + kRefChunk - 1) / kRefChunk);
        w.rdone[i] = 0;
        w.rsurv[i] = 0;
        w.rlab[i] = 0;
    }
    if (e == q && b < e) w.ritem_off[q] = (uint32_t)r;
    if (t == 0) w.counter[1] = 0;
}

// Scratch of the re-rank's selections (shared memory)
struct RefSel {
    uint32_t* hist;            // [256]
    uint32_t* wc;              // [32]
    unsigned long long* sel;   // [4]
};

// Keeps the kq smallest of the c keys in s_keys (c > kq) in s_keys[0, kq), in no order, and
// returns the kq-th smallest; the rest of [0, c) becomes ~0.  All threads.
__device__ __forceinline__ uint64_t keep_smallest(uint64_t* s_keys, int c, int kq, const RefSel& rs) {
    return block_select_smallest(s_keys, c, kq, rs.hist, rs.wc, rs.sel);
}

// Sorts s_keys[0, m) ascending (padding to the next power of two with ~0).  All threads.
__device__ __forceinline__ void sort_prefix(uint64_t* s_keys, int m) {
    const int n2 = (int)next_pow2_dev((uint32_t)max(m, 2));
    for (int i = m + threadIdx.x; i < n2; i += blockDim.x) s_keys[i] = ~0ull;
    __syncthreads();
    block_bitonic_sort(s_keys, n2);
}

// Adds the keys below the running k-th to s_keys in rounds of at most cap - kq keys; between
// rounds the buffer keeps its kq smallest.  get(i) gives key i of n; all threads.
template <typename Get>
__device__ __forceinline__ void topk_rounds(uint64_t* s_keys, int cap, int kq, int n, int* s_cnt, uint64_t* s_th,
                                            const RefSel& rs, Get get) {
    const int per_round = max(cap - kq, 1);
    for (int r0 = 0; r0 < n; r0 += per_round) {
        const int r1 = min(n, r0 + per_round);
        for (int i = r0 + (int)threadIdx.x; i < r1; i += blockDim.x) {
            const uint64_t key = get(i);
            if (key < *s_th) s_keys[atomicAdd(s_cnt, 1)] = key;
        }
        __syncthreads();
        const int c = *s_cnt;
        __syncthreads();
        if (r1 < n && c > kq) {
            const uint64_t kth = keep_smallest(s_keys, c, kq, rs);
            if (threadIdx.x == 0) {
                *s_cnt = kq;
                *s_th = kth;
            }
            __syncthreads();
        }
    }
}

__global__ void __launch_bounds__(kThreads, 5) k_refine(IndexDev D, const float* __restrict__ queries,
                                                     const float* __restrict__ data, int cap, int apply_pred,
                                                     int lbl, uint64_t q, Workspace w, float* __restrict__ out_dist,
                                                     uint64_t* __restrict__ out_ids, int k_out) {
    chain_start();
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t* s_keys = reinterpret_cast<uint64_t*>(smem);           // [cap]
    float* s_q = reinterpret_cast<float*>(s_keys + cap);             // [d]
    __shared__ float s_box[2 * kMaxDims];
    __shared__ int s_wsum[kThreads / 32];
    __shared__ int s_cnt, s_ns, s_item, s_qi, s_last;
    __shared__ uint64_t s_th;
    __shared__ uint32_t s_rb[4];
    __shared__ uint32_t s_rhist[256], s_rwc[32];
    __shared__ unsigned long long s_rsel[4];
    const RefSel rs{s_rhist, s_rwc, s_rsel};
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nw = kThreads / 32;
    const int d = D.d;
    const uint32_t n_items = w.ritem_off[q];
    int cur = -1;
    for (;;) {
        if (t < 32) {  // the item's query: the last one with ritem_off <= item, by 32-way rounds
            int item = 0;
            if (t == 0) item = (int)atomicAdd(&w.counter[1], 1u);
            item = __shfl_sync(0xffffffffu, item, 0);
            const int qf = item < (int)n_items ? warp_find_le(w.ritem_off, (int)q, (uint32_t)item) : 0;
            if (t == 0) {
                s_item = item;
                s_qi = qf;
            }
        }
        __syncthreads();
        const int item = s_item;
        if (item >= (int)n_items) break;
        const uint64_t qi = (uint64_t)s_qi;
        if ((int)qi != cur) {
            for (int i = t; i < d; i += blockDim.x) s_q[i] = queries[qi * d + i];
            if (t < 2 * lbl) s_box[t] = w.box[qi * 2 * lbl + t];
            if (t < 4) s_rb[t] = w.rank_box[qi * 4 + t];
            cur = (int)qi;
        }
        if (t == 0) {
            s_cnt = 0;
            s_ns = 0;
            s_th = ~0ull;
        }
        __syncthreads();
        const uint32_t it0 = w.ritem_off[qi], nq_items = w.ritem_off[qi + 1] - it0;
        const uint32_t c0 = (uint32_t)(item - (int)it0) * kRefChunk;
        const int nc = (int)(min(w.cand_count[qi], c0 + kRefChunk) - min(w.cand_count[qi], c0));
        const int kq = (int)q_k(w, qi);
        const bool pred_q = apply_pred && q_sched(w, qi) == 0;  // predicate-first queries already passed it
        // label ranks decide most entries: outside the rank box fails, inside the inner box passes
        const bool ranks = D.rankpack && !D.labels_nan;
        const uint32_t gd = D.rank_guard;
        uint32_t* list = sel_row(w, qi) + c0;
        // 1. the predicate survivors, compacted in place as original ids (each chunk is read
        //    before the barrier and written at or below its own start)
        uint32_t n_lab = 0;
        // a row taken whole holds valid pool rows only (the predicate pass listed them): no
        // compaction, just the ids, four lookups in flight per thread and no barrier
        const bool whole = takes_row(w, qi);
        if (whole) {
            for (int e0 = t; e0 < nc; e0 += 4 * kThreads) {
                uint32_t p[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int e = e0 + u * kThreads;
                    p[u] = e < nc ? list[e] : 0u;
                }
#pragma unroll
                for (int u = 0; u < 4; u++) p[u] = __ldg(D.ids + p[u]);
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int e = e0 + u * kThreads;
                    if (e < nc) list[e] = p[u];
                }
            }
            if (t == 0) s_ns = nc;
        }
        for (int base = 0; !whole && base < nc; base += kThreads) {
            const int e = base + t;
            bool keep = false;
            uint32_t pool = kInvalid;
            if (e < nc) {
                pool = list[e];
                keep = pool != kInvalid;
                if (keep && pred_q) {
                    bool sure = false;
                    if (ranks) {
                        const uint32_t c = __ldg(D.rankpack + pool);
                        const uint32_t to = ((c | gd) - s_rb[0]) & (s_rb[1] - c);
                        const uint32_t ti = ((c | gd) - s_rb[2]) & (s_rb[3] - c);
                        keep = (to & gd) == gd;
                        sure = (ti & gd) == gd;
                    }
                    if (keep && !sure) {
                        n_lab++;
                        const float* lab = D.labels + (uint64_t)pool * lbl;
                        for (int i = 0; i < lbl; i++) {
                            const float v = lab[i];
                            if (v < s_box[2 * i] || v > s_box[2 * i + 1]) keep = false;
                        }
                    }
                }
            }
            const unsigned bal = __ballot_sync(0xffffffffu, keep);
            if (lane == 0) s_wsum[warp] = __popc(bal);
            __syncthreads();
            int before = s_ns, tot = 0;
            for (int i = 0; i < nw; i++) {
                before += i < warp ? s_wsum[i] : 0;
                tot += s_wsum[i];
            }
            if (keep) list[before + __popc(bal & ((1u << lane) - 1))] = D.ids[pool];
            __syncthreads();
            if (t == 0) s_ns += tot;
        }
        n_lab = __reduce_add_sync(0xffffffffu, n_lab);
        if (lane == 0 && n_lab) atomicAdd(&w.rlab[qi], n_lab);
        __syncthreads();
        const int ns = s_ns;
        if (t == 0 && ns) atomicAdd(&w.rsurv[qi], (uint32_t)ns);
        // 2. exact distances in rounds of cap - kq rows: every warp takes rows of the round, the
        //    keys (distance, id) below the running k-th go to the buffer, which is sorted and cut
        //    to kq after each round
        const int per_round = max(cap - kq, 1);
        // rows 16-byte aligned with d % 4 == 0: four rows per warp at a time, 8 lanes per row,
        // 16-byte loads, four independent partial sums per lane (the gathers are latency-bound:
        // this keeps ~6 KB per warp in flight instead of one 128-byte load per lane)
        const bool vec4 = (d & 3) == 0 && (reinterpret_cast<uintptr_t>(data) & 15) == 0;
        for (int r0 = 0; r0 < ns; r0 += per_round) {
            const int r1 = min(ns, r0 + per_round);
            if (vec4) {
                const int g = lane >> 3, sl = lane & 7, d4 = d >> 2;
                const float4* q4 = reinterpret_cast<const float4*>(s_q);
                for (int i0 = r0 + warp * 4; i0 < r1; i0 += nw * 4) {
                    const int i = i0 + g;
                    const bool ok = i < r1;
                    const uint32_t id = ok ? list[i] : list[r0];
                    const float4* row = reinterpret_cast<const float4*>(data + (uint64_t)id * d);
                    float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
                    int j = sl;
                    for (; j + 24 < d4; j += 32) {
                        const float4 x0 = __ldg(row + j), x1 = __ldg(row + j + 8), x2 = __ldg(row + j + 16),
                                     x3 = __ldg(row + j + 24);
                        const float4 y0 = q4[j], y1 = q4[j + 8], y2 = q4[j + 16], y3 = q4[j + 24];
                        a0 = fmaf(y0.x - x0.x, y0.x - x0.x, a0);
                        a0 = fmaf(y0.y - x0.y, y0.y - x0.y, a0);
                        a0 = fmaf(y0.z - x0.z, y0.z - x0.z, a0);
                        a0 = fmaf(y0.w - x0.w, y0.w - x0.w, a0);
                        a1 = fmaf(y1.x - x1.x, y1.x - x1.x, a1);
                        a1 = fmaf(y1.y - x1.y, y1.y - x1.y, a1);
                        a1 = fmaf(y1.z - x1.z, y1.z - x1.z, a1);
                        a1 = fmaf(y1.w - x1.w, y1.w - x1.w, a1);
                        a2 = fmaf(y2.x - x2.x, y2.x - x2.x, a2);
                        a2 = fmaf(y2.y - x2.y, y2.y - x2.y, a2);
                        a2 = fmaf(y2.z - x2.z, y2.z - x2.z, a2);
                        a2 = fmaf(y2.w - x2.w, y2.w - x2.w, a2);
                        a3 = fmaf(y3.x - x3.x, y3.x - x3.x, a3);
                        a3 = fmaf(y3.y - x3.y, y3.y - x3.y, a3);
                        a3 = fmaf(y3.z - x3.z, y3.z - x3.z, a3);
                        a3 = fmaf(y3.w - x3.w, y3.w - x3.w, a3);
                    }
                    for (; j < d4; j += 8) {
                        const float4 x = __ldg(row + j), y = q4[j];
                        a0 = fmaf(y.x - x.x, y.x - x.x, a0);
                        a0 = fmaf(y.y - x.y, y.y - x.y, a0);
                        a0 = fmaf(y.z - x.z, y.z - x.z, a0);
                        a0 = fmaf(y.w - x.w, y.w - x.w, a0);
                    }
                    float sq = (a0 + a1) + (a2 + a3);
                    sq += __shfl_xor_sync(0xffffffffu, sq, 4);
                    sq += __shfl_xor_sync(0xffffffffu, sq, 2);
                    sq += __shfl_xor_sync(0xffffffffu, sq, 1);
                    const uint64_t key = ((uint64_t)float_key(sq) << 32) | id;
                    if (ok && sl == 0 && key < s_th) s_keys[atomicAdd(&s_cnt, 1)] = key;
                }
            } else {
                for (int i = r0 + warp; i < r1; i += nw) {
                    const uint32_t id = list[i];
                    const float* row = data + (uint64_t)id * d;
                    float sq = 0.f;
                    for (int j = lane; j < d; j += 32) {
                        const float df = s_q[j] - __ldg(row + j);
                        sq = fmaf(df, df, sq);
                    }
                    sq = warp_sum(sq);
                    const uint64_t key = ((uint64_t)float_key(sq) << 32) | id;
                    if (lane == 0 && key < s_th) s_keys[atomicAdd(&s_cnt, 1)] = key;
                }
            }
            __syncthreads();
            const int c = s_cnt;
            __syncthreads();
            if (r1 < ns && c > kq) {  // more rows follow: keep the kq best
                const uint64_t kth = keep_smallest(s_keys, c, kq, rs);
                if (t == 0) {
                    s_cnt = kq;
                    s_th = kth;
                }
                __syncthreads();
            }
        }
        int c = s_cnt;
        __syncthreads();
        if (c > kq) keep_smallest(s_keys, c, kq, rs);
        sort_prefix(s_keys, min(c, kq));
        bool write_out = nq_items == 1;
        if (!write_out) {
            // this item's best kq keys go to its partial row; the query's last item merges
            uint64_t* part = w.rpart + (uint64_t)item * k_out;
            for (int i = t; i < kq; i += blockDim.x) part[i] = i < c ? s_keys[i] : ~0ull;
            __threadfence();
            __syncthreads();
            if (t == 0) s_last = atomicAdd(&w.rdone[qi], 1u) == nq_items - 1;
            __syncthreads();
            if (s_last) {
                __threadfence();  // the other items' partial rows are visible past their counts
                if (t == 0) {
                    s_cnt = 0;
                    s_th = ~0ull;
                }
                __syncthreads();
                const uint64_t* rows = w.rpart + (uint64_t)it0 * k_out;
                topk_rounds(s_keys, cap, kq, (int)nq_items * kq, &s_cnt, &s_th, rs,
                            [&](int i) { return __ldcg(rows + (uint64_t)(i / kq) * k_out + (i % kq)); });
                c = s_cnt;
                __syncthreads();
                if (c > kq) keep_smallest(s_keys, c, kq, rs);
                sort_prefix(s_keys, min(c, kq));
                write_out = true;
            }
        }
        if (write_out) {
            for (int i = t; i < k_out; i += blockDim.x) {
                if (i < min(c, kq) && s_keys[i] != ~0ull) {
                    const uint64_t key = s_keys[i];
                    out_dist[qi * k_out + i] = key_float((uint32_t)(key >> 32));
                    out_ids[qi * k_out + i] = (uint32_t)key;
                } else {
                    out_dist[qi * k_out + i] = INFINITY;
                    out_ids[qi * k_out + i] = ~0ull;
                }
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------
// The estimate pass: which candidates of a post-filter query can be among its n_cand smallest
// ------------------------------------------------------------------------------------
// The post-filter schedule needs the n_cand smallest ADC distances of a query's candidates, a few
// percent of them.  An ADC distance is the distance to the candidate's PQ approximation, so a
// tensor-core product of queries and approximations bounds it from both sides (hdg_est.cuh):
//   k_est_thr    a threshold per query from a strided sample of its candidates' ADC distances: a
//                sample rank past n_cand's share by four standard deviations;
//   k_est_count / k_est_scan / k_est_fill   the (query, range) entries of every tile of kEstM pool
//                rows, so that a tile meets only the queries whose ranges touch it;
//   k_est        every candidate whose lower bound is not above the threshold goes to its query's
//                row, with the bound's depth below the threshold in steps;
//   k_est_pick   with v the n_cand-th smallest bound and w the most an ADC distance can exceed its
//                bound by: a candidate w and more below v is among the n_cand smallest, one more
//                than w above v is not; those in between are left open.  When v + w passes the
//                threshold (candidates outside the row could matter) the query is scanned in full;
//   k_scan_fast / k_select   the exact ADC of the open candidates and the smallest of them.
// The selection is the full scan's.  10,000 queries x 227,000 candidates x 32 subspaces (n_cand
// 9,384), estimate to select: 20.4 ms in full (a full scan, a select over every distance), 7.3 ms this way.
constexpr int kThrThreads = 512;
constexpr uint32_t kThrMax = 4096;  // sampled candidates at most
constexpr int kThrBins = 2048;

// The table is staged in BF16: the threshold only decides how many candidates are kept, and half the
// shared memory puts twice the blocks on an SM (1,417 -> 985 us at M = 96, 601 -> 658 us
// at M = 32, 10,000 queries).
template <int G>
__global__ void __launch_bounds__(kThrThreads) k_est_thr(IndexDev D, int R, const float* __restrict__ queries, Workspace w) {
    extern __shared__ __align__(16) uint32_t s_tab[];  // [G][256][16] pairs of BF16 entries
    float* s_d = reinterpret_cast<float*>(s_tab + G * kCodes * 16);     // [kThrMax]
    uint32_t* s_hist = reinterpret_cast<uint32_t*>(s_d + kThrMax);      // [kThrBins]
    uint32_t* s_pre = s_hist + kThrBins;                                  // [R + 1]
    uint32_t* s_start = s_pre + R + 1;                                    // [R]
    __shared__ unsigned long long s_scan[32];
    __shared__ float s_red[3];
    __shared__ uint32_t s_mm[2];
    __shared__ int s_bin, s_bin_lo;
    const uint64_t qi = blockIdx.x;
    const int t = threadIdx.x, lane = t & 31;
    const uint32_t N = w.qstat[qi * 4];
    const uint32_t K = w.qbud[qi];
    // sample size: the cost of a sampled candidate against the extra candidates that a coarser
    // threshold lets through, about 2.5 (5 sqrt(K N))^(2/3) of either
    uint32_t ms = 0, rank = 0, rank_lo = 1;
    if (N >= 4096 && (uint64_t)K * 3 <= N) {
        ms = (uint32_t)powf(5.f * sqrtf((float)K * (float)N), 2.f / 3.f);
        ms = min(kThrMax, max(512u, ms));
        const float r = (float)K * (float)ms / (float)N;
        rank = (uint32_t)(r + 4.f * sqrtf(r) + 4.f);
        rank_lo = (uint32_t)fmaxf(1.f, r - 5.f * sqrtf(r) - 2.f);
    }
    if (t == 0) w.prq[qi] = 0;
    if (ms == 0 || rank >= ms) return;  // block-uniform
    if (t == 0) {
        s_mm[0] = 0xffffffffu;
        s_mm[1] = 0u;
        s_red[0] = s_red[1] = s_red[2] = 0.f;
        s_bin = s_bin_lo = -1;
    }
    auto pair = [](float x, float y) {  // (rounded towards zero: no carry into infinity)
        return (__float_as_uint(x) >> 16) | (__float_as_uint(y) & 0xffff0000u);
    };
    if (w.lut16) {
        const uint2* src = reinterpret_cast<const uint2*>(reinterpret_cast<const __half*>(w.lut) + qi * G * kCodes * 32);
        for (int e = t; e < G * kCodes * 8; e += kThrThreads) {
            const uint2 v = __ldg(src + e);
            const float2 a = __half22float2(reinterpret_cast<const __half2&>(v.x)),
                         b = __half22float2(reinterpret_cast<const __half2&>(v.y));
            reinterpret_cast<uint2*>(s_tab)[e] = make_uint2(pair(a.x, a.y), pair(b.x, b.y));
        }
    } else {
        const float4* src = reinterpret_cast<const float4*>(w.lut + qi * G * kCodes * 32);
        for (int e = t; e < G * kCodes * 8; e += kThrThreads) {
            const float4 v = __ldg(src + e);
            reinterpret_cast<uint2*>(s_tab)[e] = make_uint2(pair(v.x, v.y), pair(v.z, v.w));
        }
    }
    for (int i = t; i < kThrBins; i += kThrThreads) s_hist[i] = 0;
    const uint32_t* pre = w.range_pre + qi * (R + 1);
    for (int i = t; i <= R; i += kThrThreads) s_pre[i] = pre[i];
    for (int i = t; i < R; i += kThrThreads) s_start[i] = w.range_start[qi * R + i];
    __syncthreads();
    // the query's norms (for the estimate's constants)
    {
        float qn = 0.f, q2 = 0.f, rq = 0.f;
        for (int i = t; i < (int)D.d; i += kThrThreads) {
            const __half hv = __float2half_rn(queries[qi * D.d + i]);
            const float v = queries[qi * D.d + i], h = __half2float(hv), e = v - h;
            reinterpret_cast<__half*>(w.qbf)[qi * D.d + i] = hv;  // (the coarse GEMM's BF16 copy is no longer needed)
            qn = fmaf(v, v, qn);
            q2 = fmaf(h, h, q2);
            rq = fmaf(e, e, rq);
        }
        qn = warp_sum(qn);
        q2 = warp_sum(q2);
        rq = warp_sum(rq);
        if (lane == 0 && t < (int)((D.d + 31) / 32 * 32)) {
            atomicAdd(&s_red[0], qn);
            atomicAdd(&s_red[1], q2);
            atomicAdd(&s_red[2], rq);
        }
    }
    const uint4* planes = reinterpret_cast<const uint4*>(D.codes);
    uint32_t kmin = 0xffffffffu, kmax = 0u;
    for (uint32_t i = t; i < ms; i += kThrThreads) {
        const uint32_t e = (uint32_t)(((uint64_t)i * N + N / 2) / ms);
        int lo = 0, hi = R - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (s_pre[mid] <= e) lo = mid;
            else hi = mid - 1;
        }
        const uint4* cp = planes + s_start[lo] + (e - s_pre[lo]);
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int g = 0; g < G; g++) {
            // lane r goes round from subspace r: the lanes of a warp read different banks
            const uint4 a = __ldg(cp + (uint64_t)(2 * g) * D.n), b = __ldg(cp + (uint64_t)(2 * g + 1) * D.n);
            uint32_t wv[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            rotate_words(wv, (uint32_t)lane >> 2);
            const uint32_t sh = 8u * (lane & 3);
            const unsigned short* L = reinterpret_cast<const unsigned short*>(s_tab + g * kCodes * 16);
#pragma unroll
            for (int st = 0; st < 32; st += 2) {
                const uint32_t x = __funnelshift_r(wv[st >> 2], wv[((st >> 2) + 1) & 7], sh);
                const uint32_t c0 = (x >> (8 * (st & 3))) & 255u, c1 = (x >> (8 * ((st + 1) & 3))) & 255u;
                s0 += __uint_as_float((uint32_t)L[c0 * 32 + ((lane + st) & 31)] << 16);
                s1 += __uint_as_float((uint32_t)L[c1 * 32 + ((lane + st + 1) & 31)] << 16);
            }
        }
        const float d = s0 + s1;
        s_d[i] = d;
        const uint32_t key = float_key(d);
        if (d < INFINITY) {
            kmin = min(kmin, key);
            kmax = max(kmax, key);
        }
    }
    kmin = __reduce_min_sync(0xffffffffu, kmin);
    kmax = __reduce_max_sync(0xffffffffu, kmax);
    if (lane == 0) {
        atomicMin(&s_mm[0], kmin);
        atomicMax(&s_mm[1], kmax);
    }
    __syncthreads();
    if (s_mm[0] > s_mm[1]) return;  // no finite distance
    // the threshold: the upper edge of the bin that holds the sample's rank-th distance
    const float lo = key_float(s_mm[0]), hi = key_float(s_mm[1]);
    const float inv = hi > lo ? (float)kThrBins / (hi - lo) : 0.f;
    for (uint32_t i = t; i < ms; i += kThrThreads) {
        const float d = s_d[i];
        if (d < INFINITY) atomicAdd(&s_hist[min(kThrBins - 1, max(0, (int)((d - lo) * inv)))], 1u);
    }
    __syncthreads();
    constexpr int kPer = kThrBins / kThrThreads;
    uint32_t c[kPer], sum = 0;
#pragma unroll
    for (int i = 0; i < kPer; i++) {
        c[i] = s_hist[t * kPer + i];
        sum += c[i];
    }
    unsigned long long tot = 0;
    uint32_t run = (uint32_t)block_inclusive_sum(sum, s_scan, &tot) - sum;
    auto bin_of = [&](uint32_t r, int* bin) {
        if (run < r && r <= run + sum) {
            uint32_t x = run;
            int i = 0;
            while (i < kPer - 1 && x + c[i] < r) x += c[i++];
            *bin = t * kPer + i;
        }
    };
    bin_of(rank, &s_bin);
    bin_of(rank_lo, &s_bin_lo);
    __syncthreads();
    if (t == 0 && s_bin >= 0 && s_bin_lo >= 0) {
        const float T = s_bin == kThrBins - 1 || !(inv > 0.f) ? hi : lo + (float)(s_bin + 1) / inv;
        const float qn = s_red[0], qh = sqrtf(s_red[1]) * (1.f + kEstSlack), rq = sqrtf(s_red[2]) * (1.f + kEstSlack);
        // the bounds hold for the distance itself: an ADC distance differs from it by its own
        // rounding -- FP32 sums, and with FP16 tables each entry by 2^-11 (or 2^-25)
        const float xm2 = __uint_as_float(D.decoded_max[0]), xm = __uint_as_float(D.decoded_max[1]),
                    rm = __uint_as_float(D.decoded_max[2]);
        const float adc = w.lut16 ? 1.1e-3f * T + 1e-7f * (float)D.M : kEstSlack * T;
        const float ca = 2.f * (rq + kEstAcc * (float)D.d * sqrtf(qn)) * (1.f + kEstSlack), cb = 2.f * qh;
        const float wide = 2.f * (ca * xm + cb * rm) + 4.f * kEstSlack * (qn + xm2) + 2.f * adc;
        // the steps run from the sample rank five standard deviations below n_cand's share (the
        // n_cand-th bound lies there or above, but for a rare sample) less twice the bounds' width;
        // rows are kept up to T, the width and the steps' rounding past it, so that the n_cand-th
        // bound lies that much below the threshold
        const float Tl = (inv > 0.f ? lo + (float)s_bin_lo / inv : lo) - 2.f * wide;
        const float Tb = Tl + (T + wide - Tl) * (253.f / 246.f), z = qn * (1.f - kEstSlack) - Tb;
        const float steps = 253.f / (Tb - Tl);
        const float ws = wide * steps + 4.f;    // and the steps' own rounding, on both sides
        // (a NaN or an extreme norm anywhere in the index fails these tests; FP16 entries of a distance
        // at or below T must not overflow)
        if (T < INFINITY && Tb > Tl && ws < 120.f && fabsf(z) * steps < 1e6f && qn + xm2 < 1e30f &&
            (!w.lut16 || T < 6e4f)) {
            w.est_qc[qi] = make_float4(ca, cb, z, steps);
            w.est_w[qi] = (int)ws + 1;
            w.prq[qi] = 1;
        }
    }
}

// The sure and the open candidates of each query of the pass: the kept candidates' steps counted
// per value, the value that holds the n_cand-th smallest bound, then one pass that appends the sure
// ones to the selection and the open ones -- position and pool row -- behind the row's entries.
constexpr int kPickThreads = 256;
__global__ void __launch_bounds__(kPickThreads) k_est_pick(int R, Workspace w) {
    extern __shared__ uint32_t s_pre[];  // [R + 1], then [R] range starts
    uint32_t* s_start = s_pre + R + 1;
    __shared__ uint32_t s_hist[kPickThreads / 32][256];
    __shared__ int s_v;
    __shared__ uint32_t s_in, s_open, s_cnt[2];
    const uint64_t qi = blockIdx.x;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (w.prq[qi] != 1) return;
    const uint32_t N = w.qstat[qi * 4], K = w.qbud[qi], ne = w.cand_count[qi];
    const uint64_t row = w.qoff[qi];
    const bool err = *w.gemm_err != 0;
    for (int i = lane; i < 256; i += 32) s_hist[warp][i] = 0;
    if (t == 0) {
        s_v = 0;
        s_in = s_open = s_cnt[0] = s_cnt[1] = 0;
    }
    __syncthreads();
    const int wd = w.est_w[qi];
    uint32_t* prow = w.spos + row;  // position | step << 24
    for (uint32_t e0 = t; e0 < ne; e0 += 4 * kPickThreads) {
        uint32_t x[4];
#pragma unroll
        for (int u = 0; u < 4; u++) x[u] = e0 + u * kPickThreads < ne ? prow[e0 + u * kPickThreads] : 0u;
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (e0 + u * kPickThreads < ne) atomicAdd(&s_hist[warp][x[u] >> 24], 1u);
    }
    __syncthreads();
    uint32_t c = 0;
    {  // thread t holds value 255 - t: the bounds from the smallest on
        for (int k = 0; k < kPickThreads / 32; k++) c += s_hist[k][255 - t];
        __syncthreads();
        s_hist[0][t] = c;
        __syncthreads();
        if (t < 32) {
            uint32_t sum = 0, x[8];
#pragma unroll
            for (int k = 0; k < 8; k++) sum += x[k] = s_hist[0][8 * t + k];
            uint32_t inc = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                if (t >= o) inc += y;
            }
            uint32_t run = inc - sum;
            if (run < K && K <= inc) {
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    if (run < K && K <= run + x[k]) s_v = 255 - (8 * t + k);
                    run += x[k];
                }
            }
        }
        __syncthreads();
    }
    const int v = s_v, lo = v - wd, hi = v + wd;  // open: steps lo .. hi (255 holds every smaller bound)
    {
        const int val = 255 - t;
        const uint32_t in = val > hi ? c : 0u, op = val >= lo && val <= hi ? c : 0u;
        if (in) atomicAdd(&s_in, in);
        if (op) atomicAdd(&s_open, op);
    }
    __syncthreads();
    // the open candidates' entries go behind the row's (position, step) entries
    const uint32_t n_open = s_open, n_in = s_in;
    if (err || v == 0 || lo < 1 || ne + n_open > N) {
        __syncthreads();
        if (t == 0) {
            w.prq[qi] = 0;
            w.cand_count[qi] = 0;
        }
        return;
    }
    for (int i = t; i <= R; i += kPickThreads) s_pre[i] = w.range_pre[qi * (R + 1) + i];
    for (int i = t; i < R; i += kPickThreads) s_start[i] = w.range_start[qi * R + i];
    __syncthreads();
    uint32_t* open_row = reinterpret_cast<uint32_t*>(w.dist + row) + ne;
    uint32_t* sel = w.cand_pool + w.soff[qi];
    for (uint32_t e0 = 0; e0 < ne; e0 += 4 * kPickThreads) {  // block-uniform bound
        uint32_t x[4];
#pragma unroll
        for (int u = 0; u < 4; u++) x[u] = e0 + t + u * kPickThreads < ne ? prow[e0 + t + u * kPickThreads] : 0u;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const bool v = e0 + t + u * kPickThreads < ne;
            const int val = (int)(x[u] >> 24);
            const uint32_t p = x[u] & 0xffffffu;
            const bool in = v && val > hi, op = v && val >= lo && val <= hi;
            const uint32_t a = warp_reserve(in, &s_cnt[0]), b = warp_reserve(op, &s_cnt[1]);
            if (in) sel[a] = p;
            if (op) prow[ne + b] = p;
        }
    }
    __syncthreads();
    for (uint32_t i = t; i < n_in; i += kPickThreads) sel[i] = pos_to_pool(s_pre, s_start, R, sel[i]);
    for (uint32_t i = t; i < n_open; i += kPickThreads) open_row[i] = pos_to_pool(s_pre, s_start, R, prow[ne + i]);
    if (t == 0) {
        w.est_in[qi] = n_in;
        w.est_row[qi] = ne;
        w.cand_count[qi] = n_open;
    }
}

// +1 / -1 at the first row tile of every candidate range of the pass's queries and past its last
__global__ void k_est_count(uint64_t q, int R, Workspace w, int* __restrict__ diff) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= q * R) return;
    if (w.prq[e / R] != 1) return;
    const uint32_t len = w.range_len[e], start = w.range_start[e];
    if (!len) return;
    atomicAdd(&diff[start / kEstM], 1);
    atomicAdd(&diff[(start + len - 1) / kEstM + 1], -1);
}

// Entries of every row tile (the running sum of diff), their prefix, and the prefix of their query
// tiles; cursor: a copy of the entries' prefix for the fill.  One block.
__global__ void __launch_bounds__(1024) k_est_scan(const int* __restrict__ diff, uint32_t tiles,
                                                   uint32_t* __restrict__ ent_off, uint32_t* __restrict__ nt_off,
                                                   uint32_t* __restrict__ cursor) {
    __shared__ unsigned long long s_a[32], s_b[32], s_c[32];
    const int t = threadIdx.x;
    const uint32_t per = (tiles + blockDim.x - 1) / blockDim.x, b = min(tiles, t * per), e = min(tiles, b + per);
    long long d = 0;
    for (uint32_t i = b; i < e; i++) d += diff[i];
    unsigned long long tot = 0;
    const long long c0 = (long long)block_inclusive_sum((unsigned long long)d, s_a, &tot) - d;  // (wraps like the sums)
    unsigned long long ne = 0, nt = 0;
    long long c = c0;
    for (uint32_t i = b; i < e; i++) {
        c += diff[i];
        ne += (unsigned long long)c;
        nt += (unsigned long long)(c + kEstN - 1) / kEstN;
    }
    unsigned long long pe = block_inclusive_sum(ne, s_b, &tot) - ne;
    unsigned long long pn = block_inclusive_sum(nt, s_c, &tot) - nt;
    c = c0;
    for (uint32_t i = b; i < e; i++) {
        c += diff[i];
        ent_off[i] = cursor[i] = (uint32_t)pe;
        nt_off[i] = (uint32_t)pn;
        pe += (unsigned long long)c;
        pn += (unsigned long long)(c + kEstN - 1) / kEstN;
    }
    if (e == tiles && b < e) {
        ent_off[tiles] = (uint32_t)pe;
        nt_off[tiles] = (uint32_t)pn;
    }
}

// The entries themselves.  A warp takes 32 ranges and shares their tiles out evenly: entry k of
// the warp belongs to the range whose prefix of tile counts holds k.
__global__ void __launch_bounds__(256) k_est_fill(uint64_t q, int R, Workspace w, uint32_t* __restrict__ cursor,
                                                  uint4* __restrict__ ent) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    uint32_t qi = 0, start = 0, len = 0, pre = 0;
    if (e < q * R) {
        qi = (uint32_t)(e / R);
        if (w.prq[qi] == 1) {
            len = w.range_len[e];
            start = w.range_start[e];
            pre = w.range_pre[(uint64_t)qi * (R + 1) + (uint32_t)(e % R)];
        }
    }
    const uint32_t t0 = start / kEstM, n = len ? (start + len - 1) / kEstM - t0 + 1u : 0u;
    uint32_t inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
    for (uint32_t k0 = 0; k0 < total; k0 += 32) {
        const uint32_t k = k0 + lane;
        int r = 0;  // the first lane whose inclusive prefix passes k
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const uint32_t v = __shfl_sync(0xffffffffu, inc, r + o - 1);
            if (v <= k) r += o;
        }
        r = min(r, 31);
        const uint32_t rs = __shfl_sync(0xffffffffu, start, r), rl = __shfl_sync(0xffffffffu, len, r),
                       rp = __shfl_sync(0xffffffffu, pre, r), rq = __shfl_sync(0xffffffffu, qi, r),
                       ri = __shfl_sync(0xffffffffu, inc, r), rn = __shfl_sync(0xffffffffu, n, r);
        if (k < total) {
            const uint32_t tile = rs / kEstM + (k - (ri - rn)), base = tile * kEstM;
            const uint32_t lo = max(rs, base) - base, hi = min(rs + rl, base + kEstM) - base;
            ent[atomicAdd(&cursor[tile], 1u)] = make_uint4(rq, lo | (hi << 16), rp - rs, 0u);
        }
    }
}

// ------------------------------------------------------------------------------------
// host orchestration
// ------------------------------------------------------------------------------------
static uint32_t lut_groups(const IndexDev& D) { return (D.M + 31) / 32; }

static Workspace carve(hdg_index* idx, QueryCtx& cx, uint64_t q, bool record) {
    const hdg_params& P = idx->params;
    const uint64_t l = idx->dev.l, L = idx->dev.n_lists, C = idx->dev.C;
    const uint64_t Pc = std::max<uint64_t>(1, P.n_list), Ps = std::max<uint64_t>(1, P.sub_lists);
    const uint64_t G = lut_groups(idx->dev);
    size_t off = 0;
    char* base = static_cast<char*>(cx.work.ptr);
    auto take = [&](const char* name, size_t bytes) -> void* {
        const size_t o = off;
        off += align_up(bytes ? bytes : 1, 256);
        if (record) cx.layout[name] = {o, bytes};
        return base ? base + o : nullptr;
    };
    Workspace w{};
    w.box = (float*)take("box", q * 2 * l * 4);
    w.cells = (int*)take("cells", q * 2 * l * 4);
    w.rank_box = (uint32_t*)take("rank_box", q * 4 * 4);
    w.zrange = (uint64_t*)take("zrange", q * 2 * 8);
    w.list_counts = (uint32_t*)take("list_counts", q * L * 4);
    w.cluster_counts = (uint32_t*)take("cluster_counts", q * C * 4);
    w.probe_clusters = (uint32_t*)take("probe_clusters", q * Pc * 4);
    w.probe_lists = (uint32_t*)take("probe_lists", q * Ps * 4);
    const uint64_t ns = P.is_split ? std::max<uint64_t>(1, P.n_split) : 1;
    w.range_start = (uint32_t*)take("range_start", q * Ps * ns * 4);
    w.range_len = (uint32_t*)take("range_len", q * Ps * ns * 4);
    w.range_pre = (uint32_t*)take("range_pre", q * (Ps * ns + 1) * 4);
    w.is_split = P.is_split ? 1 : 0;
    w.nsplit = (int)ns;
    w.qstat = (uint32_t*)take("qstat", q * 4 * 4);
    w.qtiles = (uint32_t*)take("row_tiles", q * 4);
    w.scal = (uint64_t*)take("scalars", 8 * 8);
    w.qoff = (uint64_t*)take("qoff", (q + 1) * 8);
    w.item_off = (uint32_t*)take("item_off", (q + 1) * 4);
    w.pitem_off = (uint32_t*)take("pre_items", (q + 1) * 4);
    w.mm = (uint32_t*)take("minmax", q * 2 * 4);
    w.nfin = (uint32_t*)take("nfin", q * 4);
    w.lab_read = (uint32_t*)take("labels_read", q * 4);
    w.rank_read = (uint32_t*)take("ranks_read", q * 4);
    w.counter = (uint32_t*)take("counter", 32);
    w.lut16 = P.lut_fp16 != 0;
    w.lut = (float*)take("lut", q * G * kCodes * 32 * (w.lut16 ? 2 : 4));
    w.cand_count = (uint32_t*)take("cand_count", q * 4);
    w.qbud = (uint32_t*)take("budget", q * 4);
    w.soff = (uint64_t*)take("sel_off", (q + 1) * 8);
    w.ritem_off = (uint32_t*)take("refine_items", (q + 1) * 4);
    w.rdone = (uint32_t*)take("refine_done", q * 4);
    w.rsurv = (uint32_t*)take("refine_rows", q * 4);
    w.rlab = (uint32_t*)take("refine_labels_read", q * 4);
    w.ldS = C + L;
    w.S = (float*)take("gemm_s", q * (C + L) * 4);
    w.qnorm = (float*)take("qnorm", q * 4);
    w.qbf = take("qbf", q * idx->dev.d * 2);
    w.gemm_err = reinterpret_cast<int*>(w.scal + 8);  // in the scalars' padding: one copy reads both
    if (record) cx.layout["gemm_err"] = {cx.layout["scalars"].first + 64, 16};
    w.feats = (float*)take("features", q * kMlpFeatures * 4);
    w.lq_ps = (uint32_t*)take("learned_nprobe", q * 4);
    w.lq_sched = (uint8_t*)take("learned_schedule", q);
    w.dist = static_cast<float*>(cx.dist_buf.ptr);
    w.spos = static_cast<uint32_t*>(cx.pos_buf.ptr);
    w.cand_pool = static_cast<uint32_t*>(cx.sel_buf.ptr);
    w.sel_cap = cx.sel_buf.bytes / 4;
    w.rpart = static_cast<uint64_t*>(cx.part_buf.ptr);
    if (!base) cx.work.bytes = std::max(cx.work.bytes, off);  // size probe
    return w;
}

// Partial rows of the refine items: at most one item per query plus one per kRefChunk
// entries of the selection buffer, k keys each.
static size_t part_bytes(const QueryCtx& cx, uint64_t q, uint32_t k) {
    return (q + (cx.sel_buf.bytes / 4) / kRefChunk + 1) * (size_t)k * 8;
}
static void invalidate_ctx_graphs(QueryCtx& cx);
static void ensure_part_buf(QueryCtx& cx, uint64_t q, uint32_t k) {
    const size_t need = part_bytes(cx, q, k);
    if (cx.part_buf.bytes >= need) return;
    invalidate_ctx_graphs(cx);
    cx.part_buf.reset();
    cx.part_buf.ensure(need);
}

// The per-candidate rows: one f32 distance and one u32 position per candidate, same capacity.
static bool resize_rows(QueryCtx& cx, size_t bytes) {
    cx.dist_buf.reset();
    cx.pos_buf.reset();
    // (dist_buf last: its size is the capacity of both)
    return cx.pos_buf.try_ensure(bytes) && cx.dist_buf.try_ensure(bytes);
}

// Rows and selection of at least the given bytes, a quarter more when the memory is there.
static void resize_candidates(QueryCtx& cx, size_t rows, size_t sel) {
    bool ok = cx.dist_buf.bytes >= rows || resize_rows(cx, rows * 5 / 4);
    if (ok && cx.sel_buf.bytes < sel) {
        cx.sel_buf.reset();
        ok = cx.sel_buf.try_ensure(sel * 5 / 4);
    }
    if (ok) return;
    for (DeviceBuffer* b : {&cx.dist_buf, &cx.pos_buf, &cx.sel_buf, &cx.est_buf}) b->reset();
    cx.sel_buf.ensure(sel);
    cx.pos_buf.ensure(rows);
    cx.dist_buf.ensure(rows);
}

static size_t workspace_bytes(hdg_index* idx, QueryCtx& cx, uint64_t q) {
    void* saved = cx.work.ptr;
    cx.work.ptr = nullptr;
    const size_t before = cx.work.bytes;
    cx.work.bytes = 0;
    carve(idx, cx, q, false);
    const size_t need = cx.work.bytes;
    cx.work.ptr = saved;
    cx.work.bytes = before;
    return need;
}

static void resolve_lazy(hdg_index* idx, QueryCtx& cx);
static void reserve_ctx(hdg_index* idx, QueryCtx& cx, uint64_t q) {
    HDG_REQUIRE(idx->built, HDG_ERR_STATE, "index not built");
    const size_t need = workspace_bytes(idx, cx, q);
    if (cx.work.ptr && cx.work.bytes >= need) return;
    resolve_lazy(idx, cx);
    cx.work.reset();
    cx.work.ensure(need);
    cx.work_queries = q;
}

// Batches of up to this many (query, point) pairs get candidate buffers for every pair (at most
// 80 MiB each for distances, positions and selection) when there is room for them, so the host need
// not read the candidate total before it enqueues the scan: one query went from 100 to 69 us without
// the wait.
constexpr uint64_t kUnsizedPairs = 16ull << 20;

// Candidate buffers of a batch whose totals are known to be at most coarse / selected entries
static void ensure_candidates(QueryCtx& cx, uint64_t q, uint32_t k, uint64_t coarse, uint64_t selected) {
    const size_t rows = std::max<uint64_t>(coarse, 1) * 4, sel = std::max<uint64_t>(selected, 1) * 4;
    if (cx.dist_buf.bytes < rows || cx.sel_buf.bytes < sel) {
        invalidate_ctx_graphs(cx);  // their distance and selection pointers die with the old buffers
        resize_candidates(cx, rows, sel);
    }
    ensure_part_buf(cx, q, k);
}

// The same for every one of `pairs` (query, point) pairs; false when the memory is not there.
static bool try_candidates(QueryCtx& cx, uint64_t q, uint32_t k, uint64_t pairs) {
    try {
        ensure_candidates(cx, q, k, pairs, pairs);
    } catch (const Error& e) {
        if (e.status != HDG_ERR_OOM) throw;
        return false;
    }
    return true;
}

// The query context of a stream (created on first use); it becomes the last one used.
static QueryCtx& query_ctx(hdg_index* idx, cudaStream_t st) {
    std::lock_guard<std::mutex> g(idx->ctx_mu);
    auto& slot = idx->ctxs[static_cast<void*>(st)];
    if (!slot) slot.reset(new QueryCtx());
    idx->last_ctx = slot.get();
    return *slot;
}

// Gives back one of the index's optional buffers: the decoded vectors (the estimate pass is left out
// from then on), then the rank planes (the packed ranks are tested instead).  No context's mutex may be
// held: none of them is enqueueing a call, which would read their addresses, while it is at work; the
// launched ones have ended when cudaFree returns.  False: nothing left to give.
static bool release_optional(hdg_index* idx) {
    std::lock_guard<std::mutex> g(idx->ctx_mu);
    std::vector<std::unique_lock<std::mutex>> held;
    for (auto& kv : idx->ctxs) held.emplace_back(kv.second->mu);
    DeviceBuffer& b = idx->decoded.ptr ? idx->decoded : idx->planes;
    if (!b.ptr) return false;
    for (auto& kv : idx->ctxs) invalidate_ctx_graphs(*kv.second);  // (they hold its address)
    if (&b == &idx->planes) idx->dev.rank_planes = nullptr;
    else idx->dev.decoded = nullptr, idx->dev.decoded_c = nullptr, idx->dev.decoded_max = nullptr;
    b.reset();
    return true;
}

// f(), again without the optional buffers where it ran out of device memory.
template <typename F>
static void with_room(hdg_index* idx, F&& f) {
    for (;;) {
        try {
            f();
            return;
        } catch (const Error& e) {
            if (e.status != HDG_ERR_OOM || !release_optional(idx)) throw;
        }
    }
}

static void reserve_once(hdg_index* idx, uint64_t q, cudaStream_t st) {
    QueryCtx& cx = query_ctx(idx, st);
    std::lock_guard<std::mutex> g(cx.mu);
    reserve_ctx(idx, cx, q);
    // a small batch's candidate buffers too, if there is room: its calls then allocate nothing
    const uint64_t pairs = q * (uint64_t)idx->dev.n, k = idx->params.topk;
    if (pairs <= kUnsizedPairs && k >= 1 && k <= 2048) try_candidates(cx, q, (uint32_t)k, pairs);
}

void reserve_workspace(hdg_index* idx, uint64_t q, cudaStream_t st) {
    with_room(idx, [&] { reserve_once(idx, q, st); });
}

FilterDev filter_dev(const hdg_index* idx) {
    FilterDev f{};
    f.l = idx->filter.l;
    f.filter_dim = (int)std::max<uint64_t>(1, idx->params.filter_dim);
    for (int i = 0; i < kMaxDims; i++) {
        f.type[i] = idx->filter.type[i];
        f.div_value[i] = idx->filter.div_value[i] ? idx->filter.div_value[i] : 1;
        f.shift_val[2 * i] = idx->filter.shift_val[2 * i];
        f.shift_val[2 * i + 1] = idx->filter.shift_val[2 * i + 1];
    }
    f.n_map = (int)idx->filter.interval_map.size();
    f.map = static_cast<const float*>(idx->map_buf.ptr);
    return f;
}

void upload_filter(hdg_index* idx) {
    const auto& m = idx->filter.interval_map;
    idx->map_buf.reset();
    idx->map_buf.ensure(std::max<size_t>(16, m.size() * 4));
    if (!m.empty()) CK(cudaMemcpy(idx->map_buf.ptr, m.data(), m.size() * 4, cudaMemcpyHostToDevice));
}

// Stage times from consecutive recorded events (the first marks the start).
static void store_stage_times(hdg_index* idx, const std::vector<cudaEvent_t>& ev,
                              const std::vector<std::string>& names) {
    std::lock_guard<std::mutex> g(idx->stats_mu);
    idx->stage_names.clear();
    idx->stage_ms.clear();
    for (size_t i = 1; i < ev.size(); i++) {
        float ms = 0;
        CK(cudaEventElapsedTime(&ms, ev[i - 1], ev[i]));
        idx->stage_names.push_back(names[i]);
        idx->stage_ms.push_back(ms);
    }
}

namespace {
// Events between the stages of one query batch.  On the plain path they are recorded on
// the stream and read by finish(); while a CUDA graph is captured (keep != nullptr) they
// become external event-record nodes of the graph, owned by its entry, and every replay
// records them again, so the stage times of each replay can be read once it completes.
struct StageTimer {
    hdg_index* idx;
    cudaStream_t st;
    bool on;
    std::vector<cudaEvent_t> ev;
    std::vector<std::string> names;
    std::vector<cudaEvent_t>* keep;
    std::vector<std::string>* keep_names;
    StageTimer(hdg_index* i, cudaStream_t s, bool enabled, std::vector<cudaEvent_t>* k = nullptr,
               std::vector<std::string>* kn = nullptr)
        : idx(i), st(s), on(enabled), keep(k), keep_names(kn) {
        mark("");
    }
    void mark(const char* name) {
        if (!on) return;
        cudaEvent_t e;
        CK(cudaEventCreate(&e));
        if (keep) {
            keep->push_back(e);
            keep_names->push_back(name);
            CK(cudaEventRecordWithFlags(e, st, cudaEventRecordExternal));
        } else {
            ev.push_back(e);
            names.push_back(name);
            CK(cudaEventRecord(e, st));
        }
    }
    void finish() {
        if (!on || keep) return;
        CK(cudaEventSynchronize(ev.back()));
        store_stage_times(idx, ev, names);
    }
    ~StageTimer() {
        for (auto e : ev) cudaEventDestroy(e);
    }
};

// Launches a kernel of the query path; with `chain`, as a programmatic dependent of the kernel before
// it on the stream: its launch and its blocks' start overlap that kernel's run.  Used for batches of
// up to kChainQueries queries, whose kernels are not much longer than a launch (one query: 67 -> 58
// us, with the prologue's searches side by side).
template <typename... P, typename... A>
void launch_next(bool chain, void (*kern)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = chain ? 1 : 0;
    CK(cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...));
}

template <typename K>
int occupancy_blocks(K kernel, int threads, size_t smem) {
    int nb = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, smem));
    return std::max(nb, 1);
}

}  // namespace

int sm_count() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        CK(cudaGetDevice(&dev));
        CK(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    }
    return n;
}

void allow_smem(const void* kernel) {
    static std::mutex mu;
    static std::map<const void*, int> fixed;  // the kernels' static shared memory (part of the code)
    int bytes;
    {
        std::lock_guard<std::mutex> g(mu);
        auto it = fixed.find(kernel);
        if (it == fixed.end()) {
            cudaFuncAttributes a;
            CK(cudaFuncGetAttributes(&a, kernel));
            it = fixed.emplace(kernel, (int)a.sharedSizeBytes).first;
        }
        bytes = (int)kBlockSmem - it->second;
    }
    CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}

struct QueryCall {
    const float* queries;
    uint64_t q;
    const float* qlabels;
    uint32_t label_cols;
    const float* data;
    uint32_t k;
    float* dist;
    uint64_t* ids;
    const uint32_t* qk;
    const uint32_t* qps;
    const uint8_t* qsched;
};

struct GraphEntry {
    uint64_t key[24];
    cudaGraphExec_t exec = nullptr;
    std::vector<cudaEvent_t> stage_ev;     // event-record nodes between the stages (break_down=1)
    std::vector<std::string> stage_names;
    uint64_t q = 0, launches = 0;
    int mode = 0;
    uint32_t k = 0;
};

struct GraphState {
    std::vector<GraphEntry> entries;
    cudaStream_t stream = nullptr;  // capture and replay stream
    cudaEvent_t ev_in = nullptr, ev_out = nullptr;
    uint64_t* pinned = nullptr;     // the last replay's scalars and GEMM status word (nine words)
    bool pending = false;
    GraphEntry last;                // description of the last replay (stats)
};

static void destroy_entry(GraphEntry& e) {
    if (e.exec) cudaGraphExecDestroy(e.exec);
    for (auto ev : e.stage_ev) cudaEventDestroy(ev);
    e.exec = nullptr;
    e.stage_ev.clear();
    e.stage_names.clear();
}

void release_graphs(GraphState* g) {
    if (!g) return;
    for (auto& e : g->entries) destroy_entry(e);
    if (g->ev_in) cudaEventDestroy(g->ev_in);
    if (g->ev_out) cudaEventDestroy(g->ev_out);
    if (g->stream) cudaStreamDestroy(g->stream);
    if (g->pinned) cudaFreeHost(g->pinned);
    delete g;
}

static void invalidate_ctx_graphs(QueryCtx& cx) {
    if (!cx.graphs) return;
    if (cx.graphs->pending) cudaEventSynchronize(cx.graphs->ev_out);
    for (auto& e : cx.graphs->entries) destroy_entry(e);
    cx.graphs->entries.clear();
    cx.graphs->pending = false;
}

void invalidate_graphs(hdg_index* idx) {
    std::lock_guard<std::mutex> g(idx->ctx_mu);
    for (auto& kv : idx->ctxs) {
        std::lock_guard<std::mutex> gc(kv.second->mu);
        invalidate_ctx_graphs(*kv.second);
    }
}

// The stats of a query from its batch scalars (scal of k_batch).
static void fill_stats(hdg_index* idx, uint64_t q, uint32_t k, int mode, uint64_t exps0, const uint64_t* sc,
                       uint64_t launches) {
    std::lock_guard<std::mutex> g(idx->stats_mu);
    const uint64_t coarse = sc[0], real = sc[1], max_row = sc[2];
    const uint32_t bb = (uint32_t)sc[4];
    float beta;
    std::memcpy(&beta, &bb, 4);
    if (mode != kPost) beta = 0.f;
    uint64_t K = k;  // the budget of a query with the batch k and the reference schedule
    if (mode == kPost) {
        if (real == 0) {
            K = max_row;
        } else {
            const float want = (float)(exps0 * (uint64_t)k) * beta;
            K = std::min<uint64_t>(want >= 1.8e19f ? ~0ull : (uint64_t)want, max_row);
        }
    } else if (mode == kL1) {
        K = exps0 * k;
    }
    idx->lazy_ctx = nullptr;  // these are the newest stats
    idx->last_ncand = K;  // no cap: the budget the reference computes is the one used
    idx->last_beta = beta;
    idx->last_q = q;
    uint32_t bits;
    std::memcpy(&bits, &beta, 4);
    const uint64_t s[10] = {q, idx->last_ncand, K, coarse, real, max_row, bits, (uint64_t)mode, launches, sc[5]};
    std::memcpy(idx->last_stats, s, sizeof(s));
}

// Reads back the scalars that the context's last call left on the device (cx.mu held) and, if
// they are still the index's newest, makes them its stats.
static void resolve_lazy(hdg_index* idx, QueryCtx& cx) {
    if (!cx.lazy.pending) return;
    cx.lazy.pending = false;
    {
        std::lock_guard<std::mutex> g(idx->stats_mu);
        if (idx->lazy_ctx != &cx) return;
    }
    uint64_t sc[8];
    CK(cudaEventSynchronize(cx.lazy.done));
    CK(cudaMemcpy(sc, cx.lazy.scal, sizeof(sc), cudaMemcpyDeviceToHost));
    fill_stats(idx, cx.lazy.q, cx.lazy.k, cx.lazy.mode, cx.lazy.exps0, sc, cx.lazy.launches);
}

// The estimate pass pays from this many candidates in the batch, on the average query and per
// selected one.  With it / without, us, at (candidates, per query, per selected): 30 M, 60,000, 6.4:
// 781 / 784; 117 M, 58,500, 6.2: 1,670 / 2,051; 74 M, 36,900, 6.7: 2,813 / 3,237; 60 M, 60,300, 21:
// 1,467 / 2,092; 46 M, 228,000, 23: 840 / 1,147; but 18 M, 36,700, 6.8: 1,161 / 1,108; 73 M, 14,600,
// 5.5: 3,499 / 3,425; 98 M, 24,600, 2.6: 2,362 / 2,345; 26 M, 5,200, 2.3: 2,314 / 2,029.
constexpr uint64_t kEstMinCands = 32ull << 20, kEstMinRow = 8192, kEstMinRatio = 6;

// Dynamic shared memory of the pass's kernels that hold a query's R candidate ranges
static size_t est_thr_smem(uint32_t G, int R) { return sizeof(uint32_t) * (G * kCodes * 16 + kThrMax + kThrBins + 2 * (size_t)R + 1); }
static size_t est_pick_smem(int R) { return sizeof(uint32_t) * (2 * (size_t)R + 1); }
// (with up to 10 KB of static tables beside them)
static bool est_fits(uint32_t G, int R) { return std::max(est_thr_smem(G, R), est_pick_smem(R)) + 10 * 1024 <= kBlockSmem; }

// Thresholds, row-tile entries (`entries` of them at most), estimates and the scan's work items of a
// batch of `cands` candidates.  False, and nothing enqueued, when its memory is not there.
static bool estimate_pass(hdg_index* idx, QueryCtx& cx, Workspace& w, const QueryCall& c, int R, uint32_t G,
                          uint64_t entries, uint64_t cands, cudaStream_t st) {
    const IndexDev& D = idx->dev;
    const uint64_t q = c.q;
    const uint32_t tiles = (D.n + kEstM - 1) / kEstM;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += align_up(bytes, 256);
        return o;
    };
    const size_t o_prq = take(q * 4), o_w = take(q * 4), o_in = take(q * 4), o_row = take(q * 4),
                 o_qc = take(q * sizeof(float4));
    const size_t o_diff = take((tiles + 1) * 4ull), o_eo = take((tiles + 1) * 4ull), o_no = take((tiles + 1) * 4ull),
                 o_cur = take((tiles + 1) * 4ull), o_ent = take(std::max<uint64_t>(entries, 1) * sizeof(uint4));
    // In the part of the rows that this batch leaves unused when it is large enough (the quarter more
    // of a batch of this size, or what a larger one left: then there may be no other memory), else in a
    // buffer of its own
    const size_t used = align_up(std::max<uint64_t>(cands, 1) * 4, 256);
    char* b = nullptr;
    if (cx.dist_buf.bytes >= used + off) {
        b = static_cast<char*>(cx.dist_buf.ptr) + used;
    } else {
        if (cx.est_buf.bytes < off) {
            cx.est_buf.reset();
            if (!cx.est_buf.try_ensure(off + off / 4) && !cx.est_buf.try_ensure(off)) return false;
        }
        b = static_cast<char*>(cx.est_buf.ptr);
    }
    w.prq = reinterpret_cast<uint32_t*>(b + o_prq);
    w.est_w = reinterpret_cast<int*>(b + o_w);
    w.est_in = reinterpret_cast<uint32_t*>(b + o_in);
    w.est_row = reinterpret_cast<uint32_t*>(b + o_row);
    w.est_qc = reinterpret_cast<float4*>(b + o_qc);
    int* diff = reinterpret_cast<int*>(b + o_diff);
    EstArgs a{};
    a.rowc = D.decoded_c;
    a.qc = w.est_qc;
    a.qb = static_cast<const uint16_t*>(w.qbf);
    a.ldq = D.d;
    a.n_rows = D.n;
    a.tiles = tiles;
    uint32_t* ent_off = reinterpret_cast<uint32_t*>(b + o_eo);
    uint32_t* nt_off = reinterpret_cast<uint32_t*>(b + o_no);
    uint32_t* cursor = reinterpret_cast<uint32_t*>(b + o_cur);
    uint4* ent = reinterpret_cast<uint4*>(b + o_ent);
    a.ent_off = ent_off;
    a.nt_off = nt_off;
    a.ent = ent;
    a.qoff = w.qoff;
    a.prow = w.spos;
    a.cnt = w.cand_count;
    CK(cudaMemsetAsync(diff, 0, (tiles + 1) * 4ull, st));
    const size_t sm = est_thr_smem(G, R);
    auto thr = [&](auto kern) {
        allow_smem(kern);
        kern<<<(unsigned)q, kThrThreads, sm, st>>>(D, R, c.queries, w);
        CK_LAUNCH();
    };
    if (G == 1) thr(k_est_thr<1>);
    else if (G == 2) thr(k_est_thr<2>);
    else thr(k_est_thr<3>);
    const unsigned blocks = (unsigned)((q * R + 255) / 256);
    k_est_count<<<blocks, 256, 0, st>>>(q, R, w, diff);
    CK_LAUNCH();
    k_est_scan<<<1, 1024, 0, st>>>(diff, tiles, ent_off, nt_off, cursor);
    CK_LAUNCH();
    k_est_fill<<<blocks, 256, 0, st>>>(q, R, w, cursor, ent);
    CK_LAUNCH();
    est_ranges(a, D.decoded, (int)D.d, w.gemm_err, st);
    allow_smem(k_est_pick);
    k_est_pick<<<(unsigned)q, kPickThreads, est_pick_smem(R), st>>>(R, w);
    CK_LAUNCH();
    k_scan_plan<<<1, 1024, 0, st>>>(q, w);
    CK_LAUNCH();
    return true;
}

// Enqueues one query batch on st.  sync_sizing: one host read after k_batch sizes the
// distance buffer and fills the stats (the plain path).  Otherwise nothing waits on the
// host (the CUDA-graph path): the distance buffer keeps its capacity, queries past it are
// cut by k_batch, and the scalars and the GEMM status word are copied to pinned memory.
static void enqueue_query(hdg_index* idx, QueryCtx& cx, const QueryCall& c, cudaStream_t st, bool sync_sizing,
                          uint64_t* pinned, uint64_t* launches_out, int* mode_out, uint64_t* coarse_out = nullptr,
                          uint64_t* sel_out = nullptr, GraphEntry* capture = nullptr) {
    const uint64_t q = c.q;
    const uint32_t k = c.k;
    HDG_REQUIRE(idx->built, HDG_ERR_STATE, "index not built");
    HDG_REQUIRE(q > 0 && q < (1ull << 31), HDG_ERR_INVALID_ARG, "query count out of range");
    HDG_REQUIRE(c.queries && c.qlabels && c.dist && c.ids, HDG_ERR_INVALID_ARG, "null pointer");
    HDG_REQUIRE(k >= 1 && k <= 2048, HDG_ERR_INVALID_ARG, "k must be in [1, 2048]");
    const hdg_params& P = idx->params;
    const IndexDev& D = idx->dev;
    const int l = (int)D.l;
    const int fd = (int)std::max<uint64_t>(1, P.filter_dim);
    HDG_REQUIRE(c.label_cols == (uint32_t)(l * fd), HDG_ERR_INVALID_ARG,
                "query label columns must equal l * filter_dim");
    const int Pc = (int)std::max<uint64_t>(1, P.n_list);
    const int Ps = (int)std::max<uint64_t>(1, P.sub_lists);
    HDG_REQUIRE(Pc <= 1024 && Ps <= 2048, HDG_ERR_UNSUPPORTED, "n_list <= 1024 and sub_lists <= 2048");
    HDG_REQUIRE(D.n_lists <= 32768, HDG_ERR_UNSUPPORTED, "at most 32768 inverted lists");
    const uint64_t exps0 = P.exps0;
    const int mode = exps0 <= 1 ? kPre : (l > 1 ? kPost : kL1);
    if (mode_out) *mode_out = mode;
    HDG_REQUIRE(mode == kPre || c.data, HDG_ERR_INVALID_ARG, "d_data is required for the re-rank");
    HDG_REQUIRE(mode != kPre || !c.qsched, HDG_ERR_INVALID_ARG,
                "per-query schedules need exps0 > 1 (the pre-filter schedule has no re-rank)");
    cx.lazy.pending = false;  // superseded by this call
    if (!cx.work.ptr || cx.work.bytes < workspace_bytes(idx, cx, q)) {
        HDG_REQUIRE(sync_sizing, HDG_ERR_STATE, "workspace too small for a captured query");
        reserve_ctx(idx, cx, q);
    }
    Workspace w = carve(idx, cx, q, true);
    const uint32_t G = lut_groups(D);
    const bool fast = (D.M % 32 == 0) && G <= 3;
    w.surv_list = fast ? 1 : 0;  // the fast path lists the predicate-first queries' survivors
    w.qk = c.qk;
    w.qps = c.qps;
    w.qsched = c.qsched;
    w.k_max = k;
    w.mode = mode;
    w.exps0 = (uint32_t)std::min<uint64_t>(exps0, 1u << 20);
    w.chunk = P.scan_chunk ? (uint32_t)std::min<uint64_t>(P.scan_chunk, 1u << 30) : kChunk;
    w.scan_items = 8 * (uint32_t)sm_count();
    w.cap = sync_sizing ? ~0ull : cx.dist_buf.bytes / 4;
    if (sync_sizing) w.sel_cap = ~0ull;  // sized after k_batch
    const FilterDev f = filter_dev(idx);
    // programmatic launches: small batches of the plain path (stage events would sit between them)
    const bool chain = sync_sizing && P.break_down == 0 && q <= kChainQueries;
    StageTimer tm(idx, st, P.break_down != 0 && (sync_sizing || capture), capture ? &capture->stage_ev : nullptr,
                  capture ? &capture->stage_names : nullptr);

    const size_t sm_pro = sizeof(uint32_t) * D.n_lists;
    if (sm_pro > 48 * 1024) allow_smem(k_prologue);
    uint64_t launches = 0;  // kernels of this query, reported in the stats
    launch_next(false, k_prologue, dim3((unsigned)q), kThreads, sm_pro, st, D, idx->grid, f, c.qlabels, (int)c.label_cols, w);
    CK_LAUNCH();
    launches++;
    tm.mark("prologue");
    const int sort_n1 = (int)next_pow2(std::max<uint32_t>(D.C, 2));
    const int sort_n2 = (int)next_pow2(std::max<uint32_t>((uint32_t)Pc * D.S_max, 2));
    const size_t sm_co = (sizeof(uint64_t) + sizeof(float)) * std::max(sort_n1, sort_n2) + sizeof(float) * D.d;
    HDG_REQUIRE(sm_co <= 200 * 1024, HDG_ERR_UNSUPPORTED, "coarse selection does not fit shared memory");
    if (sm_co > 48 * 1024)
        allow_smem(k_coarse);
    // tensor-core estimates of every query-centroid dot product, used to prune the exact
    // ranking when n_list or sub_lists leaves part of the candidates out (COARSE_BF16=1)
    const bool use_gemm = P.coarse_bf16 != 0 && D.d % 8 == 0 && (Pc < (int)D.C || Ps < Pc * (int)D.S_max);
    if (use_gemm) {
        rows_to_bf16(c.queries, q, (int)D.d, w.qbf, w.qnorm, st);
        umma_dot(w.qbf, q, D.centers_bf16, D.C, (int)D.d, w.S, w.ldS, w.gemm_err, st);
        umma_dot(w.qbf, q, D.sub_centers_bf16, D.n_lists, (int)D.d, w.S + D.C, w.ldS, w.gemm_err, st);
        launches += 3;
        tm.mark("coarse_gemm");
    } else {
        w.S = nullptr;
    }
    if (P.learned && !c.qps && !c.qsched) {
        // the learned schedule: per-query lists to probe and predicate-first flag
        HDG_REQUIRE(idx->mlp_ready, HDG_ERR_STATE, "LEARNED=1 but the index holds no trained model");
        // the features' 16 nearest centroids are pruned by the tensor-core products when present
        learned_features(idx, c.queries, q, w.box, w.cluster_counts, c.qk, k, w.feats, st, w.S, w.ldS, w.qnorm);
        learned_infer(idx, w.feats, q, w.lq_ps, w.lq_sched, mode != kPre, (uint32_t)Ps, nullptr, st);
        w.qps = w.lq_ps;
        w.qsched = mode != kPre ? w.lq_sched : nullptr;
        launches += 2;
        tm.mark("learned");
    }

    launch_next(chain && !use_gemm && !w.qps, k_coarse, dim3((unsigned)q), kCoarseThreads, sm_co, st, D, idx->grid, c.queries, Pc,
                Ps, sort_n1, sort_n2, w);
    CK_LAUNCH();
    launches++;
    tm.mark("coarse");

    // candidate offsets, work items, batch sums, beta and the per-query budgets' inputs
    launch_next(chain, k_batch, dim3(1), 1024, 0, st, q, w);
    CK_LAUNCH();
    launches++;
    uint64_t sc[10] = {0};  // the batch scalars, the GEMM status word, the row-tile sum
    // no host read: a small batch whose caller needs no totals and whose coarse stage has no
    // tensor-core status to report
    bool lazy = sync_sizing && !use_gemm && !coarse_out && P.break_down == 0 && q * (uint64_t)D.n <= kUnsizedPairs;
    if (lazy) {  // (a stream under capture is refused by the read below, as it always was)
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        CK(cudaStreamIsCapturing(st, &cap));
        lazy = cap == cudaStreamCaptureStatusNone;
    }
    const uint64_t pairs = q * (uint64_t)D.n;  // at most every point of every query
    if (lazy && !try_candidates(cx, q, k, pairs)) lazy = false;  // (its candidates may find room)
    if (sync_sizing) {
        if (lazy) {
            if (!cx.lazy.done) CK(cudaEventCreateWithFlags(&cx.lazy.done, cudaEventDisableTiming));
            CK(cudaEventRecord(cx.lazy.done, st));
        } else {
            // (one copy; to ordinary memory, since page-locking it costs a new context milliseconds)
            CK(cudaMemcpyAsync(sc, w.scal, sizeof(sc), cudaMemcpyDeviceToHost, st));
            CK(cudaStreamSynchronize(st));
            HDG_REQUIRE((uint32_t)sc[8] == 0, HDG_ERR_TIMEOUT, "tensor-core wait expired in the coarse GEMM");
            if (coarse_out) *coarse_out = sc[0];
            if (sel_out) *sel_out = sc[7];
            ensure_candidates(cx, q, k, sc[0], sc[7]);
        }
    } else {
        HDG_REQUIRE(cx.dist_buf.ptr && cx.sel_buf.ptr && cx.part_buf.bytes >= part_bytes(cx, q, k), HDG_ERR_STATE,
                    "no candidate buffers for a captured query");
    }
    w.dist = static_cast<float*>(cx.dist_buf.ptr);
    w.spos = static_cast<uint32_t*>(cx.pos_buf.ptr);
    w.cand_pool = static_cast<uint32_t*>(cx.sel_buf.ptr);
    w.rpart = static_cast<uint64_t*>(cx.part_buf.ptr);
    tm.mark("budget");

    const int pre = mode == kPre ? 1 : 0;
    // candidate ranges per query: one per probed list, or n_split per list when is_split
    const int R = Ps * w.nsplit;
    const size_t sm_tab = sizeof(uint32_t) * (2 * R + 1);
    const bool scanned = !sync_sizing || lazy || sc[3] > 0, pre_pass = fast && (pre || w.qsched);
    if (scanned) {
        if (pre_pass) {
            // the predicate pass of the predicate-first queries, then the ADC items that
            // follow from their survivors
            const bool lab4 = l == 4 && (reinterpret_cast<uintptr_t>(D.labels) & 15) == 0;
            auto launch_pre = [&](auto kern) {
                const size_t smp = sizeof(uint32_t) * kPreRingWords * (kPreThreads / 32);
                allow_smem(kern);
                const int blocks = sm_count() * occupancy_blocks(kern, kPreThreads, smp);
                kern<<<blocks, kPreThreads, smp, st>>>(D, R, l, q, w);
            };
            if (D.rank_planes) lab4 ? launch_pre(k_pre_scan<true, kPlaneTest>) : launch_pre(k_pre_scan<false, kPlaneTest>);
            else if (D.rankpack && !D.labels_nan) lab4 ? launch_pre(k_pre_scan<true, kRankTest>) : launch_pre(k_pre_scan<false, kRankTest>);
            else lab4 ? launch_pre(k_pre_scan<true, kLabelTest>) : launch_pre(k_pre_scan<false, kLabelTest>);
            CK_LAUNCH();
            k_scan_plan<<<1, 1024, 0, st>>>(q, w);
            CK_LAUNCH();
            launches += 2;
            tm.mark("predicate");
        }
        {
            // the LUTs of the queries that have ADC work items (a predicate-first query whose
            // budget takes every survivor has none)
            if (D.pq_len <= (uint32_t)kLutMaxPqLen) {
                const int slices = lut_slices(q, (int)G, sm_count());
                const size_t sm = sizeof(float) * (kCodes / slices) * D.pq_len * 33;
                allow_smem(k_lut);
                launch_next(chain && lazy && !pre_pass, k_lut, dim3((unsigned)((q + kLutQ - 1) / kLutQ), G, slices), 512, sm,
                            st, D, c.queries, q, (int)G, w.lut, w.lut16, w.item_off);
            } else {
                launch_next(false, k_lut_plain, dim3((unsigned)q, G), 256, sizeof(float) * D.d, st, D, c.queries, (int)G,
                            w.lut, w.lut16, w.item_off);
            }
            CK_LAUNCH();
            launches++;
            tm.mark("lut");
        }
        // post-filter queries with many more candidates than budget: the estimate pass (not in a
        // captured graph, whose entry count is not known)
        bool prune = sync_sizing && !lazy && mode == kPost && !w.qsched && fast && D.decoded && sc[0] >= kEstMinCands &&
                     sc[0] / q >= kEstMinRow && sc[0] >= kEstMinRatio * sc[7] && sc[2] < (1u << 24) && sc[9] < (1ull << 32) &&
                     est_fits(G, R);
        if (prune) prune = estimate_pass(idx, cx, w, c, R, G, sc[9], sc[0], st);
        if (prune) {
            launches += 7;
            tm.mark("estimate");
        }
        if (fast) {
            // threads x candidates-per-thread (SCAN_CPT, chosen by the autotuner; 0 = 1)
            const int cpt = (P.scan_cpt == 1 || P.scan_cpt == 2 || P.scan_cpt == 4) ? (int)P.scan_cpt : 1;
            const size_t sm = sizeof(float) * G * kCodes * 64 + sm_tab;
            HDG_REQUIRE(sm <= kBlockSmem, HDG_ERR_UNSUPPORTED, "scan tables exceed shared memory");
            auto launch = [&](auto kern, int nt) {
                allow_smem(kern);
                const int blocks = sm_count() * occupancy_blocks(kern, nt, sm);
                launch_next(chain && !prune, kern, dim3((unsigned)blocks), nt, sm, st, D, R, q, w);
            };
            if (G == 1) {
                if (cpt == 1) launch(k_scan_fast<1, 512, 1>, 512);
                else if (cpt == 2) launch(k_scan_fast<1, 512, 2>, 512);
                else launch(k_scan_fast<1, 256, 4>, 256);
            } else if (G == 2) {
                if (cpt == 1) launch(k_scan_fast<2, 512, 1>, 512);
                else if (cpt == 2) launch(k_scan_fast<2, 512, 2>, 512);
                else launch(k_scan_fast<2, 256, 4>, 256);
            } else {
                if (cpt == 1) launch(k_scan_fast<3, 1024, 1>, 1024);
                else if (cpt == 2) launch(k_scan_fast<3, 512, 2>, 512);
                else launch(k_scan_fast<3, 256, 4>, 256);
            }
        } else {
            const size_t sm = sizeof(float) * G * kCodes * 32 + sm_tab;
            HDG_REQUIRE(sm <= kBlockSmem, HDG_ERR_UNSUPPORTED, "scan tables exceed shared memory");
            allow_smem(k_scan_generic);
            const int blocks = sm_count() * occupancy_blocks(k_scan_generic, 512, sm);
            launch_next(chain, k_scan_generic, dim3((unsigned)blocks), 512, sm, st, D, (int)G, R, pre, l, q, w);
        }
        CK_LAUNCH();
        launches++;
    }
    tm.mark("scan");

    const int sorted_out = mode == kPre ? 1 : 0;
    const size_t sm_sel = sizeof(uint32_t) * kBins + sizeof(uint64_t) * kBCap +
                          (sorted_out ? sizeof(uint64_t) * next_pow2(std::max<uint32_t>(k, 2)) : 0) + sm_tab + 16;
    auto launch_sel = [&](auto kern, int nt) {
        allow_smem(kern);
        launch_next(chain && scanned, kern, dim3((unsigned)q), nt, sm_sel, st, D, R, (int)k, sorted_out, w, c.dist, c.ids, (int)k);
    };
    if (q <= (uint64_t)sm_count()) launch_sel(k_select<kSelThreadsFew, 8>, kSelThreadsFew);
    else launch_sel(k_select<kSelThreads, 4>, kSelThreads);
    CK_LAUNCH();
    launches++;
    tm.mark("select");
    if (mode != kPre) {
        launch_next(chain, k_refine_plan, dim3(1), 1024, 0, st, q, w);
        CK_LAUNCH();
        const int rcap = (int)next_pow2(k + 4 * kThreads);  // rounds of rcap - k exact distances
        const size_t sm_ref = sizeof(uint64_t) * rcap + sizeof(float) * D.d + 16;
        allow_smem(k_refine);
        // persistent over the refine items; no more CTAs than queries are useful for small batches
        const uint64_t blocks = std::min<uint64_t>((uint64_t)sm_count() * occupancy_blocks(k_refine, kThreads, sm_ref),
                                                   q + (cx.sel_buf.bytes / 4) / kRefChunk + 1);
        launch_next(chain, k_refine, dim3((unsigned)blocks), kThreads, sm_ref, st, D, c.queries, c.data, rcap,
                    mode == kPost ? 1 : 0, l, q, w, c.dist, c.ids, (int)k);
        CK_LAUNCH();
        launches += 2;
        tm.mark("refine");
    }
    if (!sync_sizing && pinned) {
        CK(cudaMemcpyAsync(pinned, w.scal, 9 * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    }
    if (launches_out) *launches_out = launches;
    if (lazy) {
        cx.lazy.pending = true;
        cx.lazy.scal = w.scal;
        cx.lazy.q = q;
        cx.lazy.k = k;
        cx.lazy.mode = mode;
        cx.lazy.exps0 = exps0;
        cx.lazy.launches = launches;
        std::lock_guard<std::mutex> g(idx->stats_mu);
        idx->lazy_ctx = &cx;
    } else if (sync_sizing) {
        fill_stats(idx, q, k, mode, exps0, sc, launches);
    }
    tm.finish();
}

static hdg_status finish_ctx(hdg_index* idx, QueryCtx& cx) {
    GraphState* g = cx.graphs;
    if (!g || !g->pending) return HDG_OK;
    CK(cudaEventSynchronize(g->ev_out));
    g->pending = false;
    fill_stats(idx, g->last.q, g->last.k, g->last.mode, idx->params.exps0, g->pinned, g->last.launches);
    if (!g->last.stage_ev.empty()) store_stage_times(idx, g->last.stage_ev, g->last.stage_names);
    if (static_cast<int>(g->pinned[8] & 0xffffffffu) != 0) return HDG_ERR_TIMEOUT;
    if (g->pinned[5] != 0) return HDG_ERR_OOM;
    return HDG_OK;
}

hdg_status finish_async_query(hdg_index* idx) {
    std::vector<QueryCtx*> all;
    {
        std::lock_guard<std::mutex> g(idx->ctx_mu);
        for (auto& kv : idx->ctxs) all.push_back(kv.second.get());
    }
    hdg_status worst = HDG_OK;
    for (QueryCtx* cx : all) {
        std::lock_guard<std::mutex> g(cx->mu);
        const hdg_status s = finish_ctx(idx, *cx);
        resolve_lazy(idx, *cx);
        if (worst == HDG_OK) worst = s;
    }
    return worst;
}

static void make_graph_key(const hdg_index* idx, const QueryCtx& cx, const QueryCall& c, uint64_t* key) {
    const hdg_params& P = idx->params;
    const uint64_t v[24] = {(uint64_t)c.queries, c.q, (uint64_t)c.qlabels, c.label_cols, (uint64_t)c.data, c.k,
                            (uint64_t)c.dist, (uint64_t)c.ids, (uint64_t)c.qk, (uint64_t)c.qps, (uint64_t)c.qsched,
                            (uint64_t)cx.work.ptr, cx.work.bytes, (uint64_t)cx.dist_buf.ptr,
                            cx.dist_buf.bytes, P.n_list, P.sub_lists, P.exps0, P.lut_fp16, P.coarse_bf16,
                            P.scan_cpt, P.scan_chunk, P.filter_dim, P.learned | (P.is_split << 8) | (P.n_split << 16)};
    std::memcpy(key, v, sizeof(v));
}

static void query_once(hdg_index* idx, const QueryCall& c, cudaStream_t st) {
    const uint64_t q = c.q;
    const uint32_t k = c.k;
    QueryCtx& cx = query_ctx(idx, st);
    std::lock_guard<std::mutex> lock(cx.mu);  // one query at a time per stream
    if (idx->params.query_graph == 0) {
        finish_ctx(idx, cx);
        enqueue_query(idx, cx, c, st, true, nullptr, nullptr, nullptr);
        return;
    }
    if (!cx.graphs) {
        GraphState* g = new GraphState();
        cx.graphs = g;
        CK(cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking));
        CK(cudaEventCreateWithFlags(&g->ev_in, cudaEventDisableTiming));
        CK(cudaEventCreateWithFlags(&g->ev_out, cudaEventDisableTiming));
        CK(cudaMallocHost(reinterpret_cast<void**>(&g->pinned), 16 * sizeof(uint64_t)));
        std::memset(g->pinned, 0, 16 * sizeof(uint64_t));
    }
    GraphState* g = cx.graphs;
    finish_ctx(idx, cx);  // the pinned status words are reused by this replay
    uint64_t key[24];
    make_graph_key(idx, cx, c, key);
    GraphEntry* hit = nullptr;
    for (auto& e : g->entries)
        if (std::memcmp(e.key, key, sizeof(key)) == 0) hit = &e;
    if (!hit) {
        // first call of this shape: the plain path computes this call's results and sizes
        // the buffers; the captured graph serves the next calls
        uint64_t coarse = 0, selected = 0;
        enqueue_query(idx, cx, c, st, true, nullptr, nullptr, nullptr, &coarse, &selected);
        const uint64_t need = std::max<uint64_t>(coarse, 1) * 4 * 5 / 4;  // 1.25x this batch
        const uint64_t need_sel = std::max<uint64_t>(selected, 1) * 4 * 5 / 4;
        if (cx.dist_buf.bytes < need || cx.sel_buf.bytes < need_sel) {
            invalidate_ctx_graphs(cx);
            if (cx.dist_buf.bytes < need) resize_rows(cx, need);
            if (cx.sel_buf.bytes < need_sel) {
                cx.sel_buf.reset();
                cx.sel_buf.try_ensure(need_sel);
            }
        }
        ensure_candidates(cx, q, k, coarse, selected);  // without the quarter, where it was not there
        make_graph_key(idx, cx, c, key);
        CK(cudaStreamSynchronize(st));
        GraphEntry e;
        std::memcpy(e.key, key, sizeof(key));
        cudaGraph_t graph = nullptr;
        CK(cudaStreamBeginCapture(g->stream, cudaStreamCaptureModeRelaxed));
        try {
            enqueue_query(idx, cx, c, g->stream, false, g->pinned, &e.launches, &e.mode, nullptr, nullptr, &e);
        } catch (...) {
            cudaStreamEndCapture(g->stream, &graph);
            if (graph) cudaGraphDestroy(graph);
            destroy_entry(e);
            throw;
        }
        CK(cudaStreamEndCapture(g->stream, &graph));
        const cudaError_t ie = cudaGraphInstantiate(&e.exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ie != cudaSuccess) destroy_entry(e);
        CK(ie);
        e.q = q;
        e.k = k;
        if (g->entries.size() >= 8) {
            destroy_entry(g->entries.front());
            g->entries.erase(g->entries.begin());
        }
        g->entries.push_back(e);
        return;
    }
    CK(cudaEventRecord(g->ev_in, st));
    CK(cudaStreamWaitEvent(g->stream, g->ev_in, 0));
    CK(cudaGraphLaunch(hit->exec, g->stream));
    CK(cudaEventRecord(g->ev_out, g->stream));
    CK(cudaStreamWaitEvent(st, g->ev_out, 0));
    g->last = *hit;
    g->pending = true;
    cx.lazy.pending = false;
    std::lock_guard<std::mutex> gs(idx->stats_mu);
    idx->lazy_ctx = nullptr;
}

void run_query(hdg_index* idx, const float* d_queries, uint64_t q, const float* d_query_labels,
               uint32_t label_cols, const float* d_data, uint32_t k, float* d_dist, uint64_t* d_ids,
               cudaStream_t st, const uint32_t* d_k, const uint32_t* d_nprobe, const uint8_t* d_sched) {
    const QueryCall c{d_queries, q, d_query_labels, label_cols, d_data, k, d_dist, d_ids, d_k, d_nprobe, d_sched};
    with_room(idx, [&] { query_once(idx, c, st); });
}

static void features_once(hdg_index* idx, const float* d_queries, uint64_t q, const float* d_query_labels,
                          uint32_t label_cols, const uint32_t* d_k, uint32_t k_max, float* d_feats, cudaStream_t st) {
    HDG_REQUIRE(idx->built, HDG_ERR_STATE, "index not built");
    HDG_REQUIRE(q > 0 && q < (1ull << 31), HDG_ERR_INVALID_ARG, "query count out of range");
    HDG_REQUIRE(d_queries && d_query_labels && d_feats, HDG_ERR_INVALID_ARG, "null pointer");
    const IndexDev& D = idx->dev;
    const int fd = (int)std::max<uint64_t>(1, idx->params.filter_dim);
    HDG_REQUIRE(label_cols == (uint32_t)(D.l * fd), HDG_ERR_INVALID_ARG,
                "query label columns must equal l * filter_dim");
    QueryCtx& cx = query_ctx(idx, st);
    std::lock_guard<std::mutex> lock(cx.mu);
    resolve_lazy(idx, cx);  // this call lays the workspace out for its own q
    if (!cx.work.ptr || cx.work.bytes < workspace_bytes(idx, cx, q)) reserve_ctx(idx, cx, q);
    Workspace w = carve(idx, cx, q, true);
    const FilterDev f = filter_dev(idx);
    const size_t sm_pro = sizeof(uint32_t) * D.n_lists;
    if (sm_pro > 48 * 1024) allow_smem(k_prologue);
    k_prologue<<<(unsigned)q, kThreads, sm_pro, st>>>(D, idx->grid, f, d_query_labels, (int)label_cols, w);
    CK_LAUNCH();
    learned_features(idx, d_queries, q, w.box, w.cluster_counts, d_k, k_max, d_feats, st);
}

void query_features(hdg_index* idx, const float* d_queries, uint64_t q, const float* d_query_labels,
                    uint32_t label_cols, const uint32_t* d_k, uint32_t k_max, float* d_feats, cudaStream_t st) {
    with_room(idx, [&] { features_once(idx, d_queries, q, d_query_labels, label_cols, d_k, k_max, d_feats, st); });
}

static void autotune_once(hdg_index* idx, const QueryCall& c, cudaStream_t st, float* best_ms) {
    hdg_params& P = idx->params;
    const uint64_t saved_bd = P.break_down, saved_graph = P.query_graph;
    P.break_down = 1;
    P.query_graph = 0;
    float best = INFINITY;
    uint64_t best_cpt = 1, best_chunk = kChunk;
    QueryCtx& cx = query_ctx(idx, st);
    std::unique_lock<std::mutex> lock(cx.mu);
    try {
        enqueue_query(idx, cx, c, st, true, nullptr, nullptr, nullptr);  // warm-up, buffers sized
        const uint64_t cpts[3] = {1, 2, 4};
        // the default first: another variant has to be a percent faster (on a small batch, whose items
        // are below every one of these sizes, they are all the same)
        const uint64_t chunks[4] = {kChunk, 8192, 16384, 65536};
        for (uint64_t cpt : cpts)
            for (uint64_t ch : chunks) {
                P.scan_cpt = cpt;
                P.scan_chunk = ch;
                float t = INFINITY;
                for (int rep = 0; rep < 2; rep++) {  // the faster of two runs
                    enqueue_query(idx, cx, c, st, true, nullptr, nullptr, nullptr);
                    float s = 0.f;
                    std::lock_guard<std::mutex> gs(idx->stats_mu);
                    for (size_t i = 0; i < idx->stage_names.size(); i++)
                        if (idx->stage_names[i] == "scan") s = idx->stage_ms[i];
                    t = std::min(t, s);
                }
                if (t < 0.99f * best) {
                    best = t;
                    best_cpt = cpt;
                    best_chunk = ch;
                }
            }
    } catch (...) {
        P.break_down = saved_bd;
        P.query_graph = saved_graph;
        throw;
    }
    P.scan_cpt = best_cpt;
    P.scan_chunk = best_chunk;
    P.break_down = saved_bd;
    P.query_graph = saved_graph;
    lock.unlock();
    invalidate_graphs(idx);
    if (best_ms) *best_ms = best;
}

void autotune_query(hdg_index* idx, const float* d_queries, uint64_t q, const float* d_query_labels,
                    uint32_t label_cols, const float* d_data, uint32_t k, float* d_dist, uint64_t* d_ids,
                    cudaStream_t st, float* best_ms) {
    const QueryCall c{d_queries, q, d_query_labels, label_cols, d_data, k, d_dist, d_ids, nullptr, nullptr, nullptr};
    with_room(idx, [&] { autotune_once(idx, c, st, best_ms); });
}

}  // namespace hdg
