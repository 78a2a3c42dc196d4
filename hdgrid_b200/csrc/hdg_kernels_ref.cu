// Kernel-level entry points that keep the reference kernels' data layouts, so the
// reference's known-answer tests (src/verification/test_*.cuh) can run through the GPU.
//   pq_lut          build_pq_lut_kernel            (src/index/product-quantization.cu:4-35)
//   pq_adc          compute_batched_L2_distance_kernel (product-quantization.cu:37-77)
//   label_mask      label_matrix_by_filter_indices_kernel (src/core/filter.cu:30-64)
//   recover_filters denormalize_labels_kernel      (src/core/preprocessing.cu:3-32)
//   bruteforce_knn  brute_forece_vector_search     (src/verification/ground_truth.cuh:165-232),
//                   with the filter.conf predicate instead of its hard-coded window.
#include <algorithm>
#include <cfloat>
#include <mutex>
#include <type_traits>
#include <vector>

#include <cuda_fp16.h>

#include "hdg_device.cuh"
#include "hdg_est.cuh"
#include "hdg_internal.h"

namespace hdg {

static unsigned nblk(uint64_t n, unsigned per) { return (unsigned)((n + per - 1) / per); }

// One block per query and 256 (subspace, codeword) pairs: the query index is uniform over the
// block, so an element costs one 32-bit division (it was three 64-bit ones).  Write-bound.
__global__ void k_pq_lut(const float* __restrict__ centers, const float* __restrict__ queries, uint32_t tiles,
                         uint32_t n_dim, uint32_t pq_dim, uint32_t pq_len, uint32_t n_codes,
                         float* __restrict__ lut) {
    const uint64_t q = blockIdx.x / tiles;
    const uint64_t row = (uint64_t)pq_dim * n_codes;
    const uint64_t e = (uint64_t)(blockIdx.x % tiles) * blockDim.x + threadIdx.x;
    if (e >= row) return;
    const uint32_t m = row <= 0xffffffffull ? (uint32_t)e / n_codes : (uint32_t)(e / n_codes);
    const float* c = centers + e * pq_len;
    const float* x = queries + q * n_dim + (uint64_t)m * pq_len;
    float s = 0.f;
    for (uint32_t t = 0; t < pq_len; t++) {
        if (m * pq_len + t >= n_dim) break;
        const float df = __fsub_rn(__ldg(c + t), __ldg(x + t));
        s = fmaf(df, df, s);
    }
    lut[q * row + e] = s;
}

__global__ void k_pq_adc(const uint8_t* __restrict__ codebook, uint64_t tot_data, const float* __restrict__ lut,
                         uint64_t nq, uint32_t pq_dim, uint32_t n_codes, const uint64_t* __restrict__ indices,
                         uint64_t n_cand, float* __restrict__ dist) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nq * n_cand) return;
    const uint64_t q = e / n_cand, j = e % n_cand;
    const uint64_t idx = indices ? indices[e] : j;
    if (idx >= tot_data) {
        dist[e] = FLT_MAX;
        return;
    }
    float s = 0.f;
    for (uint32_t m = 0; m < pq_dim; m++)
        s += lut[(q * pq_dim + m) * n_codes + codebook[(uint64_t)m * tot_data + idx]];
    dist[e] = s;
}

// ADC of candidates 0 .. n_cand-1 (no index list) over 256-entry tables: every query scores the
// same candidates.  A block holds the tables of QB queries in shared memory as one vector of QB
// floats per (codeword, subspace), rows of MP vectors; a warp takes 128 candidates at a time,
// stages their code bytes (coalesced rows of the column-major codebook) and gives each lane four
// consecutive ones, whose codes of a subspace are one word.  Lane r starts at subspace r and goes
// round, so the lanes of a warp read different banks whatever their codes are, and one lookup
// serves QB queries.  The (query group, tile) pairs are cut into one equal span per block, so
// that no SM is left idle by the number of groups; a block reloads the table where its span
// crosses into the next group.
// Bound: the shared-memory bandwidth of the lookups, 4 bytes per (query, candidate, subspace).
// 100 queries x 500,000 candidates x 32 subspaces: table in global memory 1,290 us, this
// kernel with one byte read per lane and a fixed number of blocks per group 436 us, as it
// stands 310 us.
template <int QB>
struct LutVec;
template <>
struct LutVec<1> {
    using T = float;
};
template <>
struct LutVec<2> {
    using T = float2;
};
template <>
struct LutVec<4> {
    using T = float4;
};
constexpr int kAdcThreads = 512, kAdcTile = 128;
static uint32_t adc_pitch(uint32_t m) { return (m + 7) / 8 * 8; }  // vectors per table row
static size_t adc_smem(uint32_t m, int qb) {
    return (size_t)256 * adc_pitch(m) * qb * 4 + (size_t)(kAdcThreads / 32) * m * kAdcTile;
}

// (a0, a1) += (b0, b1) as one packed FP32x2 add (each rounded to nearest, like two adds)
__device__ __forceinline__ void add2(float& a0, float& a1, float b0, float b1) {
    asm("{\n\t.reg .b64 ra, rb;\n\tmov.b64 ra, {%0, %1};\n\tmov.b64 rb, {%2, %3};\n\t"
        "add.rn.f32x2 ra, ra, rb;\n\tmov.b64 {%0, %1}, ra;\n\t}"
        : "+f"(a0), "+f"(a1)
        : "f"(b0), "f"(b1));
}

template <int QB>
__global__ void __launch_bounds__(kAdcThreads) k_pq_adc_all(const uint8_t* __restrict__ codebook, uint64_t tot_data,
                                                            const float* __restrict__ lut, uint64_t nq, uint32_t m,
                                                            uint32_t mp, uint64_t n_cand, float* __restrict__ dist) {
    using V = typename LutVec<QB>::T;
    extern __shared__ __align__(16) unsigned char smem_adc[];
    V* s_lut = reinterpret_cast<V*>(smem_adc);  // [256][mp]
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nw = kAdcThreads / 32;
    // [m][32] words of this warp: word `lane` of a row holds the codes of the lane's candidates
    uint32_t* s_code = reinterpret_cast<uint32_t*>(smem_adc + (size_t)256 * mp * sizeof(V)) + (size_t)warp * m * 32;
    const bool words = (tot_data & 3) == 0 && (reinterpret_cast<uintptr_t>(codebook) & 3) == 0;
    const bool vec = (n_cand & 3) == 0 && (reinterpret_cast<uintptr_t>(dist) & 15) == 0;
    const uint64_t tiles = (n_cand + kAdcTile - 1) / kAdcTile, total = (nq + QB - 1) / QB * tiles;
    const uint64_t b = blockIdx.x, nb = gridDim.x;
    uint64_t at = total / nb * b + min(b, total % nb);
    const uint64_t end = at + total / nb + (b < total % nb ? 1 : 0);
    const uint32_t start = (uint32_t)lane % m;
    while (at < end) {
        const uint64_t group = at / tiles, stop = min(end, (group + 1) * tiles), q0 = group * QB;
        const int nqb = (int)min((uint64_t)QB, nq - q0);
        __syncthreads();  // the previous group's lookups are done
        for (uint32_t e = t; e < m * 256u; e += kAdcThreads) {
            const uint32_t mm = e >> 8, c = e & 255u;
            float v[QB];
#pragma unroll
            for (int i = 0; i < QB; i++) v[i] = i < nqb ? __ldg(lut + ((q0 + i) * m + mm) * 256 + c) : 0.f;
            s_lut[c * mp + mm] = *reinterpret_cast<const V*>(v);
        }
        __syncthreads();
        for (uint64_t tile = at + warp; tile < stop; tile += nw) {
            const uint64_t j0 = (tile - group * tiles) * kAdcTile;
            const int cnt = (int)min((uint64_t)kAdcTile, n_cand - j0);
            // candidates past the data set score FLT_MAX and read no code
            const int real = j0 >= tot_data ? 0 : (int)min((uint64_t)cnt, tot_data - j0);
            __syncwarp();
            if (words && real == kAdcTile) {
                const uint32_t* src = reinterpret_cast<const uint32_t*>(codebook + j0) + lane;
#pragma unroll 4
                for (uint32_t mm = 0; mm < m; mm++) s_code[mm * 32 + lane] = __ldg(src + mm * (tot_data / 4));
            } else {
                for (uint32_t mm = 0; mm < m; mm++) {
                    uint32_t w = 0;
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const int j = 4 * lane + u;
                        if (j < real) w |= (uint32_t)__ldg(codebook + (uint64_t)mm * tot_data + j0 + j) << (8 * u);
                    }
                    s_code[mm * 32 + lane] = w;
                }
            }
            __syncwarp();
            float acc[4][QB];
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int i = 0; i < QB; i++) acc[u][i] = 0.f;
            uint32_t mm = start;
#pragma unroll 2
            for (uint32_t s = 0; s < m; s++) {
                const uint32_t w = s_code[mm * 32 + lane];
                const V* row = s_lut + mm;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const V v = row[((w >> (8 * u)) & 255u) * mp];
                    const float* f = reinterpret_cast<const float*>(&v);
                    if constexpr (QB == 1) acc[u][0] += f[0];
#pragma unroll
                    for (int i = 0; i + 1 < QB; i += 2) add2(acc[u][i], acc[u][i + 1], f[i], f[i + 1]);
                }
                mm = mm + 1 == m ? 0 : mm + 1;
            }
#pragma unroll
            for (int i = 0; i < QB; i++) {
                if (i >= nqb) break;
                float* o = dist + (q0 + i) * n_cand + j0 + 4 * lane;
                if (vec && real == kAdcTile) {
                    *reinterpret_cast<float4*>(o) = make_float4(acc[0][i], acc[1][i], acc[2][i], acc[3][i]);
                } else {
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (4 * lane + u < cnt) o[u] = 4 * lane + u < real ? acc[u][i] : FLT_MAX;
                }
            }
        }
        at = stop;
    }
}

// Label mask of candidates 0 .. n_cand-1 (no index list), at most kMaxDims label dims: a thread
// keeps the labels of four consecutive candidates in registers and tests them against up to 64
// queries' boxes from shared memory, so a label row is read once per 64 queries.  Bound: the
// mask's writes (16-byte stores when the rows are aligned).
constexpr int kMaskQ = 64, kMaskThreads = 256;
template <int LT>  // label dims; 0: l at run time
__global__ void __launch_bounds__(kMaskThreads) k_label_mask_all(const float* __restrict__ ranges,
                                                                 const float* __restrict__ labels, uint32_t l_rt,
                                                                 uint64_t n_data, uint64_t nq, uint64_t n_cand,
                                                                 uint32_t blocks_x, int32_t* __restrict__ mask) {
    constexpr int LM = LT ? LT : kMaxDims;
    const int l = LT ? LT : (int)l_rt;
    __shared__ float s_r[kMaskQ][2 * LM];
    const uint64_t q0 = (uint64_t)(blockIdx.x / blocks_x) * kMaskQ;
    const int nqb = (int)min((uint64_t)kMaskQ, nq - q0);
    for (int e = threadIdx.x; e < nqb * 2 * l; e += kMaskThreads) s_r[e / (2 * l)][e % (2 * l)] = ranges[q0 * 2 * l + e];
    __syncthreads();
    const uint64_t j0 = ((uint64_t)(blockIdx.x % blocks_x) * kMaskThreads + threadIdx.x) * 4;
    if (j0 >= n_cand) return;
    float lab[4][LM];
    bool in[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        in[u] = j0 + u < n_cand && j0 + u < n_data;
#pragma unroll
        for (int i = 0; i < LM; i++) lab[u][i] = in[u] && i < l ? __ldg(labels + (j0 + u) * l + i) : 0.f;
    }
    const bool vec = (n_cand & 3) == 0 && (reinterpret_cast<uintptr_t>(mask) & 15) == 0;
    for (int qq = 0; qq < nqb; qq++) {
        int ok[4];
#pragma unroll
        for (int u = 0; u < 4; u++) ok[u] = in[u] ? 1 : 0;
#pragma unroll
        for (int i = 0; i < LM; i++) {
            if (i >= l) break;
            const float lo = s_r[qq][2 * i], hi = s_r[qq][2 * i + 1];
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (lab[u][i] < lo || lab[u][i] > hi) ok[u] = 0;
        }
        int32_t* o = mask + (q0 + qq) * n_cand + j0;
        if (vec) {
            *reinterpret_cast<int4*>(o) = make_int4(ok[0], ok[1], ok[2], ok[3]);
        } else {
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (j0 + u < n_cand) o[u] = ok[u];
        }
    }
}

__global__ void k_label_mask(const float* __restrict__ ranges, const float* __restrict__ labels, uint32_t l,
                             uint64_t n_data, uint64_t nq, const uint64_t* __restrict__ indices,
                             uint64_t n_cand, int32_t* __restrict__ mask) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nq * n_cand) return;
    const uint64_t q = e / n_cand, j = e % n_cand;
    const uint64_t idx = indices ? indices[e] : j;
    if (idx >= n_data) {
        mask[e] = 0;
        return;
    }
    int ok = 1;
    for (uint32_t i = 0; i < l; i++) {
        const float v = labels[idx * l + i];
        if (v < ranges[q * 2 * l + 2 * i] || v > ranges[q * 2 * l + 2 * i + 1]) {
            ok = 0;
            break;
        }
    }
    mask[e] = ok;
}

__global__ void k_recover(FilterDev f, const float* __restrict__ qlabels, uint64_t nq, float* __restrict__ out) {
    const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nq) return;
    for (int i = 0; i < f.l; i++) {
        float lo, hi;
        recover_dim(f, qlabels + q * f.l * f.filter_dim, i, &lo, &hi);
        out[q * 2 * f.l + 2 * i] = lo;
        out[q * 2 * f.l + 2 * i + 1] = hi;
    }
}

void pq_lut(const float* centers, const float* queries, uint64_t nq, uint32_t n_dim, uint32_t pq_dim,
            uint32_t pq_len, uint32_t n_codes, float* lut, cudaStream_t st) {
    const uint64_t row = (uint64_t)pq_dim * n_codes, tiles = (row + 255) / 256;
    if (!nq || !row) return;
    const uint64_t step = std::max<uint64_t>(1, 0x7fffffffull / tiles);  // queries per launch (grid limit)
    for (uint64_t q0 = 0; q0 < nq; q0 += step) {
        const uint64_t nb = std::min(step, nq - q0);
        k_pq_lut<<<(unsigned)(nb * tiles), 256, 0, st>>>(centers, queries + q0 * n_dim, (uint32_t)tiles, n_dim, pq_dim,
                                                         pq_len, n_codes, lut + q0 * row);
        CK_LAUNCH();
    }
}
void pq_adc(const uint8_t* codebook, uint64_t tot_data, const float* lut, uint64_t nq, uint32_t pq_dim,
            uint32_t n_codes, const uint64_t* indices, uint64_t n_cand, float* dist, cudaStream_t st) {
    if (!nq || !n_cand) return;
    // all candidates, 256-entry tables that fit shared memory: as many queries per table as fit,
    // but no more than there are; a candidate list or another table size: k_pq_adc
    if (!indices && n_codes == 256 && pq_dim >= 1 && nq <= 0x7fffffffull) {
        auto launch = [&](auto kern, int qb) {
            const size_t sm = adc_smem(pq_dim, qb);
            allow_smem(kern);
            int occ = 0;
            CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kAdcThreads, sm));
            // one span of tiles per resident block, no block with fewer tiles than warps
            const uint64_t total = (nq + qb - 1) / qb * ((n_cand + kAdcTile - 1) / kAdcTile), nw = kAdcThreads / 32;
            const uint64_t blocks = std::min<uint64_t>((uint64_t)sm_count() * std::max(occ, 1), (total + nw - 1) / nw);
            kern<<<(unsigned)blocks, kAdcThreads, sm, st>>>(codebook, tot_data, lut, nq, pq_dim, adc_pitch(pq_dim),
                                                            n_cand, dist);
            CK_LAUNCH();
        };
        if (nq >= 3 && adc_smem(pq_dim, 4) <= kBlockSmem) return launch(k_pq_adc_all<4>, 4);
        if (nq >= 2 && adc_smem(pq_dim, 2) <= kBlockSmem) return launch(k_pq_adc_all<2>, 2);
        if (adc_smem(pq_dim, 1) <= kBlockSmem) return launch(k_pq_adc_all<1>, 1);
    }
    k_pq_adc<<<nblk(nq * n_cand, 256), 256, 0, st>>>(codebook, tot_data, lut, nq, pq_dim, n_codes, indices,
                                                      n_cand, dist);
    CK_LAUNCH();
}
void label_mask(const float* ranges, const float* labels, uint32_t l, uint64_t n_data, uint64_t nq,
                const uint64_t* indices, uint64_t n_cand, int32_t* mask, cudaStream_t st) {
    if (!nq || !n_cand) return;
    if (!indices && l >= 1 && l <= (uint32_t)kMaxDims) {
        const uint64_t bx = (n_cand + 4 * kMaskThreads - 1) / (4 * kMaskThreads), by = (nq + kMaskQ - 1) / kMaskQ;
        if (bx * by <= 0x7fffffffull) {
            auto kern = l == 4 ? k_label_mask_all<4> : k_label_mask_all<0>;
            kern<<<(unsigned)(bx * by), kMaskThreads, 0, st>>>(ranges, labels, l, n_data, nq, n_cand, (uint32_t)bx, mask);
            CK_LAUNCH();
            return;
        }
    }
    k_label_mask<<<nblk(nq * n_cand, 256), 256, 0, st>>>(ranges, labels, l, n_data, nq, indices, n_cand, mask);
    CK_LAUNCH();
}
// The interval map as a kernel argument: no device copy, allocation or synchronisation for a map
// of up to kMapArg entries (a cudaMalloc, a copy, a synchronisation and a cudaFree per call, each
// of which waits for or stalls the streams' other work, before)
struct MapArg {
    float v[kMapArg];
};
__global__ void k_recover_arg(FilterDev f, const __grid_constant__ MapArg map, const float* __restrict__ qlabels,
                              uint64_t nq, float* __restrict__ out) {
    const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nq) return;
    f.map = map.v;
    for (int i = 0; i < f.l; i++) {
        float lo, hi;
        recover_dim(f, qlabels + q * f.l * f.filter_dim, i, &lo, &hi);
        out[q * 2 * f.l + 2 * i] = lo;
        out[q * 2 * f.l + 2 * i + 1] = hi;
    }
}

void recover_filters_arg(const FilterDev& f, const float* host_map, const float* qlabels, uint64_t nq, float* ranges,
                         cudaStream_t st) {
    if (!nq) return;
    MapArg m;
    for (int i = 0; i < kMapArg; i++) m.v[i] = i < f.n_map ? host_map[i] : 0.f;
    k_recover_arg<<<nblk(nq, 128), 128, 0, st>>>(f, m, qlabels, nq, ranges);
    CK_LAUNCH();
}

void recover_filters(const FilterDev& f, const float* qlabels, uint64_t nq, float* ranges, cudaStream_t st) {
    if (!nq) return;
    k_recover<<<nblk(nq, 128), 128, 0, st>>>(f, qlabels, nq, ranges);
    CK_LAUNCH();
}

// ---- allocation-free filter recovery ---------------------------------------------------
// Scratch for the interval-map table of hdg_recover_filters_noalloc: a fixed array in the
// library's own device memory, present on every GPU that loads the library until the
// process exits.  Host code must not pass `g_noalloc_map` itself to a kernel (on the host it
// is only a stand-in symbol); it passes the device address fetched below.
static __device__ __align__(256) float g_noalloc_map[HDG_NOALLOC_MAP_MAX];

namespace {
std::mutex g_noalloc_mu;
std::vector<float*> g_noalloc_ptr;  // per device ordinal, filled on first use
}  // namespace

// Device address of the scratch array on the current device.  The first call on a device
// resolves it with cudaGetSymbolAddress (that device must be current); later calls reuse it.
static float* noalloc_map_scratch() {
    int dev = 0;
    CK(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if ((int)g_noalloc_ptr.size() <= dev) g_noalloc_ptr.resize(dev + 1, nullptr);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        CK(cudaGetSymbolAddress(&p, g_noalloc_map));
        g_noalloc_ptr[dev] = static_cast<float*>(p);
    }
    return g_noalloc_ptr[dev];
}

void recover_filters_noalloc(const FilterDev& f0, const float* host_map, const float* qlabels, uint64_t nq,
                             float* ranges, cudaStream_t st) {
    HDG_REQUIRE(f0.n_map >= 0 && f0.n_map <= HDG_NOALLOC_MAP_MAX, HDG_ERR_INVALID_ARG,
                "interval map of " + std::to_string(f0.n_map) + " entries exceeds the " +
                    std::to_string(HDG_NOALLOC_MAP_MAX) + "-entry limit of hdg_recover_filters_noalloc");
    FilterDev f = f0;
    f.map = noalloc_map_scratch();
    // the whole used prefix is rewritten every call, so nothing has to start at zero
    if (f.n_map) CK(cudaMemcpyAsync(const_cast<float*>(f.map), host_map, sizeof(float) * f.n_map,
                                    cudaMemcpyHostToDevice, st));
    recover_filters(f, qlabels, nq, ranges, st);
}

// ---- filtered exact kNN ------------------------------------------------------------------
// An item is a group of queries and a span of base rows; a block of 16 warps streams the span
// through shared memory in tiles of R rows (two tiles, copied ahead by cp.async).  A warp owns
// `own` queries (or, with fewer queries than warps, a share of every tile's rows of one query): it
// tests the tile's labels first, packs the rows that pass into a list and only then computes
// distances, one (query, row) pair per lane, in dimension order as one FMA chain.  A key below the
// query's running k-th goes to the query's buffer, which a warp sort cuts back to k when it fills.
// An item leaves its k best keys per query; k_bf_merge takes the k smallest over the spans (with one
// span, where there is no memory for the keys, they are the answer).
// Bound: with many queries the shared-memory reads of the passing rows (16 bytes per pair and four
// dimensions), with few the read of the base set.
// One block per 32 queries that computed every pair and tested the labels afterwards took 352 ms
// on 1,000 queries x 1 M x 128 (32 blocks, 10 % of the pairs pass); this takes 19.1 ms there and
// 0.31 ms for 8 queries.  Large batches go through bruteforce_est instead.
constexpr int kBfThreads = 512, kBfWarps = kBfThreads / 32;

__device__ void warp_bitonic_sort(uint64_t* keys, int n) {
    const int lane = threadIdx.x & 31;
    for (int k = 2; k <= n; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = lane; i < (n >> 1); i += 32) {
                const int lo = 2 * i - (i & (j - 1)), hi = lo + j;
                const bool up = (lo & k) == 0;
                const uint64_t a = keys[lo], b = keys[hi];
                if ((a > b) == up) {
                    keys[lo] = b;
                    keys[hi] = a;
                }
            }
            __syncwarp();
        }
}

struct BfShape {
    int rows;      // R: rows per tile (a multiple of 32)
    int pitch;     // floats per staged row (0: rows are read from global memory)
    int cap;       // keys per query buffer (a power of two, at least k + 64)
    int queries;   // queries per item
    int share;     // warps per query (queries * share = 16 * own)
    int staged_q;  // query vectors in shared memory
    uint32_t spans;
};

static size_t bf_smem(const BfShape& b, uint32_t d, uint32_t l) {
    return sizeof(uint64_t) * b.cap * std::max(b.queries * b.share, kBfWarps) + (b.staged_q ? sizeof(float) * b.queries * ((d + 3) / 4 * 4) : 0) +
           sizeof(float) * 2 * b.rows * ((size_t)b.pitch + l) + sizeof(float) * b.queries * 2 * l +
           kBfWarps * (size_t)b.rows;
}

__device__ __forceinline__ void bf_copy4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void bf_copy16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

// The squared distances of U rows per lane to one query, each one FMA chain in dimension order
// (U independent chains hide the FMA and shared-memory latency; the query's reads are shared)
template <bool VEC, int U>
__device__ __forceinline__ void bf_dist(const float* q, const float* const (&row)[U], int d, float (&acc)[U]) {
#pragma unroll
    for (int u = 0; u < U; u++) acc[u] = 0.f;
    if (VEC) {
#pragma unroll 4
        for (int j = 0; j < d / 4; j++) {
            const float4 x = reinterpret_cast<const float4*>(q)[j];
            float4 y[U];
#pragma unroll
            for (int u = 0; u < U; u++) y[u] = reinterpret_cast<const float4*>(row[u])[j];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const float e0 = x.x - y[u].x, e1 = x.y - y[u].y, e2 = x.z - y[u].z, e3 = x.w - y[u].w;
                acc[u] = fmaf(e0, e0, acc[u]);
                acc[u] = fmaf(e1, e1, acc[u]);
                acc[u] = fmaf(e2, e2, acc[u]);
                acc[u] = fmaf(e3, e3, acc[u]);
            }
        }
    } else {
#pragma unroll 4
        for (int j = 0; j < d; j++) {
            const float x = q[j];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const float e = x - row[u][j];
                acc[u] = fmaf(e, e, acc[u]);
            }
        }
    }
}

// VEC: d % 4 == 0 and 16-byte aligned base rows; LAB4: four label dims; STAGED: rows and queries in
// shared memory (else rows, and queries of extreme length, are read from global memory)
template <bool VEC, bool LAB4, bool STAGED>
__global__ void __launch_bounds__(kBfThreads) k_bruteforce(const float* __restrict__ data, uint64_t n, uint32_t d,
                                                           const float* __restrict__ labels, uint32_t l,
                                                           const float* __restrict__ queries, uint64_t nq,
                                                           const float* __restrict__ ranges, uint32_t k, BfShape b,
                                                           uint64_t* __restrict__ part, float* __restrict__ out_dist,
                                                           uint64_t* __restrict__ out_ids) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int R = b.rows, dq = (int)(d + 3) / 4 * 4;
    const int nbuf = max(b.queries * b.share, kBfWarps), own = b.queries * b.share / kBfWarps;
    uint64_t* s_buf = reinterpret_cast<uint64_t*>(smem);                        // [nbuf][cap]
    float* s_q = reinterpret_cast<float*>(s_buf + (size_t)nbuf * b.cap);        // [queries][dq]
    float* s_tile = s_q + (b.staged_q ? b.queries * dq : 0);                     // [2][R][pitch]
    float* s_lab = s_tile + 2 * (size_t)R * b.pitch;                             // [2][R][l] (R % 32: 16-byte aligned)
    float* s_rng = s_lab + 2 * (size_t)R * l;                                    // [queries][2 l]
    uint8_t* s_list = reinterpret_cast<uint8_t*>(s_rng + b.queries * 2 * l) + (size_t)warp * R;  // [R] rows that pass
    const uint64_t group = blockIdx.x / b.spans, span = blockIdx.x % b.spans;
    const uint64_t q0 = group * b.queries;
    const int nqb = (int)min((uint64_t)b.queries, nq - q0);
    for (int e = t; b.staged_q && e < b.queries * dq; e += kBfThreads) {
        const int qq = e / dq, j = e % dq;
        s_q[e] = qq < nqb && j < (int)d ? queries[(q0 + qq) * d + j] : 0.f;
    }
    for (int e = t; e < nqb * 2 * (int)l; e += kBfThreads) s_rng[e] = ranges[q0 * 2 * l + e];
    const uint64_t tiles = (n + R - 1) / R;
    const uint64_t t0 = tiles * span / b.spans, t1 = tiles * (span + 1) / b.spans;
    auto issue = [&](uint64_t tile, int st) {
        const uint64_t v0 = tile * R;
        const int rows = (int)min((uint64_t)R, n - v0);
        float* dst = s_tile + (size_t)st * R * b.pitch;
        if (STAGED) {  // a warp copies whole rows: no division per element
            for (int r = warp; r < rows; r += kBfWarps) {
                float* to = dst + (size_t)r * b.pitch;
                const float* from = data + (v0 + r) * d;
                if (VEC) {
                    for (int j = 4 * lane; j < (int)d; j += 128) bf_copy16(to + j, from + j);
                } else {
                    for (int j = lane; j < (int)d; j += 32) bf_copy4(to + j, from + j);
                }
            }
        }
        for (int e = t; e < rows * (int)l; e += kBfThreads) bf_copy4(s_lab + (size_t)st * R * l + e, labels + v0 * l + e);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the buffers of this warp: slot warp * own + i, query (warp / share) * own + i (own > 1: share 1)
    const int sub = warp % b.share, my_rows = R / b.share, r_lo = sub * my_rows;
    constexpr int kOwn = 2;
    int cnt[kOwn] = {0, 0};
    uint64_t th[kOwn] = {~0ull, ~0ull};
    if (t0 < t1) issue(t0, 0);
    for (uint64_t tile = t0; tile < t1; tile++) {
        const int st = (int)((tile - t0) & 1);
        if (tile + 1 < t1) {
            issue(tile + 1, st ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const uint64_t v0 = tile * R;
        const int rows = (int)min((uint64_t)R, n - v0);
        const float* tl = s_tile + (size_t)st * R * b.pitch;
        const float* tlab = s_lab + (size_t)st * R * l;
#pragma unroll
        for (int o = 0; o < kOwn; o++) {
            const int qq = (warp / b.share) * own + o;
            if (o >= own || qq >= nqb) continue;
            const float* rg = s_rng + qq * 2 * l;
            int np = 0;
#pragma unroll 4
            for (int r0 = r_lo; r0 < r_lo + my_rows; r0 += 32) {
                const int r = r0 + lane;
                bool ok = r < r_lo + my_rows && r < rows;
                const int rr = ok ? r : 0;
                if (LAB4) {
                    const float4 v = reinterpret_cast<const float4*>(tlab)[rr];
                    const float4 b0 = reinterpret_cast<const float4*>(rg)[0], b1 = reinterpret_cast<const float4*>(rg)[1];
                    ok = ok && !(v.x < b0.x || v.x > b0.y) && !(v.y < b0.z || v.y > b0.w) &&
                         !(v.z < b1.x || v.z > b1.y) && !(v.w < b1.z || v.w > b1.w);
                } else {
                    for (uint32_t i = 0; i < l; i++) {
                        const float v = tlab[rr * l + i];
                        if (v < rg[2 * i] || v > rg[2 * i + 1]) ok = false;
                    }
                }
                const unsigned bal = __ballot_sync(0xffffffffu, ok);
                if (ok) s_list[np + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)r;
                np += __popc(bal);
            }
            __syncwarp();
            uint64_t* buf = s_buf + (size_t)(warp * own + o) * b.cap;
            const float* q = STAGED || b.staged_q ? s_q + qq * dq : queries + (q0 + qq) * d;
            // U pairs per lane from list entry p0 on
            auto pass = [&](int p0, auto uc) {
                constexpr int U = decltype(uc)::value;
                const float* row[U];
                int r[U];
                float acc[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int p = p0 + 32 * u + lane;
                    r[u] = s_list[p < np ? p : p0];
                    row[u] = STAGED ? tl + r[u] * b.pitch : data + (v0 + r[u]) * d;
                }
                bf_dist<VEC, U>(q, row, (int)d, acc);
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const uint64_t key = ((uint64_t)float_key(acc[u]) << 32) | (uint32_t)(v0 + r[u]);
                    const bool in = p0 + 32 * u + lane < np && key < th[o];
                    const unsigned bal = __ballot_sync(0xffffffffu, in);
                    if (in) buf[cnt[o] + __popc(bal & ((1u << lane) - 1u))] = key;
                    cnt[o] += __popc(bal);
                    if (cnt[o] > b.cap - 32) {  // cut back to the k best
                        for (int i = cnt[o] + lane; i < b.cap; i += 32) buf[i] = ~0ull;
                        __syncwarp();
                        warp_bitonic_sort(buf, b.cap);
                        cnt[o] = (int)k;
                        th[o] = buf[k - 1];
                        __syncwarp();
                    }
                }
            };
            int p0 = 0;
            for (; np - p0 > 64; p0 += 128) pass(p0, std::integral_constant<int, 4>());
            for (; p0 < np; p0 += 64) {
                if (np - p0 > 32) pass(p0, std::integral_constant<int, 2>());
                else pass(p0, std::integral_constant<int, 1>());
            }
        }
        __syncthreads();  // the tile's reads are done before its buffer is refilled
    }
    // every buffer sorted, its first k keys final
#pragma unroll
    for (int o = 0; o < kOwn; o++) {
        if (o >= own) continue;
        uint64_t* buf = s_buf + (size_t)(warp * own + o) * b.cap;
        for (int i = cnt[o] + lane; i < b.cap; i += 32) buf[i] = ~0ull;
        __syncwarp();
        warp_bitonic_sort(buf, b.cap);
        for (int i = (int)k + lane; i < b.cap; i += 32) buf[i] = ~0ull;
    }
    // the warps of one query merge pairwise (k <= cap / 2)
    for (int step = 1; step < b.share; step <<= 1) {
        __syncthreads();
        if (sub % (2 * step) == 0) {
            uint64_t* buf = s_buf + (size_t)warp * b.cap;
            const uint64_t* other = buf + (size_t)step * b.cap;
            for (int i = lane; i < (int)k; i += 32) buf[b.cap - 1 - i] = other[i];
            __syncwarp();
            warp_bitonic_sort(buf, b.cap);
            for (int i = (int)k + lane; i < b.cap; i += 32) buf[i] = ~0ull;
        }
    }
    __syncwarp();
#pragma unroll
    for (int o = 0; o < kOwn; o++) {
        const int qq = (warp / b.share) * own + o;
        if (o >= own || qq >= nqb || sub) continue;
        const uint64_t* buf = s_buf + (size_t)(warp * own + o) * b.cap;
        for (int i = lane; i < (int)k; i += 32) {
            const uint64_t key = buf[i];
            if (part) {
                part[((q0 + qq) * b.spans + span) * k + i] = key;
            } else {  // one span: the answer
                out_dist[(q0 + qq) * k + i] = key != ~0ull ? key_float((uint32_t)(key >> 32)) : INFINITY;
                out_ids[(q0 + qq) * k + i] = key != ~0ull ? (uint64_t)(uint32_t)key : ~0ull;
            }
        }
    }
}

// The k smallest keys of each query's spans * k, ascending.  A query's keys come in rounds into a
// buffer of kBfMerge; once it is full, it is cut to its k smallest and the k-th bounds the rest.
constexpr int kBfMerge = 2048;
__global__ void __launch_bounds__(256) k_bf_merge(const uint64_t* __restrict__ part, uint32_t spans, uint32_t k,
                                                  float* __restrict__ out_dist, uint64_t* __restrict__ out_ids) {
    __shared__ uint64_t s_keys[kBfMerge];
    __shared__ uint32_t s_hist[256], s_wc[32];
    __shared__ unsigned long long s_sel[4];
    __shared__ int s_cnt;
    const uint64_t q = blockIdx.x;
    const uint64_t* src = part + q * spans * k;
    const uint32_t total = spans * k;
    uint64_t th = ~0ull;
    if (threadIdx.x == 0) s_cnt = 0;
    __syncthreads();
    for (uint32_t e0 = 0; e0 < total; e0 += 256) {
        const uint32_t e = e0 + threadIdx.x;
        const uint64_t key = e < total ? src[e] : ~0ull;
        if (key < th) s_keys[atomicAdd(&s_cnt, 1)] = key;
        __syncthreads();
        const int c = s_cnt;
        __syncthreads();
        if (c > kBfMerge - 256) {
            th = block_select_smallest(s_keys, c, (int)k, s_hist, s_wc, s_sel);
            if (threadIdx.x == 0) s_cnt = (int)k;
            __syncthreads();
        }
    }
    int c = s_cnt;
    __syncthreads();
    if (c > (int)k) {
        block_select_smallest(s_keys, c, (int)k, s_hist, s_wc, s_sel);
        c = (int)k;
    }
    const int n2 = (int)next_pow2_dev((uint32_t)max(c, 2));
    for (int i = c + (int)threadIdx.x; i < n2; i += blockDim.x) s_keys[i] = ~0ull;
    __syncthreads();
    block_bitonic_sort(s_keys, n2);
    for (int i = threadIdx.x; i < (int)k; i += blockDim.x) {
        const uint64_t key = i < c ? s_keys[i] : ~0ull;
        out_dist[q * k + i] = key != ~0ull ? key_float((uint32_t)(key >> 32)) : INFINITY;
        out_ids[q * k + i] = key != ~0ull ? (uint64_t)(uint32_t)key : ~0ull;
    }
}

// ---- exact kNN of a batch: tensor-core bounds first --------------------------------------------
// Many queries share the base set, so its rows meet them as a matrix product: hdg_est.cuh bounds
// every pair's distance from below, and a pair whose bound is above a valid upper bound T of the
// query's k-th distance is never read.  T comes from strided samples of the base set, each
// kBfRatio times finer than the one before: the k-th smallest exact distance among the sample's rows
// that pass is at least the k-th of the whole set.  At every level the pairs that the bounds and
// the labels leave (about kBfRatio * k per query) are computed exactly, in the same FMA chain as
// k_bruteforce; the last level is the whole set.  A query with more rows left than its list holds
// goes through k_bf_full.
// 1,000 queries x 1 M x 128: 19.1 ms with k_bruteforce, 3.0 to 3.9 ms this way (1.9 ms of it k_est, 0.9
// k_bf_exact; the scratch's allocation varies).  Vectors that FP16 cannot hold bound nothing: every query
// then goes through k_bf_full, 70 ms there (347 ms with a block per 32 queries that computed every pair).
constexpr uint64_t kBfEstQueries = 32, kBfEstPairs = 12000000;
constexpr uint64_t kBfRatio = 16;
constexpr uint64_t kBfRowsMax = 1ull << 18;  // rows converted at a time (64 MB at 128 dims)

// FP16 rows with row stride ld and their constants; one warp per row
__global__ void k_bf_rows(const float* __restrict__ data, uint32_t d, uint64_t row0, uint64_t step, uint32_t n_rows,
                          uint32_t ld, uint16_t* __restrict__ out, float4* __restrict__ cst) {
    const uint64_t r = (uint64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    const int lane = threadIdx.x & 31;
    if (r >= n_rows) return;
    const float* x = data + (row0 + r * step) * d;
    float s = 0.f, e = 0.f;
    for (uint32_t j = lane; j < ld; j += 32) {
        const float v = j < d ? __ldg(x + j) : 0.f;
        const __half h = __float2half_rn(v);
        const float df = v - __half2float(h);
        s = fmaf(v, v, s);
        e = fmaf(df, df, e);
        out[r * ld + j] = __half_as_ushort(h);
    }
    s = warp_sum(s);
    e = warp_sum(e);
    // (a norm that is not finite bounds nothing: NaN, every pair of the row is left to the exact pass)
    if (lane == 0)
        cst[r] = s < INFINITY && e < INFINITY
                     ? make_float4(s * (1.f - kEstSlack), sqrtf(s) * (1.f + kEstSlack), sqrtf(e) * (1.f + kEstSlack), 0.f)
                     : make_float4(NAN, 0.f, 0.f, 0.f);
}

// The same for the queries; no threshold yet.  qn: their squared norms.
__global__ void k_bf_queries(const float* __restrict__ queries, uint32_t d, uint32_t nq, uint32_t ld,
                             uint16_t* __restrict__ out, float4* __restrict__ qc, float* __restrict__ qn) {
    const uint64_t r = (uint64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    const int lane = threadIdx.x & 31;
    if (r >= nq) return;
    const float* x = queries + r * d;
    float s = 0.f, e = 0.f, s2 = 0.f;
    for (uint32_t j = lane; j < ld; j += 32) {
        const float v = j < d ? __ldg(x + j) : 0.f;
        const __half h = __float2half_rn(v);
        const float hv = __half2float(h), df = v - hv;
        s = fmaf(v, v, s);
        s2 = fmaf(hv, hv, s2);
        e = fmaf(df, df, e);
        out[r * ld + j] = __half_as_ushort(h);
    }
    s = warp_sum(s);
    s2 = warp_sum(s2);
    e = warp_sum(e);
    if (lane == 0) {
        const float up = 1.f + kEstSlack;
        qn[r] = s;
        qc[r] = make_float4(2.f * up * (sqrtf(e) + kEstAcc * (float)d * sqrtf(s)), 2.f * up * sqrtf(s2), -FLT_MAX, 0.f);
    }
}

// Exact distances of a query's listed rows.  Not the last level: the query's threshold from the
// k-th smallest.  Last level: the k smallest, ascending.  A thread computes one row at a time.
constexpr int kBfExactThreads = 256;
__global__ void __launch_bounds__(kBfExactThreads) k_bf_exact(const float* __restrict__ data, uint32_t n, uint32_t d,
                                                              const float* __restrict__ queries, uint32_t k,
                                                              const uint32_t* __restrict__ list, uint32_t cap,
                                                              uint32_t* __restrict__ cnt, int vec, int last,
                                                              const float* __restrict__ qn, float4* __restrict__ qc,
                                                              float* __restrict__ out_dist, uint64_t* __restrict__ out_ids) {
    extern __shared__ __align__(16) unsigned char smem_bf[];
    uint64_t* s_keys = reinterpret_cast<uint64_t*>(smem_bf);  // [cap] (a power of two at the sort: k <= 256)
    float* s_q = reinterpret_cast<float*>(s_keys + cap);       // [d]
    __shared__ uint32_t s_hist[256], s_wc[32];
    __shared__ unsigned long long s_sel[4];
    const uint64_t q = blockIdx.x;
    const int t = threadIdx.x;
    const uint32_t all = cnt[q];
    if (last && all > cap) return;  // k_bf_full's
    const int c = (int)min(all, cap);
    for (int j = t; j < (int)d; j += kBfExactThreads) s_q[j] = queries[q * d + j];
    __syncthreads();
    if (!last && t == 0) cnt[q] = 0;
    for (int e0 = t; e0 < c; e0 += 2 * kBfExactThreads) {
        uint32_t id[2];
        const float* row[2];
        float acc[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int e = e0 + u * kBfExactThreads;
            id[u] = __ldg(list + q * cap + (e < c ? e : e0));
            row[u] = data + (uint64_t)min(id[u], n - 1) * d;
        }
        if (vec) bf_dist<true, 2>(s_q, row, (int)d, acc);
        else bf_dist<false, 2>(s_q, row, (int)d, acc);
#pragma unroll
        for (int u = 0; u < 2; u++)
            if (e0 + u * kBfExactThreads < c)
                s_keys[e0 + u * kBfExactThreads] = id[u] < n ? ((uint64_t)float_key(acc[u]) << 32) | id[u] : ~0ull;
    }
    __syncthreads();
    if (!last) {
        if (c < (int)k) return;  // fewer than k rows pass in the sample: no threshold
        const uint64_t kth = block_select_smallest(s_keys, c, (int)k, s_hist, s_wc, s_sel, false);
        if (t == 0) {
            // (the exact sums' own rounding: d terms)
            const float T = key_float((uint32_t)(kth >> 32)) * (1.f + fmaxf(kEstSlack, 1.2e-7f * (float)d));
            if (T < INFINITY) qc[q].z = qn[q] * (1.f - kEstSlack) - T;
        }
        return;
    }
    const int m = min(c, (int)k);
    if (c > (int)k) block_select_smallest(s_keys, c, (int)k, s_hist, s_wc, s_sel);
    const int n2 = (int)next_pow2_dev((uint32_t)max(m, 2));
    for (int i = m + t; i < n2; i += kBfExactThreads) s_keys[i] = ~0ull;
    __syncthreads();
    block_bitonic_sort(s_keys, n2);
    for (int i = t; i < (int)k; i += kBfExactThreads) {
        const uint64_t key = i < m ? s_keys[i] : ~0ull;
        out_dist[q * k + i] = i < m && key != ~0ull ? key_float((uint32_t)(key >> 32)) : INFINITY;
        out_ids[q * k + i] = i < m && key != ~0ull ? (uint64_t)(uint32_t)key : ~0ull;
    }
}

// The queries whose last list overflowed, or every query when the tensor-core pass reports an
// expired wait: a block walks the whole base set.
__global__ void __launch_bounds__(kBfExactThreads) k_bf_full(const float* __restrict__ data, uint64_t n, uint32_t d,
                                                             const float* __restrict__ labels, uint32_t l,
                                                             const float* __restrict__ queries,
                                                             const float* __restrict__ ranges, uint32_t k, uint32_t cap,
                                                             const uint32_t* __restrict__ cnt, const int* __restrict__ err,
                                                             float* __restrict__ out_dist, uint64_t* __restrict__ out_ids) {
    __shared__ uint64_t s_keys[kBfMerge];
    __shared__ uint32_t s_hist[256], s_wc[32];
    __shared__ unsigned long long s_sel[4];
    __shared__ int s_cnt;
    const uint64_t q = blockIdx.x;
    const int t = threadIdx.x;
    if (cnt[q] <= cap && *err == 0) return;
    const float* x = queries + q * d;
    const float* rg = ranges + q * 2 * l;
    uint64_t th = ~0ull;
    if (t == 0) s_cnt = 0;
    __syncthreads();
    for (uint64_t v0 = 0; v0 < n; v0 += kBfExactThreads) {
        const uint64_t v = v0 + t;
        bool ok = v < n;
        for (uint32_t i = 0; ok && i < l; i++) {
            const float y = labels[v * l + i];
            if (y < rg[2 * i] || y > rg[2 * i + 1]) ok = false;
        }
        if (ok) {
            const float* row[1] = {data + v * d};
            float acc[1];
            bf_dist<false, 1>(x, row, (int)d, acc);
            const uint64_t key = ((uint64_t)float_key(acc[0]) << 32) | (uint32_t)v;
            if (key < th) s_keys[atomicAdd(&s_cnt, 1)] = key;
        }
        __syncthreads();
        const int c = s_cnt;
        __syncthreads();
        if (c > kBfMerge - kBfExactThreads) {
            th = block_select_smallest(s_keys, c, (int)k, s_hist, s_wc, s_sel);
            if (t == 0) s_cnt = (int)k;
            __syncthreads();
        }
    }
    int c = s_cnt;
    __syncthreads();
    if (c > (int)k) {
        block_select_smallest(s_keys, c, (int)k, s_hist, s_wc, s_sel);
        c = (int)k;
    }
    const int n2 = (int)next_pow2_dev((uint32_t)max(c, 2));
    for (int i = c + t; i < n2; i += kBfExactThreads) s_keys[i] = ~0ull;
    __syncthreads();
    block_bitonic_sort(s_keys, n2);
    for (int i = t; i < (int)k; i += kBfExactThreads) {
        const uint64_t key = i < c ? s_keys[i] : ~0ull;
        out_dist[q * k + i] = i < c ? key_float((uint32_t)(key >> 32)) : INFINITY;
        out_ids[q * k + i] = i < c ? (uint64_t)(uint32_t)key : ~0ull;
    }
}

// Stream-ordered scratch; nullptr when the memory is not there
static void* scratch(size_t bytes, cudaStream_t st) {
    void* p = nullptr;
    const cudaError_t e = cudaMallocAsync(&p, bytes, st);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        return nullptr;
    }
    CK(e);
    return p;
}

// False, and nothing enqueued, when its memory is not there.
static bool bruteforce_est(const float* data, uint64_t n, uint32_t d, const float* labels, uint32_t l,
                           const float* queries, uint32_t nq, const float* ranges, uint32_t k, float* dist,
                           uint64_t* ids, cudaStream_t st) {
    const uint32_t ld = (d + 7) / 8 * 8, cap = (uint32_t)(3 * kBfRatio * k + 2048);
    const uint64_t rows_max = std::min(n, kBfRowsMax);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += align_up(bytes, 256);
        return o;
    };
    const size_t o_rows = take(rows_max * ld * 2), o_rc = take(rows_max * sizeof(float4)), o_q = take((size_t)nq * ld * 2),
                 o_qc = take(nq * sizeof(float4)), o_qn = take(nq * 4ull), o_list = take((size_t)nq * cap * 4),
                 o_cnt = take(nq * 4ull + 4);
    char* b = static_cast<char*>(scratch(off, st));
    if (!b) return false;
    try {
        uint16_t* rows = reinterpret_cast<uint16_t*>(b + o_rows);
        uint16_t* qh = reinterpret_cast<uint16_t*>(b + o_q);
        float4* rc = reinterpret_cast<float4*>(b + o_rc);
        float4* qc = reinterpret_cast<float4*>(b + o_qc);
        float* qn = reinterpret_cast<float*>(b + o_qn);
        uint32_t* list = reinterpret_cast<uint32_t*>(b + o_list);
        uint32_t* cnt = reinterpret_cast<uint32_t*>(b + o_cnt);
        int* err = reinterpret_cast<int*>(cnt + nq);
        CK(cudaMemsetAsync(cnt, 0, nq * 4ull + 4, st));
        k_bf_queries<<<nblk(nq, 8), 256, 0, st>>>(queries, d, nq, ld, qh, qc, qn);
        CK_LAUNCH();
        EstArgs a{};
        a.rowc = rc;
        a.qc = qc;
        a.qb = qh;
        a.ldq = ld;
        a.nq = nq;
        a.labels = labels;
        a.boxes = ranges;
        a.l = (int)l;
        a.list = list;
        a.cap = cap;
        a.cnt = cnt;
        const size_t sm = sizeof(uint64_t) * cap + sizeof(float) * d;
        allow_smem(k_bf_exact);
        const int vec = d % 4 == 0 && (reinterpret_cast<uintptr_t>(data) & 15) == 0;
        uint64_t step = 1;  // the coarsest sample: as many rows as a list holds
        while ((n + step - 1) / step > cap) step *= kBfRatio;
        for (;; step /= kBfRatio) {
            const uint64_t rows_lv = (n + step - 1) / step;
            for (uint64_t r0 = 0; r0 < rows_lv; r0 += kBfRowsMax) {
                const uint32_t m = (uint32_t)std::min(kBfRowsMax, rows_lv - r0);
                k_bf_rows<<<nblk(m, 8), 256, 0, st>>>(data, d, r0 * step, step, m, ld, rows, rc);
                CK_LAUNCH();
                a.n_rows = m;
                a.tiles = (m + kEstM - 1) / kEstM;
                a.row0 = (uint32_t)(r0 * step);
                a.row_step = (uint32_t)step;
                est_all(a, rows, (int)ld, err, st);
            }
            k_bf_exact<<<nq, kBfExactThreads, sm, st>>>(data, (uint32_t)n, d, queries, k, list, cap, cnt, vec, step == 1 ? 1 : 0, qn, qc,
                                                       dist, ids);
            CK_LAUNCH();
            if (step == 1) break;
        }
        k_bf_full<<<nq, kBfExactThreads, 0, st>>>(data, n, d, labels, l, queries, ranges, k, cap, cnt, err, dist, ids);
        CK_LAUNCH();
    } catch (...) {
        cudaFreeAsync(b, st);
        throw;
    }
    CK(cudaFreeAsync(b, st));
    return true;
}

void bruteforce_knn(const float* data, uint64_t n, uint32_t d, const float* labels, uint32_t l,
                    const float* queries, uint64_t q, const float* ranges, uint32_t k, float* dist,
                    uint64_t* ids, cudaStream_t st) {
    HDG_REQUIRE(k >= 1 && k <= 256, HDG_ERR_UNSUPPORTED, "bruteforce k must be in [1, 256]");
    HDG_REQUIRE(l >= 1 && l <= (uint32_t)kMaxDims && d >= 1, HDG_ERR_INVALID_ARG, "bad dims");
    HDG_REQUIRE(n < (1ull << 32), HDG_ERR_INVALID_ARG, "n must be < 2^32");
    if (!q) return;
    // enough queries to share a pass over the base set, and enough pairs for its levels' launches
    // (k 100, d 128; this path / k_bruteforce, us: 63 x 50,000 224 / 205, 32 x 200,000 395 / 326,
    // 63 x 200,000 397 / 461, 16 x 1 M 757 / 410, 32 x 1 M 832 / 880, 63 x 1 M 842 / 1,431)
    if (q >= kBfEstQueries && q * n >= kBfEstPairs && d <= 4096) {
        uint64_t a = 0;
        for (; a < q; a += 4096) {
            const uint32_t nb = (uint32_t)std::min<uint64_t>(4096, q - a);
            if (!bruteforce_est(data, n, d, labels, l, queries + a * d, nb, ranges + a * 2 * l, k, dist + a * k, ids + a * k, st)) break;
        }
        if (a >= q) return;
        queries += a * d;  // the rest without its scratch
        ranges += a * 2 * l;
        dist += a * k;
        ids += a * k;
        q -= a;
    }
    bool vec = d % 4 == 0 && (reinterpret_cast<uintptr_t>(data) & 15) == 0;
    BfShape b{};
    // two queries per warp (32 per item: the base set is streamed once per 32 queries) while their
    // buffers are small, one for k > 128; fewer queries than warps share the warps out
    b.cap = k <= 128 ? 256 : 512;
    b.queries = k <= 128 ? 32 : 16;
    b.share = 1;
    b.staged_q = 1;
    if (q <= 16) {
        b.queries = 1;
        while ((uint64_t)b.queries < q) b.queries *= 2;
        b.share = kBfWarps / b.queries;
    }
    // the longest tile whose two buffers fit, its rows padded to an odd number of bank groups;
    // rows too long for that are read from global memory, and so are queries of extreme length
    b.pitch = vec ? (int)(d + (d / 4 % 2 ? 0 : 4)) : (int)(d | 1);
    for (b.rows = 128; b.rows >= 32 && bf_smem(b, d, l) > kBlockSmem; b.rows /= 2) {
    }
    if (b.rows < 32) {
        b.rows = 128;
        b.pitch = 0;
        if (bf_smem(b, d, l) > kBlockSmem) {
            b.staged_q = 0;
            vec = false;
        }
    }
    const size_t sm = bf_smem(b, d, l);
    // spans: of one to four items per SM, the count that leaves the last round fullest
    constexpr uint64_t kBfBatch = 65536;  // queries per launch: bounds the partial keys
    const uint64_t sms = (uint64_t)sm_count(), tiles = std::max<uint64_t>(1, (n + b.rows - 1) / b.rows);
    for (uint64_t a = 0; a < q; a += kBfBatch) {
        const uint64_t nb = std::min(kBfBatch, q - a), groups = (nb + b.queries - 1) / b.queries;
        uint64_t spans = 1;
        double fill = 0.0;
        for (uint64_t w = 1; w <= 4; w++) {
            const uint64_t c = std::min(tiles, std::max<uint64_t>(1, sms * w / groups)), items = groups * c;
            const double f = (double)items / (double)((items + sms - 1) / sms * sms);
            if (f > fill + 0.02) {
                fill = f;
                spans = c;
            }
        }
        uint64_t* part = static_cast<uint64_t*>(scratch(sizeof(uint64_t) * nb * spans * k, st));
        if (!part) spans = 1;
        b.spans = (uint32_t)spans;
        auto launch = [&](auto kern) {
            allow_smem(kern);
            kern<<<(unsigned)(groups * spans), kBfThreads, sm, st>>>(data, n, d, labels, l, queries + a * d, nb,
                                                                    ranges + a * 2 * l, k, b, part, dist + a * k, ids + a * k);
            CK_LAUNCH();
        };
        try {
            if (!b.pitch) vec ? launch(k_bruteforce<true, false, false>) : launch(k_bruteforce<false, false, false>);
            else if (vec) l == 4 ? launch(k_bruteforce<true, true, true>) : launch(k_bruteforce<true, false, true>);
            else l == 4 ? launch(k_bruteforce<false, true, true>) : launch(k_bruteforce<false, false, true>);
            if (part) {
                k_bf_merge<<<(unsigned)nb, 256, 0, st>>>(part, b.spans, k, dist + a * k, ids + a * k);
                CK_LAUNCH();
            }
        } catch (...) {
            if (part) cudaFreeAsync(part, st);
            throw;
        }
        if (part) CK(cudaFreeAsync(part, st));
    }
}

}  // namespace hdg

namespace hdg {

// ---- merge of per-data-batch results (merge_intermediate_result, src/core/merge_res.cu:18-56)
// Row r of (dist, ids) holds n_batches blocks of k results, block b from an index built on
// base rows [offset_b, ...): ids are shifted by offset_b (invalid ids stay invalid), the
// k smallest (distance, id) of the row are kept, ascending.
namespace {
__global__ void k_merge_topk(const float* __restrict__ dist, const uint64_t* __restrict__ ids, uint32_t k,
                             uint32_t nb, const uint64_t* __restrict__ offsets, int n2, float* __restrict__ out_dist,
                             uint64_t* __restrict__ out_ids) {
    extern __shared__ uint64_t s_key[];            // [n2] (distance key << 32 | slot)
    uint64_t* s_id = s_key + n2;                    // [k * nb] shifted ids
    const uint64_t r = blockIdx.x;
    const uint32_t w = k * nb;
    for (uint32_t i = threadIdx.x; i < (uint32_t)n2; i += blockDim.x) {
        uint64_t key = ~0ull;
        if (i < w) {
            const uint64_t id = ids[r * w + i];
            const bool ok = id != ~0ull;
            const uint64_t sid = ok ? id + offsets[i / k] : ~0ull;
            s_id[i] = sid;
            // ties by the shifted id: the slot order of equal distances follows the id
            key = ok ? ((uint64_t)float_key(dist[r * w + i]) << 32) | i : ~0ull;
        }
        s_key[i] = key;
    }
    __syncthreads();
    block_bitonic_sort(s_key, n2);
    // equal distance keys are ordered by slot; re-order each run of equal keys by id
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i + 1 < (uint32_t)min(n2, (int)w) && i < k; i++) {  // runs reaching the top k
            uint32_t j = i + 1;
            while (j < w && (s_key[j] >> 32) == (s_key[i] >> 32) && s_key[j] != ~0ull) j++;
            for (uint32_t a = i + 1; a < j; a++)  // insertion sort on the (short) tie run
                for (uint32_t b2 = a; b2 > i && s_id[(uint32_t)s_key[b2]] < s_id[(uint32_t)s_key[b2 - 1]]; b2--) {
                    const uint64_t tmp = s_key[b2];
                    s_key[b2] = s_key[b2 - 1];
                    s_key[b2 - 1] = tmp;
                }
            i = j - 1;
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) {
        const uint64_t key = s_key[i];
        const bool ok = key != ~0ull;
        out_dist[r * k + i] = ok ? key_float((uint32_t)(key >> 32)) : INFINITY;
        out_ids[r * k + i] = ok ? s_id[(uint32_t)key] : ~0ull;
    }
}
}  // namespace

void merge_topk(const float* dist, const uint64_t* ids, uint64_t q, uint32_t k, uint32_t nb, const uint64_t* offsets,
                float* out_dist, uint64_t* out_ids, cudaStream_t st) {
    HDG_REQUIRE(k >= 1 && nb >= 1 && (uint64_t)k * nb <= 8192, HDG_ERR_UNSUPPORTED, "k * n_batches must be <= 8192");
    const int n2 = (int)next_pow2(std::max<uint32_t>(k * nb, 2));
    const size_t sm = sizeof(uint64_t) * (n2 + (size_t)k * nb);
    allow_smem(k_merge_topk);
    k_merge_topk<<<(unsigned)q, 256, sm, st>>>(dist, ids, k, nb, offsets, n2, out_dist, out_ids);
    CK_LAUNCH();
}

}  // namespace hdg
