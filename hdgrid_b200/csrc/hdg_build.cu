// Index build: super_grid::index::build (src/index/2-level_index/Super-Grid-IVF_PQ.cu:420-646)
// re-designed for one B200.
//
//  1. label grid shape on the host (calc_grid_shape, :305-412)
//  2. PQ codebooks: per-subspace k-means(256) on a sample, then every point encoded on the
//     GPU (build_pq, src/index/product-quantization.cu:147-212)
//  3. C*S fine centroids by k-means on a sample (the reference's kmeans::fit_predict, :454-463),
//     every point assigned on the GPU; FP64 centroid sums (the only FP64 on the GPU)
//  4. the fine centroids grouped into C clusters of S by a capacity-balanced k-means (the reference's kmeans_balanced::fit_predict, :466-477)
//  5. cell coords + Morton codes of every point on the GPU (get_grid_ids_kernel :28-52,
//     encode_points_kernel zorder.cu:36-43); pool sorted by (list, Morton code, id)
//     (thrust::sort_by_key per list, :607-611, is a stable radix sort over ids in ascending order)
//  6. per-list inclusive prefix counts over the cell grid (HOPS multi_dim_scan,
//     src/core/HOPS.cu:3-74): dense, cell-major with the list index fastest, or -- when that
//     array would be large -- compressed into per-(grid row, list) change points along the diff
//     dim (compress_HOPS_data, Super-Grid-IVF_PQ.cu:209-303).
// k-means results are not pinned by any reference test (RAFT is not vendored), so the
// build uses its own seeded Lloyd iterations.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <numeric>
#include <random>
#include <type_traits>

#include "hdg_device.cuh"
#include "hdg_est.cuh"
#include "hdg_internal.h"

namespace hdg {

// ------------------------------------------------------------------------------------
// k-means kernels
// ------------------------------------------------------------------------------------

// Nearest centre of every row of X: argmin_c (|c|^2 - 2 x.c), FP32, each product one FMA chain in
// dimension order, ties to the lower centre.  Block = 256 threads, 128 rows x 128 centres per tile,
// 8 x 8 per thread from k-major shared tiles read 16 bytes at a time (64 FMAs per four reads),
// K chunks of 16 whose next chunk is loaded into registers meanwhile.  Bound: FMA issue.
// 8 x 4 per thread with 4-byte reads took 10.0 ms for 1 M x 128 rows and 1,024 centres, this 6.7 ms.
constexpr int AT_P = 128, AT_C = 128, AT_K = 16;
template <bool VEC>  // d % 4 == 0 and 16-byte aligned rows
__global__ void __launch_bounds__(256, 2) k_assign_nearest(const float* __restrict__ X, uint64_t n, int d,
                                                           const float* __restrict__ Cc,
                                                           const float* __restrict__ cnorm, int k,
                                                           int* __restrict__ out) {
    __shared__ __align__(16) float Xs[2][AT_K][AT_P + 4];
    __shared__ __align__(16) float Cs[2][AT_K][AT_C + 4];
    const int t = threadIdx.x;
    const int tx = t & 15;   // centre group (8 centres: 4 tx .. +3 and 64 + 4 tx .. +3)
    const int ty = t >> 4;   // row group (8 rows: 4 ty .. +3 and 64 + 4 ty .. +3)
    const uint64_t row0 = (uint64_t)blockIdx.x * AT_P;
    // loads: thread t takes row t % 128 of both tiles, k words (t / 128) * 8 .. + 7
    const int lr = t & 127, lk = (t >> 7) * 8;
    const uint64_t xr = min(row0 + lr, n - 1);
    float best[8];
    int besti[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        best[i] = INFINITY;
        besti[i] = 0;
    }
    const int nk = (d + AT_K - 1) / AT_K;
    float xv[8], cv[8];
    auto load = [&](int c0, int kc) {  // rows past the end repeat the last one (their results are dropped)
        const int k0 = kc * AT_K + lk;
        const float* x = X + xr * d + k0;
        const float* c = Cc + (uint64_t)min(c0 + lr, k - 1) * d + k0;
        if (VEC) {
#pragma unroll
            for (int u = 0; u < 8; u += 4) {
                const bool in = k0 + u < d;
                const float4 a = in ? __ldg(reinterpret_cast<const float4*>(x + u)) : make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 b = in ? __ldg(reinterpret_cast<const float4*>(c + u)) : make_float4(0.f, 0.f, 0.f, 0.f);
                xv[u] = a.x, xv[u + 1] = a.y, xv[u + 2] = a.z, xv[u + 3] = a.w;
                cv[u] = b.x, cv[u + 1] = b.y, cv[u + 2] = b.z, cv[u + 3] = b.w;
            }
        } else {
#pragma unroll
            for (int u = 0; u < 8; u++) {
                xv[u] = k0 + u < d ? __ldg(x + u) : 0.f;
                cv[u] = k0 + u < d ? __ldg(c + u) : 0.f;
            }
        }
    };
    auto stage = [&](int b) {
#pragma unroll
        for (int u = 0; u < 8; u++) {
            Xs[b][lk + u][lr] = xv[u];
            Cs[b][lk + u][lr] = cv[u];
        }
    };
    for (int c0 = 0; c0 < k; c0 += AT_C) {
        float acc[8][8];
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) acc[i][j] = 0.f;
        load(c0, 0);
        __syncthreads();  // the previous tile's reads are done
        stage(0);
        __syncthreads();
        for (int kc = 0; kc < nk; kc++) {
            const int b = kc & 1;
            if (kc + 1 < nk) load(c0, kc + 1);
#pragma unroll
            for (int kk = 0; kk < AT_K; kk++) {
                float x[8], c[8];
                *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(&Xs[b][kk][4 * ty]);
                *reinterpret_cast<float4*>(x + 4) = *reinterpret_cast<const float4*>(&Xs[b][kk][64 + 4 * ty]);
                *reinterpret_cast<float4*>(c) = *reinterpret_cast<const float4*>(&Cs[b][kk][4 * tx]);
                *reinterpret_cast<float4*>(c + 4) = *reinterpret_cast<const float4*>(&Cs[b][kk][64 + 4 * tx]);
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int j = 0; j < 8; j++) acc[i][j] = fmaf(x[i], c[j], acc[i][j]);
            }
            if (kc + 1 < nk) {
                stage(b ^ 1);  // last read two chunks ago, before the previous barrier
                __syncthreads();
            }
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int c = c0 + (j < 4 ? 4 * tx + j : 64 + 4 * tx + j - 4);
            if (c >= k) continue;
            const float cn = cnorm[c];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float v = cn - 2.f * acc[i][j];
                if (v < best[i]) {
                    best[i] = v;
                    besti[i] = c;
                }
            }
        }
    }
    // reduce across the 16 threads (tx) that share the same 8 rows
#pragma unroll
    for (int i = 0; i < 8; i++) {
        float v = best[i];
        int b = besti[i];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, o, 16);
            const int ob = __shfl_xor_sync(0xffffffffu, b, o, 16);
            if (ov < v || (ov == v && ob < b)) {
                v = ov;
                b = ob;
            }
        }
        const uint64_t gr = row0 + (i < 4 ? 4 * ty + i : 64 + 4 * ty + i - 4);
        if (tx == 0 && gr < n) out[gr] = b;
    }
}

static void assign_nearest(const float* X, uint64_t n, int d, const float* centers, const float* cnorm, int k, int* out,
                           cudaStream_t st) {
    const bool vec = d % 4 == 0 && ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(centers)) & 15) == 0;
    const unsigned blocks = (unsigned)((n + AT_P - 1) / AT_P);
    if (vec) k_assign_nearest<true><<<blocks, 256, 0, st>>>(X, n, d, centers, cnorm, k, out);
    else k_assign_nearest<false><<<blocks, 256, 0, st>>>(X, n, d, centers, cnorm, k, out);
}

__global__ void k_row_norms(const float* __restrict__ X, uint64_t n, int d, float* __restrict__ out) {
    const uint64_t r = (uint64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    float s = 0.f;
    for (int j = lane; j < d; j += 32) {
        const float v = X[r * d + j];
        s = fmaf(v, v, s);
    }
    s = warp_sum(s);
    if (lane == 0) out[r] = s;
}

// FP64 centroid sums (the one place the GPU computes in FP64).
__global__ void k_accumulate(const float* __restrict__ X, uint64_t n, int d,
                             const int* __restrict__ lab, double* __restrict__ sums,
                             unsigned* __restrict__ counts) {
    const uint64_t r = (uint64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    const int lane = threadIdx.x & 31;
    if (r >= n) return;
    const int c = lab[r];
    for (int j = lane; j < d; j += 32) atomicAdd(&sums[(uint64_t)c * d + j], (double)X[r * d + j]);
    if (lane == 0) atomicAdd(&counts[c], 1u);
}

__global__ void k_finalize(const double* __restrict__ sums, const unsigned* __restrict__ counts,
                           int k, int d, float* __restrict__ Cc) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (uint64_t)k * d) return;
    const unsigned cnt = counts[e / d];
    if (cnt) Cc[e] = (float)(sums[e] / (double)cnt);
}

// PQ: nearest of 256 codewords per (row, subspace), ties to the lower codeword; codebooks
// [M][256][pq_len].  A block stages the codebooks of MB subspaces (at most 64 KB) and a thread
// encodes two rows in all of them, so a codeword's broadcast read serves two rows and a row's codes
// leave as whole 16-byte pieces.  Both rows' differences and sums run as packed FP32 operations
// (each rounded like the scalar ones).  Bound: FP32 issue.  One row and subspace per thread, a
// run-time pq_len and one byte per store took 10.7 ms for 1 M x 128 and 32 subspaces, this 3.0 ms.
__device__ __forceinline__ float2 pk_sub(float2 a, float b) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %4};\n\t"
        "add.rn.f32x2 ra, ra, rb;\n\tmov.b64 {%0, %1}, ra;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(-b));
    return d;
}
__device__ __forceinline__ float2 pk_fma(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rc;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 ra, ra, rb, rc;\n\tmov.b64 {%0, %1}, ra;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
constexpr int kPqThreads = 256;
constexpr int pq_mb(int pl) { return pl <= 4 ? 16 : (pl <= 8 ? 8 : 4); }  // subspaces per block

template <int PL>
__global__ void __launch_bounds__(kPqThreads) k_pq_assign(const float* __restrict__ X, uint64_t n, int d, int M,
                                                          const float* __restrict__ cb, uint8_t* __restrict__ out,
                                                          int out_stride, int* __restrict__ out_int) {
    constexpr int MB = pq_mb(PL);
    extern __shared__ __align__(16) float s_cb[];  // [MB][256][PL]
    const int m0 = blockIdx.y * MB, mb = min(MB, M - m0);
    for (int e = threadIdx.x; e < mb * kCodes * PL; e += kPqThreads) s_cb[e] = cb[(uint64_t)m0 * kCodes * PL + e];
    __syncthreads();
    const uint64_t r0 = (uint64_t)blockIdx.x * (2 * kPqThreads) + threadIdx.x, r1 = r0 + kPqThreads;
    if (r0 >= n) return;
    const float* x0 = X + r0 * d + (uint64_t)m0 * PL;
    const float* x1 = X + (r1 < n ? r1 : r0) * d + (uint64_t)m0 * PL;
    uint32_t code0[MB / 4] = {0}, code1[MB / 4] = {0};
#pragma unroll
    for (int mm = 0; mm < MB; mm++) {
        if (mm >= mb) break;
        float2 x[PL];
#pragma unroll
        for (int t = 0; t < PL; t++) x[t] = make_float2(__ldg(x0 + mm * PL + t), __ldg(x1 + mm * PL + t));
        float b0 = INFINITY, b1 = INFINITY;
        int i0 = 0, i1 = 0;
        const float* c = s_cb + mm * kCodes * PL;
#pragma unroll 4
        for (int k = 0; k < kCodes; k++, c += PL) {
            float2 s = make_float2(0.f, 0.f);
#pragma unroll
            for (int t = 0; t < PL; t++) {
                const float2 df = pk_sub(x[t], c[t]);
                s = pk_fma(df, df, s);
            }
            if (s.x < b0) {
                b0 = s.x;
                i0 = k;
            }
            if (s.y < b1) {
                b1 = s.y;
                i1 = k;
            }
        }
        code0[mm / 4] |= (uint32_t)i0 << (8 * (mm % 4));
        code1[mm / 4] |= (uint32_t)i1 << (8 * (mm % 4));
    }
    auto put = [&](uint64_t r, const uint32_t (&code)[MB / 4]) {
        if (out) {  // (rows start at a multiple of 16 bytes: out_stride is M padded to 16)
            uint32_t* o = reinterpret_cast<uint32_t*>(out + r * out_stride + m0);
            if (mb == 16) {
                if constexpr (MB == 16) *reinterpret_cast<uint4*>(o) = make_uint4(code[0], code[1], code[2], code[3]);
            } else {  // (the padding's codes are zero)
#pragma unroll
                for (int w = 0; w < MB / 4; w++)
                    if (4 * w < mb) o[w] = code[w];
            }
        }
        if (out_int) {
#pragma unroll
            for (int mm = 0; mm < MB; mm++)
                if (mm < mb) out_int[r * M + m0 + mm] = (int)((code[mm / 4] >> (8 * (mm % 4))) & 255u);
        }
    };
    put(r0, code0);
    if (r1 < n) put(r1, code1);
}

// pq_len 1 .. 16 (checked by the build)
static void pq_assign(const float* X, uint64_t n, int d, int M, int pq_len, const float* cb, uint8_t* out, int out_stride,
                      int* out_int, cudaStream_t st) {
    auto go = [&](auto plc) {
        constexpr int PL = decltype(plc)::value;
        constexpr size_t sm = sizeof(float) * pq_mb(PL) * kCodes * PL;
        allow_smem(k_pq_assign<PL>);
        k_pq_assign<PL><<<dim3((unsigned)((n + 2 * kPqThreads - 1) / (2 * kPqThreads)),
                               (unsigned)((M + pq_mb(PL) - 1) / pq_mb(PL))),
                          kPqThreads, sm, st>>>(X, n, d, M, cb, out, out_stride, out_int);
        CK_LAUNCH();
    };
    switch (pq_len) {
#define HDG_PQ(n) \
    case n: \
        return go(std::integral_constant<int, n>())
        HDG_PQ(1);
        HDG_PQ(2);
        HDG_PQ(3);
        HDG_PQ(4);
        HDG_PQ(5);
        HDG_PQ(6);
        HDG_PQ(7);
        HDG_PQ(8);
        HDG_PQ(9);
        HDG_PQ(10);
        HDG_PQ(11);
        HDG_PQ(12);
        HDG_PQ(13);
        HDG_PQ(14);
        HDG_PQ(15);
        HDG_PQ(16);
#undef HDG_PQ
        default:
            throw Error(HDG_ERR_UNSUPPORTED, "pq_len above 16 is not supported");
    }
}

__global__ void k_pq_accumulate(const float* __restrict__ X, uint64_t n, int d, int pq_len, int M,
                                const int* __restrict__ lab, double* __restrict__ sums,
                                unsigned* __restrict__ counts) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n * (uint64_t)M) return;
    const uint64_t r = e / M;
    const int m = (int)(e % M);
    const int c = lab[e];
    const uint64_t base = ((uint64_t)m * kCodes + c) * pq_len;
    for (int t = 0; t < pq_len; t++) atomicAdd(&sums[base + t], (double)X[r * d + (uint64_t)m * pq_len + t]);
    atomicAdd(&counts[(uint64_t)m * kCodes + c], 1u);
}

__global__ void k_gather_rows(const float* __restrict__ X, int d, const uint32_t* __restrict__ rows,
                              uint64_t n_rows, float* __restrict__ out) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n_rows * d) return;
    out[e] = X[(uint64_t)rows[e / d] * d + e % d];
}

// Cell coords (shuffled order), flattened cell id and Morton code of every point
// (get_grid_ids_kernel, Super-Grid-IVF_PQ.cu:28-52; encode_points_kernel, zorder.cu:36-43).
__global__ void k_point_cells(const float* __restrict__ labels, uint64_t n, GridMeta g,
                              uint64_t* __restrict__ zcode, uint64_t* __restrict__ cell) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    int coords[kMaxDims];
    uint64_t flat = 0;
    for (int i = 0; i < g.l; i++) {
        const float x = labels[r * g.l + g.shuffle[i]];
        int c = grid_id(x, g.left[i], g.span[i], g.grid_dims[i]);
        c = c < g.grid_dims[i] - 1 ? c : g.grid_dims[i] - 1;
        if (c < 0) c = 0;
        coords[i] = c;
        flat += (uint64_t)c * g.cell_stride[i];
    }
    zcode[r] = morton_encode(coords, g.morton_dims, g.morton_max_bits, g.morton_valid_map);
    cell[r] = flat;
}

__global__ void k_count_cells(const uint64_t* __restrict__ cell, const int* __restrict__ list_of,
                              uint64_t n, uint32_t n_lists, uint32_t* __restrict__ prefix) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    atomicAdd(&prefix[cell[r] * n_lists + list_of[r]], 1u);
}

// Counts of the lists [j0, j0 + B) over every cell: dense [cells][B], list fastest.
__global__ void k_count_cells_range(const uint64_t* __restrict__ cell, const int* __restrict__ list_of, uint64_t n,
                                    uint32_t j0, uint32_t B, uint32_t* __restrict__ dense) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const uint32_t j = (uint32_t)list_of[r];
    if (j >= j0 && j < j0 + B) atomicAdd(&dense[cell[r] * B + (j - j0)], 1u);
}

// Compressed prefix rows (compress_HOPS_data, Super-Grid-IVF_PQ.cu:209-303): the grid's last
// dim of size > 1 (the diff dim, Dd cells, stride 1) runs along a row, every other dim is
// flattened into the row index t, so cell (t, z) is flat t * Dd + z.  For every (t, list j0 + b)
// of the dense inclusive prefix [cells][B] one thread walks z = 0..Dd-1 and keeps the points
// where the value changes.  Without out it writes their number to cnt[t * L + j0 + b]; with out
// it writes them as (z << 32 | value) at out + off[t * L + j0 + b].
__global__ void k_prefix_rows(const uint32_t* __restrict__ dense, uint64_t T, uint32_t Dd, uint32_t B, uint32_t j0,
                              uint32_t L, uint64_t* __restrict__ cnt, const uint64_t* __restrict__ off,
                              uint64_t* __restrict__ out) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= T * B) return;
    const uint32_t b = (uint32_t)(e % B);
    const uint64_t t = e / B, r = t * L + j0 + b;
    const uint32_t* p = dense + t * (uint64_t)Dd * B + b;
    uint64_t* o = out ? out + off[r] : nullptr;
    uint32_t prev = 0;
    uint64_t c = 0;
    uint32_t z = 0;
    for (; z + 4 <= Dd; z += 4) {  // four independent loads in flight
        uint32_t v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = __ldg(p + (uint64_t)(z + u) * B);
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (v[u] != prev) {
                if (o) o[c] = ((uint64_t)(z + u) << 32) | v[u];
                c++;
                prev = v[u];
            }
    }
    for (; z < Dd; z++) {
        const uint32_t v = __ldg(p + (uint64_t)z * B);
        if (v != prev) {
            if (o) o[c] = ((uint64_t)z << 32) | v;
            c++;
            prev = v;
        }
    }
    if (!out) cnt[r] = c;
}

// Inclusive scan along one grid dim of the cell-major [cells][lists] array.
// One thread per (outer, inner, list) line; consecutive threads = consecutive lists.
__global__ void k_scan_axis(uint32_t* __restrict__ prefix, uint64_t n_lines, uint64_t inner,
                            int axis_len, uint32_t n_lists) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n_lines) return;
    const uint64_t list = e % n_lists;
    const uint64_t line = e / n_lists;         // (outer, inner) pair
    const uint64_t in = line % inner, out = line / inner;
    const uint64_t base = (out * axis_len * inner + in) * n_lists + list;
    const uint64_t step = inner * n_lists;
    uint32_t s = 0;
    for (int a = 0; a < axis_len; a++) {
        s += prefix[base + a * step];
        prefix[base + a * step] = s;
    }
}

// Every point's label ranks packed into 32 bits: dim i's rank (thresholds at or below the
// label, by binary search) at bit i * (bits + 1).
__global__ void k_pack_ranks(const float* __restrict__ labels, uint64_t n, int l, const float* __restrict__ thr,
                             uint32_t stride, IndexDev D, uint32_t* __restrict__ out) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    uint32_t packed = 0;
    for (int i = 0; i < l; i++) {
        const float x = labels[r * l + i];
        const float* t = thr + (uint64_t)i * stride;
        uint32_t lo = 0, hi = D.rank_n[i];
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (t[mid] <= x) lo = mid + 1;
            else hi = mid;
        }
        packed |= lo << (i * (D.rank_bits + 1));
    }
    out[r] = packed;
}

// The ranks' bit planes (IndexDev::rank_planes).  A warp takes 256 rows: a ballot per plane and
// word leaves lane v the eight words of plane v, written as one 32-byte sector.
__global__ void __launch_bounds__(256) k_rank_planes(IndexDev D, uint64_t n, uint32_t* __restrict__ out) {
    const uint64_t w0 = ((uint64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * 8;  // first word
    const int lane = threadIdx.x & 31;
    if (w0 >= D.plane_words) return;
    uint32_t c[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const uint64_t r = (w0 + k) * 32 + lane;
        c[k] = r < n ? __ldg(D.rankpack + r) : 0u;
    }
    for (uint32_t i = 0; i < D.l; i++) {
        const uint32_t off = i * (D.rank_bits + 1), mask = (1u << D.rank_bits) - 1u;
        const uint32_t planes = D.rank_n[i] >> D.plane_shift;
        for (uint32_t v0 = 0; v0 < planes; v0 += 32) {
            uint32_t word[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const uint32_t x = ((c[k] >> off) & mask) >> D.plane_shift;
                word[k] = 0;
#pragma unroll
                for (uint32_t v = 0; v < 32; v++) {
                    const uint32_t b = __ballot_sync(0xffffffffu, x <= v0 + v);
                    if (lane == (int)v) word[k] = b;
                }
            }
            if (v0 + lane < planes) {
                uint4* o = reinterpret_cast<uint4*>(out + (D.plane_off[i] + v0 + lane) * D.plane_words + w0);
                o[0] = make_uint4(word[0], word[1], word[2], word[3]);
                o[1] = make_uint4(word[4], word[5], word[6], word[7]);
            }
        }
    }
}

// codes [n][chunks] (16-byte chunks, row-major) -> [chunks][n]: chunk j of point p at j*n + p
__global__ void k_interleave_codes(const uint4* __restrict__ rows, uint64_t n, uint32_t chunks,
                                   uint4* __restrict__ out) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n * chunks) return;
    const uint64_t j = i / n, p = i - j * n;
    out[i] = rows[p * chunks + j];
}

__global__ void k_gather_codes_labels(const uint8_t* __restrict__ codes_by_id, int M_pad,
                                      const float* __restrict__ labels_by_id, int l,
                                      const uint32_t* __restrict__ ids, uint64_t n,
                                      uint8_t* __restrict__ codes, float* __restrict__ labels) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    const uint64_t id = ids[r];
    const uint4* src = reinterpret_cast<const uint4*>(codes_by_id + id * M_pad);
    uint4* dst = reinterpret_cast<uint4*>(codes + r * M_pad);
    for (int v = 0; v < M_pad / 16; v++) dst[v] = src[v];
    for (int i = 0; i < l; i++) labels[r * l + i] = labels_by_id[id * l + i];
}

// A point's PQ approximation (the codewords its codes name) in FP16, and its constants for the
// distance estimates; one warp per pool row, lane = subspace (mod 32).
__global__ void k_decode_rows(IndexDev D, uint16_t* __restrict__ out, float4* __restrict__ cst,
                              uint32_t* __restrict__ mx) {
    __shared__ uint32_t s_mx[3];
    if (threadIdx.x < 3) s_mx[threadIdx.x] = 0u;
    __syncthreads();
    const uint64_t r = (uint64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    const int lane = threadIdx.x & 31;
    const int L = D.pq_len;
    float s = 0.f, e = 0.f;
    for (int m = lane; r < D.n && m < (int)D.M; m += 32) {
        const uint32_t c = D.codes[((uint64_t)(m >> 4) * D.n + r) * 16 + (m & 15)];
        const float* x = D.pq_centers + ((uint64_t)m * kCodes + c) * L;
        for (int t = 0; t < L; t++) {
            const float v = __ldg(x + t);
            const __half h = __float2half_rn(v);
            const float df = v - __half2float(h);
            s = fmaf(v, v, s);
            e = fmaf(df, df, e);
            out[r * D.d + m * L + t] = __half_as_ushort(h);
        }
    }
    s = warp_sum(s);
    e = warp_sum(e);
    if (lane == 0 && r < D.n) {
        const float4 v = make_float4(s * (1.f - kEstSlack), sqrtf(s) * (1.f + kEstSlack), sqrtf(e) * (1.f + kEstSlack), 0.f);
        cst[r] = v;
        atomicMax(&s_mx[0], __float_as_uint(v.x));  // (non-negative floats order as their bits; NaN above all)
        atomicMax(&s_mx[1], __float_as_uint(v.y));
        atomicMax(&s_mx[2], __float_as_uint(v.z));
    }
    __syncthreads();
    if (threadIdx.x < 3) atomicMax(&mx[threadIdx.x], s_mx[threadIdx.x]);
}

// ------------------------------------------------------------------------------------
// capacity-balanced groups
// ------------------------------------------------------------------------------------
// Points take the closest centre first, over all (point, centre) pairs in order of (distance, point *
// C + centre), while the centre has room: S members per centre.  That greedy assignment is the one
// stable matching of points and centres that both rank by the pair's key, so it can be found by
// proposals instead of a sort of all pairs: every point without a place proposes to its best centre
// that would not turn it away, a centre with more than S keeps its S smallest keys.  The order of
// the proposals does not change the outcome.  A host sort of the pairs per iteration took 95 ms
// for 1,024 points x 128 centres and 1.9 s for 4,096 x 512 (ten iterations), 6.4 and 109 ms this way.

// dist[i][c]: squared differences rounded and summed in dimension order
__global__ void k_group_dist(const float* __restrict__ sub, int L, int d, const float* __restrict__ centers, int C,
                             float* __restrict__ dist) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (uint64_t)L * C) return;
    // consecutive threads: consecutive centres' rows of one point
    dist[e] = seq_l2(sub + e / C * d, centers + e % C * d, d);
}

// One block.  A pair's key at a centre: float bits (distances are not negative) << 32 | point.
// thr[c]: the S-th smallest key of a full centre, past which it turns points away.  cnt [C + 1],
// mem [L]: the points at each centre, laid out anew every round.
__global__ void __launch_bounds__(1024) k_group_match(const float* __restrict__ dist, int L, int C, int S,
                                                      int* __restrict__ grp, int* __restrict__ open,
                                                      unsigned long long* __restrict__ thr, int* __restrict__ cnt,
                                                      int* __restrict__ mem) {
    __shared__ int s_open, s_w[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nw = blockDim.x >> 5;
    for (int c = t; c < C; c += blockDim.x) __stcg(thr + c, ~0ull);
    for (int i = t; i < L; i += blockDim.x) {
        grp[i] = -1;
        open[i] = i;
    }
    if (t == 0) s_open = L;
    __syncthreads();
    auto key = [&](int i, int c) {
        return ((unsigned long long)__float_as_uint(__ldg(dist + (uint64_t)i * C + c)) << 32) | (unsigned)i;
    };
    for (int n = L; n > 0;) {
        // proposals: a warp per open point, its smallest (distance, centre) among those that would take it
        for (int o = warp; o < n; o += nw) {
            const int i = open[o];
            unsigned long long best = ~0ull;
            for (int c = lane; c < C; c += 32) {
                const unsigned long long k = key(i, c);
                if (k < __ldcg(thr + c)) best = min(best, (k & 0xffffffff00000000ull) | (unsigned)c);
            }
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, s));
            if (lane == 0) grp[i] = (int)(unsigned)best;
        }
        for (int c = t; c <= C; c += blockDim.x) cnt[c] = 0;
        __syncthreads();
        for (int i = t; i < L; i += blockDim.x) atomicAdd(&cnt[grp[i]], 1);  // (every point has a place now)
        __syncthreads();
        // cnt -> the end of each centre's part of mem, then (as the parts fill from there) its start
        {
            const int per = (C + (int)blockDim.x - 1) / (int)blockDim.x, b = min(C, t * per), e = min(C, b + per);
            int sum = 0;
            for (int c = b; c < e; c++) sum += cnt[c];
            int x = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) s_w[warp] = x;
            __syncthreads();
            if (warp == 0) {
                int y = lane < nw ? s_w[lane] : 0;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int z = __shfl_up_sync(0xffffffffu, y, o);
                    if (lane >= o) y += z;
                }
                s_w[lane] = y;
            }
            __syncthreads();
            int run = x - sum + (warp ? s_w[warp - 1] : 0);
            for (int c = b; c < e; c++) {
                run += cnt[c];
                cnt[c] = run;
            }
            if (t == 0) {
                cnt[C] = L;
                s_open = 0;
            }
        }
        __syncthreads();
        for (int i = t; i < L; i += blockDim.x) mem[atomicSub(&cnt[grp[i]], 1) - 1] = i;
        __syncthreads();
        // full centres: a warp finds the S-th smallest key bit by bit from the top (the largest value
        // with fewer than S keys below it) and turns the rest away
        for (int c = warp; c < C; c += nw) {
            const int m0 = cnt[c], m1 = cnt[c + 1];
            if (m1 - m0 < S) continue;
            unsigned long long kth = 0;
            for (int b = 63; b >= 0; b--) {
                const unsigned long long cand = kth | (1ull << b);
                int below = 0;
                for (int j = m0 + lane; j < m1; j += 32) below += key(mem[j], c) < cand;
                if ((int)__reduce_add_sync(0xffffffffu, (unsigned)below) < S) kth = cand;
            }
            if (lane == 0) __stcg(thr + c, kth);
            for (int j = m0 + lane; j < m1; j += 32)
                if (key(mem[j], c) > kth) open[atomicAdd(&s_open, 1)] = mem[j];
        }
        __syncthreads();
        n = s_open;
        __syncthreads();
    }
}

// The points of each group in ascending order; one warp per group
__global__ void k_group_members(const int* __restrict__ grp, int L, int C, int S, uint32_t* __restrict__ members) {
    const int c = (int)(blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32), lane = threadIdx.x & 31;
    if (c >= C) return;
    int at = 0;
    for (int i0 = 0; i0 < L; i0 += 32) {
        const bool in = i0 + lane < L && grp[i0 + lane] == c;
        const unsigned bal = __ballot_sync(0xffffffffu, in);
        if (in) members[(uint64_t)c * S + at + __popc(bal & ((1u << lane) - 1u))] = (uint32_t)(i0 + lane);
        at += __popc(bal);
    }
}

// Group means: FP64 sums in ascending member order
__global__ void k_group_centers(const float* __restrict__ sub, int d, const uint32_t* __restrict__ members, int C, int S,
                                float* __restrict__ centers) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (uint64_t)C * d) return;
    const uint64_t c = e / d, j = e % d;
    double s = 0.0;
    for (int m = 0; m < S; m++) s += (double)sub[(uint64_t)members[c * S + m] * d + j];
    centers[e] = (float)(s / (double)S);
}

__global__ void k_to_bf16(const float* __restrict__ x, uint64_t n, __nv_bfloat16* __restrict__ y) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n) y[e] = __float2bfloat16_rn(x[e]);
}

// ------------------------------------------------------------------------------------
// stable radix sort of (u64 key, u32 value) pairs, 8 bits per pass from the lowest
// ------------------------------------------------------------------------------------
// Per pass: a digit histogram per block of kRsTile pairs, one exclusive scan over (digit, block), and
// a scatter in which a block ranks its pairs in order: a warp takes consecutive pairs, lanes with
// the same digit find one another by match, and a prefix over the warps gives the block order.
// Bound: the scatter's reads and writes of 12 bytes per pair and pass.
constexpr int kRsThreads = 256, kRsPer = 16, kRsTile = kRsThreads * kRsPer;

__global__ void __launch_bounds__(kRsThreads) k_rs_hist(const uint64_t* __restrict__ keys, uint64_t n, int shift,
                                                        uint32_t blocks, uint32_t* __restrict__ hist) {
    __shared__ uint32_t s_h[256];
    s_h[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t b0 = (uint64_t)blockIdx.x * kRsTile;
    for (int u = 0; u < kRsPer; u++) {
        const uint64_t e = b0 + u * kRsThreads + threadIdx.x;
        if (e < n) atomicAdd(&s_h[(keys[e] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[(uint64_t)threadIdx.x * blocks + blockIdx.x] = s_h[threadIdx.x];
}

// exclusive scan in place, one block
__global__ void __launch_bounds__(1024) k_rs_scan(uint32_t* __restrict__ a, uint64_t n) {
    __shared__ uint32_t s_w[32], s_run;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) s_run = 0;
    __syncthreads();
    for (uint64_t b0 = 0; b0 < n; b0 += 4096) {
        uint32_t v[4], sum = 0;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint64_t e = b0 + 4ull * t + u;
            v[u] = e < n ? a[e] : 0u;
            sum += v[u];
        }
        uint32_t x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_w[warp] = x;
        __syncthreads();
        if (warp == 0) {
            uint32_t y = s_w[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t z = __shfl_up_sync(0xffffffffu, y, o);
                if (lane >= o) y += z;
            }
            s_w[lane] = y;
        }
        __syncthreads();
        uint32_t run = s_run + x - sum + (warp ? s_w[warp - 1] : 0u);
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const uint64_t e = b0 + 4ull * t + u;
            if (e < n) a[e] = run;
            run += v[u];
        }
        __syncthreads();
        if (t == 1023) s_run = run;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kRsThreads) k_rs_scatter(const uint64_t* __restrict__ keys,
                                                           const uint32_t* __restrict__ vals, uint64_t n, int shift,
                                                           uint32_t blocks, const uint32_t* __restrict__ off,
                                                           uint64_t* __restrict__ out_keys,
                                                           uint32_t* __restrict__ out_vals) {
    constexpr int NW = kRsThreads / 32;
    __shared__ uint32_t s_c[NW][256];  // pairs of each digit so far in the warp, then before the warp
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int i = t; i < NW * 256; i += kRsThreads) (&s_c[0][0])[i] = 0;
    __syncthreads();
    // warp w holds pairs [w * 32 * kRsPer, +32 * kRsPer) of the tile, 32 per round
    const uint64_t b0 = (uint64_t)blockIdx.x * kRsTile + (uint64_t)warp * 32 * kRsPer + lane;
    uint64_t k[kRsPer];
    uint32_t rank[kRsPer];
#pragma unroll
    for (int u = 0; u < kRsPer; u++) {
        const uint64_t e = b0 + 32 * u;
        const bool v = e < n;
        k[u] = v ? keys[e] : 0ull;
        const unsigned live = __ballot_sync(0xffffffffu, v);
        const uint32_t d = (uint32_t)(k[u] >> shift) & 255u;
        const unsigned same = __match_any_sync(0xffffffffu, v ? d : 256u + lane) & live;
        uint32_t before = 0;
        if (v) before = s_c[warp][d];
        rank[u] = before + __popc(same & ((1u << lane) - 1u));
        __syncwarp();
        if (v && lane == __ffs((int)same) - 1) s_c[warp][d] = before + __popc(same);
        __syncwarp();
    }
    __syncthreads();
    {
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < NW; w++) {
            const uint32_t c = s_c[w][t];
            s_c[w][t] = run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kRsPer; u++) {
        const uint64_t e = b0 + 32 * u;
        if (e >= n) continue;
        const uint32_t d = (uint32_t)(k[u] >> shift) & 255u;
        const uint32_t at = off[(uint64_t)d * blocks + blockIdx.x] + s_c[warp][d] + rank[u];
        out_keys[at] = k[u];
        out_vals[at] = vals[e];
    }
}

__global__ void k_iota(uint32_t* __restrict__ a, uint64_t n) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n) a[e] = (uint32_t)e;
}
__global__ void k_gather_list(const int* __restrict__ list_of, const uint32_t* __restrict__ ids, uint64_t n,
                              uint64_t* __restrict__ out) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n) out[e] = (uint64_t)(uint32_t)list_of[ids[e]];
}
__global__ void k_gather_z(const uint64_t* __restrict__ z, const uint32_t* __restrict__ ids, uint64_t n,
                           uint64_t* __restrict__ out) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n) out[e] = z[ids[e]];
}
// every point's list under its new number, and the lists' sizes
__global__ void k_renumber(int* __restrict__ list_of, uint64_t n, const int* __restrict__ new_of_old,
                           uint32_t* __restrict__ sizes) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const int j = new_of_old[list_of[e]];
    list_of[e] = j;
    atomicAdd(&sizes[j], 1u);
}
__global__ void k_narrow16(const uint32_t* __restrict__ a, uint64_t n, uint16_t* __restrict__ out) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < n) out[e] = (uint16_t)a[e];
}
// Smallest and largest label of dim blockIdx.y (as ordered keys; NaN left out) and whether any is NaN
__global__ void __launch_bounds__(256) k_label_range(const float* __restrict__ labels, uint64_t n, int l,
                                                     uint32_t* __restrict__ mn, uint32_t* __restrict__ mx,
                                                     uint32_t* __restrict__ nan) {
    const int i = blockIdx.y;
    uint32_t lo = 0xffffffffu, hi = 0u, bad = 0u;
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (uint64_t)gridDim.x * blockDim.x) {
        const float x = labels[r * l + i];
        if (isnan(x)) {
            bad = 1u;
        } else {
            const uint32_t k = float_key(x);
            lo = min(lo, k);
            hi = max(hi, k);
        }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    bad = __reduce_or_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&mn[i], lo);
        atomicMax(&mx[i], hi);
        if (bad) atomicOr(nan, 1u);
    }
}
// The strided sample of one label dim as sort keys (NaN last)
__global__ void k_rank_sample(const float* __restrict__ labels, uint64_t step, uint64_t m, int l, int i,
                              uint64_t* __restrict__ keys) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= m) return;
    const float x = labels[e * step * l + i];
    keys[e] = isnan(x) ? 0xffffffffull : (uint64_t)float_key(x);
}

// ------------------------------------------------------------------------------------
// host helpers
// ------------------------------------------------------------------------------------

static unsigned blocks_for(uint64_t n, unsigned per) { return (unsigned)((n + per - 1) / per); }

// Sorts (keys, vals) by the low `bits` bits of the keys, stably; the result is in keys / vals.
struct RadixSort {
    DevMem<uint64_t> k2;
    DevMem<uint32_t> v2, hist;
    uint64_t n;
    uint32_t blocks;
    explicit RadixSort(uint64_t count)
        : k2(count), v2(count), hist(256ull * ((count + kRsTile - 1) / kRsTile)), n(count),
          blocks((uint32_t)((count + kRsTile - 1) / kRsTile)) {}
    void sort(uint64_t* keys, uint32_t* vals, int bits, cudaStream_t st) {
        uint64_t *ka = keys, *kb = k2.p;
        uint32_t *va = vals, *vb = v2.p;
        for (int shift = 0; shift < bits; shift += 8) {
            k_rs_hist<<<blocks, kRsThreads, 0, st>>>(ka, n, shift, blocks, hist.p);
            k_rs_scan<<<1, 1024, 0, st>>>(hist.p, 256ull * blocks);
            k_rs_scatter<<<blocks, kRsThreads, 0, st>>>(ka, va, n, shift, blocks, hist.p, kb, vb);
            CK_LAUNCH();
            std::swap(ka, kb);
            std::swap(va, vb);
        }
        if (ka != keys) {
            CK(cudaMemcpyAsync(keys, ka, sizeof(uint64_t) * n, cudaMemcpyDeviceToDevice, st));
            CK(cudaMemcpyAsync(vals, va, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, st));
        }
    }
};

static float ordered_float(uint32_t key) {  // the inverse of float_key
    const uint32_t u = (key & 0x80000000u) ? (key & 0x7fffffffu) : ~key;
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}

// Thresholds of one label dim from its sorted sample (NaN labels already left out): the distinct
// values when they fit in `stride` thresholds, else the sample's quantiles
static uint32_t thresholds_of(const std::vector<float>& v, uint32_t stride, float* t) {
    std::vector<float> u(v);
    u.erase(std::unique(u.begin(), u.end()), u.end());
    uint32_t m = 0;
    if (u.size() <= stride + 1) {
        for (size_t k = 1; k < u.size(); k++) t[m++] = u[k];
    } else {
        for (uint32_t k = 1; k <= stride; k++) {
            const float x = v[(size_t)((uint64_t)k * v.size() / (stride + 1))];
            if (m == 0 || x > t[m - 1]) t[m++] = x;
        }
    }
    return m;
}

// What the build still holds on the device when it uploads the index: the arena takes these
// instead of the host copies (nullptr: from the host)
struct DeviceArrays {
    const uint64_t* zcodes;
    const uint32_t* ids;
    const uint8_t* codes;    // pool-ordered rows
    const float* labels;     // pool order
    const uint32_t* prefix;  // dense counts (nullptr: the compressed rows)
    const uint64_t *prefix_off, *prefix_rows;
    uint32_t labels_nan;
};
static void upload_index_from(hdg_index* idx, cudaStream_t st, const DeviceArrays* src);

// Lloyd k-means on device rows Xs [ns x d]; centres initialised from the first k rows.
// Returns the centres (device, [k x d]).
static void kmeans_device(const float* Xs, uint64_t ns, int d, int k, int iters, std::mt19937_64& rng,
                          float* centers, cudaStream_t st) {
    DevMem<int> lab(ns);
    DevMem<float> cnorm(k);
    DevMem<double> sums((uint64_t)k * d);
    DevMem<unsigned> counts(k);
    CK(cudaMemcpyAsync(centers, Xs, sizeof(float) * k * d, cudaMemcpyDeviceToDevice, st));
    std::vector<unsigned> h_counts(k);
    for (int it = 0; it < iters; it++) {
        k_row_norms<<<blocks_for(k, 8), 256, 0, st>>>(centers, k, d, cnorm.p);
        assign_nearest(Xs, ns, d, centers, cnorm.p, k, lab.p, st);
        CK(cudaMemsetAsync(sums.p, 0, sizeof(double) * k * d, st));
        CK(cudaMemsetAsync(counts.p, 0, sizeof(unsigned) * k, st));
        k_accumulate<<<blocks_for(ns, 8), 256, 0, st>>>(Xs, ns, d, lab.p, sums.p, counts.p);
        k_finalize<<<blocks_for((uint64_t)k * d, 256), 256, 0, st>>>(sums.p, counts.p, k, d, centers);
        CK(cudaMemcpyAsync(h_counts.data(), counts.p, sizeof(unsigned) * k, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        // re-seed empty clusters from random sample rows
        for (int c = 0; c < k; c++) {
            if (h_counts[c]) continue;
            const uint64_t r = rng() % ns;
            CK(cudaMemcpyAsync(centers + (uint64_t)c * d, Xs + r * d, sizeof(float) * d,
                               cudaMemcpyDeviceToDevice, st));
        }
    }
    CK_LAUNCH();
}

// Capacity-balanced k-means of the fine centroids into C groups of exactly S members
// (stands in for RAFT kmeans_balanced, whose exact algorithm is not vendored).  sub: device [L x d]
// (L = C * S); centers: device [C x d], out; group: the centroids' groups.
static void balanced_groups(const float* sub, int L, int d, int C, int S, int iters, std::mt19937_64& rng,
                            float* centers, std::vector<int>& group, cudaStream_t st) {
    std::vector<int> perm(L);
    std::iota(perm.begin(), perm.end(), 0);
    std::shuffle(perm.begin(), perm.end(), rng);
    std::vector<uint32_t> first(perm.begin(), perm.begin() + C);
    DevMem<uint32_t> d_first(C);
    CK(cudaMemcpyAsync(d_first.p, first.data(), sizeof(uint32_t) * C, cudaMemcpyHostToDevice, st));
    k_gather_rows<<<blocks_for((uint64_t)C * d, 256), 256, 0, st>>>(sub, d, d_first.p, C, centers);
    DevMem<float> dist((uint64_t)L * C);
    DevMem<int> grp(L), open(L), cnt(C + 1), mem(L);
    DevMem<unsigned long long> thr(C);
    DevMem<uint32_t> members((uint64_t)C * S);
    for (int it = 0; it < iters; it++) {
        k_group_dist<<<blocks_for((uint64_t)L * C, 256), 256, 0, st>>>(sub, L, d, centers, C, dist.p);
        k_group_match<<<1, 1024, 0, st>>>(dist.p, L, C, S, grp.p, open.p, thr.p, cnt.p, mem.p);
        k_group_members<<<blocks_for(C, 8), 256, 0, st>>>(grp.p, L, C, S, members.p);
        k_group_centers<<<blocks_for((uint64_t)C * d, 256), 256, 0, st>>>(sub, d, members.p, C, S, centers);
        CK_LAUNCH();
    }
    group.assign(L, 0);
    if (iters) CK(cudaMemcpyAsync(group.data(), grp.p, sizeof(int) * L, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
}

// Grid shape: calc_grid_shape (Super-Grid-IVF_PQ.cu:305-412), including its integer/float
// conversions.  A dim whose span is 0 gets span 1 (the reference divides by zero there).
GridMeta compute_grid_shape(const std::vector<float>& mins, const std::vector<float>& maxs, int l,
                            uint64_t max_grids, uint64_t label_mask_bits) {
    GridMeta g;
    g.l = l;
    const uint8_t mask = (uint8_t)label_mask_bits;
    const uint8_t label_mask = (uint8_t)(~mask);
    int cnt = 0;
    for (int i = 0; i < l; i++)
        if ((label_mask >> i) & 1) cnt++;
    std::vector<std::pair<uint64_t, int>> span_pairs(l);
    for (int i = 0; i < l; i++) {
        // ceil / floor of the f32 extremes and their difference stay in f32: the reference's
        // `ceil(global_max[i]) - floor(global_min[i])` on float elements resolves to the float
        // overloads under nvcc, so a span above 2^24 is rounded to f32 before the cast
        const float mx = std::ceil(maxs[i]), mn = std::floor(mins[i]);
        HDG_REQUIRE(mn >= 0.0f, HDG_ERR_INVALID_ARG,
                    "labels must be non-negative (label dim " + std::to_string(i) + ")");
        const float diff = mx - mn;
        uint64_t span = (uint64_t)diff;
        if (span == 0) span = 1;
        span_pairs[i] = {span, i};
    }
    int main_grids = (int)std::floor(std::sqrt((double)max_grids));
    std::sort(span_pairs.begin(), span_pairs.end());
    if (l == 1) main_grids = (int)std::min<uint64_t>(max_grids, span_pairs[0].first);
    HDG_REQUIRE(main_grids >= 1, HDG_ERR_INVALID_ARG, "max_grids must be >= 1");
    int remain = 1, remain_cnt = cnt - 1, last_valid = l - 1;
    if (l > 1) remain = (int)(max_grids / (uint64_t)main_grids);
    uint8_t morton_mask = 0xff;
    std::vector<int> dims(l, 1);
    for (int i = 0; i < l; i++) {
        const int id = span_pairs[i].second;
        const uint64_t len = span_pairs[i].first;
        if ((label_mask >> id) & 1) {
            if (remain_cnt == 0) {
                last_valid = i;
                continue;
            }
            int dims_len = (int)std::min<uint64_t>(
                (uint64_t)remain,
                std::min<uint64_t>(len, (uint64_t)std::floor(std::pow((double)main_grids,
                                                                      1.0 / (double)(float)(cnt - 1)))));
            if (remain_cnt == 1) dims_len = (int)std::min<uint64_t>((uint64_t)remain, len);
            remain_cnt--;
            HDG_REQUIRE(dims_len >= 1, HDG_ERR_INVALID_ARG, "max_grids too small for the label dims");
            dims[i] = dims_len;
            remain /= dims_len;
        } else {
            morton_mask &= (uint8_t)~(1 << i);
            dims[i] = 1;
        }
    }
    dims[last_valid] = main_grids;
    g.tot_cells = 1;
    for (int i = 0; i < l; i++) {
        g.grid_dims[i] = dims[i];
        g.tot_cells *= (uint64_t)dims[i];
        g.shuffle[i] = span_pairs[i].second;
        g.span[i] = span_pairs[i].first;
        g.left[i] = (uint64_t)std::floor((double)mins[span_pairs[i].second]);
    }
    uint64_t stride = 1;
    for (int i = l - 1; i >= 0; i--) {
        g.cell_stride[i] = stride;
        stride *= (uint64_t)dims[i];
    }
    g.morton_dims = l;
    const int maxd = *std::max_element(dims.begin(), dims.end());
    g.morton_max_bits = (int)std::ceil(std::log2((double)maxd + 1));
    g.morton_valid_map = morton_mask & (uint8_t)((1u << l) - 1);
    g.diff_dim = l - 1;
    for (int i = l - 1; i >= 0; i--)
        if (dims[i] > 1) {
            g.diff_dim = i;
            break;
        }
    int valid = 0;
    for (int i = 0; i < l; i++)
        if ((g.morton_valid_map >> i) & 1) valid++;
    HDG_REQUIRE(valid * g.morton_max_bits <= 63, HDG_ERR_UNSUPPORTED,
                "Morton code wider than 63 bits; lower max_grids");
    return g;
}

// Dense prefix counts up to this size; beyond it the compressed rows.
constexpr uint64_t kDensePrefixMax = 2ull << 30;

// The compressed per-list prefix rows (the reference's compress_HOPS_data form, built per list
// from a dense HOPS scan, Super-Grid-IVF_PQ.cu:209-303, 527-583).  Lists are taken in chunks of
// B whose dense [cells][B] prefix fits a fixed budget: count, scan along every grid dim, then
// one thread per (grid row, list) keeps the change points along the diff dim.  A first round
// counts each row's change points (their exclusive sum over rows t * L + j gives the offsets),
// a second round rebuilds each chunk and writes the (z << 32 | value) pairs.
static void build_prefix_rows(const GridMeta& g, const uint64_t* d_cell, const int* d_list, uint64_t n, uint32_t L,
                              std::unique_ptr<DevMem<uint64_t>>& off, std::unique_ptr<DevMem<uint64_t>>& rows,
                              uint64_t& entries, cudaStream_t st) {
    const uint32_t Dd = (uint32_t)g.grid_dims[g.diff_dim];
    HDG_REQUIRE(g.cell_stride[g.diff_dim] == 1 && Dd >= 1 && g.tot_cells % Dd == 0, HDG_ERR_STATE,
                "diff dim of the grid is not its last dim of size > 1");
    const uint64_t T = g.tot_cells / Dd;
    const uint64_t budget = 1ull << 30;
    const uint32_t B = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(L, budget / (g.tot_cells * 4)));
    DevMem<uint32_t> dense(g.tot_cells * B);
    DevMem<uint64_t> cnt(T * L);
    auto chunk = [&](uint32_t j0, uint32_t nb, const uint64_t* off, uint64_t* out) {
        CK(cudaMemsetAsync(dense.p, 0, sizeof(uint32_t) * g.tot_cells * nb, st));
        k_count_cells_range<<<blocks_for(n, 256), 256, 0, st>>>(d_cell, d_list, n, j0, nb, dense.p);
        for (int a = 0; a < g.l; a++) {
            const uint64_t lines = g.tot_cells / (uint64_t)g.grid_dims[a] * nb;
            k_scan_axis<<<blocks_for(lines, 256), 256, 0, st>>>(dense.p, lines, g.cell_stride[a], g.grid_dims[a],
                                                                nb);
        }
        k_prefix_rows<<<blocks_for(T * nb, 128), 128, 0, st>>>(dense.p, T, Dd, nb, j0, L, cnt.p, off, out);
        CK_LAUNCH();
    };
    for (uint32_t j0 = 0; j0 < L; j0 += B) chunk(j0, std::min(B, L - j0), nullptr, nullptr);
    std::vector<uint64_t> hc(T * L);
    CK(cudaMemcpyAsync(hc.data(), cnt.p, sizeof(uint64_t) * hc.size(), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    std::vector<uint64_t> ho(T * L + 1, 0);
    for (uint64_t r = 0; r < T * L; r++) ho[r + 1] = ho[r] + hc[r];
    entries = ho.back();
    off.reset(new DevMem<uint64_t>(T * L + 1));
    rows.reset(new DevMem<uint64_t>(std::max<uint64_t>(entries, 1)));
    CK(cudaMemcpyAsync(off->p, ho.data(), sizeof(uint64_t) * (T * L + 1), cudaMemcpyHostToDevice, st));
    for (uint32_t j0 = 0; j0 < L; j0 += B) chunk(j0, std::min(B, L - j0), off->p, rows->p);
    CK(cudaStreamSynchronize(st));
}

void build_index(hdg_index* idx, const float* d_data, uint64_t n, uint32_t d, const float* d_labels,
                 uint32_t l, cudaStream_t st) {
    const hdg_params& P = idx->params;
    HDG_REQUIRE(d_data && d_labels, HDG_ERR_INVALID_ARG, "null data or labels");
    HDG_REQUIRE((int)l == idx->filter.l, HDG_ERR_INVALID_ARG,
                "label dims differ from filter.conf's l");
    HDG_REQUIRE(P.n_clusters == 256, HDG_ERR_UNSUPPORTED, "only 256-entry PQ codebooks are supported");
    HDG_REQUIRE(P.pq_dim >= 1 && d % P.pq_dim == 0, HDG_ERR_UNSUPPORTED,
                "pq_dim must divide the vector dimension");
    HDG_REQUIRE(d / P.pq_dim <= 16, HDG_ERR_UNSUPPORTED, "pq_len above 16 is not supported");
    const uint64_t C = P.clusters, S = P.sub_clusters, L = C * S;
    HDG_REQUIRE(C >= 1 && S >= 1 && L <= 65536, HDG_ERR_INVALID_ARG, "clusters*sub_clusters out of range");
    HDG_REQUIRE(n >= L && n >= 256 && n < (1ull << 32), HDG_ERR_INVALID_ARG,
                "base set must hold at least max(256, clusters*sub_clusters) points and < 2^32");
    std::mt19937_64 rng(P.seed);
    HostIndex H;  // the index's own once its arrays exist: a build that fails before leaves the old one
    H.n = n;
    H.d = d;
    H.l = l;
    H.M = P.pq_dim;
    H.M_pad = align_up(H.M, 16);
    H.pq_len = d / P.pq_dim;
    H.n_lists = L;
    H.C = C;
    const int iters = (int)(P.kmeans_iters ? P.kmeans_iters : 20);

    // ---- 1. grid shape -------------------------------------------------------------
    std::vector<float> mins(l, INFINITY), maxs(l, -INFINITY);
    uint32_t labels_nan = 0;
    {
        std::vector<uint32_t> hr(2 * l + 1, 0u);
        std::fill(hr.begin(), hr.begin() + l, 0xffffffffu);
        DevMem<uint32_t> r(2 * l + 1);
        CK(cudaMemcpyAsync(r.p, hr.data(), sizeof(uint32_t) * hr.size(), cudaMemcpyHostToDevice, st));
        k_label_range<<<dim3(std::min(blocks_for(n, 256), 1024u), l), 256, 0, st>>>(d_labels, n, (int)l, r.p, r.p + l,
                                                                                   r.p + 2 * l);
        CK_LAUNCH();
        CK(cudaMemcpyAsync(hr.data(), r.p, sizeof(uint32_t) * hr.size(), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        for (uint32_t i = 0; i < l; i++)
            if (hr[i] <= hr[l + i]) {  // (no label but NaN: the dim keeps inf / -inf)
                mins[i] = ordered_float(hr[i]);
                maxs[i] = ordered_float(hr[l + i]);
            }
        labels_nan = hr[2 * l];
    }
    H.grid = compute_grid_shape(mins, maxs, l, P.max_grids, P.label_mask);
    const GridMeta& g = H.grid;
    // per-list prefix counts: the dense cells x lists array while it stays small, else the
    // compressed rows (PREFIX_ROWS)
    const uint64_t dense_bytes = g.tot_cells * L * 4;
    const bool rows_form = P.prefix_rows == 1 || (P.prefix_rows == 0 && dense_bytes > kDensePrefixMax);
    HDG_REQUIRE(rows_form || dense_bytes <= (16ull << 30), HDG_ERR_UNSUPPORTED,
                "dense prefix-count grid (cells x lists) exceeds 16 GiB; use PREFIX_ROWS or a lower max_grids");

    // ---- sample for training ---------------------------------------------------------
    std::vector<uint32_t> perm(n);
    std::iota(perm.begin(), perm.end(), 0u);
    std::shuffle(perm.begin(), perm.end(), rng);
    const uint64_t n_train = std::min<uint64_t>(n, std::max<uint64_t>(65536, 64 * L));
    DevMem<uint32_t> d_perm(n_train);
    CK(cudaMemcpyAsync(d_perm.p, perm.data(), sizeof(uint32_t) * n_train, cudaMemcpyHostToDevice, st));
    DevMem<float> Xs(n_train * d);
    k_gather_rows<<<blocks_for(n_train * d, 256), 256, 0, st>>>(d_data, d, d_perm.p, n_train, Xs.p);

    // ---- 2. PQ codebooks + codes -----------------------------------------------------
    const int M = (int)H.M, pq_len = (int)H.pq_len;
    DevMem<float> pqc((uint64_t)M * kCodes * pq_len);
    {
        const uint64_t n_pq = std::min<uint64_t>(n_train, 65536);
        // initial codewords: first 256 sample rows' slices
        std::vector<float> init((size_t)M * kCodes * pq_len);
        std::vector<float> rows((size_t)kCodes * d);
        CK(cudaMemcpyAsync(rows.data(), Xs.p, sizeof(float) * kCodes * d, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        for (int m = 0; m < M; m++)
            for (int c = 0; c < kCodes; c++)
                for (int t = 0; t < pq_len; t++)
                    init[((size_t)m * kCodes + c) * pq_len + t] = rows[(size_t)c * d + m * pq_len + t];
        CK(cudaMemcpyAsync(pqc.p, init.data(), sizeof(float) * init.size(), cudaMemcpyHostToDevice, st));
        DevMem<int> lab(n_pq * M);
        DevMem<double> sums((uint64_t)M * kCodes * pq_len);
        DevMem<unsigned> counts((uint64_t)M * kCodes);
        std::vector<unsigned> hc((size_t)M * kCodes);
        for (int it = 0; it < iters; it++) {
            pq_assign(Xs.p, n_pq, (int)d, M, pq_len, pqc.p, nullptr, 0, lab.p, st);
            CK(cudaMemsetAsync(sums.p, 0, sizeof(double) * M * kCodes * pq_len, st));
            CK(cudaMemsetAsync(counts.p, 0, sizeof(unsigned) * M * kCodes, st));
            k_pq_accumulate<<<blocks_for(n_pq * M, 256), 256, 0, st>>>(Xs.p, n_pq, d, pq_len, M, lab.p,
                                                                      sums.p, counts.p);
            k_finalize<<<blocks_for((uint64_t)M * kCodes * pq_len, 256), 256, 0, st>>>(
                sums.p, counts.p, M * kCodes, pq_len, pqc.p);
            CK(cudaMemcpyAsync(hc.data(), counts.p, sizeof(unsigned) * hc.size(), cudaMemcpyDeviceToHost, st));
            CK(cudaStreamSynchronize(st));
            for (int m = 0; m < M; m++)
                for (int c = 0; c < kCodes; c++) {
                    if (hc[(size_t)m * kCodes + c]) continue;
                    const uint64_t r = rng() % n_pq;
                    CK(cudaMemcpyAsync(pqc.p + ((uint64_t)m * kCodes + c) * pq_len,
                                       Xs.p + r * d + (uint64_t)m * pq_len, sizeof(float) * pq_len,
                                       cudaMemcpyDeviceToDevice, st));
                }
        }
        H.pq_centers.resize((size_t)M * kCodes * pq_len);
        CK(cudaMemcpyAsync(H.pq_centers.data(), pqc.p, sizeof(float) * H.pq_centers.size(),
                           cudaMemcpyDeviceToHost, st));
    }
    DevMem<uint8_t> codes_by_id(n * H.M_pad);
    CK(cudaMemsetAsync(codes_by_id.p, 0, n * H.M_pad, st));
    pq_assign(d_data, n, (int)d, M, pq_len, pqc.p, codes_by_id.p, (int)H.M_pad, nullptr, st);
    CK_LAUNCH();

    // ---- 3. fine centroids (C*S lists) -------------------------------------------------
    DevMem<float> fine(L * d);
    kmeans_device(Xs.p, n_train, d, (int)L, iters, rng, fine.p, st);
    DevMem<int> list_of_id(n);
    {
        DevMem<float> fnorm(L);
        k_row_norms<<<blocks_for(L, 8), 256, 0, st>>>(fine.p, L, d, fnorm.p);
        assign_nearest(d_data, n, (int)d, fine.p, fnorm.p, (int)L, list_of_id.p, st);
    }
    std::vector<float> h_fine(L * d);
    CK(cudaMemcpyAsync(h_fine.data(), fine.p, sizeof(float) * L * d, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));

    // ---- 4. group the fine centroids into C clusters of S ------------------------------
    std::vector<int> group;
    {
        DevMem<float> ctr(C * d);
        balanced_groups(fine.p, (int)L, (int)d, (int)C, (int)S, std::min(iters, 10), rng, ctr.p, group, st);
        H.centers.resize(C * d);
        CK(cudaMemcpyAsync(H.centers.data(), ctr.p, sizeof(float) * C * d, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
    }
    // list order: by cluster, then by fine-centroid index (group_by_cluster_id keeps ascending ids)
    std::vector<int> new_of_old(L);
    {
        std::vector<int> order(L);
        std::iota(order.begin(), order.end(), 0);
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return group[a] < group[b]; });
        H.sub_centers.resize(L * d);
        for (uint64_t j = 0; j < L; j++) {
            new_of_old[order[j]] = (int)j;
            std::copy(h_fine.begin() + (size_t)order[j] * d, h_fine.begin() + (size_t)(order[j] + 1) * d,
                      H.sub_centers.begin() + j * d);
        }
        H.cluster_off.assign(C + 1, 0);
        for (uint64_t i = 0; i < L; i++) H.cluster_off[group[i] + 1]++;
        for (uint64_t c = 0; c < C; c++) H.cluster_off[c + 1] += H.cluster_off[c];
    }

    // ---- 5. cells, Morton codes, pool order ---------------------------------------------
    DevMem<uint64_t> zc(n), cell(n);
    k_point_cells<<<blocks_for(n, 256), 256, 0, st>>>(d_labels, n, g, zc.p, cell.p);
    // pool order: by list, Morton code, id -- a stable sort of the ids by code, then by list
    DevMem<uint32_t> dids(n);
    DevMem<uint64_t> dz(n);
    {
        DevMem<int> d_new(L);
        DevMem<uint32_t> sizes(L);
        CK(cudaMemcpyAsync(d_new.p, new_of_old.data(), sizeof(int) * L, cudaMemcpyHostToDevice, st));
        CK(cudaMemsetAsync(sizes.p, 0, sizeof(uint32_t) * L, st));
        k_renumber<<<blocks_for(n, 256), 256, 0, st>>>(list_of_id.p, n, d_new.p, sizes.p);
        k_iota<<<blocks_for(n, 256), 256, 0, st>>>(dids.p, n);
        CK(cudaMemcpyAsync(dz.p, zc.p, sizeof(uint64_t) * n, cudaMemcpyDeviceToDevice, st));
        RadixSort rs(n);
        int valid = 0, lbits = 0;
        for (int i = 0; i < g.l; i++) valid += (g.morton_valid_map >> i) & 1;
        while ((1ull << lbits) < L) lbits++;
        rs.sort(dz.p, dids.p, valid * g.morton_max_bits, st);
        k_gather_list<<<blocks_for(n, 256), 256, 0, st>>>(list_of_id.p, dids.p, n, dz.p);
        rs.sort(dz.p, dids.p, lbits, st);
        k_gather_z<<<blocks_for(n, 256), 256, 0, st>>>(zc.p, dids.p, n, dz.p);
        CK_LAUNCH();
        std::vector<uint32_t> hs(L);
        CK(cudaMemcpyAsync(hs.data(), sizes.p, sizeof(uint32_t) * L, cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        H.list_off.assign(L + 1, 0);
        for (uint64_t j = 0; j < L; j++) H.list_off[j + 1] = H.list_off[j] + hs[j];
    }

    // ---- 6. prefix counts ------------------------------------------------------------------
    DevMem<uint32_t> prefix(rows_form ? 0 : g.tot_cells * L);
    std::unique_ptr<DevMem<uint64_t>> row_off, rows;  // the compressed form
    if (rows_form) {
        build_prefix_rows(g, cell.p, list_of_id.p, n, (uint32_t)L, row_off, rows, H.prefix_entries, st);
    } else {
        CK(cudaMemsetAsync(prefix.p, 0, sizeof(uint32_t) * g.tot_cells * L, st));
        k_count_cells<<<blocks_for(n, 256), 256, 0, st>>>(cell.p, list_of_id.p, n, (uint32_t)L, prefix.p);
        for (int a = 0; a < g.l; a++) {
            const uint64_t inner = g.cell_stride[a];
            const uint64_t lines = g.tot_cells / (uint64_t)g.grid_dims[a] * L;
            k_scan_axis<<<blocks_for(lines, 256), 256, 0, st>>>(prefix.p, lines, inner, g.grid_dims[a],
                                                                (uint32_t)L);
        }
        CK_LAUNCH();
    }

    // ---- pool-ordered codes and labels ---------------------------------------------------
    DevMem<uint8_t> codes(n * H.M_pad);
    DevMem<float> labels(n * l);
    k_gather_codes_labels<<<blocks_for(n, 256), 256, 0, st>>>(codes_by_id.p, (int)H.M_pad, d_labels, (int)l, dids.p, n,
                                                             codes.p, labels.p);
    CK_LAUNCH();
    // the upload needs the pool-ordered arrays only: room for the arena beside them
    codes_by_id.reset();
    list_of_id.reset();
    zc.reset();
    cell.reset();
    Xs.reset();
    const DeviceArrays src{dz.p,       dids.p,     codes.p, labels.p, rows_form ? nullptr : prefix.p,
                           rows_form ? row_off->p : nullptr, rows_form ? rows->p : nullptr, labels_nan};
    idx->host = std::move(H);
    upload_index_from(idx, st, &src);
}

// Label-rank thresholds of n rows of l label dims (host memory, row-major [n][l]): per dim,
// the distinct values of a strided sample of at most 262,144 rows when they fit in 2^bits - 1
// thresholds (one rank per value), else the sample's quantiles (equal counts per rank); thr
// [l][2^bits - 1], n_thr [l], and each dim's smallest and largest label over every row.  NaN
// labels are left out of all of them.
void label_rank_thresholds(const float* labels, uint64_t n, int l, int bits, float* thr, uint32_t* n_thr, float* mn,
                           float* mx) {
    const uint32_t stride = (1u << bits) - 1u;
    const uint64_t step = std::max<uint64_t>(1, n / 262144);
#pragma omp parallel for
    for (int i = 0; i < l; i++) {
        std::vector<float> v;
        v.reserve(n / step + 1);
        for (uint64_t r = 0; r < n; r += step) {
            const float x = labels[r * l + i];
            if (!std::isnan(x)) v.push_back(x);
        }
        std::sort(v.begin(), v.end());
        float lo = INFINITY, hi = -INFINITY;  // over every label, not the sample
        for (uint64_t r = 0; r < n; r++) {
            const float x = labels[r * l + i];
            lo = std::min(lo, x);
            hi = std::max(hi, x);
        }
        mn[i] = lo;
        mx[i] = hi;
        const uint32_t m = thresholds_of(v, stride, thr + (size_t)i * stride);
        n_thr[i] = m;
    }
}

// The index's optional buffers (decoded vectors, rank planes) speed calls up that run without them too.
// They are kept while each takes at most a quarter of the memory that is free, and given back to a
// call that has no room otherwise (release_optional).
struct OptionalRoom {
    size_t free = 0;
    OptionalRoom() {
        size_t total = 0;
        CK(cudaMemGetInfo(&free, &total));
    }
    bool keep(DeviceBuffer& b, uint64_t bytes) {
        if (bytes > free / 4 || !b.try_ensure(bytes)) return false;
        free -= bytes;
        return true;
    }
};
constexpr uint64_t kDecodedMax = 16ull << 30;
constexpr uint64_t kPlanes = 512, kPlanesMax = 8ull << 30;  // label-rank bit planes: at most 64 bytes per point
constexpr uint64_t kDecodedMinPoints = 16384;  // smaller sets never reach the estimate pass

// Copy the host index into one device arena and fill idx->dev.
void upload_index(hdg_index* idx, cudaStream_t st) { upload_index_from(idx, st, nullptr); }

// src: arrays that the build still holds on the device, copied there instead of from the host
static void upload_index_from(hdg_index* idx, cudaStream_t st, const DeviceArrays* src) {
    idx->built = false;      // until every array is in place
    invalidate_graphs(idx);  // captured graphs hold the old arrays' addresses
    HostIndex& H = idx->host;
    // element counts of the large arrays, wherever they are
    const uint64_t n_dense = src ? (src->prefix ? H.grid.tot_cells * H.n_lists : 0) : H.prefix.size();
    const uint64_t n_off = src ? (src->prefix_off ? H.grid.tot_cells / (uint64_t)H.grid.grid_dims[H.grid.diff_dim] * H.n_lists + 1 : 0)
                               : H.prefix_off.size();
    if (!src) H.prefix_entries = H.prefix_rows.size();
    const uint64_t n_rows = n_off ? H.prefix_entries : 0;
    struct Part {
        const void* src;
        size_t bytes;
        void** dst;
    };
    uint16_t* cb = nullptr;
    uint16_t* scb = nullptr;
    float* cn = nullptr;
    IndexDev& D = idx->dev;
    D = IndexDev();
    std::vector<std::pair<size_t, size_t>> offs;
    size_t total = 0;
    auto reserve = [&](size_t bytes) {
        const size_t o = total;
        total += align_up(bytes ? bytes : 1, 256);
        return o;
    };
    const size_t o_c = reserve(H.centers.size() * 4), o_sc = reserve(H.sub_centers.size() * 4);
    const size_t o_cb = reserve(H.centers.size() * 2), o_scb = reserve(H.sub_centers.size() * 2);
    const size_t o_cn = reserve((H.C + H.n_lists) * 4);
    const size_t o_co = reserve(H.cluster_off.size() * 4), o_lo = reserve(H.list_off.size() * 4);
    GridMeta gp = H.grid;
    // label-rank thresholds, so that a rank box is about as tight as the labels
    const int rbits = H.n ? rank_bits_for((int)H.l) : 0;
    const uint32_t rstride = rbits ? (1u << rbits) - 1u : 0u;
    std::vector<float> rthr((size_t)H.l * rstride);
    uint32_t rn[kMaxDims] = {0};
    float rmin[kMaxDims] = {0.f}, rmax[kMaxDims] = {0.f};
    if (rbits && !src) {
        label_rank_thresholds(H.labels.data(), H.n, (int)H.l, rbits, rthr.data(), rn, rmin, rmax);
    } else if (rbits) {
        // the same from the device's labels: the strided sample sorted there, dim by dim
        const uint64_t step = std::max<uint64_t>(1, H.n / 262144), m = (H.n + step - 1) / step;
        const uint32_t l = (uint32_t)H.l;
        DevMem<uint64_t> keys(m);
        DevMem<uint32_t> vals(m);
        RadixSort rs(m);
        std::vector<uint64_t> hk(m);
        std::vector<float> v;
        std::vector<uint32_t> hr(2 * l + 1, 0u);
        std::fill(hr.begin(), hr.begin() + l, 0xffffffffu);
        DevMem<uint32_t> rg(2 * l + 1);
        CK(cudaMemcpyAsync(rg.p, hr.data(), sizeof(uint32_t) * hr.size(), cudaMemcpyHostToDevice, st));
        k_label_range<<<dim3(std::min(blocks_for(H.n, 256), 1024u), l), 256, 0, st>>>(src->labels, H.n, (int)l, rg.p, rg.p + l,
                                                                                     rg.p + 2 * l);
        CK_LAUNCH();
        CK(cudaMemcpyAsync(hr.data(), rg.p, sizeof(uint32_t) * hr.size(), cudaMemcpyDeviceToHost, st));
        for (uint32_t i = 0; i < l; i++) {
            k_rank_sample<<<blocks_for(m, 256), 256, 0, st>>>(src->labels, step, m, (int)l, (int)i, keys.p);
            k_iota<<<blocks_for(m, 256), 256, 0, st>>>(vals.p, m);
            CK_LAUNCH();
            rs.sort(keys.p, vals.p, 32, st);
            CK(cudaMemcpyAsync(hk.data(), keys.p, sizeof(uint64_t) * m, cudaMemcpyDeviceToHost, st));
            CK(cudaStreamSynchronize(st));
            v.clear();
            for (uint64_t k : hk) {
                if (k == 0xffffffffull) break;  // NaN labels sort last
                v.push_back(ordered_float((uint32_t)k));
            }
            rn[i] = thresholds_of(v, rstride, rthr.data() + (size_t)i * rstride);
            const bool any = hr[i] <= hr[l + i];
            rmin[i] = any ? ordered_float(hr[i]) : INFINITY;
            rmax[i] = any ? ordered_float(hr[l + i]) : -INFINITY;
        }
    }
    const size_t o_z = reserve(H.n * 8), o_id = reserve(H.n * 4);
    const size_t o_pk = reserve(rbits ? H.n * 4 : 0), o_rt = reserve(rthr.size() * 4);
    const size_t o_code = reserve(H.n * H.M_pad + 64), o_lab = reserve(H.n * H.l * 4);
    // a dense prefix count never exceeds its list's size: 16 bits suffice when no list passes 65535
    uint32_t max_list = 0;
    for (uint64_t j = 0; j + 1 < H.list_off.size(); j++) max_list = std::max(max_list, H.list_off[j + 1] - H.list_off[j]);
    const bool pre16 = n_dense && max_list <= 0xffffu;
    const size_t o_pq = reserve(H.pq_centers.size() * 4), o_pre = reserve(n_dense * (pre16 ? 2 : 4));
    const size_t o_poff = reserve(n_off * 8), o_prow = reserve(n_rows * 8);
    idx->planes.reset();
    idx->decoded.reset();
    idx->arena.reset();
    idx->arena.ensure(total);
    char* base = static_cast<char*>(idx->arena.ptr);
    auto up = [&](size_t off, const void* src, size_t bytes) {
        if (bytes) CK(cudaMemcpyAsync(base + off, src, bytes, cudaMemcpyHostToDevice, st));
        return base + off;
    };
    auto keep = [&](size_t off, const void* dev, const void* host, size_t bytes) {
        if (dev && bytes) CK(cudaMemcpyAsync(base + off, dev, bytes, cudaMemcpyDeviceToDevice, st));
        else up(off, host, bytes);
        return base + off;
    };
    D.centers = (const float*)up(o_c, H.centers.data(), H.centers.size() * 4);
    D.sub_centers = (const float*)up(o_sc, H.sub_centers.data(), H.sub_centers.size() * 4);
    cb = (uint16_t*)(base + o_cb);
    scb = (uint16_t*)(base + o_scb);
    cn = (float*)(base + o_cn);
    D.cluster_off = (const uint32_t*)up(o_co, H.cluster_off.data(), H.cluster_off.size() * 4);
    D.list_off = (const uint32_t*)up(o_lo, H.list_off.data(), H.list_off.size() * 4);
    D.zcodes = (const uint64_t*)keep(o_z, src ? src->zcodes : nullptr, H.zcodes.data(), H.n * 8);
    D.ids = (const uint32_t*)keep(o_id, src ? src->ids : nullptr, H.ids.data(), H.n * 4);
    D.labels_nan = src ? src->labels_nan : std::any_of(H.labels.begin(), H.labels.end(), [](float v) { return std::isnan(v); }) ? 1u : 0u;
    {
        // pool-ordered rows -> 16-byte chunk planes (the scan's coalesced layout)
        DevMem<uint8_t> rows(src ? 0 : std::max<size_t>(H.codes.size(), 16));
        if (H.n) {
            if (!src) CK(cudaMemcpyAsync(rows.p, H.codes.data(), H.codes.size(), cudaMemcpyHostToDevice, st));
            const uint64_t chunks = H.M_pad / 16;
            k_interleave_codes<<<blocks_for(H.n * chunks, 256), 256, 0, st>>>(
                reinterpret_cast<const uint4*>(src ? src->codes : rows.p), H.n, (uint32_t)chunks, reinterpret_cast<uint4*>(base + o_code));
            CK_LAUNCH();
        }
        CK(cudaStreamSynchronize(st));
        D.codes = (const uint8_t*)(base + o_code);
    }
    D.labels = (const float*)keep(o_lab, src ? src->labels : nullptr, H.labels.data(), H.n * H.l * 4);
    D.rank_bits = (uint32_t)rbits;
    D.rank_stride = rstride;
    D.rank_guard = 0;
    for (int i = 0; i < kMaxDims; i++) {
        D.rank_n[i] = i < (int)H.l ? rn[i] : 0u;
        D.rank_min[i] = i < (int)H.l ? rmin[i] : 0.f;
        D.rank_max[i] = i < (int)H.l ? rmax[i] : 0.f;
    }
    for (int i = 0; rbits && i < (int)H.l; i++) D.rank_guard |= 1u << (i * (rbits + 1) + rbits);
    D.rank_thr = rbits ? (const float*)up(o_rt, rthr.data(), rthr.size() * 4) : nullptr;
    D.rankpack = rbits ? reinterpret_cast<const uint32_t*>(base + o_pk) : nullptr;
    if (rbits) {
        k_pack_ranks<<<blocks_for(H.n, 256), 256, 0, st>>>(D.labels, H.n, (int)H.l, D.rank_thr, rstride, D,
                                                         reinterpret_cast<uint32_t*>(base + o_pk));
        CK_LAUNCH();
        CK(cudaStreamSynchronize(st));  // rthr is read by the copy
    }
    D.pq_centers = (const float*)up(o_pq, H.pq_centers.data(), H.pq_centers.size() * 4);
    if (n_off) {  // the compressed rows form
        D.prefix = nullptr;
        D.prefix16 = nullptr;
        D.prefix_off = (const uint64_t*)keep(o_poff, src ? src->prefix_off : nullptr, H.prefix_off.data(), n_off * 8);
        D.prefix_rows = (const uint64_t*)keep(o_prow, src ? src->prefix_rows : nullptr, H.prefix_rows.data(), n_rows * 8);
    } else {
        D.prefix = nullptr;
        D.prefix16 = nullptr;
        if (pre16 && src && src->prefix) {
            k_narrow16<<<blocks_for(n_dense, 256), 256, 0, st>>>(src->prefix, n_dense, reinterpret_cast<uint16_t*>(base + o_pre));
            CK_LAUNCH();
            D.prefix16 = reinterpret_cast<const uint16_t*>(base + o_pre);
        } else if (pre16) {
            std::vector<uint16_t> p16(H.prefix.size());
#pragma omp parallel for
            for (int64_t i = 0; i < (int64_t)H.prefix.size(); i++) p16[i] = (uint16_t)H.prefix[i];
            D.prefix16 = (const uint16_t*)up(o_pre, p16.data(), p16.size() * 2);
            CK(cudaStreamSynchronize(st));  // p16 is read by the copy
        } else {
            D.prefix = (const uint32_t*)keep(o_pre, src ? src->prefix : nullptr, H.prefix.data(), n_dense * 4);
        }
        D.prefix_off = D.prefix_rows = nullptr;
    }
    k_to_bf16<<<blocks_for(H.centers.size(), 256), 256, 0, st>>>(D.centers, H.centers.size(),
                                                                reinterpret_cast<__nv_bfloat16*>(cb));
    k_to_bf16<<<blocks_for(H.sub_centers.size(), 256), 256, 0, st>>>(
        D.sub_centers, H.sub_centers.size(), reinterpret_cast<__nv_bfloat16*>(scb));
    k_row_norms<<<blocks_for(H.C, 8), 256, 0, st>>>(D.centers, H.C, (int)H.d, cn);
    k_row_norms<<<blocks_for(H.n_lists, 8), 256, 0, st>>>(D.sub_centers, H.n_lists, (int)H.d, cn + H.C);
    D.centers_bf16 = cb;
    D.sub_centers_bf16 = scb;
    D.cnorm = cn;
    D.n = (uint32_t)H.n;
    D.d = (uint32_t)H.d;
    D.l = (uint32_t)H.l;
    D.M = (uint32_t)H.M;
    D.M_pad = (uint32_t)H.M_pad;
    D.pq_len = (uint32_t)H.pq_len;
    D.n_lists = (uint32_t)H.n_lists;
    D.C = (uint32_t)H.C;
    D.S_max = 0;
    for (uint64_t c = 0; c < H.C; c++)
        D.S_max = std::max<uint32_t>(D.S_max, H.cluster_off[c + 1] - H.cluster_off[c]);
    OptionalRoom room;
    // the ranks' bit planes: up to kPlanes of them in all, a bit of resolution less for as long as
    // they would take more than kPlanesMax bytes
    if (rbits && !D.labels_nan) {
        D.plane_words = align_up((H.n + 31) / 32, 8);
        D.plane_shift = 0;
        while ((H.l << rbits) >> D.plane_shift > kPlanes) D.plane_shift++;
        uint64_t planes = 0;
        for (;; D.plane_shift++) {
            planes = 0;
            for (uint64_t i = 0; i < H.l; i++) {
                D.plane_off[i] = (uint32_t)planes;
                planes += rn[i] >> D.plane_shift;
            }
            if (planes * D.plane_words * 4 <= kPlanesMax) break;
        }
        // (without room for them the predicate pass tests the packed ranks, one candidate at a time)
        if (room.keep(idx->planes, std::max<uint64_t>(planes * D.plane_words * 4, 16))) {
            k_rank_planes<<<blocks_for(D.plane_words, 64), 256, 0, st>>>(D, H.n, static_cast<uint32_t*>(idx->planes.ptr));
            CK_LAUNCH();
            D.rank_planes = static_cast<const uint32_t*>(idx->planes.ptr);
        }
    }
    // the estimate pass of the post-filter scan reads the points' PQ approximations as tensor-core
    // operands (2 d + 16 bytes per point; not kept past kDecodedMax, where the full scan runs, nor with one
    // label dim, whose schedule has no such scan)
    const uint64_t dec = align_up((uint64_t)H.n * H.d * 2, 256);
    if (H.l > 1 && H.d % 8 == 0 && H.M % 32 == 0 && H.M <= 96 && H.M * H.pq_len == H.d && H.n >= kDecodedMinPoints &&
        dec <= kDecodedMax && room.keep(idx->decoded, dec + (uint64_t)H.n * sizeof(float4) + 16)) {
        const uint64_t cst = (uint64_t)H.n * sizeof(float4);
        char* p = static_cast<char*>(idx->decoded.ptr);
        uint32_t* mx = reinterpret_cast<uint32_t*>(p + dec + cst);
        CK(cudaMemsetAsync(mx, 0, 16, st));
        k_decode_rows<<<blocks_for(H.n, 8), 256, 0, st>>>(D, reinterpret_cast<uint16_t*>(p),
                                                         reinterpret_cast<float4*>(p + dec), mx);
        CK_LAUNCH();
        D.decoded_max = mx;
        D.decoded = reinterpret_cast<const uint16_t*>(p);
        D.decoded_c = reinterpret_cast<const float4*>(p + dec);
    }
    idx->grid = gp;
    uint32_t hm[3] = {0, 0, 0};
    if (D.decoded) CK(cudaMemcpyAsync(hm, D.decoded_max, sizeof(hm), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    CK_LAUNCH();
    if (D.decoded) {
        // Rounding to FP16 leaves a residual of about 2^-12 of a vector.  One past 2^-6 (components above
        // 65,504 or among FP16's subnormals) makes every bound useless: a batch would pay for thresholds and
        // tiles before its full scan (1,500 queries x 60,000 candidates: 3.1 ms beside 3.5).
        float xm, rm;
        std::memcpy(&xm, &hm[1], 4);
        std::memcpy(&rm, &hm[2], 4);
        if (!(rm <= xm * 0x1p-6f && xm < INFINITY)) {
            idx->decoded.reset();
            D.decoded = nullptr;
            D.decoded_c = nullptr;
            D.decoded_max = nullptr;
        }
    }
    idx->built = true;
    (void)offs;
    // the device holds the one copy from here on
    std::vector<uint32_t>().swap(H.ids);
    std::vector<uint32_t>().swap(H.prefix);
    std::vector<uint64_t>().swap(H.prefix_off);
    std::vector<uint64_t>().swap(H.prefix_rows);
    std::vector<uint64_t>().swap(H.zcodes);
    std::vector<uint8_t>().swap(H.codes);
    std::vector<float>().swap(H.labels);
}

HostIndex fetch_host(const hdg_index* idx) {
    HostIndex H = idx->host;
    const IndexDev& D = idx->dev;
    auto down = [](auto& v, const void* src, uint64_t count) {
        v.resize(count);
        if (count) CK(cudaMemcpy(v.data(), src, count * sizeof(v[0]), cudaMemcpyDeviceToHost));
    };
    down(H.ids, D.ids, H.n);
    down(H.zcodes, D.zcodes, H.n);
    down(H.labels, D.labels, H.n * H.l);
    {  // chunk planes back to rows
        std::vector<uint8_t> planes;
        down(planes, D.codes, H.n * H.M_pad);
        H.codes.resize(H.n * H.M_pad);
        const uint64_t chunks = H.M_pad / 16;
#pragma omp parallel for
        for (int64_t r = 0; r < (int64_t)H.n; r++)
            for (uint64_t j = 0; j < chunks; j++)
                std::memcpy(&H.codes[(uint64_t)r * H.M_pad + 16 * j], &planes[(j * H.n + (uint64_t)r) * 16], 16);
    }
    const uint64_t cells = H.grid.tot_cells * H.n_lists;
    if (D.prefix_off) {
        down(H.prefix_off, D.prefix_off, H.grid.tot_cells / (uint64_t)H.grid.grid_dims[H.grid.diff_dim] * H.n_lists + 1);
        down(H.prefix_rows, D.prefix_rows, H.prefix_entries);
    } else if (D.prefix16) {
        std::vector<uint16_t> p16;
        down(p16, D.prefix16, cells);
        H.prefix.assign(p16.begin(), p16.end());
    } else {
        down(H.prefix, D.prefix, cells);
    }
    return H;
}

}  // namespace hdg
