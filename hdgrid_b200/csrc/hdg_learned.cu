// Learned per-query schedule: query features and a BF16 MLP (48 -> 128 -> 128 -> 2) with
// hand-written forward, backward and Adam kernels.
//
// The network predicts, per query, z0 = log2 of the number of inverted lists to probe and
// z1 = the logit of the predicate-first flag (1: label predicate inside the ADC pass, a budget
// of exps0 * k and an exact re-rank; 0: the index's own schedule,
// Super-Grid-IVF_PQ.cu:1151-1241).  It replaces the batch-wide n_list / sub_lists choice of
// super_grid::index::query for each query; the plain schedule stays the fallback.
//
// Precision: weights, inputs and hidden activations are rounded to BF16 (round to nearest
// even), every dot product accumulates in FP32, the optimiser keeps FP32 master weights.
//
// Features (48 per query, all scale-free):
//   [0, 8)   normalised filter bounds (lo, hi) of label dims 0..3: (x - left) / span in [0, 1]
//   [8, 12)  log10 of the normalised box width of dims 0..3, divided by 7
//   [12, 28) the 16 nearest coarse-centroid distances: log1p(d_0), then log1p(d_j) - log1p(d_0)
//   [28, 44) filtered point counts of those 16 clusters (the grid-cell histogram counts of the
//            query's cell box summed over each cluster's lists), log1p(count) / log1p(N)
//   [44]     log1p(filtered points over all lists) / log1p(N)   (selectivity estimate)
//   [45]     fraction of clusters holding any filtered point
//   [46]     k of the query / 100
//   [47]     log1p(filtered points of the 16 nearest clusters) / log1p(N)
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <random>
#include <type_traits>
#include <vector>

#include "hdg_device.cuh"
#include "hdg_internal.h"

namespace hdg {

namespace {

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

struct Params {
    const float* master;          // fp32 parameters (biases are read from here)
    const __nv_bfloat16* w;       // bf16 copies of the parameters (weights are read from here)
};

// ---- features --------------------------------------------------------------------------
// One 128-thread block per query (its phases are serial; small blocks keep more queries in flight)
__global__ void __launch_bounds__(128) k_features(IndexDev D, GridMeta g, const float* __restrict__ queries,
                                                  const float* __restrict__ box, const uint32_t* __restrict__ cc,
                                                  const uint32_t* __restrict__ qk, uint32_t k_max, int sort_n,
                                                  const float* __restrict__ S, uint64_t ldS,
                                                  const float* __restrict__ qnorm, float* __restrict__ feats) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t* s_keys = reinterpret_cast<uint64_t*>(smem);         // [sort_n]
    uint32_t* s_cand = reinterpret_cast<uint32_t*>(s_keys + sort_n);  // [sort_n]
    float* s_q = reinterpret_cast<float*>(s_cand + sort_n);        // [d]
    float* s_lo = s_q + D.d;                                         // [sort_n] the bands' lows
    __shared__ int s_ncand;
    __shared__ float s_bound;
    __shared__ float s_f[kMlpFeatures];
    __shared__ uint32_t s_hist[256], s_wc[32];
    __shared__ unsigned long long s_sel[4];
    __shared__ unsigned long long s_tot;
    __shared__ unsigned s_nz;
    const uint64_t qi = blockIdx.x;
    const int t = threadIdx.x, d = D.d, C = D.C, l = g.l;
    for (int i = t; i < d; i += blockDim.x) s_q[i] = queries[qi * d + i];
    if (t == 0) {
        s_tot = 0;
        s_nz = 0;
    }
    __syncthreads();
    unsigned long long tot = 0;
    unsigned nz = 0;
    for (int c = t; c < sort_n; c += blockDim.x) {
        if (c < C) {
            const uint32_t n = cc[qi * C + c];
            tot += n;
            nz += n > 0;
        } else {
            s_keys[c] = ~0ull;
        }
    }
    // centroid distances, one warp per centroid: the lanes read a row with coalesced loads
    // (the features only rank and log-scale these distances; no summation order is implied)
    // Four centroids per warp and step keep four independent row loads in flight; each
    // centroid's sum is formed exactly as with one per step (per-lane FMA chain, warp sum).
    const int lane = t & 31, warp = t >> 5, nw = blockDim.x >> 5;
    // With the coarse stage's tensor-core products S, only a centroid whose lower bound lies
    // within the 16th smallest upper bound can be among the 16 nearest (the 16 with the
    // smallest upper bounds are at or below it), so only those get exact distances: the same
    // 16 keys, each computed the same way
    const int kn = min(16, C);
    int n_ex = C;
    if (S) {
        for (int c = t; c < sort_n; c += blockDim.x) {
            uint64_t key = ~0ull;
            if (c < C) {
                float lo, hi;
                coarse_band(qnorm[qi], D.cnorm[c], S[qi * ldS + c], &lo, &hi);
                key = ((uint64_t)float_key(hi) << 32) | (uint32_t)c;
                s_lo[c] = lo;
            }
            s_keys[c] = key;
        }
        if (t == 0) s_ncand = 0;
        __syncthreads();
        // (only the k-th is needed: the keys stay in place)
        const uint64_t kth = block_select_smallest(s_keys, sort_n, kn, s_hist, s_wc, s_sel, false);
        if (t == 0) s_bound = key_float((uint32_t)(kth >> 32));
        __syncthreads();
        for (int c = t; c < sort_n; c += blockDim.x) {
            if (c < C && s_lo[c] <= s_bound) s_cand[atomicAdd(&s_ncand, 1)] = (uint32_t)c;
            s_keys[c] = ~0ull;
        }
        __syncthreads();
        n_ex = s_ncand;
    }
    auto cid = [&](int k) { return S ? (int)s_cand[k] : k; };
    constexpr int kCU = 4;
    for (int c0 = warp; c0 < n_ex; c0 += kCU * nw) {
        const float* row[kCU];
        float sq[kCU];
#pragma unroll
        for (int u = 0; u < kCU; u++) {
            row[u] = D.centers + (uint64_t)cid(min(c0 + u * nw, n_ex - 1)) * d;
            sq[u] = 0.f;
        }
        for (int i = lane; i < d; i += 32) {
            const float qv = s_q[i];
#pragma unroll
            for (int u = 0; u < kCU; u++) {
                const float df = qv - __ldg(row[u] + i);
                sq[u] = fmaf(df, df, sq[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < kCU; u++) {
            const float v = warp_sum(sq[u]);
            if (lane == 0 && c0 + u * nw < n_ex) {
                const int c = cid(c0 + u * nw);
                s_keys[c] = ((uint64_t)float_key(v) << 32) | (uint32_t)c;
            }
        }
    }
    atomicAdd(&s_tot, tot);
    atomicAdd(&s_nz, nz);
    __syncthreads();
    // the 16 nearest centroids (keys distinct: the centroid index is their low word), in order
    block_select_smallest(s_keys, sort_n, kn, s_hist, s_wc, s_sel);
    block_bitonic_sort(s_keys, (int)next_pow2_dev((uint32_t)max(kn, 2)));
    const float lnN = logf(1.f + (float)D.n);
    if (t < 16) {
        const int j = min(t, C - 1);
        const float dj = key_float((uint32_t)(s_keys[j] >> 32));
        const float d0 = key_float((uint32_t)(s_keys[0] >> 32));
        s_f[12 + t] = t == 0 ? log1pf(d0) : log1pf(dj) - log1pf(d0);
        const uint32_t c = (uint32_t)s_keys[j];
        s_f[28 + t] = t < C ? log1pf((float)cc[qi * C + c]) / lnN : 0.f;
    } else if (t < 20) {
        const int i = t - 16;  // original label dim
        float lo = 0.f, hi = 1.f;
        if (i < l) {
            int sd = 0;
            for (int s = 0; s < l; s++)
                if (g.shuffle[s] == i) sd = s;
            const float left = (float)g.left[sd], span = fmaxf((float)g.span[sd], 1.f);
            lo = fminf(fmaxf((box[qi * 2 * l + 2 * i] - left) / span, 0.f), 1.f);
            hi = fminf(fmaxf((box[qi * 2 * l + 2 * i + 1] - left) / span, 0.f), 1.f);
        }
        s_f[2 * i] = lo;
        s_f[2 * i + 1] = hi;
        s_f[8 + i] = log10f(fmaxf(hi - lo, 1e-7f)) / 7.f;
    }
    __syncthreads();
    if (t == 0) {
        float near = 0.f;
        for (int j = 0; j < 16 && j < C; j++) near += (float)cc[qi * C + (uint32_t)s_keys[j]];
        s_f[44] = log1pf((float)s_tot) / lnN;
        s_f[45] = (float)s_nz / (float)C;
        s_f[46] = (float)(qk ? max(1u, min(qk[qi], k_max)) : k_max) / 100.f;
        s_f[47] = log1pf(near) / lnN;
    }
    __syncthreads();
    if (t < kMlpFeatures) feats[qi * kMlpFeatures + t] = s_f[t];
}

// ---- forward and backward ----------------------------------------------------------------
// One kernel for inference and for a training step's whole forward and backward pass: 256
// threads, one tile of TS samples at a time, persistent over the tiles.  The weights are staged
// once per block, unit-major with rows padded by one word (49 and 129), so that both the staging
// writes and the reads of unit t's row across the threads are conflict-free.  Activations are
// unit-major rows of TS samples padded by 4 words: 16-byte reads, 8 consecutive rows on
// different banks.
//
// Training (GRAD): the tile's activations never leave shared memory.  The loss gradient, the
// two hidden gradients and the tile's share of every weight gradient follow from them, the
// weight gradients in registers (8 x 8 of W2 and 8 x 3 of W1 per thread) across the block's
// tiles; each block writes one partial row of all parameters, which k_grad_reduce sums.  A
// separate pass per layer, each output one serial sum over the batch, took 4.2 ms at 4,096 rows
// (one chain of dependent FMAs and loads per weight, 128 blocks, eight allocations a call);
// gradients plus a forward call now take 78 us together.
// Bound: FMA issue of one block per SM (about 2 M FMAs per 32 samples) and, below one tile per
// SM, the latency of one tile.
struct FwdOut {
    float* z;            // [n x 2]
    uint32_t* nprobe;    // inference: per-query lists to probe
    uint8_t* sched;      // inference: per-query schedule flag
    int allow_sched;
    uint32_t max_probe;
    const float* y;      // training: targets [rows x 2]
    const uint32_t* rows;  // training: row of sample b in x and y (nullptr: b)
    float* part;         // training: [blocks x kMlpParams] partial gradients
    double* loss;        // training: [blocks] partial loss sums
};

constexpr int kFwdThreads = 256;

template <int TS, bool GRAD>
constexpr size_t forward_smem() {
    return sizeof(float) * ((kMlpFeatures + 1) * kMlpHidden + (kMlpHidden + 1) * kMlpHidden + kMlpOut * kMlpHidden +
                            (kMlpFeatures + (GRAD ? 3 : 2) * kMlpHidden) * (TS + 4) + kMlpOut * TS);
}

template <int TS, bool GRAD>
__global__ void __launch_bounds__(kFwdThreads) k_mlp(Params P, const float* __restrict__ x, uint64_t n, FwdOut o) {
    constexpr int S1 = kMlpFeatures + 1, S2 = kMlpHidden + 1;  // padded weight rows
    constexpr int SH = TS + 4;                                 // activation rows
    constexpr int TH = TS / 2;                                 // samples per thread in a hidden layer
    extern __shared__ __align__(16) float sm[];
    float* xs = sm;                                    // [48][SH]: feature-major inputs
    float* h1 = xs + kMlpFeatures * SH;                // [128][SH]: unit-major activations
    float* h2 = h1 + kMlpHidden * SH;                  // [128][SH]
    float* g2 = h2 + kMlpHidden * SH;                  // [128][SH] (GRAD): gradient at hidden 2
    float* dz = g2 + (GRAD ? kMlpHidden * SH : 0);     // [2][TS] loss gradient at the outputs
    float* w1p = dz + kMlpOut * TS;                    // [128][49]: unit-major W1
    float* w2p = w1p + kMlpHidden * S1;                // [128][129]
    float* w3 = w2p + kMlpHidden * S2;                 // [2][128]
    __shared__ double s_loss[kFwdThreads / 32];
    const int t = threadIdx.x, u = t & (kMlpHidden - 1), half = t / kMlpHidden;
    for (int e = t; e < kMlpHidden * kMlpFeatures; e += kFwdThreads)
        w1p[(e / kMlpFeatures) * S1 + e % kMlpFeatures] = __bfloat162float(P.w[kMlpW1 + e]);
    for (int e = t; e < kMlpHidden * kMlpHidden; e += kFwdThreads)
        w2p[(e / kMlpHidden) * S2 + e % kMlpHidden] = __bfloat162float(P.w[kMlpW2 + e]);
    for (int e = t; e < kMlpOut * kMlpHidden; e += kFwdThreads) w3[e] = __bfloat162float(P.w[kMlpW3 + e]);
    const float bias1 = P.master[kMlpB1 + u], bias2 = P.master[kMlpB2 + u];
    // acc[b] = sum over r of w[r * ws] * in[r][b], in order r = 0, 1, ..., for this thread's half
    // of the samples (read four at a time as broadcasts)
    auto layer = [&](const float* w, int ws, const float* in, int rows, float (&acc)[TH]) {
#pragma unroll
        for (int b = 0; b < TH; b++) acc[b] = 0.f;
#pragma unroll 4
        for (int r = 0; r < rows; r++) {
            const float wv = w[r * ws];
            const float4* v = reinterpret_cast<const float4*>(in + r * SH + half * TH);
#pragma unroll
            for (int b4 = 0; b4 < TH / 4; b4++) {
                const float4 a = v[b4];
                acc[4 * b4] = fmaf(wv, a.x, acc[4 * b4]);
                acc[4 * b4 + 1] = fmaf(wv, a.y, acc[4 * b4 + 1]);
                acc[4 * b4 + 2] = fmaf(wv, a.z, acc[4 * b4 + 2]);
                acc[4 * b4 + 3] = fmaf(wv, a.w, acc[4 * b4 + 3]);
            }
        }
    };
    auto put = [&](float* row, const float (&v)[TH]) {
#pragma unroll
        for (int b4 = 0; b4 < TH / 4; b4++)
            reinterpret_cast<float4*>(row + half * TH)[b4] =
                make_float4(v[4 * b4], v[4 * b4 + 1], v[4 * b4 + 2], v[4 * b4 + 3]);
    };
    // GRAD: the block's weight gradients so far.  Rows to*8 .. +7 (outputs), columns ti + 16 k
    const int ti = t & 15, to = t >> 4;
    float gw2[GRAD ? 8 : 1][8], gw1[GRAD ? 8 : 1][3];
    float gw3 = 0.f, gb = 0.f, gb3 = 0.f;  // W3[half][u]; b1 (half 0) or b2 (half 1) of unit u; b3[t]
    double lsum = 0.0;
    if constexpr (GRAD) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
#pragma unroll
            for (int k = 0; k < 8; k++) gw2[i][k] = 0.f;
#pragma unroll
            for (int k = 0; k < 3; k++) gw1[i][k] = 0.f;
        }
    }
    // tile share of dW[to*8 + i][ti + 16 k] = sum_b dy[row][b] * in[col][b]
    auto outer = [&](const float* dy, const float* in, auto& acc, auto kc) {
        constexpr int K = decltype(kc)::value;
#pragma unroll 1
        for (int b4 = 0; b4 < TS / 4; b4++) {
            float4 dv[8], av[K];
#pragma unroll
            for (int i = 0; i < 8; i++) dv[i] = reinterpret_cast<const float4*>(dy + (to * 8 + i) * SH)[b4];
#pragma unroll
            for (int k = 0; k < K; k++) av[k] = reinterpret_cast<const float4*>(in + (ti + 16 * k) * SH)[b4];
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int k = 0; k < K; k++) {
                    acc[i][k] = fmaf(dv[i].x, av[k].x, acc[i][k]);
                    acc[i][k] = fmaf(dv[i].y, av[k].y, acc[i][k]);
                    acc[i][k] = fmaf(dv[i].z, av[k].z, acc[i][k]);
                    acc[i][k] = fmaf(dv[i].w, av[k].w, acc[i][k]);
                }
        }
    };
    auto row_of = [&](uint64_t b) -> uint64_t { return GRAD && o.rows ? (uint64_t)o.rows[b] : b; };
    for (uint64_t b0 = (uint64_t)blockIdx.x * TS; b0 < n; b0 += (uint64_t)gridDim.x * TS) {
        __syncthreads();  // the weights are staged; the previous tile's reads are done
        for (int e = t; e < TS * kMlpFeatures; e += kFwdThreads) {
            const int b = e / kMlpFeatures, i = e % kMlpFeatures;
            xs[i * SH + b] = b0 + b < n ? bf16r(x[row_of(b0 + b) * kMlpFeatures + i]) : 0.f;
        }
        __syncthreads();
        float acc[TH];
        layer(w1p + u * S1, 1, xs, kMlpFeatures, acc);
#pragma unroll
        for (int b = 0; b < TH; b++) acc[b] = bf16r(fmaxf(acc[b] + bias1, 0.f));
        put(h1 + u * SH, acc);
        __syncthreads();
        layer(w2p + u * S2, 1, h1, kMlpHidden, acc);
#pragma unroll
        for (int b = 0; b < TH; b++) acc[b] = bf16r(fmaxf(acc[b] + bias2, 0.f));
        put(h2 + u * SH, acc);
        __syncthreads();
        if (t < TS * kMlpOut) {
            const int b = t >> 1, c = t & 1;
            float z = 0.f;
#pragma unroll 8
            for (int j2 = 0; j2 < kMlpHidden; j2++) z = fmaf(w3[c * kMlpHidden + j2], h2[j2 * SH + b], z);
            z += P.master[kMlpB3 + c];
            const uint64_t bi = b0 + b;
            if (bi < n) {
                if (o.z) o.z[bi * kMlpOut + c] = z;
                if (c == 0 && o.nprobe) {
                    const float p = exp2f(fminf(fmaxf(z, 0.f), 20.f));
                    o.nprobe[bi] = (uint32_t)min((float)o.max_probe, fmaxf(1.f, rintf(p)));
                }
                if (c == 1 && o.sched) o.sched[bi] = (o.allow_sched && z > 0.f) ? 1 : 0;
            }
            if constexpr (GRAD) {
                // loss = mean over the batch of (z0 - y0)^2 + BCE(sigmoid(z1), y1); a tile's missing
                // samples have gradient 0
                float g = 0.f;
                if (bi < n) {
                    const float yv = o.y[row_of(bi) * kMlpOut + c];
                    const float inv = 1.f / (float)n;
                    if (c == 0) {
                        g = 2.f * (z - yv) * inv;
                        lsum += (double)(z - yv) * (z - yv);
                    } else {
                        const float s = 1.f / (1.f + expf(-z));
                        g = (s - yv) * inv;
                        // numerically stable BCE with logits: max(z,0) - z*y + log(1 + exp(-|z|))
                        lsum += (double)(fmaxf(z, 0.f) - z * yv + log1pf(expf(-fabsf(z))));
                    }
                }
                dz[c * TS + b] = g;
            }
        }
        if constexpr (GRAD) {
            __syncthreads();
            // hidden 2: g2[u][b] = (dz[0][b] W3[0][u] + dz[1][b] W3[1][u]) where h2 > 0; W3 and b3
            {
                const float w30 = w3[u], w31 = w3[kMlpHidden + u];
                float g[TH], s = 0.f;
#pragma unroll
                for (int b = 0; b < TH; b++) {
                    const int bb = half * TH + b;
                    g[b] = h2[u * SH + bb] > 0.f ? fmaf(dz[TS + bb], w31, dz[bb] * w30) : 0.f;
                }
                put(g2 + u * SH, g);
#pragma unroll
                for (int b = 0; b < TS; b++) s = fmaf(dz[half * TS + b], h2[u * SH + b], s);
                gw3 += s;
                if (t < kMlpOut) {
                    float sb = 0.f;
#pragma unroll
                    for (int b = 0; b < TS; b++) sb += dz[t * TS + b];
                    gb3 += sb;
                }
            }
            __syncthreads();
            // hidden 1: sum over o of g2[o][b] W2[o][u] where h1 > 0, kept in h2's place (its last
            // readers are behind the barrier)
            layer(w2p + u, S2, g2, kMlpHidden, acc);
#pragma unroll
            for (int b = 0; b < TH; b++) acc[b] = h1[u * SH + half * TH + b] > 0.f ? acc[b] : 0.f;
            put(h2 + u * SH, acc);
            outer(g2, h1, gw2, std::integral_constant<int, 8>());
            __syncthreads();
            outer(h2, xs, gw1, std::integral_constant<int, 3>());
            const float* gr = (half ? g2 : h2) + u * SH;
            float s = 0.f;
#pragma unroll
            for (int b = 0; b < TS; b++) s += gr[b];
            gb += s;
        }
    }
    if constexpr (GRAD) {
        float* p = o.part + (uint64_t)blockIdx.x * kMlpParams;
#pragma unroll
        for (int i = 0; i < 8; i++) {
#pragma unroll
            for (int k = 0; k < 8; k++) p[kMlpW2 + (to * 8 + i) * kMlpHidden + ti + 16 * k] = gw2[i][k];
#pragma unroll
            for (int k = 0; k < 3; k++) p[kMlpW1 + (to * 8 + i) * kMlpFeatures + ti + 16 * k] = gw1[i][k];
        }
        p[kMlpW3 + half * kMlpHidden + u] = gw3;
        p[(half ? kMlpB2 : kMlpB1) + u] = gb;
        if (t < kMlpOut) p[kMlpB3 + t] = gb3;
        for (int k = 16; k > 0; k >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, k);
        if ((t & 31) == 0) s_loss[t >> 5] = lsum;
        __syncthreads();
        if (t == 0) {
            double l = 0.0;
            for (int k = 0; k < kFwdThreads / 32; k++) l += s_loss[k];
            o.loss[blockIdx.x] = l;
        }
    }
}

// One Adam update (b1, b2, eps; c1, c2 the bias corrections); lr 0 with m = nullptr: none.
struct AdamStep {
    float *p, *m, *v;
    float lr, b1, b2, eps, c1, c2;
    __nv_bfloat16* pw;
};

// Gradient = sum of the blocks' partial rows, then the Adam update when a.m is given.  32
// parameters per block, 8 threads each over every 8th row (up to 19 loads in flight per thread),
// in a fixed order.  Bound: the partial rows' L2 reads (13 MB at 148 rows).
__global__ void __launch_bounds__(256) k_grad_reduce(const float* __restrict__ part, int nb,
                                                     const double* __restrict__ lpart, uint64_t n, int accumulate,
                                                     float* __restrict__ grad, double* __restrict__ loss, AdamStep a) {
    __shared__ float s_p[8][33];
    const int lane = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (i < kMlpParams) {
#pragma unroll 4
        for (int r = y; r < nb; r += 8) s += __ldcg(part + (uint64_t)r * kMlpParams + i);
    }
    s_p[y][lane] = s;
    __syncthreads();
    if (y == 0 && i < kMlpParams) {
        float g = ((s_p[0][lane] + s_p[1][lane]) + (s_p[2][lane] + s_p[3][lane])) +
                  ((s_p[4][lane] + s_p[5][lane]) + (s_p[6][lane] + s_p[7][lane]));
        if (grad) grad[i] = g;
        if (a.m) {
            const float mi = a.b1 * a.m[i] + (1.f - a.b1) * g;
            const float vi = a.b2 * a.v[i] + (1.f - a.b2) * g * g;
            a.m[i] = mi;
            a.v[i] = vi;
            const float pi = a.p[i] - a.lr * (mi / a.c1) / (sqrtf(vi / a.c2) + a.eps);
            a.p[i] = pi;
            a.pw[i] = __float2bfloat16_rn(pi);
        }
    }
    if (blockIdx.x == 0 && y == 1) {  // the mean loss of the batch
        double l = 0.0;
        for (int r = lane; r < nb; r += 32) l += __ldcg(lpart + r);
        for (int k = 16; k > 0; k >>= 1) l += __shfl_xor_sync(0xffffffffu, l, k);
        if (lane == 0) *loss = (accumulate ? *loss : 0.0) + l / (double)n;
    }
}

__global__ void k_to_bf16_params(const float* __restrict__ p, int n, __nv_bfloat16* __restrict__ pw) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) pw[i] = __float2bfloat16_rn(p[i]);
}

// model buffer: master | adam m | adam v (fp32, kMlpParams each) | bf16 copy
struct ModelPtrs {
    float *master, *m, *v;
    __nv_bfloat16* w;
};

ModelPtrs model_ptrs(hdg_index* idx) {
    if (!idx->mlp.ptr) {
        idx->mlp.ensure(sizeof(float) * 3 * kMlpParams + sizeof(__nv_bfloat16) * kMlpParams + 256);
        CK(cudaMemset(idx->mlp.ptr, 0, idx->mlp.bytes));
    }
    float* base = static_cast<float*>(idx->mlp.ptr);
    ModelPtrs p;
    p.master = base;
    p.m = base + kMlpParams;
    p.v = base + 2 * kMlpParams;
    p.w = reinterpret_cast<__nv_bfloat16*>(base + 3 * kMlpParams);
    return p;
}

// Blocks of a pass over n samples in tiles of ts: one per SM at most (the staged weights fill it)
int mlp_blocks(uint64_t n, int ts) { return (int)std::min<uint64_t>((n + ts - 1) / ts, (uint64_t)sm_count()); }

// Tile size for n samples: a tile costs a fixed part (about 12 samples' worth: staging, barriers,
// the output layer's chain) plus its samples, and the pass lasts as long as the block with the
// most tiles; the smallest such time wins.
int mlp_tile(uint64_t n) {
    int best = 8;
    uint64_t cost = ~0ull;
    for (int ts : {8, 16, 32}) {
        const uint64_t tiles = (n + ts - 1) / ts, rounds = (tiles + sm_count() - 1) / sm_count();
        if (rounds * (ts + 12) < cost) {
            cost = rounds * (ts + 12);
            best = ts;
        }
    }
    return best;
}

template <bool GRAD>
int launch_mlp(const ModelPtrs& mp, const float* x, uint64_t n, const FwdOut& o, cudaStream_t st) {
    auto go = [&](auto tsc) {
        constexpr int TS = decltype(tsc)::value;
        constexpr size_t sm = forward_smem<TS, GRAD>();
        allow_smem(k_mlp<TS, GRAD>);
        const int blocks = std::max(1, mlp_blocks(n, TS));
        k_mlp<TS, GRAD><<<blocks, kFwdThreads, sm, st>>>(Params{mp.master, mp.w}, x, n, o);
        CK_LAUNCH();
        return blocks;
    };
    const int ts = mlp_tile(n);
    if (ts == 8) return go(std::integral_constant<int, 8>());
    if (ts == 16) return go(std::integral_constant<int, 16>());
    return go(std::integral_constant<int, 32>());
}

// Scratch of a training pass, kept in the index (14 MB at most): one partial gradient row and
// loss sum per block, then the batch loss.
struct TrainScratch {
    float* part;
    double *lpart, *loss;
};
TrainScratch train_scratch(hdg_index* idx) {
    const size_t rows = (size_t)sm_count(), part = align_up(rows * kMlpParams * sizeof(float), 256);
    idx->mlp_work.ensure(part + (rows + 1) * sizeof(double));
    char* b = static_cast<char*>(idx->mlp_work.ptr);
    TrainScratch t;
    t.part = reinterpret_cast<float*>(b);
    t.lpart = reinterpret_cast<double*>(b + part);
    t.loss = t.lpart + rows;
    return t;
}

// Forward, backward and the summed gradient (into grad when given) of one batch; with a.m, the
// Adam update too.  accumulate: the batch's mean loss is added to *s.loss instead of stored.
void train_pass(const ModelPtrs& mp, const TrainScratch& s, const float* x, const float* y, const uint32_t* rows,
                uint64_t n, int accumulate, float* grad, const AdamStep& a, cudaStream_t st) {
    const FwdOut o{nullptr, nullptr, nullptr, 0, 0, y, rows, s.part, s.lpart};
    const int nb = launch_mlp<true>(mp, x, n, o, st);
    k_grad_reduce<<<(kMlpParams + 31) / 32, 256, 0, st>>>(s.part, nb, s.lpart, n, accumulate, grad, s.loss, a);
    CK_LAUNCH();
}

}  // namespace

void learned_features(hdg_index* idx, const float* d_queries, uint64_t q, const float* box, const uint32_t* cc,
                      const uint32_t* qk, uint32_t k_max, float* feats, cudaStream_t st, const float* S, uint64_t ldS,
                      const float* qnorm) {
    const IndexDev& D = idx->dev;
    const int sort_n = (int)next_pow2(std::max<uint32_t>(D.C, 16));
    const size_t sm = (sizeof(uint64_t) + sizeof(uint32_t) + sizeof(float)) * sort_n + sizeof(float) * D.d;
    HDG_REQUIRE(sm <= 200 * 1024, HDG_ERR_UNSUPPORTED, "feature kernel does not fit shared memory");
    allow_smem(k_features);
    k_features<<<(unsigned)q, 128, sm, st>>>(D, idx->grid, d_queries, box, cc, qk, k_max, sort_n, S, ldS, qnorm,
                                             feats);
    CK_LAUNCH();
}

void learned_infer(hdg_index* idx, const float* feats, uint64_t q, uint32_t* nprobe, uint8_t* sched, int allow_sched,
                   uint32_t max_probe, float* z, cudaStream_t st) {
    HDG_REQUIRE(idx->mlp_ready, HDG_ERR_STATE, "no trained model in this index");
    const ModelPtrs mp = model_ptrs(idx);
    launch_mlp<false>(mp, feats, q, FwdOut{z, nprobe, sched, allow_sched, max_probe, nullptr, nullptr, nullptr, nullptr},
                      st);
}

void mlp_init(hdg_index* idx, uint64_t seed) {
    const ModelPtrs mp = model_ptrs(idx);
    std::vector<float> p(kMlpParams, 0.f);
    std::mt19937_64 rng(seed);
    auto fill = [&](int off, int fan_in, int count) {  // He-uniform for the ReLU layers
        const float a = std::sqrt(6.f / (float)fan_in);
        std::uniform_real_distribution<float> u(-a, a);
        for (int i = 0; i < count; i++) p[off + i] = u(rng);
    };
    fill(kMlpW1, kMlpFeatures, kMlpHidden * kMlpFeatures);
    fill(kMlpW2, kMlpHidden, kMlpHidden * kMlpHidden);
    fill(kMlpW3, kMlpHidden, kMlpOut * kMlpHidden);
    mlp_set(idx, p.data(), kMlpParams);
}

void mlp_set(hdg_index* idx, const float* host, size_t count) {
    HDG_REQUIRE(count == (size_t)kMlpParams, HDG_ERR_INVALID_ARG, "wrong parameter count for the MLP");
    const ModelPtrs mp = model_ptrs(idx);
    CK(cudaMemcpy(mp.master, host, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice));
    CK(cudaMemset(mp.m, 0, sizeof(float) * 2 * kMlpParams));
    k_to_bf16_params<<<(kMlpParams + 255) / 256, 256>>>(mp.master, kMlpParams, mp.w);
    CK_LAUNCH();
    CK(cudaDeviceSynchronize());
    idx->mlp_step = 0;
    idx->mlp_ready = true;
}

void mlp_get(hdg_index* idx, float* host, size_t count) {
    HDG_REQUIRE(idx->mlp_ready, HDG_ERR_STATE, "no model in this index");
    HDG_REQUIRE(count == (size_t)kMlpParams, HDG_ERR_INVALID_ARG, "wrong parameter count for the MLP");
    const ModelPtrs mp = model_ptrs(idx);
    CK(cudaMemcpy(host, mp.master, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost));
}

void mlp_forward(hdg_index* idx, const float* d_x, uint64_t n, float* d_z, cudaStream_t st) {
    HDG_REQUIRE(idx->mlp_ready, HDG_ERR_STATE, "no model in this index");
    const ModelPtrs mp = model_ptrs(idx);
    launch_mlp<false>(mp, d_x, n, FwdOut{d_z, nullptr, nullptr, 0, 0, nullptr, nullptr, nullptr, nullptr}, st);
}

double mlp_gradients(hdg_index* idx, const float* d_x, const float* d_y, uint64_t n, float* d_grad, cudaStream_t st) {
    HDG_REQUIRE(idx->mlp_ready, HDG_ERR_STATE, "no model in this index");
    HDG_REQUIRE(n > 0, HDG_ERR_INVALID_ARG, "empty batch");
    const ModelPtrs mp = model_ptrs(idx);
    std::lock_guard<std::mutex> lock(idx->mlp_mu);  // the scratch serves one call at a time
    const TrainScratch ts = train_scratch(idx);
    train_pass(mp, ts, d_x, d_y, nullptr, n, 0, d_grad, AdamStep{}, st);
    double h = 0.0;
    CK(cudaMemcpyAsync(&h, ts.loss, sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    return h;
}

double mlp_train(hdg_index* idx, const float* d_x, const float* d_y, uint64_t n, uint32_t epochs, uint32_t batch,
                 float lr, uint64_t seed, cudaStream_t st) {
    HDG_REQUIRE(idx->mlp_ready, HDG_ERR_STATE, "initialise or load the model first");
    HDG_REQUIRE(n > 0 && batch > 0 && epochs > 0, HDG_ERR_INVALID_ARG, "empty training run");
    const ModelPtrs mp = model_ptrs(idx);
    const uint64_t B = std::min<uint64_t>(batch, n);
    std::lock_guard<std::mutex> lock(idx->mlp_mu);
    const TrainScratch ts = train_scratch(idx);
    DevMem<uint32_t> perm(n);
    std::vector<uint32_t> order(n);
    for (uint64_t i = 0; i < n; i++) order[i] = (uint32_t)i;
    std::mt19937_64 rng(seed);
    double last = 0.0;
    for (uint32_t ep = 0; ep < epochs; ep++) {
        std::shuffle(order.begin(), order.end(), rng);
        CK(cudaMemcpyAsync(perm.p, order.data(), sizeof(uint32_t) * n, cudaMemcpyHostToDevice, st));
        uint64_t steps = 0;
        for (uint64_t s = 0; s + B <= n || (s < n && steps == 0); s += B) {
            const uint64_t nb = std::min<uint64_t>(B, n - s);
            idx->mlp_step++;
            const float b1 = 0.9f, b2 = 0.999f;
            const float c1 = 1.f - std::pow(b1, (float)idx->mlp_step), c2 = 1.f - std::pow(b2, (float)idx->mlp_step);
            train_pass(mp, ts, d_x, d_y, perm.p + s, nb, steps > 0, nullptr,
                       AdamStep{mp.master, mp.m, mp.v, lr, b1, b2, 1e-8f, c1, c2, mp.w}, st);
            steps++;
        }
        double h = 0.0;
        CK(cudaMemcpyAsync(&h, ts.loss, sizeof(double), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        last = h / (double)std::max<uint64_t>(steps, 1);
    }
    return last;
}

}  // namespace hdg
