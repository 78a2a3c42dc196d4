// Distance estimates on the tensor cores (hdg_est.cuh).
//
// Persistent, one CTA per SM, 20 warps: 0-15 epilogue (two groups of eight, taking turns at the
// items), 16 MMA issue and TMEM, 17 the rows by TMA (a tile's rows are consecutive), 18-19 the
// queries by cp.async (any queries, gathered by id into the 128-byte-swizzled layout).  A work item
// is one tile of 128 rows x 128 queries; every CTA takes an equal, consecutive span of them, so
// successive items share their rows in L2.  K runs in chunks of 64 through a ring of stages (full
// barriers: one for the TMA bytes, one for the two gathering warps; the tcgen05.commit of a
// chunk's MMAs frees its stage).  Four accumulators of 128 TMEM columns keep the MMAs ahead.
//
// Epilogue of an item: thread = row, loop over columns (queries), two at a time in packed FP32
// FMAs against the queries' constants, broadcast from shared memory; a ballot per column and warp
// gives the column's 128-bit mask.  One thread per column then reserves the kept rows' slots with
// one atomic, whose latency runs under the group's next item, after whose masks the group writes
// the kept rows, shared out evenly over its threads (a prefix over the columns, the n-th set bit).
// Bound: the epilogue's issue slots, 12,700 warp instructions per item at about 2 per clock.
// 154,000 items of K = 128 (10,000 queries x 227,000 candidates): 6.6 ms with one epilogue group
// and a warp per column writing its kept rows (15,000 instructions, 35 % issue), 4.1 ms with two
// groups and the even sharing, 5.0 ms with the steps as well.  A thread per column walking its mask
// took 11.4 ms (64-deep loops where a query is near); TMA gather4 instead of cp.async left this
// case alone and took 0.9 ms more at K = 384.  Every wait is bounded: on expiry the kernel sets
// *err, lets its copies land, frees TMEM and returns.
#include <cuda.h>

#include <algorithm>

#include "hdg_est.cuh"
#include "hdg_internal.h"
#include "hdg_umma.cuh"

namespace hdg {

namespace {

constexpr int kEpiThreads = 256, kGroups = 2, kAccs = 4;  // threads per epilogue group
constexpr int kEstThreads = kGroups * kEpiThreads + 128;
constexpr uint32_t kChunkBytes = 128 * 64 * 2;  // one 128 x 64 FP16 operand chunk
constexpr int kMaxStages = 4;
// ring stages: the steps of two pending items per group take the fourth stage's room
constexpr int est_stages(bool ranges) { return ranges ? 3 : 4; }
constexpr int kSlots = 3;  // column constants: read through the group's following item

struct EstGroup {  // of one epilogue group
    float4 ab[kSlots][kEstN / 2];    // {a0, a1, b0, b1} of a pair of columns
    float4 zs[kSlots][kEstN / 2];    // {z0, z1, steps0, steps1}
    float2 sb[kSlots][kEstN / 2];    // the steps' bias: 2^23 + 1 - z * steps
    uint64_t off[kSlots][kEstN];     // ranges: the query's row offset
    uint32_t qid[kSlots][kEstN];
    uint32_t delta[kSlots][kEstN];
    uint32_t lohi[kSlots][kEstN];
    uint4 mask[2][kEstN];
    uint32_t base[2][kEstN];         // the query's slot of its first kept row
    uint32_t pre[2][kEstN];          // kept rows of the columns before, within the column's warp
    uint32_t wsum[2][kEstN / 32];    // kept rows of 32 columns
};
struct EstShared {
    EstGroup grp[kGroups];
    uint64_t full_a[kMaxStages], full_b[kMaxStages], empty[kMaxStages], acc_full[kAccs], acc_empty[kAccs];
    uint32_t tmem;
    int fail;
};

// a bounded wait that also gives up once another role has failed
__device__ __forceinline__ bool est_wait(EstShared& s, uint64_t& bar, uint32_t parity) {
    const uint32_t b = smem_u32(&bar);
    for (long long it = 0; it < kSpinLimit; it++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred P1;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, P1;\n\t}"
            : "=r"(done)
            : "r"(b), "r"(parity)
            : "memory");
        if (done) return true;
        if (*(volatile int*)&s.fail) return false;
    }
    *(volatile int*)&s.fail = 1;
    return false;
}
__device__ __forceinline__ void est_arrive(uint64_t& bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&bar)) : "memory");
}
__device__ __forceinline__ void est_commit(uint64_t& bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&bar))
                 : "memory");
}
__device__ __forceinline__ void epi_bar(int group) { asm volatile("bar.sync %0, 256;" ::"r"(1 + group) : "memory"); }
// (d0, d1) = (a0, a1) * (b0, b1) + (c0, c1), each rounded like one fmaf
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rc;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 ra, ra, rb, rc;\n\tmov.b64 {%0, %1}, ra;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(addr));
}
__device__ __forceinline__ void tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// The items of this CTA in order: row tile t, its query tile j
template <bool RANGES>
struct Walk {
    const EstArgs& a;
    uint32_t t = 0, j = 0, nt = 0;  // nt: query tiles of row tile t
    uint32_t e0 = 0, n_ent = 0;     // its entries
    __device__ Walk(const EstArgs& args) : a(args) {}
    __device__ uint32_t total() const {
        return RANGES ? a.nt_off[a.tiles] : a.tiles * ((a.nq + kEstN - 1) / kEstN);
    }
    __device__ void load() {
        if (RANGES) {
            e0 = a.ent_off[t];
            n_ent = a.ent_off[t + 1] - e0;
            nt = (n_ent + kEstN - 1) / kEstN;
        }
    }
    __device__ void seek(uint32_t item) {
        if (RANGES) {  // the tile whose query tiles hold the item: the last one with nt_off <= item
            uint32_t lo = 0, hi = a.tiles - 1;
            while (lo < hi) {
                const uint32_t mid = lo + (hi - lo + 1) / 2;
                if (a.nt_off[mid] <= item) lo = mid;
                else hi = mid - 1;
            }
            t = lo;
            j = item - a.nt_off[t];
            load();
        } else {
            nt = (a.nq + kEstN - 1) / kEstN;
            n_ent = a.nq;
            t = item / nt;
            j = item % nt;
        }
    }
    __device__ void next() {  // (called only while items are left: a later tile with entries exists)
        if (++j < nt) return;
        j = 0;
        do {
            t++;
            load();
        } while (RANGES && nt == 0);
    }
};

template <bool RANGES, int LT>
__global__ void __launch_bounds__(kEstThreads, 1) k_est(const __grid_constant__ CUtensorMap map_rows, EstArgs a, int d,
                                                        int nk, int* __restrict__ err) {
    extern __shared__ unsigned char est_smem[];
    // [stages][rows chunk, queries chunk], then the shared block, then the label boxes or the steps
    unsigned char* ring = est_smem + (1024 - (smem_u32(est_smem) & 1023)) % 1024;
    constexpr int kEstStages = est_stages(RANGES);
    EstShared& s = *reinterpret_cast<EstShared*>(ring + kEstStages * 2 * kChunkBytes);
    unsigned char* tail = reinterpret_cast<unsigned char*>(&s) + (sizeof(EstShared) + 15) / 16 * 16;
    float* s_box = reinterpret_cast<float*>(tail);  // [group][2][column][2 l] label boxes (!RANGES)
    unsigned char* s_step = tail;                   // [group][2][column][row] steps (RANGES)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rbase = smem_u32(ring);
    constexpr int kMmaWarp = kGroups * kEpiThreads / 32;
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem)),
                     "r"(kAccs * kEstN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        s.fail = 0;
        auto init = [](uint64_t& b, uint32_t n) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&b)), "r"(n));
        };
        for (int i = 0; i < kEstStages; i++) {
            init(s.full_a[i], 1);
            init(s.full_b[i], 2);
            init(s.empty[i], 1);
        }
        for (int i = 0; i < kAccs; i++) {
            init(s.acc_full[i], 1);
            init(s.acc_empty[i], kEpiThreads / 32);
        }
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = s.tmem;
    Walk<RANGES> w(a);
    const uint32_t total = w.total(), nb = gridDim.x, b = blockIdx.x;
    const uint32_t first = total / nb * b + min(b, total % nb), items = total / nb + (b < total % nb ? 1u : 0u);
    if (items) w.seek(first);

    if (warp == kMmaWarp + 1) {
        // ---- the rows: one thread, TMA ----
        if (lane == 0) {
            uint32_t g = 0;
            bool ok = true;
            for (uint32_t i = 0; i < items && ok; i++) {
                for (int kc = 0; kc < nk; kc++, g++) {
                    const uint32_t st = g % kEstStages;
                    if (!est_wait(s, s.empty[st], ((g / kEstStages) & 1u) ^ 1u)) {
                        ok = false;
                        break;
                    }
                    const uint32_t bar = smem_u32(&s.full_a[st]);
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kChunkBytes)
                                 : "memory");
                    tma_load_2d(rbase + st * 2 * kChunkBytes, &map_rows, kc * 64, (int)(w.t * kEstM), bar);
                }
                if (ok && i + 1 < items) w.next();
            }
            if (!ok)  // the loads in flight land before the shared memory is given back
                for (uint32_t h = g > kEstStages ? g - kEstStages : 0; h < g; h++)
                    mbar_wait(smem_u32(&s.full_a[h % kEstStages]), (h / kEstStages) & 1u);
        }
    } else if (warp >= kMmaWarp + 2) {
        // ---- the queries: two warps, thread p copies 16-byte unit p % 8 of rows p / 8 + 8 r ----
        const int p = tid - 32 * (kMmaWarp + 2), unit = p & 7, row0 = p >> 3;
        uint32_t g = 0;
        constexpr uint32_t kLag = RANGES ? 1 : 2;  // stages whose copies may be in flight
        bool ok = true;
        auto landed = [&](uint32_t h) {  // stage h's copies of this warp have landed
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) est_arrive(s.full_b[h % kEstStages]);
        };
        for (uint32_t i = 0; i < items && ok; i++) {
            uint32_t src[16];
            const uint32_t c0 = w.j * kEstN;
#pragma unroll
            for (int r = 0; r < 16; r++) {
                const uint32_t c = c0 + row0 + 8 * r;
                src[r] = c < w.n_ent ? (RANGES ? __ldg(&a.ent[w.e0 + c].x) : c) : 0xffffffffu;
            }
            for (int kc = 0; kc < nk; kc++, g++) {
                const uint32_t st = g % kEstStages;
                ok = __all_sync(0xffffffffu, est_wait(s, s.empty[st], ((g / kEstStages) & 1u) ^ 1u));
                if (!ok) break;
                const uint32_t dst = rbase + st * 2 * kChunkBytes + kChunkBytes;
                const int k = kc * 64 + unit * 8;
#pragma unroll
                for (int r = 0; r < 16; r++) {
                    const int row = row0 + 8 * r;
                    const bool v = src[r] != 0xffffffffu && k < d;
                    const uint16_t* from = v ? a.qb + (uint64_t)src[r] * a.ldq + k : a.qb;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                                     dst + (uint32_t)(row * 128 + ((unit ^ (row & 7)) << 4))),
                                 "l"(from), "r"(v ? 16 : 0)
                                 : "memory");
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                if (g >= kLag) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(kLag) : "memory");
                    landed(g - kLag);
                }
            }
            if (ok && i + 1 < items) w.next();
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (ok)
            for (uint32_t h = g > kLag ? g - kLag : 0; h < g; h++) landed(h);
    } else if (warp == kMmaWarp) {
        // ---- MMA issue: one thread ----
        if (lane == 0) {
            // F32 accumulate, FP16 A and B, both K-major
            constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(kEstN >> 3) << 17) | ((uint32_t)(kEstM >> 4) << 24);
            uint32_t g = 0;
            bool ok = true;
            for (uint32_t i = 0; i < items && ok; i++) {
                const uint32_t acc = i % kAccs;
                if (!est_wait(s, s.acc_empty[acc], ((i / kAccs) & 1u) ^ 1u)) break;
                asm volatile("tcgen05.fence::after_thread_sync;");
                for (int kc = 0; kc < nk; kc++, g++) {
                    const uint32_t st = g % kEstStages, ph = (g / kEstStages) & 1u;
                    if (!est_wait(s, s.full_a[st], ph) || !est_wait(s, s.full_b[st], ph)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;");
                    const uint32_t sa = rbase + st * 2 * kChunkBytes, sb = sa + kChunkBytes;
#pragma unroll
                    for (int ks = 0; ks < 4; ks++) {
                        const uint64_t da = umma_desc_sw128(sa + ks * 32), db = umma_desc_sw128(sb + ks * 32);
                        const uint32_t add = (kc > 0 || ks > 0) ? 1u : 0u;
                        asm volatile(
                            "{\n\t.reg .pred p;\n\t"
                            "setp.ne.b32 p, %4, 0;\n\t"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem + acc * kEstN),
                            "l"(da), "l"(db), "r"(kIdesc), "r"(add));
                    }
                    est_commit(s.empty[st]);
                }
                if (ok) est_commit(s.acc_full[acc]);
            }
            // the MMAs issued so far end before their operands and TMEM are given back
            if (g) {
                const uint32_t h = g - 1;
                mbar_wait(smem_u32(&s.empty[h % kEstStages]), (h / kEstStages) & 1u);
            }
        }
    } else {
        // ---- epilogue: group `group` takes items group, group + kGroups, ... ----
        const int group = warp / (kEpiThreads / 32), gt = tid - group * kEpiThreads;  // thread in the group
        const int gw = gt >> 5, rl = (gw & 3) * 32 + lane, half = gw >> 2;
        EstGroup& G = s.grp[group];
        const int l = RANGES ? 0 : (LT ? LT : a.l);
        constexpr int LM = RANGES ? 1 : (LT ? LT : kMaxDims);
        float* box0 = s_box + (size_t)group * 2 * kEstN * 2 * l;
        unsigned char* step0 = s_step + (size_t)group * 2 * kEstN * kEstM;
        // the next item's row and column constants, loaded one item ahead
        float4 rc = make_float4(INFINITY, 0.f, 0.f, 0.f), cc = make_float4(0.f, 0.f, INFINITY, 0.f);
        uint32_t qid = 0, lohi = 0, delta = 0;
        uint64_t off = 0;
        float lab[LM];
        auto fetch = [&]() {
            const uint32_t row = w.t * kEstM + rl;
            rc = row < a.n_rows ? __ldg(a.rowc + row) : make_float4(INFINITY, 0.f, 0.f, 0.f);
            if constexpr (!RANGES) {
                const uint64_t br = (uint64_t)a.row0 + (uint64_t)min(row, a.n_rows - 1) * a.row_step;
#pragma unroll
                for (int i = 0; i < LM; i++) lab[i] = i < l ? __ldg(a.labels + br * l + i) : 0.f;
            }
            if (gt < kEstN) {
                const uint32_t c = w.j * kEstN + gt;
                cc = make_float4(0.f, 0.f, INFINITY, 0.f);
                qid = 0xffffffffu;  // a column without a query keeps nothing
                lohi = 0;
                if (c < w.n_ent) {
                    if (RANGES) {
                        const uint4 e = __ldg(a.ent + w.e0 + c);
                        qid = e.x;
                        lohi = e.y;
                        delta = e.z;
                        off = __ldg(a.qoff + qid);
                    } else {
                        qid = c;
                    }
                    cc = __ldg(a.qc + qid);
                }
            }
        };
        auto skip = [&](uint32_t i, uint32_t n) {  // n items on from item i, as far as there are items
            for (uint32_t k = 0; k < n && i + k + 1 < items; k++) w.next();
        };
        skip(0, (uint32_t)group);
        if ((uint32_t)group < items) fetch();
        uint32_t base_reg = 0, prev_row0 = 0;
        bool ok = true;
        // the kept rows of the group's item number n, shared out evenly: kept row f of the item
        // is bit f - (the kept rows of the columns before) of its column's mask
        auto write_kept = [&](uint32_t n, uint32_t row0) {
            const int ms = n & 1, cs = n % kSlots;
            const uint32_t s0 = G.wsum[ms][0], s1 = s0 + G.wsum[ms][1], s2 = s1 + G.wsum[ms][2], all = s2 + G.wsum[ms][3];
            for (uint32_t f = gt; f < all; f += kEpiThreads) {
                const int q4 = (f >= s0) + (f >= s1) + (f >= s2);
                const uint32_t k = f - (q4 == 0 ? 0u : (q4 == 1 ? s0 : (q4 == 2 ? s1 : s2)));
                int c = 32 * q4;  // the last of the 32 columns with pre <= k
#pragma unroll
                for (int st = 16; st > 0; st >>= 1)
                    if (G.pre[ms][c + st] <= k) c += st;
                const uint4 m = G.mask[ms][c];
                uint32_t bit = k - G.pre[ms][c];  // the bit's rank in the mask
                const uint32_t slot = G.base[ms][c] + bit;
                const uint32_t p0 = __popc(m.x), p1 = p0 + __popc(m.y), p2 = p1 + __popc(m.z);
                const int wd = (bit >= p0) + (bit >= p1) + (bit >= p2);
                uint32_t x = wd == 0 ? m.x : (wd == 1 ? m.y : (wd == 2 ? m.z : m.w));
                bit -= wd == 0 ? 0u : (wd == 1 ? p0 : (wd == 2 ? p1 : p2));
                uint32_t at = 0;  // the position of set bit number `bit` of x
#pragma unroll
                for (int st = 16; st > 0; st >>= 1) {
                    const uint32_t below = __popc(x & ((1u << st) - 1u));
                    if (bit >= below) {
                        bit -= below;
                        at += st;
                        x >>= st;
                    }
                }
                const uint32_t row = row0 + 32u * wd + at;
                if (RANGES) {
                    const uint64_t o = G.off[cs][c] + slot;
                    a.prow[o] = (row + G.delta[cs][c]) |
                                ((uint32_t)step0[((size_t)ms * kEstN + c) * kEstM + 32 * wd + at] << 24);
                } else if (slot < a.cap) {
                    a.list[(uint64_t)G.qid[cs][c] * a.cap + slot] = a.row0 + row * a.row_step;
                }
            }
        };
        uint32_t n = 0;  // the group's items so far
        for (uint32_t i = group; i < items; i += kGroups, n++) {
            const int cs = n % kSlots, ms = n & 1;
            const uint32_t row0 = w.t * kEstM, acc = i % kAccs;
            if (gt < kEstN) {
                float* ab = reinterpret_cast<float*>(&G.ab[cs][gt >> 1]);
                ab[gt & 1] = cc.x;
                ab[2 + (gt & 1)] = cc.y;
                float* zs = reinterpret_cast<float*>(&G.zs[cs][gt >> 1]);
                zs[gt & 1] = cc.z;
                zs[2 + (gt & 1)] = cc.w;
                // (2^23 + 1: the sum's low byte is the rounded step, never below zero for a kept row)
                if (RANGES) reinterpret_cast<float*>(&G.sb[cs][gt >> 1])[gt & 1] = fmaf(-cc.z, cc.w, 8388609.f);
                G.qid[cs][gt] = qid;
                if (RANGES) {
                    G.off[cs][gt] = off;
                    G.delta[cs][gt] = delta;
                    G.lohi[cs][gt] = lohi;
                }
            }
            if constexpr (!RANGES) {  // the columns' label boxes (read in this item only)
                const uint32_t c0 = w.j * kEstN;
                float* bx = box0 + (size_t)ms * kEstN * 2 * l;
                for (int e = gt; e < kEstN * 2 * l; e += kEpiThreads)
                    bx[e] = c0 + e / (2 * l) < a.nq ? __ldg(a.boxes + (uint64_t)c0 * 2 * l + e) : 0.f;
            }
            const float2 xn = make_float2(-rc.x, -rc.x), xm = make_float2(rc.y, rc.y), rx = make_float2(rc.z, rc.z);
            float lb[LM];
#pragma unroll
            for (int k = 0; k < LM; k++) lb[k] = RANGES ? 0.f : lab[k];
            epi_bar(group);
            if (i + kGroups < items) {
                skip(i, kGroups);
                fetch();
            }
            if (ok) ok = est_wait(s, s.acc_full[acc], (i / kAccs) & 1u);
            ok = __all_sync(0xffffffffu, ok);
            asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll 1
            for (int h = 0; h < 2; h++) {
                const int cb = half * 64 + h * 32;
                const uint32_t taddr = tmem + ((uint32_t)((gw & 3) * 32) << 16) + acc * kEstN + (uint32_t)cb;
#pragma unroll
                for (int hh = 0; hh < 2; hh++) {
                    uint32_t v[16];
                    tmem_ld16(taddr + 16 * hh, v);
                    tmem_wait();
                    if (h == 1 && hh == 1) {  // this warp has read its part of the accumulator
                        asm volatile("tcgen05.fence::before_thread_sync;");
                        __syncwarp();
                        if (lane == 0) est_arrive(s.acc_empty[acc]);
                    }
#pragma unroll
                    for (int c = 0; c < 16; c += 2) {
                        const int col = cb + 16 * hh + c;
                        const float4 q = G.ab[cs][col >> 1];
                        const float4 z = G.zs[cs][col >> 1];
                        float2 x = fma2(make_float2(2.f, 2.f),
                                        make_float2(__uint_as_float(v[c]), __uint_as_float(v[c + 1])), xn);
                        x = fma2(make_float2(q.x, q.y), xm, x);
                        x = fma2(make_float2(q.z, q.w), rx, x);
                        float2 st = x;
                        if (RANGES) {
                            st = fma2(x, make_float2(z.z, z.w), G.sb[cs][col >> 1]);
                            st.x = fminf(st.x, 8388608.f + 255.f);
                            st.y = fminf(st.y, 8388608.f + 255.f);
                        }
#pragma unroll
                        for (int u = 0; u < 2; u++) {
                            bool keep = !((u ? x.y : x.x) < (u ? z.y : z.x));  // (NaN: no bound, kept)
                            unsigned bal = __ballot_sync(0xffffffffu, keep);
                            if constexpr (!RANGES) {
                                if (bal) {
                                    const float* bx = box0 + ((size_t)ms * kEstN + col + u) * 2 * l;
#pragma unroll
                                    for (int k = 0; k < LM; k++)
                                        if (k < l && (lb[k] < bx[2 * k] || lb[k] > bx[2 * k + 1])) keep = false;
                                    bal = __ballot_sync(0xffffffffu, keep);
                                }
                            }
                            if (lane == 0)
                                reinterpret_cast<uint32_t*>(&G.mask[ms][col + u])[gw & 3] = bal;
                            if (RANGES && keep)
                                step0[((size_t)ms * kEstN + col + u) * kEstM + rl] =
                                    (unsigned char)__float_as_uint(u ? st.y : st.x);
                        }
                    }
                }
            }
            if (n > 0 && gt < kEstN) G.base[ms ^ 1][gt] = base_reg;
            epi_bar(group);
            if (n > 0) write_kept(n - 1, prev_row0);
            if (gt < kEstN) {
                uint4 m = G.mask[ms][gt];
                if (G.qid[cs][gt] == 0xffffffffu || !ok) {
                    m = make_uint4(0u, 0u, 0u, 0u);
                    G.mask[ms][gt] = m;
                } else if (RANGES || row0 + kEstM > a.n_rows) {
                    // the rows of the entry's range, or those that the last tile has: a bound that is not
                    // finite keeps its whole column, the rows past the end with it
                    const uint32_t r = RANGES ? G.lohi[cs][gt] : (a.n_rows - row0) << 16;
                    const int lo = (int)(r & 0xffffu), hi = (int)(r >> 16);
                    auto part = [&](uint32_t x, int k) {
                        const int a0 = min(max(lo - 32 * k, 0), 32), a1 = min(max(hi - 32 * k, 0), 32);
                        const uint32_t below = a1 >= 32 ? ~0u : (1u << a1) - 1u, skip0 = a0 >= 32 ? ~0u : (1u << a0) - 1u;
                        return x & below & ~skip0;
                    };
                    m = make_uint4(part(m.x, 0), part(m.y, 1), part(m.z, 2), part(m.w, 3));
                    G.mask[ms][gt] = m;
                }
                const uint32_t kept = __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
                if (kept) base_reg = atomicAdd(a.cnt + G.qid[cs][gt], kept);
                uint32_t inc = kept;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o) inc += y;
                }
                G.pre[ms][gt] = inc - kept;
                if (lane == 31) G.wsum[ms][gw] = inc;
            }
            prev_row0 = row0;
        }
        if (n > 0) {
            epi_bar(group);
            if (gt < kEstN) G.base[(n - 1) & 1][gt] = base_reg;
            epi_bar(group);
            write_kept(n - 1, prev_row0);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (tid == 0 && s.fail) atomicExch(err, 1);
    if (warp == kMmaWarp)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kAccs * kEstN));
}

template <bool RANGES, int LT>
void launch_est(const EstArgs& a, const void* rows, int ld, int* err, cudaStream_t st) {
    const CUtensorMap map = bf16_rows_map(rows, a.n_rows, ld, kEstM);
    const size_t sm = 1024 + (size_t)est_stages(RANGES) * 2 * kChunkBytes + sizeof(EstShared) + 16 +
                      (RANGES ? (size_t)kGroups * 2 * kEstN * kEstM : sizeof(float) * kGroups * 2 * kEstN * 2 * a.l);
    auto kern = k_est<RANGES, LT>;
    allow_smem(kern);
    kern<<<(unsigned)sm_count(), kEstThreads, sm, st>>>(map, a, ld, (ld + 63) / 64, err);
    CK_LAUNCH();
}

}  // namespace

void est_ranges(const EstArgs& a, const void* rows, int ld, int* err, cudaStream_t st) {
    launch_est<true, 0>(a, rows, ld, err, st);
}
void est_all(const EstArgs& a, const void* rows, int ld, int* err, cudaStream_t st) {
    if (!a.n_rows || !a.nq) return;
    if (a.l == 4) launch_est<false, 4>(a, rows, ld, err, st);
    else launch_est<false, 0>(a, rows, ld, err, st);
}

}  // namespace hdg
