// Distance estimates on the tensor cores (hdg_est.cuh).
//
// Persistent, one CTA per SM, 12 warps: 0-7 epilogue, 8 MMA issue and TMEM, 9 the rows by TMA
// (a tile's rows are consecutive), 10-11 the queries by cp.async (any queries, gathered by id into
// the 128-byte-swizzled layout).  A work item is one tile of 128 rows x 128 queries; every CTA
// takes an equal, consecutive span of them, so successive items share their rows in L2.  K runs in
// chunks of 64 through a ring of stages (full barriers: one for the TMA bytes, one for the two
// gathering warps; the tcgen05.commit of a chunk's MMAs frees its stage).  Two accumulators of 128
// TMEM columns let the MMAs of item i + 1 run under the epilogue of item i.
//
// Epilogue of item i: thread = row, loop over columns (queries): three FMAs and a compare per pair
// against the query's constants, broadcast from shared memory; a ballot per column and warp gives
// the column's 128-bit mask.  One thread per column then reserves the kept rows' slots with one
// atomic, whose latency runs under item i + 1; after that item's masks the rows of item i are
// written, a warp per column, consecutive slots by consecutive lanes.
// Bound: the epilogue's issue slots (about 8 instructions per 32 pairs and the writes); the MMAs
// take half of that at K = 128.  Every wait is bounded: on expiry the kernel sets *err, lets its
// copies land, frees TMEM and returns.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "hdg_est.cuh"
#include "hdg_internal.h"
#include "hdg_umma.cuh"

namespace hdg {

namespace {

constexpr int kEstThreads = 384, kEpiThreads = 256;
constexpr uint32_t kChunkBytes = 128 * 64 * 2;  // one 128 x 64 bf16 operand chunk
constexpr int kEstStages = 5;
constexpr int kSlots = 3;  // column constants: read through the following item

struct EstShared {
    float4 col[kSlots][kEstN];
    uint64_t off[kSlots][kEstN];     // ranges: the query's row offset
    uint32_t qid[kSlots][kEstN];
    uint32_t delta[kSlots][kEstN];
    uint32_t lohi[kSlots][kEstN];
    uint4 mask[2][kEstN];
    uint32_t base[2][kEstN];
    uint64_t full_a[kEstStages], full_b[kEstStages], empty[kEstStages], acc_full[2], acc_empty[2];
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
__device__ __forceinline__ void epi_bar() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,"
        "%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

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
    // [stages][rows chunk, queries chunk], then the shared block, then (LT) the label boxes
    unsigned char* ring = est_smem + (1024 - (smem_u32(est_smem) & 1023)) % 1024;
    EstShared& s = *reinterpret_cast<EstShared*>(ring + kEstStages * 2 * kChunkBytes);
    float* s_box = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(&s) + (sizeof(EstShared) + 15) / 16 * 16);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rbase = smem_u32(ring);
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem)),
                     "r"(2 * kEstN));
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
        for (int i = 0; i < 2; i++) {
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

    if (warp == 9) {
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
    } else if (warp >= 10) {
        // ---- the queries: two warps, thread p copies 16-byte unit p % 8 of rows p / 8 + 8 r ----
        const int p = tid - 320, unit = p & 7, row0 = p >> 3;
        uint32_t g = 0;
        constexpr uint32_t kLag = 2;  // stages whose copies may be in flight
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
    } else if (warp == 8) {
        // ---- MMA issue: one thread ----
        if (lane == 0) {
            constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kEstN >> 3) << 17) |
                                        ((uint32_t)(kEstM >> 4) << 24);
            uint32_t g = 0;
            bool ok = true;
            for (uint32_t i = 0; i < items && ok; i++) {
                const uint32_t acc = i & 1u;
                if (!est_wait(s, s.acc_empty[acc], ((i >> 1) & 1u) ^ 1u)) break;
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
        // ---- epilogue ----
        const int rl = (warp & 3) * 32 + lane, half = warp >> 2;
        const unsigned lt = (1u << lane) - 1u;
        const int l = RANGES ? 0 : (LT ? LT : a.l);
        constexpr int LM = RANGES ? 1 : (LT ? LT : kMaxDims);
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
            if (tid < kEstN) {
                const uint32_t c = w.j * kEstN + tid;
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
        if (items) fetch();
        uint32_t base_reg = 0, prev_row0 = 0;
        bool ok = true;
        auto write_kept = [&](uint32_t i, uint32_t row0) {  // the kept rows of item i
            const int ms = i & 1, cs = i % kSlots;
#pragma unroll 1
            for (int c = warp * 16; c < warp * 16 + 16; c++) {
                const uint4 m = s.mask[ms][c];
                if (!(m.x | m.y | m.z | m.w)) continue;
                const uint32_t word[4] = {m.x, m.y, m.z, m.w};
                uint32_t at = s.base[ms][c];
                const uint32_t q = s.qid[cs][c];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if ((word[k] >> lane) & 1u) {
                        const uint32_t slot = at + __popc(word[k] & lt), row = row0 + 32 * k + lane;
                        if (RANGES) {
                            const uint64_t o = s.off[cs][c] + slot;
                            a.prow[o] = row + s.delta[cs][c];
                            a.drow[o] = row;
                        } else if (slot < a.cap) {
                            a.list[(uint64_t)q * a.cap + slot] = a.row0 + row * a.row_step;
                        }
                    }
                    at += __popc(word[k]);
                }
            }
        };
        for (uint32_t i = 0; i < items; i++) {
            const int cs = i % kSlots, ms = i & 1;
            const uint32_t row0 = w.t * kEstM;
            if (tid < kEstN) {
                s.col[cs][tid] = cc;
                s.qid[cs][tid] = qid;
                if (RANGES) {
                    s.off[cs][tid] = off;
                    s.delta[cs][tid] = delta;
                    s.lohi[cs][tid] = lohi;
                }
            }
            if constexpr (!RANGES) {  // the columns' label boxes (read in this item only)
                const uint32_t c0 = w.j * kEstN;
                float* bx = s_box + (size_t)ms * kEstN * 2 * l;
                for (int e = tid; e < kEstN * 2 * l; e += kEpiThreads)
                    bx[e] = c0 + e / (2 * l) < a.nq ? __ldg(a.boxes + (uint64_t)c0 * 2 * l + e) : 0.f;
            }
            const float xn = rc.x, xm = rc.y, rx = rc.z;
            float lb[LM];
#pragma unroll
            for (int k = 0; k < LM; k++) lb[k] = RANGES ? 0.f : lab[k];
            epi_bar();
            if (i + 1 < items) {
                w.next();
                fetch();
            }
            if (ok) ok = est_wait(s, s.acc_full[ms], (i >> 1) & 1u);
            ok = __all_sync(0xffffffffu, ok);
            asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int cb = half * 64 + h * 32;
                uint32_t v[32];
                tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(ms * kEstN + cb), v);
                if (h == 1) {  // this warp has read its part of the accumulator
                    asm volatile("tcgen05.fence::before_thread_sync;");
                    __syncwarp();
                    if (lane == 0) est_arrive(s.acc_empty[ms]);
                }
                uint32_t mine = 0;
#pragma unroll
                for (int c = 0; c < 32; c++) {
                    const float4 q = s.col[cs][cb + c];
                    float x = fmaf(2.f, __uint_as_float(v[c]), -xn);
                    x = fmaf(q.x, xm, x);
                    x = fmaf(q.y, rx, x);
                    bool keep = !(x < q.z);  // (NaN: no bound, kept)
                    unsigned bal = __ballot_sync(0xffffffffu, keep);
                    if constexpr (!RANGES) {
                        if (bal) {
                            const float* bx = s_box + ((size_t)ms * kEstN + cb + c) * 2 * l;
#pragma unroll
                            for (int k = 0; k < LM; k++)
                                if (k < l && (lb[k] < bx[2 * k] || lb[k] > bx[2 * k + 1])) keep = false;
                            bal = __ballot_sync(0xffffffffu, keep);
                        }
                    }
                    if (lane == c) mine = bal;
                }
                reinterpret_cast<uint32_t*>(&s.mask[ms][cb + lane])[warp & 3] = ok ? mine : 0u;
            }
            if (i > 0 && tid < kEstN) s.base[ms ^ 1][tid] = base_reg;
            epi_bar();
            if (tid < kEstN) {
                uint4 m = s.mask[ms][tid];
                if (s.qid[cs][tid] == 0xffffffffu) {
                    m = make_uint4(0u, 0u, 0u, 0u);
                    s.mask[ms][tid] = m;
                } else if (RANGES) {  // the rows of the entry's range
                    const uint32_t r = s.lohi[cs][tid];
                    const int lo = (int)(r & 0xffffu), hi = (int)(r >> 16);
                    auto part = [&](uint32_t x, int k) {
                        const int a0 = min(max(lo - 32 * k, 0), 32), a1 = min(max(hi - 32 * k, 0), 32);
                        const uint32_t below = a1 >= 32 ? ~0u : (1u << a1) - 1u, skip = a0 >= 32 ? ~0u : (1u << a0) - 1u;
                        return x & below & ~skip;
                    };
                    m = make_uint4(part(m.x, 0), part(m.y, 1), part(m.z, 2), part(m.w, 3));
                    s.mask[ms][tid] = m;
                }
                const uint32_t n = __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
                if (n) base_reg = atomicAdd(a.cnt + s.qid[cs][tid], n);
            }
            if (i > 0) write_kept(i - 1, prev_row0);
            prev_row0 = row0;
        }
        if (items) {
            epi_bar();
            if (tid < kEstN) s.base[(items - 1) & 1][tid] = base_reg;
            epi_bar();
            write_kept(items - 1, prev_row0);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (tid == 0 && s.fail) atomicExch(err, 1);
    if (warp == 8) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kEstN));
}

template <bool RANGES, int LT>
void launch_est(const EstArgs& a, const void* rows, int ld, int* err, cudaStream_t st) {
    const CUtensorMap map = bf16_rows_map(rows, a.n_rows, ld, kEstM);
    const size_t sm = 1024 + (size_t)kEstStages * 2 * kChunkBytes + sizeof(EstShared) + 16 +
                      (RANGES ? 0 : sizeof(float) * 2 * kEstN * 2 * a.l);
    auto kern = k_est<RANGES, LT>;
    CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
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
