// qg_gbwide.cu -- column group-by (int64 SUM + COUNT per key, optionally only
// rows with lo2 <= val2 <= hi2) whose keys spread too widely for a window
// (hashed ids): partitioned by key range, so that the output needs no sort.
//
// The reference chain this answers for: sort -> label -> scan -> write ->
// parallelAggregate (kernel/aggregation/1/group_by_cu_op_dp.cl:89-716).
//
//   1. k_gbd_range (qg_gbdense.cu)  the exact key range
//   2. k_gbw_rows   the rows that take part as records (key << 32 | value), and
//                   how many fall in each of up to 256 equal parts of the range
//   3. k_gbw_plan   the parts' first rows; whether the parts are even enough
//   4. one radix pass (qg_sort.cu) puts the records in part order
//   5. k_gbw_merge  one CTA per part: hash table in shared memory, the distinct
//                   keys sorted there, their place from a look-back over the
//                   parts, written in ascending key order
// The two-pass path (qg_groupby.cu) spills misses into 1024 buckets per SM and
// sorts the groups in four passes afterwards: calls of 64K rows took 160 us (52
// here), of 1M rows 150 to 220 (64 to 72), of 8M rows in 1M groups 390 (190).  It
// stays for keys that fill the parts unevenly (a frequent key, clusters) and for
// more groups than the parts' tables hold.  Of the 190 us the range takes 14, the
// rows 27, the plan 6, the pass 37 (bandwidth) and the merge 92: 1.9 clocks a row
// and SM of shared-memory probes and atomics, in two waves of 152 CTAs.
#include <algorithm>
#include <stddef.h>
#include "qg_cta_sort.cuh"
#include "qg_internal.cuh"
#include "qg_keytable.cuh"
#include "qg_sort.cuh"

namespace {

constexpr int GW_PARTS = 256;
constexpr int GW_THREADS = 256;  // k_gbw_rows
constexpr int GW_ROUNDS = 4;
constexpr int GW_WARPS = GW_THREADS / 32;
constexpr int GW_TILE = GW_THREADS * GW_ROUNDS * 4;  // 4096 rows
constexpr int GW_SLOTS = 8192;
constexpr uint32_t GW_PROBES = 64;
constexpr uint32_t GW_UNEVEN = 8;  // a part with more than this many times its share ends the attempt
static_assert(GW_ROUNDS * GW_WARPS == 32, "one warp scans the tile's pieces");
static_assert(GW_SLOTS <= QG_CS_MAX, "the distinct keys are sorted by qg_cta_sort");

struct GwState {
    unsigned long long rows;  // records
    uint32_t verdict;         // a qg_gbw_result
    uint32_t full;            // a part had more distinct keys than its table takes
    uint32_t base[GW_PARTS + 1];
    RsPass pass;
};

// Part of key k: (k - kmin) >> shift, below 2^parts_log2.
__device__ __forceinline__ int gw_shift(uint32_t span, int parts_log2) { return max(0, 32 - parts_log2 - __clz(span)); }

// PRED: the rows that take part are compacted per tile and appended in any
// order; else record i is row i.
template <bool PRED>
__global__ void __launch_bounds__(GW_THREADS, 4)
k_gbw_rows(const int32_t *__restrict__ key, const int32_t *__restrict__ val, const int32_t *__restrict__ val2,
           int32_t lo2, int32_t hi2, long long n, const uint32_t *__restrict__ range, uint32_t window, int parts_log2,
           const uint32_t *__restrict__ seems, unsigned long long *__restrict__ rec, uint32_t *__restrict__ hist,
           unsigned long long *__restrict__ rows, uint4 *__restrict__ clear, long long clear_n) {
    qg_chain();
    __shared__ uint32_t s_h[GW_PARTS], s_woff[32], s_cnt;
    __shared__ unsigned long long s_base;
    __shared__ unsigned long long s_row[PRED ? GW_TILE : 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t kmin = ~range[0], span = range[1] - kmin, lt = qg_lanemask_lt();
    if (span < window || (seems && *seems)) return;  // a window holds the keys; too few groups or too many
    const int shift = gw_shift(span, parts_log2);
    for (long long j = (long long)blockIdx.x * GW_THREADS + tid; j < clear_n; j += (long long)gridDim.x * GW_THREADS)
        clear[j] = make_uint4(0, 0, 0, 0);  // the radix pass's status words
    s_h[tid] = 0;
    __syncthreads();
    const long long ntiles = (n + GW_TILE - 1) / GW_TILE;
    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const long long base = t * GW_TILE;
        int4 kv[GW_ROUNDS], pv[GW_ROUNDS];
        uint32_t fl = 0;
#pragma unroll
        for (int r = 0; r < GW_ROUNDS; r++) {
            const long long i = base + (long long)(r * GW_THREADS + tid) * 4;
            if (i + 3 < n) {
                kv[r] = qg_ldg_stream(reinterpret_cast<const int4 *>(key + i));
                pv[r] = qg_ldg_stream(reinterpret_cast<const int4 *>(val + i));
                uint32_t f = 15u;
                if (PRED) {
                    const int4 w = qg_ldg_stream(reinterpret_cast<const int4 *>(val2 + i));
                    f = (uint32_t)((w.x >= lo2) & (w.x <= hi2)) | ((uint32_t)((w.y >= lo2) & (w.y <= hi2)) << 1) |
                        ((uint32_t)((w.z >= lo2) & (w.z <= hi2)) << 2) | ((uint32_t)((w.w >= lo2) & (w.w <= hi2)) << 3);
                }
                fl |= f << (4 * r);
            } else {
                int k[4] = {0, 0, 0, 0}, p[4] = {0, 0, 0, 0};
                for (int j = 0; j < 4; j++)
                    if (i + j < n) {
                        k[j] = key[i + j];
                        p[j] = val[i + j];
                        if (!PRED || ((val2[i + j] >= lo2) & (val2[i + j] <= hi2))) fl |= 1u << (4 * r + j);
                    }
                kv[r] = make_int4(k[0], k[1], k[2], k[3]);
                pv[r] = make_int4(p[0], p[1], p[2], p[3]);
            }
        }
        if (PRED) {
            uint32_t lpre[GW_ROUNDS];
#pragma unroll
            for (int r = 0; r < GW_ROUNDS; r++) {
                uint32_t c = 0, tot = 0;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const uint32_t b = __ballot_sync(QG_FULL_MASK, (fl >> (4 * r + j)) & 1u);
                    c += __popc(b & lt);
                    tot += __popc(b);
                }
                lpre[r] = c;
                if (lane == 0) s_woff[r * GW_WARPS + warp] = tot;
            }
            __syncthreads();
            if (warp == 0) {
                const uint32_t x = s_woff[lane];
                uint32_t inc = x;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t y = __shfl_up_sync(QG_FULL_MASK, inc, d);
                    if (lane >= d) inc += y;
                }
                s_woff[lane] = inc - x;
                if (lane == 31) {
                    s_cnt = inc;
                    s_base = inc ? atomicAdd(rows, (unsigned long long)inc) : 0ull;
                }
            }
            __syncthreads();
#pragma unroll
            for (int r = 0; r < GW_ROUNDS; r++) {
                uint32_t pos = s_woff[r * GW_WARPS + warp] + lpre[r];
                const int kk[4] = {kv[r].x, kv[r].y, kv[r].z, kv[r].w}, pp[4] = {pv[r].x, pv[r].y, pv[r].z, pv[r].w};
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if ((fl >> (4 * r + j)) & 1u) s_row[pos++] = (unsigned long long)(uint32_t)kk[j] << 32 | (uint32_t)pp[j];
            }
            __syncthreads();
            const uint32_t cnt = s_cnt;
            const unsigned long long at = s_base;
            for (uint32_t i = tid; i < cnt; i += GW_THREADS) {
                const unsigned long long v = s_row[i];
                rec[at + i] = v;
                atomicAdd(&s_h[((uint32_t)(v >> 32) - kmin) >> shift], 1u);
            }
            __syncthreads();
        } else {
#pragma unroll
            for (int r = 0; r < GW_ROUNDS; r++) {
                const long long i = base + (long long)(r * GW_THREADS + tid) * 4;
                const uint32_t kk[4] = {(uint32_t)kv[r].x, (uint32_t)kv[r].y, (uint32_t)kv[r].z, (uint32_t)kv[r].w};
                const uint32_t pp[4] = {(uint32_t)pv[r].x, (uint32_t)pv[r].y, (uint32_t)pv[r].z, (uint32_t)pv[r].w};
                if (i + 3 < n) {
                    uint4 *o = reinterpret_cast<uint4 *>(rec + i);
                    o[0] = make_uint4(pp[0], kk[0], pp[1], kk[1]);
                    o[1] = make_uint4(pp[2], kk[2], pp[3], kk[3]);
                }
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if ((fl >> (4 * r + j)) & 1u) {
                        if (i + 3 >= n) rec[i + j] = (unsigned long long)kk[j] << 32 | pp[j];
                        atomicAdd(&s_h[(kk[j] - kmin) >> shift], 1u);
                    }
            }
        }
    }
    __syncthreads();
    if (s_h[tid]) atomicAdd(&hist[tid], s_h[tid]);
}

// One CTA of GW_PARTS threads.  The histogram and the row counter are cleared
// for their next user.
__global__ void __launch_bounds__(GW_PARTS)
k_gbw_plan(const uint32_t *__restrict__ range, uint32_t window, int parts_log2, const uint32_t *__restrict__ seems,
           uint32_t *__restrict__ hist, unsigned long long *__restrict__ rows, GwState *__restrict__ W, const unsigned long long *r0,
           unsigned long long *r1, uint32_t *status) {
    qg_chain();
    __shared__ uint32_t ws[GW_PARTS / 32], wm[GW_PARTS / 32];
    const int d = threadIdx.x, lane = d & 31, w = d >> 5;
    const uint32_t kmin = ~range[0], span = range[1] - kmin;
    const uint32_t c = hist[d];
    hist[d] = 0;
    uint32_t inc = c;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
        const uint32_t x = __shfl_up_sync(QG_FULL_MASK, inc, k);
        if (lane >= k) inc += x;
    }
    const uint32_t mx = __reduce_max_sync(QG_FULL_MASK, c);
    if (lane == 31) ws[w] = inc;
    if (lane == 0) wm[w] = mx;
    __syncthreads();
    uint32_t off = 0, all = 0, most = 0;
    for (int i = 0; i < GW_PARTS / 32; i++) {
        off += i < w ? ws[i] : 0u;
        all += ws[i];
        most = max(most, wm[i]);
    }
    W->base[d] = off + inc - c;
    if (d != 0) return;
    W->base[GW_PARTS] = all;
    W->rows = all;
    W->full = 0;
    *rows = 0;
    const bool even = most <= 16384u || ((unsigned long long)most << parts_log2) <= (unsigned long long)GW_UNEVEN * all;
    const uint32_t g = seems ? *seems : 0u;
    const uint32_t verdict = span < window ? QG_GBW_NARROW : g == QG_GBW_SEEMS_FEW ? QG_GBW_FEW
                             : even && g != QG_GBW_SEEMS_MANY ? QG_GBW_DONE : QG_GBW_OTHER;
    W->verdict = verdict;
    W->pass = RsPass{r0, r1, status, nullptr, verdict == QG_GBW_DONE ? 1u : 0u, (uint32_t)gw_shift(span, parts_log2), kmin, 0u};
}

// One CTA per part (numbered in start order).  A part's rows are added to the
// table with two 32-bit adds, the sums as halves of the values; a part of more
// than 65536 rows keeps the sum as two words with a carry instead.
__global__ void __launch_bounds__(QG_CS_THREADS, 1)
k_gbw_merge(GwState *__restrict__ W, const unsigned long long *__restrict__ rec, uint32_t slots,
            int32_t *__restrict__ gkey, long long *__restrict__ gsum, long long *__restrict__ gcnt, long long cap,
            uint32_t *__restrict__ range, volatile long long *d_num, volatile uint32_t *result, qg_lookback lb) {
    qg_chain();
    extern __shared__ __align__(16) unsigned char gw_raw[];
    __shared__ uint32_t s_tile, s_epoch, s_full, s_n, s_excl, s_tmp[16];
    const int tid = threadIdx.x, lane = tid & 31;
    if (blockIdx.x == 0 && tid < 2) range[tid] = 0;  // the words of k_gbd_range, read by the kernels before
    if (W->verdict != QG_GBW_DONE) {
        if (blockIdx.x == 0 && tid == 0) *result = W->verdict;
        return;
    }
    unsigned long long *ord = reinterpret_cast<unsigned long long *>(gw_raw);
    const uint32_t pitch = slots + 4;  // entry `slots`: key 0xffffffff, the free mark
    uint32_t *hk = reinterpret_cast<uint32_t *>(ord + slots), *hc = hk + pitch, *hl = hc + pitch, *hh = hl + pitch;
    uint32_t(*whist)[256] = reinterpret_cast<uint32_t(*)[256]>(hh + pitch);
    qg_lb_begin_dyn(lb, &s_tile, &s_epoch);
    const uint32_t part = s_tile;
    const uint32_t rb = W->base[part], rn = W->base[part + 1] - rb;
    uint4 *z = reinterpret_cast<uint4 *>(hk);
    for (uint32_t i = tid; i < pitch; i += QG_CS_THREADS) {
        const uint32_t x = i < pitch / 4 ? QG_KT_FREE : 0u;
        z[i] = make_uint4(x, x, x, x);
    }
    if (tid == 0) s_full = s_n = 0;
    __syncthreads();
    const uint32_t mask = slots - 1;
    const bool halves = rn <= 65536u;
    uint32_t fresh = 0;  // counted by qg_kt_find, not used here
    auto add = [&](uint32_t h, int32_t v) {
        atomicAdd(&hc[h], 1u);
        if (halves) {
            atomicAdd(&hl[h], (uint32_t)v & 0xffffu);
            const int32_t up = v >> 16;
            if (up) atomicAdd(&hh[h], (uint32_t)up);
        } else {
            const uint32_t old = atomicAdd(&hl[h], (uint32_t)v);
            const uint32_t up = (uint32_t)(v >> 31) + (old + (uint32_t)v < old ? 1u : 0u);
            if (up) atomicAdd(&hh[h], up);
        }
    };
    constexpr int U = 4;
    for (uint32_t i0 = tid; i0 < rn; i0 += U * QG_CS_THREADS) {
        unsigned long long v[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t i = i0 + u * QG_CS_THREADS;
            v[u] = i < rn && i >= i0 ? __ldcs(rec + rb + i) : 0ull;
        }
        uint32_t k[U], h[U], live = 0;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t i = i0 + u * QG_CS_THREADS;
            k[u] = (uint32_t)(v[u] >> 32);
            if (i < rn && i >= i0) live |= 1u << u;
        }
        if (qg_kt_find<U>(hk, mask, k, live, h, GW_PROBES, fresh)) {
#pragma unroll
            for (int u = 0; u < U; u++)
                if ((live >> u) & 1u) add(h[u], (int32_t)(uint32_t)v[u]);
        } else {
            s_full = 1;
        }
        if (*(volatile uint32_t *)&s_full) break;
    }
    __syncthreads();
    const bool full = s_full != 0;
    uint32_t g = 0, top = 0;
    if (!full) {
        for (uint32_t i = tid; i < slots; i += QG_CS_THREADS) {  // whole warps: slots >= 1024
            const bool used = hc[i] != 0;
            const uint32_t m = __ballot_sync(QG_FULL_MASK, used);
            uint32_t at = 0;
            if (lane == 0 && m) at = atomicAdd(&s_n, (uint32_t)__popc(m));
            at = __shfl_sync(QG_FULL_MASK, at, 0);
            if (used) ord[at + __popc(m & qg_lanemask_lt())] = (unsigned long long)hk[i] << 32 | i;
        }
        __syncthreads();
        g = s_n;
        top = hc[slots] ? 1u : 0u;  // key 0xffffffff comes last
    } else if (tid == 0) {
        *(volatile uint32_t *)&W->full = 1u;
        __threadfence();  // before the part's count, which the last part waits for
    }
    if (tid < 256) {  // the place among the parts, while nothing is sorted yet
        const uint32_t excl = qg_lb_wide_exclusive<8>(lb, part, s_epoch, g + top, s_tmp);
        if (tid == 0) s_excl = excl;
    }
    if (!full) qg_cta_sort(ord, whist, g);
    else __syncthreads();
    const long long base = s_excl;
    for (uint32_t r = tid; r < g + top; r += QG_CS_THREADS) {
        if (base + r >= cap) break;
        const uint32_t i = r < g ? (uint32_t)ord[r] : slots;
        gkey[base + r] = r < g ? (int32_t)(ord[r] >> 32) : -1;
        gsum[base + r] = halves ? (long long)hl[i] + ((long long)(int32_t)hh[i] << 16)
                                : (long long)((unsigned long long)hh[i] << 32 | hl[i]);
        gcnt[base + r] = hc[i];
    }
    if (tid == 0 && part == gridDim.x - 1) {
        *d_num = base + g + top;
        *result = qg_ld_relaxed_u32(&W->full) ? QG_GBW_OTHER : QG_GBW_DONE;
    }
    qg_lb_finish_dyn(lb, part, gridDim.x - 1, s_epoch);
}

size_t gw_smem(uint32_t slots) { return (size_t)slots * 8 + 4 * (slots + 4) * 4 + 32 * 1024; }

}  // namespace

// Distinct keys a part of 2^parts_log2 may expect, for the tables' sizes.
static int64_t gw_expected(int64_t n, int64_t cap, int parts_log2) { return std::min(n, cap) >> parts_log2; }

// Few groups among many rows stay in the two-pass path's per-SM tables, and its one
// pass over the rows wins; here each part's CTA meets its rows one a clock.  Hashed
// ids, two-pass / this path: 4M rows in 64 groups 168 / 133 us; 8M in 64 178 / 201,
// in 512 190 / 161; 16M in 512 213 / 277, in 2048 251 / 255, in 8192 413 / 249; 32M in
// 2048 314 / 461, in 8192 582 / 446.  The line in distinct keys of a 4096-row sample
// (5000 equally frequent keys show 2800):
static uint32_t gw_few_limit(int64_t n) {
    return n < 6'000'000 ? 0u : (uint32_t)std::min<int64_t>((n - 6'000'000) / 5500, 2700);
}

// Many groups among very many rows: a part's table is half full and its CTA meets a row
// in two clocks, where the two-pass path spills sequentially.  1M groups, two-pass /
// this path: 45M rows 1017 / 919 us, 60M 1257 / 1275, 100M 1950 / 2336; 400K groups,
// 100M rows 1697 / 1424.  The sample tells 100K groups (3890 bits) from 1M (3960), cap
// has to say the rest.
static uint32_t gw_many_limit(int64_t rows, int64_t cap) {
    return rows > 56'000'000 && gw_expected(rows, cap, 8) > 2700 ? 3925u : 0xffffffffu;
}

bool qg_gbw_few(int64_t n, int64_t groups) { return groups <= gw_few_limit(n) * 3 / 2; }

bool qg_gbw_applies(int64_t n, int64_t cap) {
    return n > QG_GBS_MAX_ROWS && n < (1LL << 30) && gw_expected(n, cap, 8) <= GW_SLOTS * 5 / 8;
}

qg_status qg_gbw_launch(qg_ctx *ctx, const int32_t *key, const int32_t *val, const int32_t *val2, int32_t lo2,
                        int32_t hi2, int64_t n, int32_t *gkey, int64_t *gsum, int64_t *gcnt, int64_t cap,
                        volatile long long *d_num, volatile uint32_t *result) {
    const size_t rb = qg_align_up((size_t)n * 8, 256), words = qg_radix_status_words(n);
    char *aux, *scr;
    QG_TRY(qg_aux(ctx, 2 * rb, &aux));
    QG_TRY(qg_scratch(ctx, qg_align_up(sizeof(GwState), 256) + words * 4, &scr));
    unsigned long long *r0 = (unsigned long long *)aux, *r1 = (unsigned long long *)(aux + rb);
    GwState *W = (GwState *)scr;
    uint32_t *status = (uint32_t *)(scr + qg_align_up(sizeof(GwState), 256));
    // 128 parts (one wave of CTAs) while their tables take the keys, else 256
    const int plog2 = gw_expected(n, cap, 7) <= 3000 ? 7 : 8;
    uint32_t slots = 1024;
    while (slots < GW_SLOTS && slots < 2 * gw_expected(n, cap, plog2) + 512) slots <<= 1;
    const uint32_t window = QG_GBD_WINDOW;
    const bool pred = val2 != nullptr;
    uint32_t *range = ctx->ctl->gbd, *hist = ctx->ctl->shist;
    static qg_per_device site;
    QG_TRY(qg_allow_smem(ctx, site, k_gbw_merge, gw_smem(GW_SLOTS)));
    qg_lookback lb;
    QG_TRY(qg_lb_make(ctx, GW_PARTS, QG_SITE_GROUPBY, &lb));
    const uint32_t limit = gw_few_limit(n), *seems = limit ? &ctx->ctl->gbw_groups : nullptr;
    QG_TRY(qg_gbd_range(ctx, key, n, limit, gw_many_limit(pred ? n / 2 : n, cap)));  // a predicate: half the rows, say
    const unsigned grid = (unsigned)std::min<long long>(qg_ceil_div(n, GW_TILE), 4LL * ctx->sm_count);
    QG_TRY(qg_launch_chained(ctx, "k_gbw_rows", (pred ? k_gbw_rows<true> : k_gbw_rows<false>), grid, GW_THREADS, 0,
                             key, val, val2, lo2, hi2, n, range, window, plog2, seems, r0, hist, &ctx->ctl->gbw_rows,
                             (uint4 *)status, (long long)(words / 4)));
    QG_TRY(qg_launch_chained(ctx, "k_gbw_plan", k_gbw_plan, 1, GW_PARTS, 0, range, window, plog2, seems, hist,
                             &ctx->ctl->gbw_rows, W, r0, r1, status));
    QG_TRY(qg_radix_pass_planned(ctx, &W->pass, W->base, n, &W->rows));
    return qg_launch_chained(ctx, "k_gbw_merge", k_gbw_merge, 1u << plog2, QG_CS_THREADS, gw_smem(slots), W, r1, slots,
                             gkey, (long long *)gsum, (long long *)gcnt, cap, range, d_num, result, lb);
}
