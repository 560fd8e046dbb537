// qg_jdirect.cu -- join + filter + sort with a dense build side, by counting:
// the path of qg_join_filter_sort for small and middling inputs.
//
// Reference operators this replaces: buildHashTable / probeHashTable and the
// filter + bitonic sort of the matches (kernel/hj_filter_sort/1/
// hj_filter_sort_op.cl:25-109, :117-564).
//
// When R's keys are unique and spread over at most 2 nR values, a table entry
// per key value of the span holds R's payload and a count.  Because the output
// is ordered by key and the order among equal keys is free, a probe row's
// place is its key's first place (a scan of the counts) plus the number of
// rows of that key counted before it, so nothing is partitioned or sorted:
//   1. k_jd_range  R's key range
//   2. k_jd_fill   entries = 0
//   3. k_jd_table  entries of R's keys = (payload, JD_HERE); a key met twice ends
//                  the attempt, before S is read
//   4. k_jd_count  S rows that pass the filter: one 64-bit atomic on the key's
//                  entry returns R's payload (does the key match?) and the
//                  row's number among its key's rows; (key, payload, number)
//                  are appended
//   5. k_jd_scan   counts -> first places; every key and its R payload are
//                  written as often as counted
//   6. k_jd_write  every appended row's S payload to its place
// Six launches (four for a small build side, k_jd_build) and one wait.  Where the
// scattered accesses leave L2, the rows are partitioned first (qg_jpart.cu).  A key with
// more than JD_KEY_ROWS rows ends the attempt: its atomics would queue at one
// word, and the partitioned form treats such keys apart.
#include <algorithm>
#include <stddef.h>
#include "qg_internal.cuh"
#include "qg_join.cuh"

namespace {

// Words of ctl->jd.  The first two are zero between calls: the smallest key is
// kept as the largest complement.
enum {
    JD_NKMIN = 0, JD_KMAX = 1, // ~(smallest key), largest key (unsigned)
    JD_OK = QG_JD_OK,           // a qg_jd_result: QG_JD_DONE while nothing speaks against the path
    JD_KMIN = 5, JD_SPAN = 6,   // first key and number of key values of the table
    JD_ROWS = 7,                // appended rows
};

constexpr int JD_THREADS = 256;
constexpr uint32_t JD_KEY_ROWS = 4096;  // rows of one key, at most
constexpr uint32_t JD_HERE = 0x80000000u;  // in an entry's count: R has the key

__global__ void __launch_bounds__(JD_THREADS)
k_jd_range(const int32_t *__restrict__ rkey, long long nR, uint32_t *jd) {
    qg_chain();
    __shared__ uint32_t s[2];
    if (threadIdx.x < 2) s[threadIdx.x] = 0;
    __syncthreads();
    uint32_t m[2] = {0, 0};
    auto row = [&](int32_t k) {
        m[0] = max(m[0], ~(uint32_t)k);
        m[1] = max(m[1], (uint32_t)k);
    };
    const long long stride = (long long)gridDim.x * JD_THREADS;
    const long long t0 = (long long)blockIdx.x * JD_THREADS + threadIdx.x;
    const long long nv = ((uintptr_t)rkey & 15) == 0 ? nR / 4 : 0;
    for (long long i = t0; i < nv; i += stride) {
        const int4 k = __ldg(reinterpret_cast<const int4 *>(rkey) + i);
        row(k.x);
        row(k.y);
        row(k.z);
        row(k.w);
    }
    for (long long i = 4 * nv + t0; i < nR; i += stride) row(__ldg(rkey + i));
#pragma unroll
    for (int j = 0; j < 2; j++) {
        m[j] = __reduce_max_sync(QG_FULL_MASK, m[j]);
        if ((threadIdx.x & 31) == 0) atomicMax(&s[j], m[j]);
    }
    __syncthreads();
    if (threadIdx.x < 2) atomicMax(&jd[JD_NKMIN + threadIdx.x], s[threadIdx.x]);
}

__global__ void __launch_bounds__(JD_THREADS)
k_jd_fill(unsigned long long *__restrict__ E, long long nR, uint32_t *__restrict__ jd) {
    qg_chain();
    const uint32_t kmin = ~jd[JD_NKMIN], kmax = jd[JD_KMAX];
    const unsigned long long w = (unsigned long long)(kmax - kmin) + 1ull;
    const bool ok = w <= 2ull * (unsigned long long)nR;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        jd[JD_OK] = ok ? QG_JD_DONE : QG_JD_SPARSE;
        jd[JD_KMIN] = kmin;
        jd[JD_SPAN] = ok ? (uint32_t)w : 0u;
        jd[JD_ROWS] = 0;
    }
    if (!ok) return;
    ulonglong2 *E2 = reinterpret_cast<ulonglong2 *>(E);  // one entry past an odd span is part of the buffer
    for (unsigned long long i = (unsigned long long)blockIdx.x * JD_THREADS + threadIdx.x; i < (w + 1) / 2;
         i += (unsigned long long)gridDim.x * JD_THREADS)
        E2[i] = make_ulonglong2(0ull, 0ull);
}

// R's payload into its key's entry; true: another row of the key was there before.
// (With an exchange instead of a store a table of 1M rows takes 14 us, 12 before.
// Counting the entries afterwards found duplicates only when all of S had been
// counted, 16M rows 60 us in vain.)
__device__ __forceinline__ bool jd_put(unsigned long long *e, uint32_t pay) {
    return (uint32_t)atomicExch(e, (unsigned long long)pay << 32 | JD_HERE) & JD_HERE;
}

__global__ void __launch_bounds__(JD_THREADS)
k_jd_table(const int32_t *__restrict__ rkey, const int32_t *__restrict__ rpay, long long nR,
           unsigned long long *__restrict__ E, uint32_t *__restrict__ jd) {
    qg_chain();
    if (blockIdx.x == 0 && threadIdx.x < 2) jd[JD_NKMIN + threadIdx.x] = 0;  // k_jd_fill has read them
    if (jd[JD_OK] != QG_JD_DONE) return;
    const uint32_t kmin = jd[JD_KMIN];
    constexpr int U = 4;  // rows in flight per thread
    const long long stride = (long long)gridDim.x * JD_THREADS;
    bool twice = false;
    for (long long i0 = (long long)blockIdx.x * JD_THREADS + threadIdx.x; i0 < nR; i0 += U * stride) {
        uint32_t k[U], p[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long long i = i0 + u * stride;
            k[u] = i < nR ? (uint32_t)__ldg(rkey + i) - kmin : 0u;
            p[u] = i < nR ? (uint32_t)__ldg(rpay + i) : 0u;
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i0 + u * stride < nR) twice |= jd_put(E + k[u], p[u]);
    }
    if (twice) jd[JD_OK] = QG_JD_TWICE;
}

// The three steps above in one CTA: with so few rows the launches are what costs.
// Joins with 256 to 2048 build rows 53 -> 48 us; with 4096 one SM takes as long as
// the three launches (52), with 8192 longer (55 / 52).
constexpr int JD_ONE_THREADS = 1024, JD_ONE_PER = 2;
constexpr int64_t JD_ONE_R = JD_ONE_THREADS * JD_ONE_PER;
__global__ void __launch_bounds__(JD_ONE_THREADS, 1)
k_jd_build(const int32_t *__restrict__ rkey, const int32_t *__restrict__ rpay, uint32_t nR,
           unsigned long long *__restrict__ E, uint32_t *__restrict__ jd) {
    qg_chain();
    __shared__ uint32_t s[2];
    const uint32_t tid = threadIdx.x;
    uint32_t k[JD_ONE_PER], p[JD_ONE_PER], lo = 0xffffffffu, hi = 0;
    if (tid == 0) {
        s[0] = 0xffffffffu;
        s[1] = 0;
    }
#pragma unroll
    for (int j = 0; j < JD_ONE_PER; j++) {
        const uint32_t i = j * JD_ONE_THREADS + tid;
        if (i >= nR) break;
        k[j] = (uint32_t)__ldg(rkey + i);
        p[j] = (uint32_t)__ldg(rpay + i);
        lo = min(lo, k[j]);
        hi = max(hi, k[j]);
    }
    __syncthreads();
    lo = __reduce_min_sync(QG_FULL_MASK, lo);
    hi = __reduce_max_sync(QG_FULL_MASK, hi);
    if ((tid & 31) == 0) {
        atomicMin(&s[0], lo);
        atomicMax(&s[1], hi);
    }
    __syncthreads();
    const uint32_t kmin = s[0];
    const unsigned long long w = (unsigned long long)(s[1] - kmin) + 1ull;
    const bool ok = w <= 2ull * nR;
    if (tid == 0) {
        jd[JD_OK] = ok ? QG_JD_DONE : QG_JD_SPARSE;
        jd[JD_KMIN] = kmin;
        jd[JD_SPAN] = ok ? (uint32_t)w : 0u;
        jd[JD_ROWS] = 0;
    }
    if (!ok) return;
    ulonglong2 *E2 = reinterpret_cast<ulonglong2 *>(E);  // one entry past an odd span is part of the buffer
    for (uint32_t i = tid; i < ((uint32_t)w + 1) / 2; i += JD_ONE_THREADS) E2[i] = make_ulonglong2(0ull, 0ull);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < JD_ONE_PER; j++)
        if (j * JD_ONE_THREADS + tid < nR && jd_put(E + (k[j] - kmin), p[j])) jd[JD_OK] = QG_JD_TWICE;
}

// S rows, 4096 per tile (persistent CTAs): the rows that pass the filter and
// lie in the key span are compacted in shared memory, take one place range of
// the append list per tile, and then their atomics, four in flight per thread.
// A row whose key R lacks keeps its place with the number JD_NONE.
constexpr int JD_ROUNDS = 4;
constexpr int JD_TILE = JD_THREADS * JD_ROUNDS * 4;
constexpr int JD_WARPS = JD_THREADS / 32;
constexpr uint32_t JD_NONE = 0xffffffffu;
static_assert(JD_ROUNDS * JD_WARPS == 32, "one warp scans the tile's pieces");

__global__ void __launch_bounds__(JD_THREADS, 4)
k_jd_count(const int32_t *__restrict__ skey, const int32_t *__restrict__ spay, long long n, int32_t slo, int32_t shi,
           unsigned long long *__restrict__ E, uint32_t *__restrict__ jd, uint32_t *__restrict__ ak,
           uint32_t *__restrict__ ap, uint32_t *__restrict__ an) {
    qg_chain();
    __shared__ uint32_t s_woff[JD_ROUNDS * JD_WARPS], s_base, s_cnt, s_stop;
    __shared__ unsigned long long s_row[JD_TILE];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // Other CTAs may store to the verdict meanwhile, so one thread reads it for all:
    // a CTA leaves whole, here and in the loop, or not at all.
    if (tid == 0) s_stop = qg_ld_relaxed_u32(&jd[JD_OK]) != QG_JD_DONE;
    __syncthreads();
    if (s_stop) return;
    const uint32_t lt = qg_lanemask_lt(), kmin = jd[JD_KMIN], span = jd[JD_SPAN];
    const long long ntiles = (n + JD_TILE - 1) / JD_TILE;
    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const long long base = t * JD_TILE;
        int4 kv[JD_ROUNDS], pv[JD_ROUNDS];
#pragma unroll
        for (int r = 0; r < JD_ROUNDS; r++) {
            const long long idx = base + (long long)(r * JD_THREADS + tid) * 4;
            if (idx + 3 < n) {
                kv[r] = qg_ldg_stream(reinterpret_cast<const int4 *>(skey + idx));
                pv[r] = qg_ldg_stream(reinterpret_cast<const int4 *>(spay + idx));
            } else {
                int tk[4] = {0, 0, 0, 0}, tp[4] = {0, 0, 0, 0};
                for (int j = 0; j < 4; j++)
                    if (idx + j < n) { tk[j] = skey[idx + j]; tp[j] = spay[idx + j]; }
                kv[r] = make_int4(tk[0], tk[1], tk[2], tk[3]);
                pv[r] = make_int4(tp[0], tp[1], tp[2], tp[3]);
            }
        }
        uint32_t fl = 0, lpre[JD_ROUNDS];
#pragma unroll
        for (int r = 0; r < JD_ROUNDS; r++) {
            const long long idx = base + (long long)(r * JD_THREADS + tid) * 4;
            const int32_t kk[4] = {kv[r].x, kv[r].y, kv[r].z, kv[r].w}, pp[4] = {pv[r].x, pv[r].y, pv[r].z, pv[r].w};
            uint32_t c = 0, tot = 0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const bool f = (idx + j < n) & (pp[j] >= slo) & (pp[j] <= shi) & ((uint32_t)kk[j] - kmin < span);
                const uint32_t b = __ballot_sync(QG_FULL_MASK, f);
                c += __popc(b & lt);
                tot += __popc(b);
                fl |= (uint32_t)f << (4 * r + j);
            }
            lpre[r] = c;
            if (lane == 0) s_woff[r * JD_WARPS + warp] = tot;
        }
        __syncthreads();
        if (warp == 0) {  // exclusive offsets of the tile's (round, warp) pieces; one atomic for the tile
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
                s_base = inc ? atomicAdd(&jd[JD_ROWS], inc) : 0u;
                s_stop = qg_ld_relaxed_u32(&jd[JD_OK]) != QG_JD_DONE;
            }
        }
        __syncthreads();
        if (s_stop) return;  // a key with too many rows was met
#pragma unroll
        for (int r = 0; r < JD_ROUNDS; r++) {
            uint32_t pos = s_woff[r * JD_WARPS + warp] + lpre[r];
            const int32_t kk[4] = {kv[r].x, kv[r].y, kv[r].z, kv[r].w}, pp[4] = {pv[r].x, pv[r].y, pv[r].z, pv[r].w};
#pragma unroll
            for (int j = 0; j < 4; j++)
                if ((fl >> (4 * r + j)) & 1u) s_row[pos++] = (unsigned long long)((uint32_t)kk[j] - kmin) << 32 | (uint32_t)pp[j];
        }
        __syncthreads();
        const uint32_t cnt = s_cnt, at = s_base;
        constexpr int U = 4;
        bool heavy = false;
        for (uint32_t i0 = tid; i0 < cnt; i0 += U * JD_THREADS) {
            unsigned long long e[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t i = i0 + u * JD_THREADS;
                e[u] = i < cnt ? atomicAdd(E + (s_row[i] >> 32), 1ull) : 0ull;
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const uint32_t i = i0 + u * JD_THREADS;
                if (i >= cnt) break;
                ak[at + i] = (uint32_t)(s_row[i] >> 32);
                ap[at + i] = (uint32_t)s_row[i];
                const uint32_t seen = (uint32_t)e[u] & ~JD_HERE;
                an[at + i] = (uint32_t)e[u] & JD_HERE ? seen : JD_NONE;
                heavy |= seen >= JD_KEY_ROWS;
            }
        }
        if (heavy) jd[JD_OK] = QG_JD_HOT;
        __syncthreads();  // the shared words are rewritten by the next tile
    }
}

// Counts of the table's entries -> first places (in the entries' low words),
// 256 * PER entries per tile with a look-back over the tiles; a warp writes the keys
// and R payloads of 32 entries at a time, consecutively.
template <int PER>
__global__ void __launch_bounds__(JD_THREADS)
k_jd_scan(unsigned long long *__restrict__ E, const uint32_t *__restrict__ jd, uint32_t *__restrict__ ok,
          uint32_t *__restrict__ oa, long long cap, long long *__restrict__ d_count, volatile uint32_t *result,
          qg_lookback lb) {
    qg_chain();
    __shared__ uint32_t s_tile, s_epoch, s_w[JD_WARPS], s_tmp[2 * JD_WARPS];
    qg_lb_begin_dyn(lb, &s_tile, &s_epoch);
    const uint32_t tile = s_tile, kmin = jd[JD_KMIN], verdict = jd[JD_OK];
    const uint32_t span = verdict == QG_JD_DONE ? jd[JD_SPAN] : 0u;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t base = tile * (PER * JD_THREADS) + warp * (PER * 32);
    unsigned long long e[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const uint32_t i = base + j * 32 + lane;
        e[j] = i < span ? __ldcg(E + i) : 0ull;
    }
    uint32_t pre[PER], sum = 0;  // counted rows before the entry, among the warp's
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const uint32_t c = (uint32_t)e[j] & JD_HERE ? (uint32_t)e[j] & ~JD_HERE : 0u;
        uint32_t inc = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t x = __shfl_up_sync(QG_FULL_MASK, inc, d);
            if (lane >= d) inc += x;
        }
        pre[j] = sum + inc - c;
        sum += __shfl_sync(QG_FULL_MASK, inc, 31);
    }
    if (lane == 0) s_w[warp] = sum;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < JD_WARPS; w++) {
        before += w < warp ? s_w[w] : 0u;
        total += s_w[w];
    }
    const uint32_t excl = qg_lb_wide_exclusive<JD_WARPS>(lb, tile, s_epoch, total, s_tmp);
#pragma unroll
    for (int j = 0; j < PER; j++) {
        const uint32_t i = base + j * 32 + lane;
        const uint32_t first = excl + before + pre[j];
        if (i < span) E[i] = (e[j] & 0xffffffff00000000ull) | first;
        // the 32 entries' output rows: row q belongs to the last entry that starts at or before q
        const uint32_t c = (uint32_t)e[j] & JD_HERE ? (uint32_t)e[j] & ~JD_HERE : 0u;
        const uint32_t p0 = __shfl_sync(QG_FULL_MASK, first, 0);
        const uint32_t rel = first - p0, rows = __shfl_sync(QG_FULL_MASK, rel + c, 31);
        for (uint32_t q0 = 0; q0 < rows; q0 += 32) {
            const uint32_t q = q0 + lane;
            int at = 0;
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) {
                const uint32_t x = __shfl_sync(QG_FULL_MASK, rel, at + d);
                if (x <= q) at += d;
            }
            const uint32_t pay = __shfl_sync(QG_FULL_MASK, (uint32_t)(e[j] >> 32), at);
            const long long o = (long long)p0 + q;
            if (q < rows && o < cap) {
                ok[o] = kmin + base + j * 32 + at;
                oa[o] = pay;
            }
        }
    }
    if (tid == 0 && tile == gridDim.x - 1) {
        *d_count = (long long)excl + total;
        if (result) *result = verdict;
    }
    qg_lb_finish_dyn(lb, tile, gridDim.x - 1, s_epoch);
}

__global__ void __launch_bounds__(JD_THREADS)
k_jd_write(const unsigned long long *__restrict__ E, const uint32_t *__restrict__ jd, const uint32_t *__restrict__ ak,
           const uint32_t *__restrict__ ap, const uint32_t *__restrict__ an, uint32_t *__restrict__ ob, long long cap) {
    qg_chain();
    if (jd[JD_OK] != QG_JD_DONE) return;
    const long long n = jd[JD_ROWS], stride = (long long)gridDim.x * JD_THREADS;
    constexpr int U = 4;
    for (long long i0 = (long long)blockIdx.x * JD_THREADS + threadIdx.x; i0 < n; i0 += U * stride) {
        uint32_t k[U], p[U], m[U], e[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long long i = i0 + u * stride;
            k[u] = i < n ? __ldcs(ak + i) : 0u;
            p[u] = i < n ? __ldcs(ap + i) : 0u;
            m[u] = i < n ? __ldcs(an + i) : JD_NONE;
        }
#pragma unroll
        for (int u = 0; u < U; u++) e[u] = m[u] != JD_NONE ? __ldg(reinterpret_cast<const uint32_t *>(E + k[u])) : 0u;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long long o = (long long)e[u] + m[u];
            if (m[u] != JD_NONE && o < cap) ob[o] = p[u];
        }
    }
}

unsigned jd_grid(qg_ctx *ctx, long long work, int per_block, int per_sm) {
    return (unsigned)std::max<long long>(1, std::min<long long>((work + per_block - 1) / per_block, (long long)ctx->sm_count * per_sm));
}

}  // namespace

size_t qg_jd_bytes(int64_t nR, int64_t nS) {
    return qg_align_up(((size_t)2 * nR + 2) * 8, 256) + 3 * qg_align_up((size_t)nS * 4, 256);
}

qg_status qg_jd_launch(qg_ctx *ctx, char *work, const int32_t *rkey, const int32_t *rpay, int64_t nR,
                       const int32_t *skey, const int32_t *spay, int64_t nS, int32_t slo, int32_t shi, uint32_t *out_key,
                       uint32_t *out_rpay, uint32_t *out_spay, int64_t cap, long long *d_count, volatile uint32_t *result) {
    unsigned long long *E = (unsigned long long *)work;
    const size_t eb = qg_align_up(((size_t)2 * nR + 2) * 8, 256), ab = qg_align_up((size_t)nS * 4, 256);
    uint32_t *ak = (uint32_t *)(work + eb), *ap = (uint32_t *)(work + eb + ab), *an = (uint32_t *)(work + eb + 2 * ab);
    uint32_t *jd = ctx->ctl->jd;
    if (nR <= JD_ONE_R) {
        qg_pre_launch(ctx);
        k_jd_build<<<1, JD_ONE_THREADS, 0, ctx->stream>>>(rkey, rpay, (uint32_t)nR, E, jd);
        QG_TRY(qg_check_launch(ctx, "k_jd_build"));
    } else {
        qg_pre_launch(ctx);
        k_jd_range<<<jd_grid(ctx, nR, 4 * JD_THREADS, 4), JD_THREADS, 0, ctx->stream>>>(rkey, nR, jd);
        QG_TRY(qg_check_launch(ctx, "k_jd_range"));
        QG_TRY(qg_launch_chained(ctx, "k_jd_fill", k_jd_fill, jd_grid(ctx, nR, 2 * JD_THREADS, 8), JD_THREADS, 0, E,
                                 nR, jd));
        QG_TRY(qg_launch_chained(ctx, "k_jd_table", k_jd_table, jd_grid(ctx, nR, JD_THREADS, 8), JD_THREADS, 0, rkey,
                                 rpay, nR, E, jd));
    }
    QG_TRY(qg_launch_chained(ctx, "k_jd_count", k_jd_count, jd_grid(ctx, nS, JD_TILE, 4), JD_THREADS, 0, skey, spay,
                             nS, slo, shi, E, jd, ak, ap, an));
    // few entries: more, smaller tiles (2K build rows 15 us with 16 entries per lane)
    const int per = nR <= (1 << 18) ? 2 : 16;
    const long long tiles = qg_ceil_div(2 * nR, per * JD_THREADS);
    qg_lookback lb;
    QG_TRY(qg_lb_make(ctx, tiles, QG_SITE_JOIN_PROBE, &lb));
    if (per == 2) {
        QG_TRY(qg_launch_chained(ctx, "k_jd_scan", k_jd_scan<2>, (unsigned)tiles, JD_THREADS, 0, E, jd, out_key,
                                 out_rpay, cap, d_count, result, lb));
    } else {
        // Not chained: CTAs that wait for the count are placed wherever its first CTAs end,
        // several to an SM, and then run there (265K build rows, 17M probe rows: 186 us a
        // call, chained 199 to 215).
        qg_pre_launch(ctx);
        k_jd_scan<16><<<(unsigned)tiles, JD_THREADS, 0, ctx->stream>>>(E, jd, out_key, out_rpay, cap, d_count, result, lb);
        QG_TRY(qg_check_launch(ctx, "k_jd_scan"));
    }
    return qg_launch_chained(ctx, "k_jd_write", k_jd_write, jd_grid(ctx, nS / 4, JD_THREADS, 8), JD_THREADS, 0, E, jd,
                             ak, ap, an, out_spay, cap);
}
