// qg_jpart.cu -- join + filter + sort of large probe inputs with a dense build
// side: one partition step fused with the filter, then one CTA per key range.
//
// Reference operators this replaces: partition / partitionGroup and
// buildHashTable / probeHashTable with the filter and bitonic sort of the matches
// (kernel/hj_filter_sort/1/hj_filter_sort_op.cl:25-109, :117-564).
//
// R stands in key order as a payload table (qg_pjoin.cu, k_pj_rtab), so the probe
// rows only have to be brought in key order.  The partitioned form filters them
// into a list, moves the list twice (8 bits a pass) and sorts buckets of 4096 rows:
// every selected row is written four times.  Here it is written twice:
//   1. k_jp_sample  1/64 of S: selected rows per 1/4096 of the key span
//   2. k_jp_plan    the number of buckets (about 16K rows each), and whether rows
//                   and keys spread evenly enough over them
//   3. k_jp_part    S rows that pass the filter, tile by tile, to their buckets'
//                   places (fixed room per bucket, places from a counter)
//   4. k_jp_join    one CTA per bucket: rows per key counted in shared memory,
//                   first places, S payloads put in key order, output written
//                   with consecutive addresses
// A bucket that outgrows its room ends the attempt, and the rows are filtered and
// partitioned as before.
// R 16M, S 256M, 61M rows joined: calls of 1764 us take 1356 (64M: 583 -> 405).
// k_jp_part takes 687 of them (2.5 GB, 374 at the copy rate): 332 to read and
// select alone, 205 more to collect and order a tile, 150 for the stores, in runs
// of five rows.  k_jp_join takes 414 (1.2 GB, 180): counting waits for its loads
// while the SM's other CTA writes.  The list, its two moves and the bucket sort
// took 478 + 554 + 427.
#include <algorithm>
#include <stddef.h>
#include "qg_internal.cuh"
#include "qg_join.cuh"

namespace {

constexpr int JP_THREADS = 512;        // k_jp_join
constexpr int JP_WARPS = JP_THREADS / 32;
constexpr int JPP_THREADS = 1024;      // k_jp_part
constexpr int JPP_WARPS = JPP_THREADS / 32;
constexpr int JP_BINS = 4096;          // of the sample
constexpr uint32_t JP_MAX_NB = 6144;   // buckets
constexpr int JP_WPT = JP_MAX_NB / 2 / JPP_THREADS;  // pairs of buckets per thread
constexpr uint32_t JP_BUCKET = 16384;  // rows per bucket aimed at
constexpr uint32_t JP_CAP = 22528;     // room of a bucket in rows; its payloads fit in shared memory
constexpr uint32_t JP_TILE = 19968;    // selected rows collected before they are moved
constexpr int JP_SEG = JP_TILE / JPP_WARPS;
constexpr int JP_VECS = 2;             // 16-byte vectors of S keys that a lane looks at together
constexpr int JP_STEP = 128 * JP_VECS;           // S rows that a warp looks at together
constexpr int JP_KPT = 9;              // keys of a bucket per thread; odd, so that the threads' runs of words share no bank
constexpr uint32_t JP_KEYS = JP_KPT * JP_THREADS;
constexpr uint32_t JP_ABSENT = 0x80000000u;
constexpr int JP_CHUNK = 1024;         // S rows per sampled run of 16
static_assert(2 * JP_WPT * JPP_THREADS == (int)JP_MAX_NB && JP_WPT % 2 == 1, "the scan over the buckets");
static_assert(JP_TILE < 32768 && JP_CAP < 32768, "16-bit places and differences");
static_assert(JP_CAP % 2 == 0, "two rows per load");

struct JpPlan {
    uint32_t ok, over, done;  // the plan stands; some bucket's room was too small; the outputs hold the result
    uint32_t nb, mul;         // buckets; bucket of key offset x: (x * mul) >> 32
    uint32_t kmin, span;
    uint32_t pad;
    unsigned long long cursor[JP_MAX_NB / 2];  // rows placed in each of two buckets
    uint32_t hist[JP_BINS];
};

__device__ __forceinline__ uint32_t jp_mul(uint32_t parts, uint32_t span) {
    return (uint32_t)(((unsigned long long)parts << 32) / span);  // parts < span
}
// First key offset of bucket b.
__device__ __forceinline__ uint32_t jp_first(uint32_t b, uint32_t nb, uint32_t mul, uint32_t span) {
    if (b >= nb) return span;
    return (uint32_t)min((((unsigned long long)b << 32) + mul - 1) / mul, (unsigned long long)span);
}

__device__ __forceinline__ bool jp_dense(const qg_jp_r &r, uint32_t *kmin, uint32_t *span) {
    unsigned long long distinct = *reinterpret_cast<const unsigned long long *>(r.flags + PJ_F_DISTINCT);
    *kmin = r.range[0];
    *span = r.range[1] - r.range[0] + 1u;  // at most 2 nR
    return r.flags[PJ_F_DENSE] && distinct == (unsigned long long)r.nR && *span > 65536u;
}

__global__ void __launch_bounds__(1024)
k_jp_sample(const int32_t *__restrict__ skey, const int32_t *__restrict__ spay, long long chunks, int32_t slo,
            int32_t shi, qg_jp_r r, JpPlan *__restrict__ P) {
    qg_chain();
    __shared__ uint32_t h[JP_BINS];
    uint32_t kmin, span;
    if (!jp_dense(r, &kmin, &span)) return;
    for (int i = threadIdx.x; i < JP_BINS; i += 1024) h[i] = 0;
    __syncthreads();
    const uint32_t mul = jp_mul(JP_BINS, span);
    const long long stride = (long long)gridDim.x * 1024;
    for (long long i = (long long)blockIdx.x * 1024 + threadIdx.x; i < 4 * chunks; i += stride) {
        const long long c = i >> 2;  // four vectors at a place of the chunk that varies
        const long long v = c * (JP_CHUNK / 4) + (qg_hash32((uint32_t)c) & (JP_CHUNK / 16 - 1)) * 4 + (i & 3);
        const int4 k = __ldg(reinterpret_cast<const int4 *>(skey) + v), p = __ldg(reinterpret_cast<const int4 *>(spay) + v);
        const uint32_t kk[4] = {(uint32_t)k.x, (uint32_t)k.y, (uint32_t)k.z, (uint32_t)k.w};
        const int32_t pp[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
        for (int j = 0; j < 4; j++)
            if ((pp[j] >= slo) & (pp[j] <= shi) & (kk[j] - kmin < span)) atomicAdd(&h[__umulhi(kk[j] - kmin, mul)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < JP_BINS; i += 1024)
        if (h[i]) atomicAdd(&P->hist[i], h[i]);
}

// One CTA.  room: rows that the buckets may take together.
__global__ void __launch_bounds__(1024)
k_jp_plan(long long nS, long long chunks, long long room, qg_jp_r r, JpPlan *__restrict__ P) {
    qg_chain();
    __shared__ uint32_t cum[JP_BINS + 1], ws[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t kmin, span;
    const bool dense = jp_dense(r, &kmin, &span);
    const uint4 c = reinterpret_cast<const uint4 *>(P->hist)[tid];
    const uint32_t mine = c.x + c.y + c.z + c.w;
    uint32_t inc = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t x = __shfl_up_sync(QG_FULL_MASK, inc, d);
        if (lane >= d) inc += x;
    }
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    uint32_t at = __reduce_add_sync(QG_FULL_MASK, lane < warp ? ws[lane] : 0u) + inc - mine;
    cum[4 * tid] = at;
    cum[4 * tid + 1] = at += c.x;
    cum[4 * tid + 2] = at += c.y;
    cum[4 * tid + 3] = at += c.z;
    if (tid == 1023) cum[JP_BINS] = at + c.w;
    for (uint32_t i = tid; i < JP_MAX_NB / 2; i += 1024) P->cursor[i] = 0;
    __syncthreads();
    const float ratio = (float)nS / (16.f * (float)chunks), rows = ratio * (float)cum[JP_BINS];
    const uint32_t nb = max((uint32_t)(rows / JP_BUCKET), (uint32_t)(span / (JP_KEYS - 100))) + 1u;
    bool ok = dense && nb <= JP_MAX_NB && (long long)nb * JP_CAP <= room;
    const uint32_t mul = ok ? jp_mul(nb, span) : 1u;
    if (ok) {
        // rows at the buckets' borders, linear within a bin
        const float per = (float)JP_BINS / (float)span;
        auto below = [&](uint32_t x) {
            const float f = (float)x * per;
            const uint32_t b = min((uint32_t)f, (uint32_t)JP_BINS - 1);
            return (float)cum[b] + (f - (float)b) * (float)(cum[b + 1] - cum[b]);
        };
        for (uint32_t b = tid; b < nb; b += 1024) {
            const uint32_t k0 = jp_first(b, nb, mul, span), k1 = jp_first(b + 1, nb, mul, span);
            // Refused only when the sample's count less three times its error says so:
            // of 3750 evenly filled buckets some lie 4.6 errors above the mean, and that
            // alone refused one input in fifty, at the price of the slower path.
            const float x = below(k1) - below(k0);
            if ((x - 3.f * sqrtf(x)) * ratio > JP_CAP * (15.f / 16) || k1 - k0 > JP_KEYS) ok = false;
        }
    }
    ok = __syncthreads_and(ok);
    if (tid == 0) {
        P->ok = ok;
        P->over = P->done = 0;
        P->nb = nb;
        P->mul = mul;
        P->kmin = kmin;
        P->span = span;
    }
}

struct JpTile {
    unsigned long long row[JP_TILE];  // key offset << 32 | payload
    uint16_t perm[JP_TILE];           // rows in bucket order
    uint32_t cnt[JP_MAX_NB / 2];      // rows per bucket, then places: two buckets to a word
    int16_t delta[JP_MAX_NB];         // from a place in the tile to one in the bucket
};

// Each warp looks at S rows on its own, 256 at a time, appends the selected ones to
// its part of the tile in shared memory and counts their buckets; when a warp's
// part is full, the CTA puts the tile in bucket order, so that a warp's stores
// cover fewer lines.  One CTA of 1024 threads with a tile of 20K rows: two of 512
// with 9K rows take 735 us instead of 687 (runs of two to three rows), and so does
// a tile that the warps share through a counter.  The places come from one atomic
// per tile and pair of buckets, issued so that a warp's fall in two lines (with a
// sector each they took twice the time).  More rows in flight per warp spill.
__global__ void __launch_bounds__(JPP_THREADS, 1)
k_jp_part(const int32_t *__restrict__ skey, const int32_t *__restrict__ spay, uint32_t n, int32_t slo, int32_t shi,
          JpPlan *__restrict__ P, unsigned long long *__restrict__ out) {
    qg_chain();
    extern __shared__ __align__(16) unsigned char jp_raw[];
    JpTile &S = *reinterpret_cast<JpTile *>(jp_raw);
    __shared__ uint32_t s_rows, s_w[JPP_WARPS];
    if (!P->ok) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t lt = qg_lanemask_lt(), kmin = P->kmin, span = P->span, mul = P->mul;
    for (uint32_t i = tid; i < JP_MAX_NB / 2; i += JPP_THREADS) S.cnt[i] = 0;
    __syncthreads();
    constexpr int V = JP_VECS;
    auto load = [&](uint32_t t, int4 (&k)[V], int4 (&p)[V]) {
#pragma unroll
        for (int v = 0; v < V; v++) {
            const uint32_t i = t * JP_STEP + v * 128 + lane * 4;
            if (i + 3 < n) {
                k[v] = qg_ldg_stream(reinterpret_cast<const int4 *>(skey + i));
                p[v] = qg_ldg_stream(reinterpret_cast<const int4 *>(spay + i));
            } else {  // a row past the end has a key that is not selected
                const int none = (int)(kmin - 1u);
                k[v] = make_int4(i < n ? skey[i] : none, i + 1 < n ? skey[i + 1] : none, i + 2 < n ? skey[i + 2] : none, none);
                p[v] = make_int4(i < n ? spay[i] : 0, i + 1 < n ? spay[i + 1] : 0, i + 2 < n ? spay[i + 2] : 0, 0);
            }
        }
    };
    const uint32_t width = (uint32_t)shi - (uint32_t)slo, keys = slo <= shi ? span : 0u;
    // one more row of a bucket: the number before
    auto count = [&](uint32_t b) {
        const uint32_t sh = 16 * (b & 1u);
        return (atomicAdd(&S.cnt[b >> 1], 1u << sh) >> sh) & 0xffffu;
    };
    unsigned long long *seg = S.row + warp * JP_SEG;  // the warp's part of the tile
    uint32_t have = 0;                                // rows in it
    // Appends and counts the selected rows; false: there is no room for them.
    auto append = [&](const int4 (&k)[V], const int4 (&p)[V]) -> bool {
        uint32_t m[4 * V], pre[4 * V], tot = 0;
#pragma unroll
        for (int j = 0; j < 4 * V; j++) {
            const int4 &kv = k[j >> 2], &pv = p[j >> 2];
            const int kj = (j & 3) == 0 ? kv.x : (j & 3) == 1 ? kv.y : (j & 3) == 2 ? kv.z : kv.w;
            const int pj = (j & 3) == 0 ? pv.x : (j & 3) == 1 ? pv.y : (j & 3) == 2 ? pv.z : pv.w;
            m[j] = __ballot_sync(QG_FULL_MASK, ((uint32_t)pj - (uint32_t)slo <= width) & ((uint32_t)kj - kmin < keys));
            pre[j] = tot;
            tot += __popc(m[j]);
        }
        if (have + tot > (uint32_t)JP_SEG) return false;
#pragma unroll
        for (int j = 0; j < 4 * V; j++) {
            const int4 &kv = k[j >> 2], &pv = p[j >> 2];
            const int kj = (j & 3) == 0 ? kv.x : (j & 3) == 1 ? kv.y : (j & 3) == 2 ? kv.z : kv.w;
            const int pj = (j & 3) == 0 ? pv.x : (j & 3) == 1 ? pv.y : (j & 3) == 2 ? pv.z : pv.w;
            if ((m[j] >> lane) & 1u) {
                const uint32_t off = (uint32_t)kj - kmin;
                seg[have + pre[j] + __popc(m[j] & lt)] = (unsigned long long)off << 32 | (uint32_t)pj;
                count(__umulhi(off, mul));
            }
        }
        have += tot;
        return true;
    };
    int4 kq[V], pq[V];  // the next step's rows
    const uint32_t steps = (n + JP_STEP - 1) / JP_STEP, stride = gridDim.x * JPP_WARPS;
    uint32_t t = blockIdx.x * JPP_WARPS + warp;
    if (t < steps) load(t, kq, pq);
    for (;;) {
        bool wait = false;
        while (t < steps) {
            if (!append(kq, pq)) {
                wait = true;
                break;
            }
            t += stride;
            if (t < steps) load(t, kq, pq);
        }
        const bool more = __syncthreads_or(wait);
        unsigned long long g[JP_WPT];
        uint32_t sum = 0;
        bool over = false;
#pragma unroll
        for (int j = 0; j < JP_WPT; j++) {
            const uint32_t c = S.cnt[j * JPP_THREADS + tid];
            g[j] = c ? atomicAdd(&P->cursor[j * JPP_THREADS + tid], (unsigned long long)(c >> 16) << 32 | (c & 0xffffu)) : 0ull;
            const uint32_t x = S.cnt[tid * JP_WPT + j];
            sum += (x >> 16) + (x & 0xffffu);
        }
        uint32_t inc = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t x = __shfl_up_sync(QG_FULL_MASK, inc, d);
            if (lane >= d) inc += x;
        }
        if (lane == 31) s_w[warp] = inc;
        __syncthreads();
        uint32_t at = __reduce_add_sync(QG_FULL_MASK, lane < warp ? s_w[lane] : 0u) + inc - sum;
#pragma unroll
        for (int j = 0; j < JP_WPT; j++) {
            const uint32_t c = S.cnt[j * JPP_THREADS + tid];
            over |= (uint32_t)g[j] + (c & 0xffffu) > JP_CAP || (uint32_t)(g[j] >> 32) + (c >> 16) > JP_CAP;
        }
        if (__syncthreads_or(over)) {
            if (tid == 0) *(volatile uint32_t *)&P->over = 1u;
            return;
        }
#pragma unroll
        for (int j = 0; j < JP_WPT; j++) {
            const uint32_t x = S.cnt[tid * JP_WPT + j];
            S.cnt[tid * JP_WPT + j] = at | (at + (x & 0xffffu)) << 16;
            at += (x & 0xffffu) + (x >> 16);
        }
        if (tid == JPP_THREADS - 1) s_rows = at;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < JP_WPT; j++) {
            const uint32_t w = j * JPP_THREADS + tid, x = S.cnt[w];
            const uint32_t d0 = (uint32_t)g[j] - (x & 0xffffu), d1 = (uint32_t)(g[j] >> 32) - (x >> 16);
            reinterpret_cast<uint32_t *>(S.delta)[w] = (d0 & 0xffffu) | d1 << 16;
        }
        __syncthreads();
        for (uint32_t i = lane; i < have; i += 32)
            S.perm[count(__umulhi((uint32_t)(seg[i] >> 32), mul))] = (uint16_t)(warp * JP_SEG + i);
        have = 0;
        __syncthreads();
        for (uint32_t p = tid; p < s_rows; p += JPP_THREADS) {
            const unsigned long long v = S.row[S.perm[p]];
            const uint32_t b = __umulhi((uint32_t)(v >> 32), mul);
            out[b * JP_CAP + p + (int32_t)S.delta[b]] = v;
        }
        for (uint32_t i = tid; i < JP_MAX_NB / 2; i += JPP_THREADS) S.cnt[i] = 0;
        __syncthreads();
        if (!more) return;
    }
}

struct JpBucket {
    uint32_t cnt[JP_KEYS];   // rows per key, then places
    uint32_t pay[JP_CAP];    // S payloads in key order
    uint2 list[JP_WARPS][32];
};

// A bucket at a time per CTA (tickets in bucket order; persistent, the number of
// buckets being known on the device only).  The rows are read twice, the second
// time from L2.  Counting, moving and writing overlap between the two CTAs of an SM.
__global__ void __launch_bounds__(JP_THREADS, 2)
k_jp_join(JpPlan *__restrict__ P, const unsigned long long *__restrict__ rows, qg_jp_r r, uint32_t *__restrict__ ok,
          uint32_t *__restrict__ oa, uint32_t *__restrict__ ob, long long cap, volatile long long *d_count,
          volatile uint32_t *result, qg_lookback lb) {
    qg_chain();
    extern __shared__ __align__(16) unsigned char jp_raw[];
    JpBucket &S = *reinterpret_cast<JpBucket *>(jp_raw);
    __shared__ uint32_t s_tile, s_epoch, s_excl, s_w[JP_WARPS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t lt = qg_lanemask_lt();
    if (!P->ok || P->over) {  // the same for all CTAs: only k_jp_part sets it
        if (blockIdx.x == 0 && tid == 0) *result = P->ok ? QG_JP_OVER : QG_JP_REFUSED;
        return;
    }
    const uint32_t nb = P->nb, kmin = P->kmin, sent = r.flags[PJ_F_SENT], by_sent = r.flags[PJ_F_SENT_OK];
    for (;;) {
        qg_lb_begin_dyn(lb, &s_tile, &s_epoch);  // (a barrier: the bucket before is done with)
        const uint32_t b = s_tile;
        if (b >= nb) break;
        const uint32_t klo = jp_first(b, nb, P->mul, P->span), nk = jp_first(b + 1, nb, P->mul, P->span) - klo;
        const uint32_t n = reinterpret_cast<const uint32_t *>(P->cursor)[b];
        const unsigned long long *in = rows + (size_t)b * JP_CAP;
        // R's payloads of the keys j * JP_THREADS + tid
        uint32_t pay[JP_KPT], absent = 0;
#pragma unroll
        for (int j = 0; j < JP_KPT; j++) {
            const uint32_t k = j * JP_THREADS + tid, off = klo + k;
            pay[j] = k < nk ? __ldg(r.T + off) : 0u;
            if (k < nk && !by_sent && !((__ldg(r.bitmap + (off >> 5)) >> (off & 31u)) & 1u)) absent |= 1u << j;
        }
        for (uint32_t i = tid; i < nk; i += JP_THREADS) S.cnt[i] = 0;
        __syncthreads();
        // f(row) of every row of the bucket, two per load, 2 * U of them in flight per thread
        auto scan_rows = [&](auto &&f) {
            constexpr int U = 3;
            for (uint32_t i0 = 2 * tid; i0 < n; i0 += 2 * U * JP_THREADS) {
                ulonglong2 v[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const uint32_t i = i0 + u * 2 * JP_THREADS;
                    if (i < n) v[u] = __ldcg(reinterpret_cast<const ulonglong2 *>(in + i));  // JP_CAP is even: in bounds
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const uint32_t i = i0 + u * 2 * JP_THREADS;
                    if (i < n) f(v[u].x);
                    if (i + 1 < n) f(v[u].y);
                }
            }
        };
        scan_rows([&](unsigned long long v) {
            const uint32_t k = (uint32_t)(v >> 32) - klo;
            atomicAdd(&S.cnt[k], 1u);
        });
        __syncthreads();
        // counts -> first places; the keys that R lacks are marked and take none
#pragma unroll
        for (int j = 0; j < JP_KPT; j++) {
            const uint32_t k = j * JP_THREADS + tid;
            if (by_sent && k < nk && pay[j] == sent) absent |= 1u << j;
            if ((absent >> j) & 1u) {
                if (S.cnt[k]) S.cnt[k] = JP_ABSENT;
                else absent ^= 1u << j;
            }
        }
        const bool some_absent = __syncthreads_or(absent);
        uint32_t c[JP_KPT], sum = 0;
#pragma unroll
        for (int j = 0; j < JP_KPT; j++) {
            const uint32_t k = tid * JP_KPT + j;
            c[j] = k < nk ? S.cnt[k] : 0u;
            sum += c[j] & ~JP_ABSENT;
        }
        uint32_t inc = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t x = __shfl_up_sync(QG_FULL_MASK, inc, d);
            if (lane >= d) inc += x;
        }
        if (lane == 31) s_w[warp] = inc;
        __syncthreads();
        uint32_t at = __reduce_add_sync(QG_FULL_MASK, lane < warp ? s_w[lane] : 0u) + inc - sum;
        const uint32_t total = __reduce_add_sync(QG_FULL_MASK, lane < JP_WARPS ? s_w[lane] : 0u);
        if (tid == 0) qg_lb_publish_agg(lb, b, s_epoch, total);
#pragma unroll
        for (int j = 0; j < JP_KPT; j++) {
            const uint32_t k = tid * JP_KPT + j;
            if (k < nk) S.cnt[k] = at | (c[j] & JP_ABSENT);
            at += c[j] & ~JP_ABSENT;
        }
        __syncthreads();
        scan_rows([&](unsigned long long v) {
            const uint32_t k = (uint32_t)(v >> 32) - klo;
            if (!(some_absent && (S.cnt[k] & JP_ABSENT))) S.pay[atomicAdd(&S.cnt[k], 1u)] = (uint32_t)v;
        });
        if (warp == 0) {
            const uint32_t excl = qg_lb_warp_lookback(lb, b, s_epoch, total);
            if (lane == 0) s_excl = excl;
        }
        __syncthreads();  // a key's word is now the place after its last row
        const long long o0 = s_excl;
        for (uint32_t i = tid; i < total; i += JP_THREADS)
            if (o0 + i < cap) ob[o0 + i] = S.pay[i];
        // 32 keys a warp: row q belongs to the last key with rows that starts at or
        // before q, so a bit per start and a list of those keys give it
#pragma unroll
        for (int j = 0; j < JP_KPT; j++) {
            const uint32_t kb = j * JP_THREADS + warp * 32, k = kb + lane;
            if (kb >= nk) break;
            const uint32_t end = S.cnt[min(k, nk - 1)] & ~JP_ABSENT;
            const uint32_t first = k == 0 ? 0u : S.cnt[min(k, nk) - 1] & ~JP_ABSENT;
            const uint32_t p0 = __shfl_sync(QG_FULL_MASK, first, 0), rows32 = __shfl_sync(QG_FULL_MASK, end, 31) - p0;
            const bool some = end > first;
            const uint32_t m = __ballot_sync(QG_FULL_MASK, some);
            __syncwarp();
            if (some) S.list[warp][__popc(m & lt)] = make_uint2(kmin + klo + k, pay[j]);
            __syncwarp();
            const uint32_t rel = some ? first - p0 : 0xffffffffu;
            uint32_t seen = 0;  // keys with rows that start before q0
            for (uint32_t q0 = 0; q0 < rows32; q0 += 32) {
                const uint32_t starts = __reduce_or_sync(QG_FULL_MASK, rel - q0 < 32u ? 1u << (rel - q0) : 0u);
                const uint32_t q = q0 + lane;
                const long long o = o0 + p0 + q;
                if (q < rows32 && o < cap) {
                    const uint2 x = S.list[warp][seen + __popc(starts & (lt | 1u << lane)) - 1];
                    ok[o] = x.x;
                    oa[o] = x.y;
                }
                seen += __popc(starts);
            }
        }
        if (tid == 0 && b == nb - 1) {
            *d_count = o0 + total;
            P->done = 1;
            *result = QG_JP_DONE;
        }
    }
    qg_lb_end(lb);
}

}  // namespace

size_t qg_jp_bytes() { return qg_align_up(sizeof(JpPlan), 256); }

const uint32_t *qg_jp_done(const char *work) { return &reinterpret_cast<const JpPlan *>(work)->done; }

qg_status qg_jp_launch(qg_ctx *ctx, char *work, const qg_jp_r &r, const int32_t *skey, const int32_t *spay, int64_t nS,
                       int32_t slo, int32_t shi, unsigned long long *rows, int64_t room, uint32_t *out_key,
                       uint32_t *out_rpay, uint32_t *out_spay, int64_t cap, volatile long long *d_count,
                       volatile uint32_t *result) {
    JpPlan *P = (JpPlan *)work;
    static qg_per_device sites[2];
    QG_TRY(qg_allow_smem(ctx, sites[0], k_jp_part, sizeof(JpTile)));
    QG_TRY(qg_allow_smem(ctx, sites[1], k_jp_join, sizeof(JpBucket)));
    qg_lookback lb;
    QG_TRY(qg_lb_make(ctx, JP_MAX_NB, QG_SITE_PJ_BUCKET, &lb));
    QG_TRY_CUDA(ctx, cudaMemsetAsync(P, 0, sizeof(JpPlan), ctx->stream), "plan");
    const long long chunks = nS / JP_CHUNK;
    qg_pre_launch(ctx);
    k_jp_sample<<<(unsigned)ctx->sm_count, 1024, 0, ctx->stream>>>(skey, spay, chunks, slo, shi, r, P);
    QG_TRY(qg_check_launch(ctx, "k_jp_sample"));
    QG_TRY(qg_launch_chained(ctx, "k_jp_plan", k_jp_plan, 1, 1024, 0, nS, chunks, room, r, P));
    QG_TRY(qg_launch_chained(ctx, "k_jp_part", k_jp_part, (unsigned)ctx->sm_count, JPP_THREADS, sizeof(JpTile), skey,
                             spay, (uint32_t)nS, slo, shi, P, rows));
    return qg_launch_chained(ctx, "k_jp_join", k_jp_join, 2 * (unsigned)ctx->sm_count, JP_THREADS, sizeof(JpBucket), P,
                             rows, r, out_key, out_rpay, out_spay, cap, d_count, result, lb);
}
