// qg_sort.cu -- LSD radix sort by an unsigned 32-bit key.
//
// Replaces the reference's bitonic sort (bitonicSortShared +
// bitonicMergeGlobal, kernel/aggregation/1/group_by_cu_op_dp.cl:89-291,
// driven by radixSortImpl_sm, host/host/testSort.cpp:24-136), which needs a
// power-of-two n >= 2048 and O(n log^2 n) global passes.  Here:
//   1. one histogram pass counts the 8-bit digits of every key position (or
//      the producer of the data counted them already, as the join probe does);
//   2. positions where all keys share one digit are skipped: a record sort is planned
//      on the device, and such a position's launch leaves at once; sorts whose digit
//      counts the host has anyway leave its launch out;
//   3. each remaining position is one "onesweep" pass: a tile is ranked by
//      digit in shared memory (warp ballots give peer masks), its per-digit
//      global offsets come from a decoupled look-back over earlier tiles, and
//      the tile is reordered in shared memory so that each digit's run is
//      written with consecutive addresses.
// Every pass is stable, so the LSD composition is a correct sort; the order
// among equal keys is input order (the reference's is unspecified).
//
// Two item layouts:
//   REC: 64-bit items, key = high 32 bits (a Record uint2 {x, y} read as one
//        little-endian u64 has y in the high word).
//   KV3: three u32 columns (key, a, b) -- the join output (key, R.payload,
//        S.payload).
#include <string.h>
#include <algorithm>
#include <utility>
#include <vector>
#include "qg_internal.cuh"
#include "qg_sort.cuh"
#include "qg_part.cuh"

namespace {

constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_ITEMS = 20;
constexpr int RS_CTAS = 3;  // per SM
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;  // 5120
constexpr int RS_LB = 8;  // predecessors read per look-back round

constexpr uint32_t ST_AGG = 1u << 30;
constexpr uint32_t ST_PRE = 2u << 30;
constexpr uint32_t ST_VAL = (1u << 30) - 1;

__global__ void __launch_bounds__(256)
k_radix_hist(const uint32_t *__restrict__ kin, const unsigned long long *__restrict__ rin,
             long long n, uint32_t key_off, int npos, uint32_t *__restrict__ ghist,
             unsigned long long *__restrict__ copy, uint4 *__restrict__ clear, long long clear_n) {
    qg_chain();
    __shared__ uint32_t sh[4][QG_RADIX];
    for (int i = threadIdx.x; i < 4 * QG_RADIX; i += blockDim.x) (&sh[0][0])[i] = 0;
    __syncthreads();
    // Four items per thread and round, all loaded before any is counted: with
    // one load in flight per thread the kernel waited on DRAM latency
    // (long-scoreboard stalls, 41 % of DRAM bandwidth).
    constexpr int U = 4;
    const long long stride = (long long)gridDim.x * blockDim.x;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (long long j = i; j < clear_n; j += stride) clear[j] = make_uint4(0, 0, 0, 0);  // the first pass's status words
    for (; i + (U - 1) * stride < n; i += U * stride) {
        uint32_t k[U];
        if (kin) {
#pragma unroll
            for (int u = 0; u < U; u++) k[u] = __ldg(kin + i + u * stride);
        } else {
            unsigned long long v[U];
#pragma unroll
            for (int u = 0; u < U; u++) v[u] = __ldg(rin + i + u * stride);
#pragma unroll
            for (int u = 0; u < U; u++) {
                if (copy) copy[i + u * stride] = v[u];  // records: optionally a copy for the passes to start from
                k[u] = (uint32_t)(v[u] >> 32);
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t ku = k[u] - key_off;
            for (int p = 0; p < npos; p++) atomicAdd(&sh[p][(ku >> (8 * p)) & 255u], 1u);
        }
    }
    for (; i < n; i += stride) {
        uint32_t k;
        if (kin) {
            k = __ldg(kin + i) - key_off;
        } else {
            const unsigned long long v = __ldg(rin + i);
            if (copy) copy[i] = v;
            k = (uint32_t)(v >> 32) - key_off;
        }
        for (int p = 0; p < npos; p++) atomicAdd(&sh[p][(k >> (8 * p)) & 255u], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < npos * QG_RADIX; i += blockDim.x) {
        uint32_t c = (&sh[0][0])[i];
        if (c) atomicAdd(&ghist[i], c);
    }
}

// A record sort planned on the device: per key position its digit bases and
// what its pass does.
struct RsPlan {
    RsPass pass[5];  // the four positions, and the copy back of an in-place sort
    uint32_t base[4 * QG_RADIX];
};

template <bool KV3, bool SIDE = false>
struct RsSmem {
    uint32_t whist[RS_WARPS][QG_RADIX];  // a warp's items per digit, then where its items of the digit go in the tile
    uint32_t goff[QG_RADIX];
    uint32_t wsum[RS_WARPS];
    // REC: v holds the u64 items; KV3: v holds (a, b) pairs and k the keys
    unsigned long long v[RS_TILE];
    uint32_t k[KV3 ? RS_TILE : 1];
    uint16_t bid[SIDE ? RS_TILE : 1];  // REC with a bucket-id sidecar: the reordered ids
};

// Radix digit of a key: ((k - key_off) >> shift) & 255.
__device__ __forceinline__ uint32_t rs_digit(uint32_t k, uint32_t key_off, int shift) {
    return (uint32_t)((unsigned long long)(k - key_off) >> shift) & 255u;  // shift may exceed 31
}

// Rank of the lane's item among the warp's items of its digit: earlier steps'
// items (hist, this warp's counters) plus lower lanes'.  Stable.  RANK as in
// k_radix_pass; ALL: every lane holds an item.
template <int RANK, bool ALL>
__device__ __forceinline__ uint32_t rs_rank(uint32_t d, bool valid, uint32_t *hist, uint32_t lt, int lane) {
    uint32_t peers;
    if (RANK == 1) {
        peers = __match_any_sync(QG_FULL_MASK, valid ? d : 256u);  // the tail's invalid lanes share 256
    } else if (RANK == 3) {
        peers = __match_any_sync(QG_FULL_MASK, valid ? d >> 4 : 16u);  // the tail's invalid lanes share 16
#pragma unroll
        for (int b = 0; b < 4; b++) {
            const uint32_t bal = __ballot_sync(QG_FULL_MASK, (d >> b) & 1u);
            peers &= ((d >> b) & 1u) ? bal : ~bal;
        }
    } else if (RANK == 4) {
        peers = __match_any_sync(QG_FULL_MASK, valid ? d >> 4 : 16u) &
                __match_any_sync(QG_FULL_MASK, valid ? d & 15u : 16u);
    } else {
        peers = ALL ? QG_FULL_MASK : __ballot_sync(QG_FULL_MASK, valid);
#pragma unroll
        for (int b = 0; b < 8; b++) {
            const uint32_t bal = __ballot_sync(QG_FULL_MASK, (d >> b) & 1u);
            peers &= ((d >> b) & 1u) ? bal : ~bal;
        }
    }
    const uint32_t before = (ALL || valid) ? hist[d] : 0u;
    __syncwarp();
    const uint32_t rank = before + __popc(peers & lt);
    if ((ALL || valid) && lane == 31 - __clz(peers)) hist[d] = rank + 1u;  // the highest peer's rank is the last
    __syncwarp();
    return rank;
}

// A tile whose pass is the identity (one digit value holds every item): copied.
template <bool KV3, bool SIDE>
__device__ __forceinline__ void rs_copy_tile(const qg_sort_bufs &src, const qg_sort_bufs &dst, long long n) {
    // every load of the tile before any store (the buffers are distinct,
    // which the compiler cannot see)
    const int tid = threadIdx.x;
    const long long b0 = (long long)blockIdx.x * RS_TILE;
    const int cnt = (int)min((long long)RS_TILE, n - b0);
    unsigned long long v[RS_ITEMS];
    uint32_t kk[KV3 ? RS_ITEMS : 1];
#pragma unroll
    for (int i = 0; i < RS_ITEMS; i++) {
        const int j = i * RS_THREADS + tid;
        if (j < cnt) {
            if (KV3) {
                kk[i] = __ldcs(src.k + b0 + j);
                v[i] = ((unsigned long long)__ldcs(src.b + b0 + j) << 32) | __ldcs(src.a + b0 + j);
            } else {
                v[i] = __ldcs(src.rec + b0 + j);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < RS_ITEMS; i++) {
        const int j = i * RS_THREADS + tid;
        if (j < cnt) {
            if (KV3) {
                dst.k[b0 + j] = kk[i];
                dst.a[b0 + j] = (uint32_t)v[i];
                dst.b[b0 + j] = (uint32_t)(v[i] >> 32);
            } else {
                dst.rec[b0 + j] = v[i];
                if (SIDE && dst.bid) dst.bid[b0 + j] = src.bid[b0 + j];
            }
        }
    }
}

// One tile of a pass.  ALL: a full tile, with no bounds checks per item.
template <bool KV3, bool SIDE, int RANK, bool ALL>
__device__ __forceinline__ void rs_tile(RsSmem<KV3, SIDE> &S, const qg_sort_bufs &src, const qg_sort_bufs &dst,
                                        uint32_t n, int cnt, int shift, uint32_t key_off, const uint32_t *__restrict__ dbase,
                                        uint32_t *__restrict__ status, qg_control *ctl, uint32_t spin_limit) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t tile = blockIdx.x;  // started in index order; the status words are cleared before every pass
    const long long base = (long long)tile * RS_TILE;
    const int w0 = warp * 32 * RS_ITEMS + lane;  // the lane's first item in the tile
    const uint32_t lt = qg_lanemask_lt();

    // REC items carry their key in the high word, so only KV3 keeps a key
    // array.  The digit is taken from the key again where it is needed, so two
    // items' ranks share a word; a sidecar's digit is kept beside the rank.
    uint32_t key[KV3 ? RS_ITEMS : 1];
    unsigned long long val[RS_ITEMS];
    uint32_t rd[SIDE ? RS_ITEMS : RS_ITEMS / 2];  // SIDE: digit << 24 | rank; else rank << 16 (odd item) | rank
    // All loads are issued before any ranking: __syncwarp orders memory, so
    // a load placed after one in program order cannot be hoisted above it,
    // and interleaving would pay one DRAM latency per item.
#pragma unroll
    for (int i = 0; i < RS_ITEMS; i++) {
        const int j = w0 + i * 32;
        val[i] = 0;
        if (KV3) key[i] = 0;
        if (SIDE) rd[i] = 0;
        if (ALL || j < cnt) {
            if (KV3) {
                key[i] = __ldcs(src.k + base + j);
                val[i] = ((unsigned long long)__ldcs(src.b + base + j) << 32) | __ldcs(src.a + base + j);
            } else {
                val[i] = __ldcs(src.rec + base + j);
                if (SIDE) rd[i] = __ldcs(src.bid + base + j);  // the bucket id, until its digit replaces it
            }
        }
    }
#pragma unroll
    for (int i = 0; i < RS_ITEMS; i++) {
        const bool valid = ALL || w0 + i * 32 < cnt;
        const uint32_t ki = KV3 ? key[i] : (uint32_t)(val[i] >> 32);
        const uint32_t d = SIDE ? (rd[i] >> shift) & 255u : rs_digit(ki, key_off, shift);
        uint32_t rank = 0;
        if constexpr (RANK == 2) {
            if (valid) rank = atomicAdd(&S.whist[0][d], 1u);
        } else {
            rank = rs_rank<RANK, ALL>(d, valid, S.whist[warp], lt, lane);
        }
        if (SIDE) rd[i] = d << 24 | rank;
        else if (i & 1) rd[i >> 1] |= rank << 16;
        else rd[i >> 1] = rank;
    }
    __syncthreads();
    uint32_t total, dstart;  // the tile's items of digit tid, and its first place in the tile
    {
        // Thread t owns digit t: where each warp's items of the digit go in the
        // tile (first place of the digit, then the earlier warps' items).
        total = 0;
        if constexpr (RANK == 2) {
            total = S.whist[0][tid];  // ranks are tile-wide already
        } else {
#pragma unroll
            for (int w = 0; w < RS_WARPS; w++) total += S.whist[w][tid];
        }
        // The tile's counts go out before its items are staged: successors
        // read them meanwhile.
        qg_st_relaxed_u32(status + (size_t)tile * QG_RADIX + tid, (tile == 0 ? ST_PRE : ST_AGG) | total);
        uint32_t inc = total;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            uint32_t x = __shfl_up_sync(QG_FULL_MASK, inc, d);
            if (lane >= d) inc += x;
        }
        if (lane == 31) S.wsum[warp] = inc;
        __syncthreads();
        uint32_t woff = 0;
        for (int w = 0; w < warp; w++) woff += S.wsum[w];
        dstart = woff + inc - total;
        uint32_t run = dstart;
        if constexpr (RANK == 2) {
            S.whist[0][tid] = run;
        } else {
#pragma unroll
            for (int w = 0; w < RS_WARPS; w++) {
                const uint32_t c = S.whist[w][tid];
                S.whist[w][tid] = run;
                run += c;
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RS_ITEMS; i++) {
        const int j = w0 + i * 32;
        if (ALL || j < cnt) {
            const uint32_t ki = KV3 ? key[i] : (uint32_t)(val[i] >> 32);
            const uint32_t d = SIDE ? rd[i] >> 24 : rs_digit(ki, key_off, shift);
            const uint32_t rank = SIDE ? rd[i] & 0xffffffu : (rd[i >> 1] >> (16 * (i & 1))) & 0xffffu;
            const uint32_t pos = S.whist[RANK == 2 ? 0 : warp][d] + rank;
            S.v[pos] = val[i];
            if (KV3) S.k[pos] = key[i];
            if (SIDE) S.bid[pos] = __ldg(src.bid + base + j);  // read again: no register held
        }
    }
    {
        // Look-back for digit t over earlier tiles, after the staging has freed
        // the items' registers.  RS_LB predecessors' words are loaded together,
        // so a chain of tiles that only published counts costs one L2 round
        // trip per RS_LB tiles.
        uint32_t excl = 0;
        if (tile > 0) {
            int j = (int)tile - 1;
            bool done = false;
            while (!done) {
                uint32_t w[RS_LB];
#pragma unroll
                for (int u = 0; u < RS_LB; u++)
                    w[u] = (j - u >= 0) ? qg_ld_relaxed_u32(status + (size_t)(j - u) * QG_RADIX + tid) : ST_PRE;
#pragma unroll
                for (int u = 0; u < RS_LB; u++) {
                    if (done) break;
                    uint32_t spins = 0;
                    while (!(w[u] & (ST_AGG | ST_PRE))) {
                        if (spins >= spin_limit) {
                            qg_record_error(ctl, QG_ERR_TIMEOUT, QG_SITE_SORT_LOOKBACK);
                            w[u] = ST_PRE;
                            break;
                        }
                        spins++;
                        __nanosleep(32);
                        w[u] = qg_ld_relaxed_u32(status + (size_t)(j - u) * QG_RADIX + tid);
                    }
                    excl += w[u] & ST_VAL;
                    if (w[u] & ST_PRE) done = true;
                }
                j -= RS_LB;
            }
            qg_st_relaxed_u32(status + (size_t)tile * QG_RADIX + tid, ST_PRE | ((excl + total) & ST_VAL));
        }
        S.goff[tid] = dbase[tid] + excl - dstart;
    }
    __syncthreads();
    // Out, each digit's run with consecutive addresses.  The digit is taken
    // from the key (or id) again: cheaper than a byte array of digits, whose
    // scattered stores cost shared-memory wavefronts.  A pass after one whose look-back
    // gave up (reported as QG_ERR_TIMEOUT) reads items that are not the ones counted, so
    // a place may lie past the end: those are dropped.
    auto put = [&](int p) {
        const unsigned long long v = S.v[p];
        const uint32_t k = KV3 ? S.k[p] : (uint32_t)(v >> 32);
        const uint32_t d = SIDE ? ((uint32_t)S.bid[p] >> shift) & 255u : rs_digit(k, key_off, shift);
        const uint32_t g = S.goff[d] + (uint32_t)p;
        if (g >= n) return;
        if (KV3) {
            dst.k[g] = k;
            dst.a[g] = (uint32_t)v;
            dst.b[g] = (uint32_t)(v >> 32);
        } else {
            dst.rec[g] = v;
            if (SIDE && dst.bid) dst.bid[g] = S.bid[p];
        }
    };
    if (ALL) {
#pragma unroll
        for (int i = 0; i < RS_ITEMS; i++) put(i * RS_THREADS + tid);
    } else {
        for (int p = tid; p < cnt; p += RS_THREADS) put(p);
    }
}

// Three CTAs per SM (80 registers, 5120 items each): one CTA's load phase
// overlaps another's ranking and writes.  The shared-memory pipe (74 % busy in
// the form before: two table reads, a digit byte and an 8-byte scatter per
// item) and the instructions per item bound it, so the tile's digit starts are
// folded into the warps' counters, the digit is taken from the key again
// instead of a byte array, full tiles have no bounds checks, and the look-back
// runs after the staging, when its predecessors have had longer to publish.
// A pass over 16M records 113 -> 88 us, over the join's 61M 386 -> 276 us.
// Four CTAs of 4096 items took 293 us there, 512- and 1024-thread CTAs 309 and
// 355, 8 items per thread 379, a look-back window of 16 or 32 was no faster.
// SIDE: the digit is bits of the bucket id in the source's sidecar (REC only),
// else radix bits of the key.
// RANK: how an item's rank within its digit is found -- 0 eight warp ballots,
// 1 one match instruction, 3 one match instruction on the digit's high four
// bits (at most 16 groups, where match is fast) and four ballots on the low
// four, 4 a match on each half (stable all four), 2 one shared-memory atomic
// on the tile's digit counter (not stable: for a first LSD pass whose order
// among equal digits nothing after it needs).
template <bool KV3, bool SIDE, int RANK = 0>
__global__ void __launch_bounds__(RS_THREADS, RS_CTAS)
k_radix_pass(qg_sort_bufs src, qg_sort_bufs dst, long long n, int shift, uint32_t key_off,
             const uint32_t *__restrict__ dbase, uint32_t *__restrict__ status, qg_control *ctl, uint32_t spin_limit,
             const unsigned long long *__restrict__ d_n, const uint32_t *__restrict__ trivial,
             const RsPass *__restrict__ plan, const qg_sort_range *__restrict__ range) {
    qg_chain();
    extern __shared__ __align__(16) unsigned char rs_raw[];
    static_assert(!(KV3 && SIDE), "no sidecar with three columns");
    RsSmem<KV3, SIDE> &S = *reinterpret_cast<RsSmem<KV3, SIDE> *>(rs_raw);
    // Item count known only on the device (graph-captured sorts): the grid
    // covers the bound n, and CTAs past the real count leave at once (no
    // tile before them waits on them).
    if (d_n && *d_n < (unsigned long long)n) n = (long long)*d_n;
    const long long left = n - (long long)blockIdx.x * RS_TILE;
    if (left <= 0) return;
    bool copy = trivial && __ldg(trivial);
    if (plan) {  // planned on the device
        const uint32_t mode = plan->mode;
        if (mode == 0) return;
        copy = mode == 2;
        src.rec = const_cast<unsigned long long *>(plan->src);
        dst.rec = plan->dst;
        status = plan->status;
        shift = (int)plan->shift;
        key_off = plan->key_off;
        if (plan->clear) plan->clear[(size_t)blockIdx.x * QG_RADIX + threadIdx.x] = 0;
    }
    if (range) {  // three columns: the pass runs or not, and reads a or b, by the key range's positions
        const int left = (int)range->npos - shift / 8;
        if (left <= 0) return;
        key_off = range->key_off;
        if (left & 1) {
            const qg_sort_bufs t = src;
            src = dst;
            dst = t;
        }
    }
    if (copy) {  // one digit value holds every item: a stable pass is the identity
        rs_copy_tile<KV3, SIDE>(src, dst, n);
        return;
    }
    for (int i = threadIdx.x; i < RS_WARPS * QG_RADIX; i += RS_THREADS) (&S.whist[0][0])[i] = 0;
    __syncthreads();
    if (left >= RS_TILE)
        rs_tile<KV3, SIDE, RANK, true>(S, src, dst, (uint32_t)n, RS_TILE, shift, key_off, dbase, status, ctl, spin_limit);
    else
        rs_tile<KV3, SIDE, RANK, false>(S, src, dst, (uint32_t)n, (int)left, shift, key_off, dbase, status, ctl, spin_limit);
}

}  // namespace

int qg_sort_positions(int bits) {
    int npos = (bits + 7) / 8;
    if (npos < 1) npos = 1;
    if (npos > 4) npos = 4;
    return npos;
}

static int rs_hist_grid(qg_ctx *ctx, long long n) {
    // 2048 threads per SM at 32 registers
    return (int)std::min<long long>((n + 255) / 256, (long long)ctx->sm_count * 8);
}

qg_status qg_radix_histogram(qg_ctx *ctx, const qg_sort_bufs &src, bool kv3, long long n,
                             uint32_t key_off, int npos, uint32_t *d_hist) {
    QG_TRY_CUDA(ctx, cudaMemsetAsync(d_hist, 0, 4 * QG_RADIX * 4, ctx->stream), "memset hist");
    if (n == 0) return QG_OK;
    qg_pre_launch(ctx);
    k_radix_hist<<<rs_hist_grid(ctx, n), 256, 0, ctx->stream>>>(kv3 ? src.k : nullptr, kv3 ? nullptr : src.rec,
                                                   n, key_off, npos, d_hist, nullptr, nullptr, 0);
    return qg_check_launch(ctx, "k_radix_hist");
}

int qg_sort_plan(const uint32_t *h_hist, int npos, long long n, int *passes, uint32_t *bases) {
    int np = 0;
    for (int p = 0; p < npos; p++) {
        bool trivial = false;
        uint32_t run = 0;
        for (int d = 0; d < QG_RADIX; d++) {
            uint32_t c = h_hist[p * QG_RADIX + d];
            if ((long long)c == n) trivial = true;
            bases[p * QG_RADIX + d] = run;
            run += c;
        }
        if (!trivial) passes[np++] = p;
    }
    return np;
}

using rs_kernel = void (*)(qg_sort_bufs, qg_sort_bufs, long long, int, uint32_t, const uint32_t *, uint32_t *,
                           qg_control *, uint32_t, const unsigned long long *, const uint32_t *, const RsPass *,
                           const qg_sort_range *);

// The pass kernel of a ranking form (see k_radix_pass); form 2 for records only.
template <bool KV3, bool SIDE>
static rs_kernel rs_pick(int rank) {
    if constexpr (!KV3)
        if (rank == 2) return k_radix_pass<KV3, SIDE, 2>;
    return rank == 1 ? k_radix_pass<KV3, SIDE, 1> : rank == 3 ? k_radix_pass<KV3, SIDE, 3>
         : rank == 4 ? k_radix_pass<KV3, SIDE, 4> : k_radix_pass<KV3, SIDE, 0>;
}

template <bool KV3, bool SIDE>
static qg_status rs_set_attr(qg_ctx *ctx) {
    static qg_per_device sites[5];
    for (int rank = 0; rank < 5; rank++)
        QG_TRY(qg_allow_smem(ctx, sites[rank], rs_pick<KV3, SIDE>(rank), sizeof(RsSmem<KV3, SIDE>)));
    return QG_OK;
}

// Ranking by match instruction for a pass with at most 16 digit values in
// use (the top pass of narrow keys): measured faster there (the 64M-record
// sort of 20-bit keys, 1.30 -> 1.22 ms over its passes), while passes with
// many digit values were slower with it (the join's partition passes 1.10 ->
// 1.38 ms) and keep the eight ballots.
// Stable ranking of the passes with many digit values: -1 the default (3),
// else forced -- 0 eight ballots, 3 a match on the high four bits and four
// ballots, 4 a match on each half (ANDed).  Measured on GB300 with 0 / 3 / 4:
// the 64M-record sort of a fresh unsorted copy, passes 1.290 / 1.265 /
// 1.437 ms; the join's stable partition pass 0.778 / 0.766 / 0.855 ms.  (Form
// 4 had looked fastest when the sort was timed re-sorting its own sorted
// output, where a warp's items share their high digits.)
static int g_rs_stable_rank = -1;

extern "C" QG_API qg_status qg_sort_set_rank(int mode) {
    if (mode != -1 && mode != 0 && mode != 3 && mode != 4) return QG_ERR_INVALID;
    g_rs_stable_rank = mode;
    return QG_OK;
}

static bool rs_few_digits(const uint32_t *hb, long long n) {
    int used = 0;
    for (int d = 0; d < QG_RADIX; d++) {
        const unsigned long long hi = d + 1 < QG_RADIX ? hb[d + 1] : (unsigned long long)n;
        used += hi > hb[d];
    }
    return used <= 16;
}

qg_status qg_radix_passes_pf(qg_ctx *ctx, bool kv3, qg_sort_bufs a, qg_sort_bufs b, long long n,
                             const qg_part_fn &pf, const int *passes, int np, const uint32_t *h_bases,
                             bool *result_in_b, bool first_unstable) {
    *result_in_b = false;
    if (np == 0 || n <= 1) return QG_OK;
    if (n >= (1LL << 30)) return QG_ERR_UNSUPPORTED;
    // REC items with a bucket-id sidecar: digits come from the sidecar, whatever
    // the partition function (it was evaluated once, when the ids were written).
    const bool side = !kv3 && a.bid != nullptr && b.bid != nullptr;
    if (pf.learned && !side) return QG_ERR_UNSUPPORTED;
    const long long tiles = (n + RS_TILE - 1) / RS_TILE;
    size_t need = 4 * QG_RADIX * 4 + (size_t)tiles * QG_RADIX * 4;
    char *scr;
    QG_TRY(qg_scratch(ctx, need, &scr));
    uint32_t *dbase = (uint32_t *)scr;
    uint32_t *status = dbase + 4 * QG_RADIX;
    // 4 KB of digit bases, in stream order before the passes that read them.
    QG_TRY(qg_stage_bases(ctx, h_bases, dbase));
    const size_t smem = kv3 ? sizeof(RsSmem<true>) : side ? sizeof(RsSmem<false, true>) : sizeof(RsSmem<false>);
    if (kv3) QG_TRY((rs_set_attr<true, false>(ctx)));
    else if (side) QG_TRY((rs_set_attr<false, true>(ctx)));
    else QG_TRY((rs_set_attr<false, false>(ctx)));
    bool in_a = true;
    for (int i = 0; i < np; i++) {
        const int p = passes[i];
        QG_TRY_CUDA(ctx, cudaMemsetAsync(status, 0, (size_t)tiles * QG_RADIX * 4, ctx->stream), "memset status");
        const qg_sort_bufs &s = in_a ? a : b;
        qg_sort_bufs d = in_a ? b : a;
        if (side && i == np - 1) d.bid = nullptr;  // the last pass's ids are not read again
        const int shift = side ? 8 * p : pf.shift + 8 * p;
        const bool m = rs_few_digits(h_bases + p * QG_RADIX, n);
        // the first pass of a caller that needs only the grouping need not be stable
        const int sr = g_rs_stable_rank >= 0 ? g_rs_stable_rank : 3;
        const int rk = (first_unstable && i == 0 && !kv3) ? 2 : (m ? 1 : sr);
        const rs_kernel kern = kv3 ? rs_pick<true, false>(rk) : side ? rs_pick<false, true>(rk) : rs_pick<false, false>(rk);
        QG_TRY(qg_launch_chained(ctx, "k_radix_pass", kern, (unsigned)tiles, RS_THREADS, smem, s, d, n, shift,
                                 side ? 0u : pf.kmin, dbase + p * QG_RADIX, status, ctx->ctl, ctx->spin_limit, nullptr,
                                 nullptr, nullptr, nullptr));
        in_a = !in_a;
    }
    *result_in_b = !in_a;
    return QG_OK;
}

// Exclusive digit bases of every position from a device histogram [npos][256];
// trivial[p] = 1 when one digit value holds every item of position p (that
// pass is then a copy).
__global__ void k_radix_bases(const uint32_t *__restrict__ hist, int npos, uint32_t *__restrict__ bases,
                              uint32_t *__restrict__ trivial) {
    qg_chain();
    __shared__ uint32_t ws[QG_RADIX / 32], wm[QG_RADIX / 32];
    const int d = threadIdx.x, lane = d & 31, w = d >> 5;
    for (int p = 0; p < npos; p++) {
        const uint32_t c = hist[p * QG_RADIX + d];
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
        uint32_t off = 0;
        for (int i = 0; i < w; i++) off += ws[i];
        bases[p * QG_RADIX + d] = off + inc - c;
        if (d == 0) {
            uint32_t tot = 0, big = 0;
            for (int i = 0; i < QG_RADIX / 32; i++) {
                tot += ws[i];
                big = max(big, wm[i]);
            }
            trivial[p] = big == tot ? 1u : 0u;
        }
        __syncthreads();
    }
}

qg_status qg_radix_passes_dev(qg_ctx *ctx, bool kv3, qg_sort_bufs a, qg_sort_bufs b, long long n_bound,
                              const unsigned long long *d_n, const uint32_t *d_hist, int npos, uint32_t key_off,
                              char *work, bool *result_in_b) {
    *result_in_b = false;
    if (n_bound <= 1 || npos <= 0) return QG_OK;
    if (npos > 4) return QG_ERR_INVALID;  // the work area holds four status regions
    if (n_bound >= (1LL << 30)) return QG_ERR_UNSUPPORTED;
    const long long tiles = (n_bound + RS_TILE - 1) / RS_TILE;
    uint32_t *dbase = (uint32_t *)work;
    uint32_t *trivial = dbase + 4 * QG_RADIX;  // [4], in a 256-byte slot
    uint32_t *status = trivial + 64;           // [npos][tiles][256]: one region per pass, cleared at once
    const size_t st_words = (size_t)tiles * QG_RADIX;
    const size_t smem = kv3 ? sizeof(RsSmem<true>) : sizeof(RsSmem<false>);
    if (kv3) QG_TRY((rs_set_attr<true, false>(ctx)));
    else QG_TRY((rs_set_attr<false, false>(ctx)));
    QG_TRY(qg_launch_chained(ctx, "k_radix_bases", k_radix_bases, 1, QG_RADIX, 0, d_hist, npos, dbase, trivial));
    QG_TRY_CUDA(ctx, cudaMemsetAsync(status, 0, (size_t)npos * st_words * 4, ctx->stream), "memset status");
    bool in_a = true;
    for (int p = 0; p < npos; p++) {
        const qg_sort_bufs &s = in_a ? a : b;
        const qg_sort_bufs &d = in_a ? b : a;
        uint32_t *stp = status + (size_t)p * st_words;
        const rs_kernel kern = kv3 ? rs_pick<true, false>(3) : rs_pick<false, false>(3);
        QG_TRY(qg_launch_chained(ctx, "k_radix_pass", kern, (unsigned)tiles, RS_THREADS, smem, s, d, n_bound, 8 * p,
                                 key_off, dbase + p * QG_RADIX, stp, ctx->ctl, ctx->spin_limit, d_n, trivial + p,
                                 nullptr, nullptr));
        in_a = !in_a;
    }
    *result_in_b = !in_a;
    return QG_OK;
}

qg_status qg_radix_passes_range(qg_ctx *ctx, qg_sort_bufs a, qg_sort_bufs b, long long n_bound,
                                const unsigned long long *d_n, const uint32_t *d_hist, const qg_sort_range *range,
                                char *work) {
    if (n_bound <= 1) return QG_OK;
    if (n_bound >= (1LL << 30)) return QG_ERR_UNSUPPORTED;
    const long long tiles = (n_bound + RS_TILE - 1) / RS_TILE;
    uint32_t *dbase = (uint32_t *)work;
    uint32_t *trivial = dbase + 4 * QG_RADIX;  // (not used: a pass whose digits are all equal is an ordinary one)
    uint32_t *status = trivial + 64;           // [4][tiles][256]
    const size_t st_words = (size_t)tiles * QG_RADIX;
    QG_TRY((rs_set_attr<true, false>(ctx)));
    QG_TRY(qg_launch_chained(ctx, "k_radix_bases", k_radix_bases, 1, QG_RADIX, 0, d_hist, 4, dbase, trivial));
    QG_TRY_CUDA(ctx, cudaMemsetAsync(status, 0, 4 * st_words * 4, ctx->stream), "memset status");
    const rs_kernel kern = rs_pick<true, false>(3);
    for (int p = 0; p < 4; p++) {
        QG_TRY(qg_launch_chained(ctx, "k_radix_pass", kern, (unsigned)tiles, RS_THREADS, sizeof(RsSmem<true>), a, b,
                                 n_bound, 8 * p, 0u, dbase + p * QG_RADIX, status + (size_t)p * st_words, ctx->ctl,
                                 ctx->spin_limit, d_n, nullptr, nullptr, range));
    }
    return QG_OK;
}

size_t qg_radix_dev_work_bytes(long long n_bound) {
    return 4 * QG_RADIX * 4 + 256 + 4 * (size_t)((n_bound + RS_TILE - 1) / RS_TILE) * QG_RADIX * 4;
}

qg_status qg_radix_passes(qg_ctx *ctx, bool kv3, qg_sort_bufs a, qg_sort_bufs b, long long n,
                          uint32_t key_off, const int *passes, int np, const uint32_t *h_bases,
                          bool *result_in_b) {
    qg_part_fn pf{0, key_off, 0, nullptr};
    return qg_radix_passes_pf(ctx, kv3, a, b, n, pf, passes, np, h_bases, result_in_b, false);
}

// Plan of a record sort from its digit counts (cleared for the next sort): the
// digit bases, and for every position with more than one digit value a pass
// from the last one's output, so that the final one lands in `out`.  In place
// (in == out) an odd number of passes starts from the copy that the histogram
// kernel made in tmp (pre_copy), else ends in tmp and is copied back.
__global__ void __launch_bounds__(QG_RADIX)
k_radix_plan(uint32_t *__restrict__ hist, const unsigned long long *in, unsigned long long *out,
             unsigned long long *tmp, bool pre_copy, uint32_t *status, size_t status_words, long long n, RsPlan *plan,
             volatile uint32_t *h_passes) {
    qg_chain();
    __shared__ uint32_t ws[4][QG_RADIX / 32], wm[4][QG_RADIX / 32];
    const int d = threadIdx.x, lane = d & 31, w = d >> 5;
    uint32_t c[4], inc[4];
#pragma unroll
    for (int p = 0; p < 4; p++) {
        c[p] = hist[p * QG_RADIX + d];
        hist[p * QG_RADIX + d] = 0;
        inc[p] = c[p];
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const uint32_t x = __shfl_up_sync(QG_FULL_MASK, inc[p], k);
            if (lane >= k) inc[p] += x;
        }
        const uint32_t mx = __reduce_max_sync(QG_FULL_MASK, c[p]);
        if (lane == 31) ws[p][w] = inc[p];
        if (lane == 0) wm[p][w] = mx;
    }
    __syncthreads();
    bool act[4];
    int np = 0;
#pragma unroll
    for (int p = 0; p < 4; p++) {
        uint32_t off = 0, big = 0;
        for (int i = 0; i < QG_RADIX / 32; i++) {
            off += i < w ? ws[p][i] : 0u;
            big = max(big, wm[p][i]);
        }
        plan->base[p * QG_RADIX + d] = off + inc[p] - c[p];
        act[p] = (long long)big != n;
        np += act[p];
    }
    if (d != 0) return;
    const bool odd = (np & 1) != 0, same = in == out;
    const unsigned long long *from = same && odd && pre_copy ? tmp : in;
    const bool to_tmp = same && odd && !pre_copy;  // the last pass ends in tmp
    int left = np, q = 0;
#pragma unroll
    for (int p = 0; p < 4; p++) {
        RsPass &P = plan->pass[p];
        P = RsPass{nullptr, nullptr, nullptr, nullptr, 0u, 8u * p, 0u, 0u};
        if (!act[p]) continue;
        left--;
        unsigned long long *to = ((left & 1) != 0) == to_tmp ? out : tmp;
        P.src = from;
        P.dst = to;
        P.status = status + (size_t)(q & 1) * status_words;
        P.clear = left ? status + (size_t)((q + 1) & 1) * status_words : nullptr;
        P.mode = 1u;
        from = to;
        q++;
    }
    if (np == 0 && !same) plan->pass[0] = RsPass{in, out, nullptr, nullptr, 2u, 0u, 0u, 0u};
    plan->pass[4] = RsPass{tmp, out, nullptr, nullptr, to_tmp ? 2u : 0u, 0u, 0u, 0u};
    *h_passes = (uint32_t)np;
}

// Sorts n REC items of `in` by key into `out` (may be `in`), tmp (n items) as
// the ping-pong buffer; `in` is not written otherwise.  Nothing is read back:
// one histogram, the plan and a launch per key position, those with a single
// digit value leaving at once (a host plan cost a copy of the counts, the wait
// and an upload, 30 us per sort, and a memset of the status words per pass:
// each pass clears the next one's).
qg_status qg_sort_rec(qg_ctx *ctx, const unsigned long long *in, unsigned long long *out, unsigned long long *tmp,
                      long long n) {
    if (n <= 0) return QG_OK;
    if (n >= (1LL << 30)) return QG_ERR_UNSUPPORTED;
    const long long tiles = (n + RS_TILE - 1) / RS_TILE;
    const size_t words = (size_t)tiles * QG_RADIX;
    char *scr;
    QG_TRY(qg_scratch(ctx, qg_align_up(sizeof(RsPlan), 256) + 2 * words * 4, &scr));
    RsPlan *plan = (RsPlan *)scr;
    uint32_t *status = (uint32_t *)(scr + qg_align_up(sizeof(RsPlan), 256));
    // In place, an odd number of passes ends in tmp.  When the context's last
    // in-place sort took an odd number, the histogram kernel (bound by its
    // shared-memory atomics, not by DRAM) also copies the records to tmp, and
    // the passes start there; otherwise a copy back follows.
    const bool same = in == out;
    const bool pre_copy = same && ctx->sort_odd_passes;
    QG_TRY((rs_set_attr<false, false>(ctx)));
    qg_pre_launch(ctx);
    k_radix_hist<<<rs_hist_grid(ctx, n), 256, 0, ctx->stream>>>(nullptr, in, n, 0u, 4, ctx->ctl->shist,
                                                                pre_copy ? tmp : nullptr, (uint4 *)status,
                                                                (long long)(words / 4));
    QG_TRY(qg_check_launch(ctx, "k_radix_hist"));
    QG_TRY(qg_launch_chained(ctx, "k_radix_plan", k_radix_plan, 1, QG_RADIX, 0, ctx->ctl->shist, in, out, tmp,
                             pre_copy, status, words, n, plan, &ctx->hres->passes));
    // Keys that are all equal need no pass.  Five launches that find nothing to do take
    // longer than one look at the plan when there are many tiles (64M records 343 us a
    // call, 294 with the look), so it is looked at after a sort that had none.
    if (same && ctx->sort_no_passes && tiles > 2000) {
        QG_TRY_CUDA(ctx, cudaStreamSynchronize(ctx->stream), "sync");
        if (ctx->hres->passes == 0) return QG_OK;
    }
    const rs_kernel kern = rs_pick<false, false>(g_rs_stable_rank >= 0 ? g_rs_stable_rank : 3);
    for (int p = 0; p < (same && !pre_copy ? 5 : 4); p++) {
        QG_TRY(qg_launch_chained(ctx, "k_radix_pass", kern, (unsigned)tiles, RS_THREADS, sizeof(RsSmem<false>),
                                 qg_sort_bufs{}, qg_sort_bufs{}, n, 8 * p, 0u, plan->base + (p & 3) * QG_RADIX,
                                 nullptr, ctx->ctl, ctx->spin_limit, nullptr, nullptr, &plan->pass[p], nullptr));
    }
    return QG_OK;
}

size_t qg_radix_status_words(long long n_bound) { return (size_t)((n_bound + RS_TILE - 1) / RS_TILE) * QG_RADIX; }

qg_status qg_radix_pass_planned(qg_ctx *ctx, const RsPass *plan, const uint32_t *dbase, long long n_bound,
                                const unsigned long long *d_n) {
    if (n_bound >= (1LL << 30)) return QG_ERR_UNSUPPORTED;
    QG_TRY((rs_set_attr<false, false>(ctx)));
    return qg_launch_chained(ctx, "k_radix_pass", k_radix_pass<false, false, 2>,
                             (unsigned)((n_bound + RS_TILE - 1) / RS_TILE), RS_THREADS, sizeof(RsSmem<false>),
                             qg_sort_bufs{}, qg_sort_bufs{}, n_bound, 0, 0u, dbase, nullptr, ctx->ctl, ctx->spin_limit,
                             d_n, nullptr, plan, nullptr);
}

// After the sort's stream has been waited for: remember an in-place sort's passes.
void qg_sort_remember(qg_ctx *ctx) {
    ctx->sort_odd_passes = (ctx->hres->passes & 1u) != 0;
    ctx->sort_no_passes = ctx->hres->passes == 0;
}

extern "C" QG_API qg_status qg_sort_rec_by_y(qg_ctx *ctx, void *records, int64_t n) {
    if (!ctx || n < 0 || (n > 0 && !records)) return QG_ERR_INVALID;
    if (((uintptr_t)records) & 7) return QG_ERR_INVALID;
    if (n <= 1) return QG_OK;
    if (n >= (1LL << 30)) return QG_ERR_UNSUPPORTED;
    char *tmp = nullptr;
    QG_TRY(qg_aux(ctx, (size_t)n * 8, &tmp));
    QG_TRY(qg_sort_rec(ctx, (unsigned long long *)records, (unsigned long long *)records, (unsigned long long *)tmp, n));
    QG_TRY(qg_ctx_check(ctx));
    qg_sort_remember(ctx);
    return QG_OK;
}
