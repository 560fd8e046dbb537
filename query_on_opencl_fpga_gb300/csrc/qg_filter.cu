// qg_filter.cu -- stable range filter.
//
// Reference chain replaced (kernel/filter/filter_op.cl, host/host/testFilter.cpp:92-154):
//   filterImpl_map_kernel (:6-31)       mark[i] = lo <= (int)Rin[i].y <= hi
//   ScanLargeArrays/prefixSum/blockAddition (:51-207)  exclusive scan of mark
//   filterImpl_outSize_kernel (:211-215) count = mark[n-1] + scan[n-1]
//   filterImpl_write_kernel (:220-238)   Rout[scan[i]] = Rin[i] if mark[i]
// The reference moves each row through HBM about six times and launches
// 2*pass+3 kernels.  Here one kernel counts the selected rows with 128-bit
// loads, gets each CTA's output offset from one exchange of counts, and writes
// the selected rows in input order (stable, as the reference's scatter is).
#include <algorithm>
#include "qg_internal.cuh"

namespace {

constexpr int FT_THREADS = 256;
constexpr int FT_WARPS = FT_THREADS / 32;
constexpr int FT_LB_WARPS = 4;  // warps doing the look-back: 128 predecessors per round

// Two phases in one launch (records, and the default column form below 2^22 rows).
// The rows are cut into units of four 128-bit loads per lane of a warp, and every warp
// owns a contiguous range of units:
//   phase 1: the warp reads its keys (or records) and counts the selected rows,
//            with no exchange between warps; it keeps each row's predicate bit,
//            and the selected records themselves as far as they fit;
//   exchange: one count per CTA, a wide look-back over the CTAs before it
//            (CTAs are numbered as they start, so they are running);
//   phase 2: the warp writes the kept records, then walks the other units
//            backwards from its end position, all in input order.  Columns read
//            payloads of lanes with a selected row only; records are read again,
//            the last unit from registers and the most recent ones from L2.
// What bounds it is the memory's pace in both phases plus one exchange per
// launch: neither a chain of look-backs, tile by tile (what records had:
// 5M of them, 40 % kept, 30.8 us, now 21; columns of 16M rows in 4096-row tiles
// with a look-back each 67, now 34), nor a second launch (columns of 300K rows 18 us
// in two, 13).  One CTA per SM: with four to eight smaller ones
// the exchange took longer (49 us with six).  Loading a unit ahead did not help.
// Keeping records spares their second read (16M, 10 % selected: 48.8 -> 34.1 us),
// unless most would not fit anyway (40M, 90 %: 161 -> 170).  A column's payloads
// would be waited for after its keys: 2 % selected 36.7 -> 34.0, but 25 % 38.3 -> 41.7.
// The selected rows pass through shared memory so that a warp's stores are
// consecutive (16M rows, 90 % kept: 87 -> 53 us).
constexpr int F2_MAX_WARPS = 32;  // one CTA of up to 1024 threads per SM
constexpr int F2_MIN_WARPS = 8;   // the look-back's warps
constexpr int F2_LOADS = 4;       // 128-bit loads per lane and unit
constexpr int F2_SUNITS = 16;     // units of a warp whose predicate bits stay in shared memory

template <bool REC>
struct F2 {
    static constexpr int PER = REC ? 2 : 4;                      // rows per 128-bit load
    static constexpr int UNIT = 32 * F2_LOADS * PER;             // rows per unit
    static constexpr uint32_t FM = (1u << PER) - 1u;             // predicate bits of one load
    static constexpr int SEG = 512;  // rows of a warp's shared memory: a unit's, or selected records kept
};

// Lane's load r of unit u: rows [idx, idx + PER), zero past the end.
template <bool REC>
__device__ __forceinline__ int4 f2_load(const int32_t *__restrict__ src, long long idx, long long n) {
    constexpr int PER = F2<REC>::PER, WORDS = 4 / PER;  // words per row
    if (idx + PER <= n) return qg_ldg_stream(reinterpret_cast<const int4 *>(src + idx * WORDS));
    int t[4] = {0, 0, 0, 0};
    for (int j = 0; j < 4; j++)
        if (idx + j / WORDS < n) t[j] = src[idx * WORDS + j];
    return make_int4(t[0], t[1], t[2], t[3]);
}

template <bool REC>
__device__ __forceinline__ uint32_t f2_flags(const int4 &k, long long idx, long long n, int32_t lo, int32_t hi) {
    if (REC)
        return (uint32_t)((k.y >= lo) & (k.y <= hi) & (idx + 0 < n)) |
               ((uint32_t)((k.w >= lo) & (k.w <= hi) & (idx + 1 < n)) << 1);
    return (uint32_t)((k.x >= lo) & (k.x <= hi) & (idx + 0 < n)) |
           ((uint32_t)((k.y >= lo) & (k.y <= hi) & (idx + 1 < n)) << 1) |
           ((uint32_t)((k.z >= lo) & (k.z <= hi) & (idx + 2 < n)) << 2) |
           ((uint32_t)((k.w >= lo) & (k.w <= hi) & (idx + 3 < n)) << 3);
}

// A unit's selected rows before this lane's load r; returns the unit's total.  One
// scan over the lanes of the four loads' counts, a byte each: a ballot and two
// population counts per row took 37.4 us instead of 34.2 (16M rows, 10 % selected).
template <bool REC>
__device__ __forceinline__ uint32_t f2_places(uint32_t fl, uint32_t (&pre)[F2_LOADS]) {
    constexpr int PER = F2<REC>::PER;
    static_assert(F2_LOADS == 4 && 32 * PER < 256, "a byte per load");
    const int lane = threadIdx.x & 31;
    uint32_t c = 0;
#pragma unroll
    for (int r = 0; r < F2_LOADS; r++) c |= (uint32_t)__popc((fl >> (PER * r)) & F2<REC>::FM) << (8 * r);
    uint32_t inc = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t x = __shfl_up_sync(QG_FULL_MASK, inc, d);
        if (lane >= d) inc += x;
    }
    const uint32_t all = __shfl_sync(QG_FULL_MASK, inc, 31);
    inc -= c;
    uint32_t tot = 0;
#pragma unroll
    for (int r = 0; r < F2_LOADS; r++) {
        pre[r] = tot + ((inc >> (8 * r)) & 255u);
        tot += (all >> (8 * r)) & 255u;
    }
    return tot;
}

template <bool REC>
__global__ void __launch_bounds__(32 * F2_MAX_WARPS, 1)
k_filter_two(const int32_t *__restrict__ src, const int32_t *__restrict__ pay, long long n, long long units,
             int32_t lo, int32_t hi, int2 *__restrict__ out, long long cap, long long *__restrict__ d_count,
             uint16_t *__restrict__ spill, qg_lookback lb) {
    constexpr int PER = F2<REC>::PER, UNIT = F2<REC>::UNIT;
    // per warp: a unit's selected rows on their way out, or records kept; per thread: predicate bits
    extern __shared__ __align__(16) unsigned char f2_raw[];
    __shared__ uint32_t s_tile, s_epoch, s_excl, s_cnt[F2_MAX_WARPS], s_tmp[2 * F2_MIN_WARPS];
    const uint32_t nw = blockDim.x >> 5;
    int2 *stage = reinterpret_cast<int2 *>(f2_raw) + (size_t)(threadIdx.x >> 5) * F2<REC>::SEG;
    uint16_t *s_mask = reinterpret_cast<uint16_t *>(reinterpret_cast<int2 *>(f2_raw) + (size_t)nw * F2<REC>::SEG);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    qg_lb_begin_dyn(lb, &s_tile, &s_epoch);
    const uint32_t tile = s_tile;
    const long long W = (long long)gridDim.x * nw, gw = (long long)tile * nw + warp;
    const long long ub = units * gw / W, ue = units * (gw + 1) / W;
    int4 v[F2_LOADS];
    uint32_t cnt = 0, fl = 0, kept = 0;
    long long ur = ub;  // the rows of units [ub, ur) are kept, the others' counted
    if (REC) {
        const long long most = 4 * F2<REC>::SEG / max(ue - ub, 1ll);
        for (; ur < ue; ur++) {
            const long long r0 = ur * UNIT + lane * PER;
#pragma unroll
            for (int r = 0; r < F2_LOADS; r++) v[r] = f2_load<REC>(src, r0 + r * 32 * PER, n);
            fl = 0;
#pragma unroll
            for (int r = 0; r < F2_LOADS; r++) fl |= f2_flags<REC>(v[r], r0 + r * 32 * PER, n, lo, hi) << (PER * r);
            uint32_t pre[F2_LOADS];
            const uint32_t tot = f2_places<REC>(fl, pre);
            if (kept + tot > (uint32_t)F2<REC>::SEG || (ur == ub && tot > most)) break;
#pragma unroll
            for (int r = 0; r < F2_LOADS; r++) {
                uint32_t pos = kept + pre[r];
                if ((fl >> (PER * r)) & 1u) stage[pos++] = make_int2(v[r].x, v[r].y);
                if ((fl >> (PER * r)) & 2u) stage[pos] = make_int2(v[r].z, v[r].w);
            }
            kept += tot;
        }
    }
    for (long long u = ur; u < ue; u++) {
        const long long r0 = u * UNIT + lane * PER;
#pragma unroll
        for (int r = 0; r < F2_LOADS; r++) v[r] = f2_load<REC>(src, r0 + r * 32 * PER, n);
        fl = 0;
#pragma unroll
        for (int r = 0; r < F2_LOADS; r++) fl |= f2_flags<REC>(v[r], r0 + r * 32 * PER, n, lo, hi) << (PER * r);
        cnt += __popc(fl);
        // only this thread reads its bits back
        if (u - ub < F2_SUNITS) s_mask[(u - ub) * blockDim.x + tid] = (uint16_t)fl;
        else spill[u * 32 + lane] = (uint16_t)fl;
    }
    cnt = __reduce_add_sync(QG_FULL_MASK, cnt) + kept;
    if (lane == 0) s_cnt[warp] = cnt;
    __syncthreads();
    const uint32_t wc = lane < (int)nw ? s_cnt[lane] : 0u;
    const uint32_t before = __reduce_add_sync(QG_FULL_MASK, lane < warp ? wc : 0u);
    if (warp < F2_MIN_WARPS) {
        const uint32_t total = __reduce_add_sync(QG_FULL_MASK, wc);
        const uint32_t e = qg_lb_wide_exclusive<F2_MIN_WARPS>(lb, tile, s_epoch, total, s_tmp);
        if (tid == 0) {
            s_excl = e;
            if (tile == gridDim.x - 1) *d_count = (long long)e + total;
        }
    }
    __syncthreads();
    long long end = (long long)s_excl + before + cnt;  // one past the warp's last output row
    if (REC) {
        const long long start = end - cnt;
        const uint32_t lim = start >= cap ? 0u : (uint32_t)min((long long)kept, cap - start);
        __syncwarp();
        for (uint32_t i = lane; i < lim; i += 32) out[start + i] = stage[i];
        __syncwarp();
    }
    for (long long u = ue - 1; u >= ur; u--) {
        const long long r0 = u * UNIT + lane * PER;
        if (u < ue - 1) {
            fl = u - ub < F2_SUNITS ? (uint32_t)s_mask[(u - ub) * blockDim.x + tid] : (uint32_t)spill[u * 32 + lane];
            if (!__any_sync(QG_FULL_MASK, fl != 0u)) continue;
        }
        if (!REC || u < ue - 1) {
#pragma unroll
            for (int r = 0; r < F2_LOADS; r++) {
                v[r] = make_int4(0, 0, 0, 0);
                if ((fl >> (PER * r)) & F2<REC>::FM) v[r] = f2_load<REC>(REC ? src : pay, r0 + r * 32 * PER, n);
            }
        }
        uint32_t pre[F2_LOADS];
        const uint32_t tot = f2_places<REC>(fl, pre);
        // through shared memory, so that the warp's stores are consecutive
#pragma unroll
        for (int r = 0; r < F2_LOADS; r++) {
            uint32_t pos = pre[r];
            const int x[4] = {v[r].x, v[r].y, v[r].z, v[r].w};
#pragma unroll
            for (int j = 0; j < PER; j++)
                if ((fl >> (PER * r + j)) & 1u)
                    stage[pos++] = REC ? make_int2(x[2 * j & 3], x[(2 * j + 1) & 3])
                                       : make_int2((int)(r0 + r * 32 * PER + j), x[j]);
        }
        __syncwarp();
        end -= tot;
        const uint32_t lim = end >= cap ? 0u : (uint32_t)min((long long)tot, cap - end);
        for (uint32_t i = lane; i < lim; i += 32) out[end + i] = stage[i];
        __syncwarp();
    }
    qg_lb_finish_dyn(lb, tile, gridDim.x - 1, s_epoch);
}

// Records whose output lies over the input, beginning at or before it: one pass, a
// look-back per 4096-record tile.  A tile's rows go to places of its own and earlier
// tiles' rows, and those were loaded before their counts were published, so nothing is
// overwritten that is still to be read.  A copy of the input for k_filter_two took
// longer (1.0 selected: 16M records 110 us a call, 99 so; 40M 264 / 227).
constexpr int FR_ROUNDS = 8;  // 128-bit loads per thread

__global__ void __launch_bounds__(FT_THREADS, 5)
k_filter_rec(const int4 *in, long long n, int32_t lo, int32_t hi, int2 *out, long long cap, long long *d_count,
             qg_lookback lb) {
    constexpr int TILE = FT_THREADS * FR_ROUNDS * 2;
    __shared__ uint32_t s_tile, s_epoch, s_excl, s_woff[FR_ROUNDS * FT_WARPS], s_tmp[2 * FT_LB_WARPS + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long base = (long long)blockIdx.x * TILE;
    const uint32_t lt = qg_lanemask_lt();
    int4 v[FR_ROUNDS];
    // every load of the tile before the first ballot
#pragma unroll
    for (int r = 0; r < FR_ROUNDS; r++) {
        const long long idx = base + (long long)(r * FT_THREADS + tid) * 2;
        v[r] = make_int4(0, 0, 0, 0);
        if (idx + 1 < n) {
            v[r] = __ldcs(in + (idx >> 1));
        } else if (idx < n) {
            const int2 a = reinterpret_cast<const int2 *>(in)[idx];
            v[r] = make_int4(a.x, a.y, 0, 0);
        }
    }
    qg_lb_begin(lb, &s_tile, &s_epoch);
    uint32_t fl = 0, lpre[FR_ROUNDS];  // bits 2r, 2r + 1: the round's records
#pragma unroll
    for (int r = 0; r < FR_ROUNDS; r++) {
        const uint32_t f = f2_flags<true>(v[r], base + (long long)(r * FT_THREADS + tid) * 2, n, lo, hi);
        const uint32_t b0 = __ballot_sync(QG_FULL_MASK, f & 1u), b1 = __ballot_sync(QG_FULL_MASK, f & 2u);
        lpre[r] = __popc(b0 & lt) + __popc(b1 & lt);
        if (lane == 0) s_woff[r * FT_WARPS + warp] = __popc(b0) + __popc(b1);
        fl |= f << (2 * r);
    }
    qg_tile_offsets_wide<FR_ROUNDS * FT_WARPS, FT_LB_WARPS>(s_woff, lb, blockIdx.x, s_epoch, &s_excl, s_tmp, d_count,
                                                            gridDim.x - 1);
    const long long excl = s_excl;
#pragma unroll
    for (int r = 0; r < FR_ROUNDS; r++) {
        long long pos = excl + s_woff[r * FT_WARPS + warp] + lpre[r];
        if ((fl >> (2 * r)) & 1u) {
            if (pos < cap) out[pos] = make_int2(v[r].x, v[r].y);
            pos++;
        }
        if (((fl >> (2 * r + 1)) & 1u) && pos < cap) out[pos] = make_int2(v[r].z, v[r].w);
    }
    qg_lb_finish(lb, blockIdx.x, gridDim.x - 1, s_epoch);
}

// The default column filter of larger inputs: the two phases in two launches, the
// launch boundary being their exchange.  In k_filter_two a warp writes the rows it
// has counted, so rows selected close together (a time range of a sorted table) are
// written by a few SMs: 40M sorted rows, 1 % selected 109 us a call, 59 here (16M 60
// / 40, 4M 32 / 30).  Here the write phase deals the units out one by one to all
// warps; it reads the predicate bits (64 bytes per unit) instead of the keys.  For
// rows selected evenly both take the same (16M rows, 10 %: 46 / 45 us; 40M 74 / 75,
// 1 % 69 / 72); below 4M rows one launch is 1 to 2 us faster.  As the keys are not
// read again, the output may lie over them.
//   per: units per range, which one warp of the count phase takes;
//   upre: selected rows of the range before the unit; rtot: of the range.
constexpr int FC_WARPS = 32;  // k_filter_count, one CTA per SM
constexpr int FW_WARPS = 28;  // k_filter_write: 72 registers; 24 warps take 48 us instead of 42, 32 spill
constexpr int FW_EACH = 12;   // ranges per thread, at most
constexpr int64_t F2_TWO_ROWS = 1 << 22;

__global__ void __launch_bounds__(32 * FC_WARPS, 1)
k_filter_count(const int32_t *__restrict__ key, long long n, uint32_t units, uint32_t per, int32_t lo, int32_t hi,
               uint16_t *__restrict__ mask, uint32_t *__restrict__ upre, uint32_t *__restrict__ rtot) {
    constexpr int PER = F2<false>::PER, UNIT = F2<false>::UNIT;
    qg_chain();
    const int lane = threadIdx.x & 31;
    const uint32_t range = blockIdx.x * FC_WARPS + (threadIdx.x >> 5);
    const long long ub = (long long)range * per, ue = min(ub + per, (long long)units);
    uint32_t run = 0;
    for (long long u = ub; u < ue; u++) {
        const long long r0 = u * UNIT + lane * PER;
        int4 v[F2_LOADS];
#pragma unroll
        for (int r = 0; r < F2_LOADS; r++) v[r] = f2_load<false>(key, r0 + r * 32 * PER, n);
        uint32_t fl = 0;
#pragma unroll
        for (int r = 0; r < F2_LOADS; r++) fl |= f2_flags<false>(v[r], r0 + r * 32 * PER, n, lo, hi) << (PER * r);
        mask[u * 32 + lane] = (uint16_t)fl;
        if (lane == 0) upre[u] = run;
        run += __reduce_add_sync(QG_FULL_MASK, __popc(fl));
    }
    if (lane == 0) rtot[range] = run;
}

__global__ void __launch_bounds__(32 * FW_WARPS, 1)
k_filter_write(const uint16_t *__restrict__ mask, const uint32_t *__restrict__ upre, const uint32_t *__restrict__ rtot,
               uint32_t ranges, const int32_t *__restrict__ pay, long long n, uint32_t units, uint32_t per,
               int2 *__restrict__ out, long long cap, long long *__restrict__ d_count) {
    constexpr int PER = F2<false>::PER, UNIT = F2<false>::UNIT;
    qg_chain();
    extern __shared__ __align__(16) unsigned char f2_raw[];
    __shared__ uint32_t s_w[FW_WARPS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int2 *stage = reinterpret_cast<int2 *>(f2_raw) + (size_t)warp * F2<false>::SEG;
    uint32_t *s_base = reinterpret_cast<uint32_t *>(reinterpret_cast<int2 *>(f2_raw) + (size_t)FW_WARPS * F2<false>::SEG);
    const uint32_t W = gridDim.x * FW_WARPS;
    uint32_t u = blockIdx.x * FW_WARPS + warp;
    // the bits two units ahead, the payloads of lanes with a selected row one unit
    // ahead (16M rows, 10 %: 46.5 us without the payloads, 45)
    uint32_t fl = 0, up = 0, fn = 0, pn = 0;
    if (u < units) {
        fl = mask[(size_t)u * 32 + lane];
        up = upre[u];
    }
    {  // the ranges' first output rows
        uint32_t c[FW_EACH], sum = 0;
        const uint32_t b0 = tid * FW_EACH;
#pragma unroll
        for (int i = 0; i < FW_EACH; i += 4) {  // (ranges is a multiple of four)
            const uint4 x = b0 + i < ranges ? __ldg(reinterpret_cast<const uint4 *>(rtot + b0 + i)) : make_uint4(0, 0, 0, 0);
            c[i] = x.x;
            c[i + 1] = x.y;
            c[i + 2] = x.z;
            c[i + 3] = x.w;
        }
#pragma unroll
        for (int i = 0; i < FW_EACH; i++) {
            const uint32_t x = c[i];
            c[i] = sum;
            sum += x;
        }
        uint32_t inc = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t x = __shfl_up_sync(QG_FULL_MASK, inc, d);
            if (lane >= d) inc += x;
        }
        if (lane == 31) s_w[warp] = inc;
        __syncthreads();
        const uint32_t at = __reduce_add_sync(QG_FULL_MASK, lane < warp ? s_w[lane] : 0u) + inc - sum;
#pragma unroll
        for (int i = 0; i < FW_EACH; i++)
            if (b0 + i < ranges) s_base[b0 + i] = at + c[i];
        if (blockIdx.x == 0 && tid == 32 * FW_WARPS - 1) *d_count = (long long)at + sum;
        __syncthreads();
    }
    auto load = [&](int4 (&v)[F2_LOADS], uint32_t unit, uint32_t f) {
        const long long r0 = (long long)unit * UNIT + lane * PER;
#pragma unroll
        for (int r = 0; r < F2_LOADS; r++) {
            v[r] = make_int4(0, 0, 0, 0);
            if ((f >> (PER * r)) & F2<false>::FM) v[r] = f2_load<false>(pay, r0 + r * 32 * PER, n);
        }
    };
    int4 vn[F2_LOADS];
    load(vn, u, fl);
    if (u + W < units) {
        fn = mask[(size_t)(u + W) * 32 + lane];
        pn = upre[u + W];
    }
    while (u < units) {
        const uint32_t f = fl, p = up, next = u + W;
        int4 v[F2_LOADS];
#pragma unroll
        for (int r = 0; r < F2_LOADS; r++) v[r] = vn[r];
        fl = fn;
        up = pn;
        if (next < units) load(vn, next, fl);
        fn = 0;
        if (next + W < units) {
            fn = mask[(size_t)(next + W) * 32 + lane];
            pn = upre[next + W];
        }
        if (__any_sync(QG_FULL_MASK, f != 0u)) {
            const long long r0 = (long long)u * UNIT + lane * PER;
            uint32_t pre[F2_LOADS];
            const uint32_t tot = f2_places<false>(f, pre);
#pragma unroll
            for (int r = 0; r < F2_LOADS; r++) {
                uint32_t pos = pre[r];
                const int x[4] = {v[r].x, v[r].y, v[r].z, v[r].w};
#pragma unroll
                for (int j = 0; j < PER; j++)
                    if ((f >> (PER * r + j)) & 1u) stage[pos++] = make_int2((int)(r0 + r * 32 * PER + j), x[j]);
            }
            __syncwarp();
            const long long at = (long long)s_base[u / per] + p;
            const uint32_t lim = at >= cap ? 0u : (uint32_t)min((long long)tot, cap - at);
            for (uint32_t i = lane; i < lim; i += 32) out[at + i] = stage[i];
            __syncwarp();
        }
        u = next;
    }
}

// Columns: int32 key and payload, four rows per 128-bit load.  Output is the
// int32 pair (row id, payload).  The tile id is taken from the control
// block's tile counter (the CTAs' start order), so a tile only ever waits for
// tiles that are already running.
template <int ROUNDS>
__global__ void __launch_bounds__(FT_THREADS, 5)
k_filter_cols(const int32_t *__restrict__ key, const int32_t *__restrict__ pay, long long n,
              int32_t lo, int32_t hi, int2 *__restrict__ out, long long cap,
              long long *__restrict__ d_count, qg_lookback lb) {
    constexpr int TILE = FT_THREADS * ROUNDS * 4;
    __shared__ uint32_t s_tile, s_epoch, s_excl;
    __shared__ uint32_t s_woff[ROUNDS * FT_WARPS];
    qg_lb_begin_dyn(lb, &s_tile, &s_epoch);
    const uint32_t tile = s_tile;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long base = (long long)tile * TILE;
    const uint32_t lt = qg_lanemask_lt();

    int4 kv[ROUNDS], pv[ROUNDS];
    uint32_t fl = 0;  // bit 4r+j
    uint32_t lpre[ROUNDS];
    // All loads first, then the predicates and ballots.
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        long long idx = base + (long long)(r * FT_THREADS + tid) * 4;
        if (idx + 3 < n) {
            kv[r] = qg_ldg_stream(reinterpret_cast<const int4 *>(key + idx));
            pv[r] = qg_ldg_stream(reinterpret_cast<const int4 *>(pay + idx));
        } else {
            int t[4] = {0, 0, 0, 0}, p[4] = {0, 0, 0, 0};
            for (int j = 0; j < 4; j++)
                if (idx + j < n) { t[j] = key[idx + j]; p[j] = pay[idx + j]; }
            kv[r] = make_int4(t[0], t[1], t[2], t[3]);
            pv[r] = make_int4(p[0], p[1], p[2], p[3]);
        }
    }
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        long long idx = base + (long long)(r * FT_THREADS + tid) * 4;
        uint32_t f = 0;
        f |= (uint32_t)((kv[r].x >= lo) & (kv[r].x <= hi) & (idx + 0 < n)) << 0;
        f |= (uint32_t)((kv[r].y >= lo) & (kv[r].y <= hi) & (idx + 1 < n)) << 1;
        f |= (uint32_t)((kv[r].z >= lo) & (kv[r].z <= hi) & (idx + 2 < n)) << 2;
        f |= (uint32_t)((kv[r].w >= lo) & (kv[r].w <= hi) & (idx + 3 < n)) << 3;
        uint32_t c = 0, tot = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            uint32_t b = __ballot_sync(QG_FULL_MASK, (f >> j) & 1u);
            c += __popc(b & lt);
            tot += __popc(b);
        }
        lpre[r] = c;
        if (lane == 0) s_woff[r * FT_WARPS + warp] = tot;
        fl |= f << (4 * r);
    }
    __shared__ uint32_t s_tmp[2 * FT_LB_WARPS + 1];
    qg_tile_offsets_wide<ROUNDS * FT_WARPS, FT_LB_WARPS>(s_woff, lb, tile, s_epoch, &s_excl, s_tmp,
                                                         d_count, gridDim.x - 1);
    const long long excl = s_excl;
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        long long pos = excl + s_woff[r * FT_WARPS + warp] + lpre[r];
        const long long idx = base + (long long)(r * FT_THREADS + tid) * 4;
        const int kk[4] = {pv[r].x, pv[r].y, pv[r].z, pv[r].w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if ((fl >> (4 * r + j)) & 1u) {
                if (pos < cap) out[pos] = make_int2((int32_t)(idx + j), kk[j]);
                pos++;
            }
        }
    }
    qg_lb_finish_dyn(lb, tile, gridDim.x - 1, s_epoch);
}

constexpr int COL_ROUNDS = 4;   // 4096 rows per tile

// Persistent column filter: each CTA streams tiles of 4096 rows (keys and
// payloads, 32 KB) through a 3-stage shared-memory ring filled by the bulk-copy
// (TMA) engine, so the next tiles are in flight while a tile's look-back
// resolves.  Tile ids come from the context's atomic counter in the order the
// CTAs ask for them; a CTA processes its tiles in increasing order, so every
// tile's predecessors belong to running CTAs and the look-back always ends.
constexpr int FP_THREADS = 256;
constexpr int FP_WARPS = FP_THREADS / 32;
constexpr int FP_TILE = 4096;
constexpr int FP_ROUNDS = FP_TILE / FP_THREADS;  // 16: one row per thread per round
constexpr int FP_STAGES = 3;

struct FpSmem {
    int32_t k[FP_STAGES][FP_TILE];
    int32_t p[FP_STAGES][FP_TILE];
    unsigned long long bar[FP_STAGES];
    uint32_t tile_of[FP_STAGES];
    uint32_t pending[FP_STAGES];  // a copy (or arrival) was issued into the stage and not yet seen to land
    uint32_t phase[FP_STAGES];    // phases of the stage's barrier seen to complete
    uint32_t broken;              // a wait gave up: no more copies, every later tile read from global
    uint32_t woff[FP_ROUNDS * FP_WARPS];
    uint32_t bal[FP_ROUNDS * FP_WARPS];
    uint32_t lbtmp[2 * FT_LB_WARPS + 1];
    uint32_t excl, epoch;
};

__device__ __forceinline__ void fp_issue(FpSmem &S, int s, const int32_t *key, const int32_t *pay,
                                         long long n, uint32_t t) {
    const long long base = (long long)t * FP_TILE;
    long long rows = n - base;
    if (rows > FP_TILE) rows = FP_TILE;
    const uint32_t bytes = (uint32_t)(rows & ~3LL) * 4u;
    if (bytes) {
        qg_mbar_arrive_expect_tx(&S.bar[s], 2 * bytes);
        qg_bulk_g2s(S.k[s], key + base, bytes, &S.bar[s]);
        qg_bulk_g2s(S.p[s], pay + base, bytes, &S.bar[s]);
    } else {
        qg_mbar_arrive(&S.bar[s]);
    }
}

__global__ void __launch_bounds__(FP_THREADS)
k_filter_cols_tma(const int32_t *__restrict__ key, const int32_t *__restrict__ pay, long long n,
                  int32_t lo, int32_t hi, int2 *__restrict__ out, long long cap,
                  long long *__restrict__ d_count, qg_lookback lb, uint32_t num_tiles) {
    extern __shared__ __align__(128) unsigned char fp_raw[];
    FpSmem &S = *reinterpret_cast<FpSmem *>(fp_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t lt = qg_lanemask_lt();
    if (tid == 0) {
        for (int s = 0; s < FP_STAGES; s++) qg_mbar_init(&S.bar[s], 1);
        qg_mbar_fence_init();
        S.epoch = *(volatile uint32_t *)&lb.ctl->epoch;
        S.broken = 0;
        for (int s = 0; s < FP_STAGES; s++) {
            const uint32_t t = atomicAdd(&lb.ctl->tile_ctr, 1u);
            S.tile_of[s] = t;
            S.phase[s] = 0;
            S.pending[s] = t < num_tiles ? 1u : 0u;
            if (t < num_tiles) fp_issue(S, s, key, pay, n, t);
        }
    }
    __syncthreads();
    for (uint32_t it = 0;; it++) {
        const int s = (int)(it % FP_STAGES);
        const uint32_t t = S.tile_of[s];
        if (t >= num_tiles) break;
        // Bounded wait for the stage's copy.  The CTA uses the staged tile only
        // when every thread saw it land; otherwise it reports QG_ERR_TIMEOUT,
        // reads this and every later tile from global memory, issues no more
        // copies, and never reads a stage whose copy it did not see land.
        const bool waited = !S.broken && S.pending[s];
        bool landed = false;
        if (waited) {
            const uint32_t parity = S.phase[s] & 1u;
            uint32_t w = 0;
            landed = true;
            while (!qg_mbar_try_wait(&S.bar[s], parity)) {
                if (++w >= lb.spin_limit) {
                    landed = false;
                    break;
                }
            }
        }
        const bool all = __syncthreads_and(landed) != 0;
        const bool some = __syncthreads_or(landed) != 0;
        if (waited && tid == 0) {
            if (!all) {
                qg_record_error(lb.ctl, QG_ERR_TIMEOUT, lb.site);
                S.broken = 1;
            }
            if (some) {  // the copy completed (a thread saw its phase end)
                S.pending[s] = 0;
                S.phase[s]++;
            }
        }
        const long long base = (long long)t * FP_TILE;
        long long rows_l = n - base;
        const int rows = rows_l > FP_TILE ? FP_TILE : (int)rows_l;
        const int bulk_rows = (waited && all) ? (rows & ~3) : 0;
#pragma unroll
        for (int r = 0; r < FP_ROUNDS; r++) {
            const int row = r * FP_THREADS + tid;
            bool f = false;
            if (row < rows) {
                const int32_t k = row < bulk_rows ? S.k[s][row] : key[base + row];
                f = (k >= lo) & (k <= hi);
            }
            const uint32_t b = __ballot_sync(QG_FULL_MASK, f);
            if (lane == 0) {
                S.woff[r * FP_WARPS + warp] = __popc(b);
                S.bal[r * FP_WARPS + warp] = b;
            }
        }
        qg_tile_offsets_wide<FP_ROUNDS * FP_WARPS, FT_LB_WARPS>(S.woff, lb, t, S.epoch, &S.excl,
                                                                S.lbtmp, d_count, num_tiles - 1);
        const long long excl = S.excl;
#pragma unroll
        for (int r = 0; r < FP_ROUNDS; r++) {
            const uint32_t b = S.bal[r * FP_WARPS + warp];
            if ((b >> lane) & 1u) {
                const int row = r * FP_THREADS + tid;
                const long long pos = excl + S.woff[r * FP_WARPS + warp] + __popc(b & lt);
                const int32_t pv = row < bulk_rows ? S.p[s][row] : pay[base + row];
                if (pos < cap) out[pos] = make_int2((int32_t)(base + row), pv);
            }
        }
        __syncthreads();
        if (tid == 0) {
            const uint32_t t2 = atomicAdd(&lb.ctl->tile_ctr, 1u);
            S.tile_of[s] = t2;
            if (t2 < num_tiles && !S.broken && !S.pending[s]) {
                fp_issue(S, s, key, pay, n, t2);
                S.pending[s] = 1;
            }
        }
        __syncthreads();
    }
    // A copy still in flight into this CTA's shared memory must land before the
    // CTA exits (only after a wait gave up): wait for it, again with a limit --
    // its own, not the caller's poll limit, which may be 0 (a copy from valid
    // memory lands within microseconds; the limit only bounds the loop).
    if (tid == 0 && S.broken) {
        constexpr uint32_t DRAIN_POLLS = 1u << 22;
        for (int s = 0; s < FP_STAGES; s++) {
            if (!S.pending[s]) continue;
            for (uint32_t w = 0; w < DRAIN_POLLS && !qg_mbar_try_wait(&S.bar[s], S.phase[s] & 1u); w++) {
            }
        }
    }
    __syncthreads();
    qg_lb_end(lb);
}

}  // namespace

static qg_status finish_count(qg_ctx *ctx, int64_t cap, int64_t *out_n) {
    long long h = 0;
    QG_TRY(qg_host_count(ctx, &h));
    *out_n = h;
    if (h > cap) return QG_ERR_CAPACITY;
    return QG_OK;
}

// Launch of k_filter_two: a warp per unit until every SM is full, then
// contiguous ranges.  `spill` holds the predicate bits of a warp's units past
// the 16 it keeps in shared memory (above 20M records on 152 SMs, or 40M column rows).
template <bool REC>
static qg_status f2_launch(qg_ctx *ctx, const int32_t *src, const int32_t *pay, int64_t n, int32_t lo, int32_t hi,
                           void *out, int64_t cap, long long *d_count) {
    const long long units = qg_ceil_div(n, F2<REC>::UNIT);
    const long long warps = std::max<long long>(F2_MIN_WARPS, std::min<long long>(F2_MAX_WARPS, qg_ceil_div(units, ctx->sm_count)));
    const long long grid = std::min<long long>(qg_ceil_div(units, warps), ctx->sm_count);
    qg_lookback lb;
    QG_TRY(qg_lb_make(ctx, grid, QG_SITE_FILTER, &lb));
    const long long per_warp = qg_ceil_div(units, grid * warps);  // a warp's units, at most
    uint16_t *spill = nullptr;
    if (per_warp > F2_SUNITS) {
        char *scr;
        QG_TRY(qg_scratch(ctx, (size_t)units * 64, &scr));
        spill = (uint16_t *)scr;
    }
    const size_t smem = (size_t)warps * (F2<REC>::SEG * 8 + std::min<long long>(per_warp, F2_SUNITS) * 64);
    static qg_per_device site;
    QG_TRY(qg_allow_smem(ctx, site, k_filter_two<REC>, F2_MAX_WARPS * (F2<REC>::SEG * 8 + F2_SUNITS * 64)));
    qg_pre_launch(ctx);
    k_filter_two<REC><<<(unsigned)grid, (unsigned)(32 * warps), smem, ctx->stream>>>(src, pay, n, units, lo, hi,
                                                                                    (int2 *)out, cap, d_count, spill, lb);
    return qg_check_launch(ctx, REC ? "k_filter_two_rec" : "k_filter_two");
}

static size_t f2_two_bytes(qg_ctx *ctx, int64_t n) {
    return (size_t)qg_ceil_div(n, F2<false>::UNIT) * 68 + 512 + (size_t)ctx->sm_count * FC_WARPS * 4;
}
// Whether the scratch arena holds the bits, or may grow (not while a graph is captured).
static bool f2_two_fits(qg_ctx *ctx, int64_t n) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    return f2_two_bytes(ctx, n) <= ctx->scratch_bytes ||
           (cudaStreamIsCapturing(ctx->stream, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone);
}

static qg_status f2_launch_two(qg_ctx *ctx, const int32_t *key, const int32_t *pay, int64_t n, int32_t lo, int32_t hi,
                               void *out, int64_t cap, long long *d_count) {
    const uint32_t units = (uint32_t)qg_ceil_div(n, F2<false>::UNIT);
    const long long sms = std::min<long long>(ctx->sm_count, FW_EACH * FW_WARPS);  // ranges fit the write phase's threads
    const uint32_t gc = (uint32_t)std::min<long long>(qg_ceil_div(units, FC_WARPS), sms), ranges = gc * FC_WARPS;
    const uint32_t gw = (uint32_t)std::min<long long>(qg_ceil_div(units, FW_WARPS), ctx->sm_count);
    const uint32_t per = (uint32_t)qg_ceil_div(units, ranges);
    const size_t mb = qg_align_up((size_t)units * 64, 256), ub = qg_align_up((size_t)units * 4, 256);
    char *scr;
    QG_TRY(qg_scratch(ctx, f2_two_bytes(ctx, n), &scr));
    uint16_t *mask = (uint16_t *)scr;
    uint32_t *upre = (uint32_t *)(scr + mb), *rtot = (uint32_t *)(scr + mb + ub);
    const size_t smem = (size_t)FW_WARPS * F2<false>::SEG * 8 + (size_t)ranges * 4;
    static qg_per_device site;
    QG_TRY(qg_allow_smem(ctx, site, k_filter_write, smem));
    qg_pre_launch(ctx);
    k_filter_count<<<gc, 32 * FC_WARPS, 0, ctx->stream>>>(key, n, units, per, lo, hi, mask, upre, rtot);
    QG_TRY(qg_check_launch(ctx, "k_filter_count"));
    return qg_launch_chained(ctx, "k_filter_write", k_filter_write, gw, 32 * FW_WARPS, smem, mask, upre, rtot, ranges, pay,
                             n, units, per, (int2 *)out, cap, d_count);
}

// The count of an empty input: the host word directly, a device word in stream order.
static qg_status qg_zero_count(qg_ctx *ctx, long long *d_count) {
    if (d_count == (long long *)&ctx->hres->count) ctx->hres->count = 0;
    else QG_TRY_CUDA(ctx, cudaMemsetAsync(d_count, 0, sizeof(long long), ctx->stream), "memset");
    return QG_OK;
}

qg_status qg_filter_rec_launch(qg_ctx *ctx, const void *in, int64_t n, int32_t lo, int32_t hi,
                               void *out, int64_t cap, long long *d_count) {
    if (n == 0) {
        return qg_zero_count(ctx, d_count);
    }
    if (((uintptr_t)in & 15) != 0 || ((uintptr_t)out & 7) != 0) return QG_ERR_INVALID;
    // k_filter_two reads rows again that other CTAs' writes may have reached by then.
    if (qg_overlap(out, (size_t)std::min(cap, n) * 8, in, (size_t)n * 8)) {
        if ((uintptr_t)out <= (uintptr_t)in) {
            const int64_t tiles = qg_ceil_div(n, FT_THREADS * FR_ROUNDS * 2);
            qg_lookback lb;
            QG_TRY(qg_lb_make(ctx, tiles, QG_SITE_FILTER, &lb));
            qg_pre_launch(ctx);
            k_filter_rec<<<(unsigned)tiles, FT_THREADS, 0, ctx->stream>>>((const int4 *)in, n, lo, hi, (int2 *)out, cap,
                                                                         d_count, lb);
            return qg_check_launch(ctx, "k_filter_rec");
        }
        char *tmp;  // the output begins inside the input: filtered from a copy
        QG_TRY(qg_aux(ctx, (size_t)n * 8, &tmp));
        QG_TRY_CUDA(ctx, cudaMemcpyAsync(tmp, in, (size_t)n * 8, cudaMemcpyDeviceToDevice, ctx->stream), "copy");
        in = tmp;
    }
    return f2_launch<true>(ctx, (const int32_t *)in, nullptr, n, lo, hi, out, cap, d_count);
}

static int g_filter_variant = 2;  // two phases: fastest measured at every size

qg_status qg_filter_cols_launch(qg_ctx *ctx, const int32_t *key, const int32_t *pay, int64_t n,
                                int32_t lo, int32_t hi, int32_t *out, int64_t cap,
                                long long *d_count) {
    constexpr int TILE = FT_THREADS * COL_ROUNDS * 4;
    if (n == 0) {
        return qg_zero_count(ctx, d_count);
    }
    if (((uintptr_t)key & 15) || ((uintptr_t)pay & 15) || ((uintptr_t)out & 7))
        return QG_ERR_INVALID;
    int64_t tiles = qg_ceil_div(n, TILE);
    if (tiles > 0x7fffffff || n > 0x7fffffffLL) return QG_ERR_UNSUPPORTED;
    const int variant = qg_effective_variant(ctx, QG_STEER_FILTER, g_filter_variant);
    if (variant == 2) {
        // k_filter_two writes rows while other CTAs still read keys
        const bool over = qg_overlap(out, (size_t)std::min(cap, n) * 8, key, (size_t)n * 4);
        if (over || (n >= F2_TWO_ROWS && f2_two_fits(ctx, n))) {
            const qg_status st = f2_launch_two(ctx, key, pay, n, lo, hi, out, cap, d_count);
            if (st != QG_ERR_OOM || over) return st;  // no room for the bits: nothing was launched
        }
        return f2_launch<false>(ctx, key, pay, n, lo, hi, out, cap, d_count);
    }
    qg_lookback lb;
    QG_TRY(qg_lb_make(ctx, tiles, QG_SITE_FILTER, &lb));
    if (variant == 1) {
        static qg_per_device site;
        QG_TRY(qg_allow_smem(ctx, site, k_filter_cols_tma, sizeof(FpSmem)));
        const long long ftiles = qg_ceil_div(n, FP_TILE);
        const int grid = (int)(ftiles < ctx->sm_count * 2LL ? ftiles : ctx->sm_count * 2LL);
        qg_pre_launch(ctx);
        k_filter_cols_tma<<<grid, FP_THREADS, sizeof(FpSmem), ctx->stream>>>(
            key, pay, n, lo, hi, (int2 *)out, cap, d_count, lb, (uint32_t)ftiles);
        return qg_check_launch(ctx, "k_filter_cols_tma");
    }
    qg_pre_launch(ctx);
    k_filter_cols<COL_ROUNDS><<<(unsigned)tiles, FT_THREADS, 0, ctx->stream>>>(
        key, pay, n, lo, hi, (int2 *)out, cap, d_count, lb);
    return qg_check_launch(ctx, "k_filter_cols");
}

// 0: one tile per CTA, rows staged in registers, decoupled look-back;
// 1: persistent CTAs with a bulk-copy ring; 2: two phases (count, write)
// around one exchange (all bit-identical; chosen by measurement).
int qg_filter_default_variant() { return g_filter_variant; }

extern "C" QG_API qg_status qg_filter_set_variant(int variant) {
    if (variant < 0 || variant > 2) return QG_ERR_INVALID;
    g_filter_variant = variant;
    return QG_OK;
}

extern "C" {

QG_API qg_status qg_filter_range_rec_async(qg_ctx *ctx, const void *in, int64_t n, int32_t lo,
                                           int32_t hi, void *out, int64_t cap, int64_t *d_out_n) {
    if (!ctx || n < 0 || cap < 0 || !d_out_n || (n > 0 && (!in || !out))) return QG_ERR_INVALID;
    if (n >= (1LL << 32)) return QG_ERR_UNSUPPORTED;
    return qg_filter_rec_launch(ctx, in, n, lo, hi, out, cap, (long long *)d_out_n);
}

QG_API qg_status qg_filter_range_rec(qg_ctx *ctx, const void *in, int64_t n, int32_t lo,
                                     int32_t hi, void *out, int64_t cap, int64_t *out_n) {
    if (!ctx || !out_n) return QG_ERR_INVALID;
    long long *d_count = (long long *)&ctx->hres->count;  // the kernel stores the count in host memory
    QG_TRY(qg_filter_range_rec_async(ctx, in, n, lo, hi, out, cap, (int64_t *)d_count));
    return finish_count(ctx, cap, out_n);
}

QG_API qg_status qg_filter_cols_async(qg_ctx *ctx, const int32_t *key, const int32_t *pay,
                                      int64_t n, int32_t lo, int32_t hi, int32_t *out, int64_t cap,
                                      int64_t *d_out_n) {
    if (!ctx || n < 0 || cap < 0 || !d_out_n || (n > 0 && (!key || !pay || !out)))
        return QG_ERR_INVALID;
    return qg_filter_cols_launch(ctx, key, pay, n, lo, hi, out, cap, (long long *)d_out_n);
}

QG_API qg_status qg_filter_cols(qg_ctx *ctx, const int32_t *key, const int32_t *pay, int64_t n,
                                int32_t lo, int32_t hi, int32_t *out, int64_t cap,
                                int64_t *out_n) {
    if (!ctx || !out_n) return QG_ERR_INVALID;
    // With a cost model attached the variant is its choice for this size; the
    // selectivity estimate is the predicate's share of the int32 range.
    qg_steer_call sc;
    qg_steer_begin(ctx, QG_STEER_FILTER, n, 0, ((double)hi - (double)lo + 1.0) / 4294967296.0, &sc);
    long long *d_count = (long long *)&ctx->hres->count;  // the kernel stores the count in host memory
    qg_status st = qg_filter_cols_async(ctx, key, pay, n, lo, hi, out, cap, (int64_t *)d_count);
    if (st == QG_OK) st = finish_count(ctx, cap, out_n);
    qg_steer_end(ctx, &sc, st);
    return st;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Column filter that allocates nothing.
//
// For callers that cannot allocate device memory themselves -- code running
// inside an allocator or memory-pool callback, in a process whose device
// memory is carved up by a framework that forbids extra cudaMalloc calls, or
// on a path that must never block on the allocator -- and so cannot create a
// qg_ctx (qg_ctx_create allocates its control block and scratch).  The
// look-back status words and the control block this kernel needs live in the
// file-scope device array below instead, sized for at most
// QG_NOALLOC_MAX_ROWS rows; every GPU that loads the library holds it
// (about 128 KB) until the process exits.
//
// Host code only sees a stand-in for the array, not its device address, so
// the first call on a device (with that device current) looks the address up
// with cudaGetSymbolAddress and keeps it; make that first call before any
// stream capture.  Every call shares the one array: the counters and the
// status words the call uses are cleared at the start of each call (stream
// ordered), and calls that overlap on the GPU (on different streams, or from
// different threads without ordering) race on it.
// ---------------------------------------------------------------------------
#define QG_NOALLOC_MAX_ROWS (1LL << 26)
#define QG_NOALLOC_TILE (FT_THREADS * COL_ROUNDS * 4)
#define QG_NOALLOC_MAX_TILES ((QG_NOALLOC_MAX_ROWS + QG_NOALLOC_TILE - 1) / QG_NOALLOC_TILE)
#define QG_NOALLOC_MAX_DEVICES 64

struct qg_noalloc_scratch {
    qg_control ctl;
    unsigned long long status[QG_NOALLOC_MAX_TILES];
};
static_assert((long long)QG_NOALLOC_MAX_TILES * QG_NOALLOC_TILE >= QG_NOALLOC_MAX_ROWS,
              "no-alloc status words cover the largest accepted input");

static __device__ __align__(256) qg_noalloc_scratch g_noalloc_scratch;

// Device address of g_noalloc_scratch per device, looked up by the first call
// on that device.  A cudaDeviceReset (or any teardown of the device's primary
// context) makes the remembered address stale; qg_noalloc_forget() drops it.
static qg_noalloc_scratch *g_noalloc_addr[QG_NOALLOC_MAX_DEVICES];
// Polls a look-back wait of the no-alloc filter makes before it gives up.
static uint32_t g_noalloc_spin = 1u << 22;

extern "C" QG_API qg_status qg_noalloc_set_spin_limit(uint32_t polls) {
    g_noalloc_spin = polls;
    return QG_OK;
}

extern "C" QG_API qg_status qg_noalloc_forget(void) {
    for (int i = 0; i < QG_NOALLOC_MAX_DEVICES; i++) g_noalloc_addr[i] = nullptr;
    return QG_OK;
}

// Reports a device-side error of the call through the count (as -code) and
// clears the error word for the next call.
__global__ void k_noalloc_report(qg_noalloc_scratch *s, long long *d_count) {
    const int e = s->ctl.err;
    if (e) {
        *d_count = -(long long)e;
        s->ctl.err = 0;
        s->ctl.err_site = 0;
    }
}

extern "C" QG_API qg_status qg_filter_cols_noalloc(const int32_t *key, const int32_t *pay, int64_t n,
                                                   int32_t lo, int32_t hi, int32_t *out,
                                                   int64_t cap, int64_t *d_out_n, void *stream) {
    constexpr int TILE = QG_NOALLOC_TILE;
    if (n < 0 || cap < 0 || !d_out_n || (n > 0 && (!key || !pay || !out))) return QG_ERR_INVALID;
    if (n > QG_NOALLOC_MAX_ROWS || (n + TILE - 1) / TILE > QG_NOALLOC_MAX_TILES) return QG_ERR_UNSUPPORTED;
    if (((uintptr_t)key & 15) || ((uintptr_t)pay & 15) || ((uintptr_t)out & 7) ||
        ((uintptr_t)d_out_n & 7))
        return QG_ERR_INVALID;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= QG_NOALLOC_MAX_DEVICES) {
        cudaGetLastError();
        return QG_ERR_CUDA;
    }
    if (!g_noalloc_addr[dev]) {  // set-up, once per device
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) {
            cudaGetLastError();
            return QG_ERR_CUDA;
        }
        g_noalloc_addr[dev] = (qg_noalloc_scratch *)p;
    }
    qg_noalloc_scratch *s = g_noalloc_addr[dev];
    cudaStream_t st = (cudaStream_t)stream;
    if (n == 0)
        return cudaMemsetAsync(d_out_n, 0, sizeof(long long), st) == cudaSuccess ? QG_OK : QG_ERR_CUDA;
    const long long tiles = (n + TILE - 1) / TILE;
    // Counters and error word start at zero; status words of this call's
    // tiles are cleared so nothing from an earlier call can be read as ready.
    if (cudaMemsetAsync(&s->ctl, 0, sizeof(qg_control), st) != cudaSuccess ||
        cudaMemsetAsync(s->status, 0, (size_t)tiles * sizeof(unsigned long long), st) != cudaSuccess) {
        cudaGetLastError();
        return QG_ERR_CUDA;
    }
    qg_lookback lb{s->status, &s->ctl, g_noalloc_spin, QG_SITE_FILTER};
    k_filter_cols<COL_ROUNDS><<<(unsigned)tiles, FT_THREADS, 0, st>>>(
        key, pay, n, lo, hi, (int2 *)out, cap, (long long *)d_out_n, lb);
    k_noalloc_report<<<1, 1, 0, st>>>(s, (long long *)d_out_n);
    if (cudaGetLastError() != cudaSuccess) return QG_ERR_CUDA;
    return QG_OK;
}
