// qg_gbsmall.cu -- column group-by (int64 SUM + COUNT per key, optionally only
// rows with lo2 <= val2 <= hi2) of a small input in one CTA and one launch.
//
// The reference chain this answers for: sort -> label -> scan -> write ->
// parallelAggregate (kernel/aggregation/1/group_by_cu_op_dp.cl:89-716).
//
// A few thousand rows cost the dense-window path (qg_gbdense.cu) four dependent
// launches of 6 to 12 us each, all latency.  Here the rows are aggregated in a
// hash table in shared memory, whatever their keys' range, and the distinct
// keys are sorted there.  A table that fills up (more distinct keys than it
// takes) is reported and the caller takes the general paths.
//
// A 10K-row call in 500 groups 57 -> 40 us, hashed ids (keys of no window) 150
// -> 40.  One SM adds 2K to 4K rows a microsecond: at 16K rows a call takes 41
// (64 groups) to 54 us (4096), the dense-window path's three launches 41 whatever
// the groups and hashed ids 51 on theirs, so larger inputs go there.
#include <algorithm>
#include "qg_cta_sort.cuh"
#include "qg_internal.cuh"
#include "qg_keytable.cuh"

namespace {

constexpr int GS_THREADS = 1024;
constexpr int GS_WARPS = GS_THREADS / 32;
constexpr int GS_SLOTS = 8192;      // at most; a power of two
static_assert(GS_THREADS == QG_CS_THREADS && GS_SLOTS <= QG_CS_MAX, "the distinct keys are sorted by qg_cta_sort");
constexpr uint32_t GS_PROBES = 32;  // slots looked at before the table counts as full
// Distinct keys among the first 4096 rows, and among the rows of any later
// round, above which the table is given up: it is likely to fill, and the
// general paths should not wait for that.
constexpr uint32_t GS_FIRST_MOST = 3000, GS_MOST = 5000;

// A sum is kept as two 32-bit words: the values' low halves and (signed) high
// halves, each exact for up to GS_MAX_ROWS rows, so an add needs no carry.
struct GsSlot {
    uint32_t *key, *cnt, *lo, *hi;
};

template <bool PRED>
__global__ void __launch_bounds__(GS_THREADS, 1)
k_gb_small(const int32_t *__restrict__ key, const int32_t *__restrict__ val, const int32_t *__restrict__ val2,
           int32_t lo2, int32_t hi2, int n, uint32_t slots, int32_t *__restrict__ gkey, long long *__restrict__ gsum,
           long long *__restrict__ gcnt, long long cap, volatile long long *d_num, volatile uint32_t *full) {
    // with more slots than rows a row always finds its slot
    const uint32_t probes = (uint32_t)n < slots ? slots : GS_PROBES;
    extern __shared__ __align__(16) unsigned char gs_raw[];
    __shared__ uint32_t s_full, s_n;  // s_n: distinct keys of the whole rounds, then of the table
    unsigned long long *ord = reinterpret_cast<unsigned long long *>(gs_raw);  // [slots] key << 32 | slot
    const uint32_t pitch = slots + 4;  // entry `slots`: key 0xffffffff, the free mark
    const GsSlot T{reinterpret_cast<uint32_t *>(ord + slots), reinterpret_cast<uint32_t *>(ord + slots) + pitch,
                   reinterpret_cast<uint32_t *>(ord + slots) + 2 * pitch,
                   reinterpret_cast<uint32_t *>(ord + slots) + 3 * pitch};
    uint32_t(*whist)[256] = reinterpret_cast<uint32_t(*)[256]>(T.hi + pitch);  // [GS_WARPS] the sort's counters
    const int tid = threadIdx.x, lane = tid & 31;
    // the first vectors in flight while the table is cleared
    const int nv = n >> 2;
    const int4 *k4 = reinterpret_cast<const int4 *>(key), *v4 = reinterpret_cast<const int4 *>(val),
               *w4 = reinterpret_cast<const int4 *>(val2);
    int4 kn = make_int4(0, 0, 0, 0), vn = kn, wn = kn;
    if (tid < nv) {
        kn = k4[tid];
        vn = v4[tid];
        if (PRED) wn = w4[tid];
    }
    uint4 *kz = reinterpret_cast<uint4 *>(T.key), *cz = reinterpret_cast<uint4 *>(T.cnt);
    for (uint32_t i = tid; i < pitch / 4; i += GS_THREADS) kz[i] = make_uint4(QG_KT_FREE, QG_KT_FREE, QG_KT_FREE, QG_KT_FREE);
    for (uint32_t i = tid; i < 3 * (pitch / 4); i += GS_THREADS) cz[i] = make_uint4(0, 0, 0, 0);
    if (tid == 0) s_full = s_n = 0;
    __syncthreads();
    const uint32_t mask = slots - 1;
    uint32_t fresh = 0;  // keys this thread was the first to see
    auto add = [&](uint32_t h, int32_t v) {
        atomicAdd(&T.cnt[h], 1u);
        atomicAdd(&T.lo[h], (uint32_t)v & 0xffffu);
        const int32_t up = v >> 16;
        if (up) atomicAdd(&T.hi[h], (uint32_t)up);
    };
    for (int q = tid; q < nv; q += GS_THREADS) {
        const int4 kk = kn, vv = vn, ww = wn;
        if (q + GS_THREADS < nv) {
            kn = k4[q + GS_THREADS];
            vn = v4[q + GS_THREADS];
            if (PRED) wn = w4[q + GS_THREADS];
        }
        const int32_t vs[4] = {vv.x, vv.y, vv.z, vv.w}, ws[4] = {ww.x, ww.y, ww.z, ww.w};
        const uint32_t ks[4] = {(uint32_t)kk.x, (uint32_t)kk.y, (uint32_t)kk.z, (uint32_t)kk.w};
        uint32_t h[4], live = 0;
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (!PRED || ((ws[j] >= lo2) & (ws[j] <= hi2))) live |= 1u << j;
        if (qg_kt_find<4>(T.key, mask, ks, live, h, probes, fresh)) {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if ((live >> j) & 1u) add(h[j], vs[j]);
        } else {
            s_full = 1;
        }
        if (q - tid + 2 * GS_THREADS <= nv) {  // every thread has this round and the next
            const uint32_t f = __reduce_add_sync(QG_FULL_MASK, fresh);
            if (lane == 0 && f) atomicAdd(&s_n, f);
            fresh = 0;
            __syncthreads();
            // (no thread writes either word between the two barriers)
            const bool stop = s_full || s_n > (q < GS_THREADS ? GS_FIRST_MOST : GS_MOST);
            if (__syncthreads_or(stop)) {  // all threads leave, or none
                s_full = 1;
                break;
            }
        }
    }
    if (tid < (n & 3)) {
        const int i = nv * 4 + tid;
        if (!PRED || ((val2[i] >= lo2) & (val2[i] <= hi2))) {
            const uint32_t k[1] = {(uint32_t)key[i]};
            uint32_t h[1];
            if (qg_kt_find<1>(T.key, mask, k, 1u, h, probes, fresh)) add(h[0], val[i]);
            else s_full = 1;
        }
    }
    __syncthreads();
    if (s_full) {
        if (tid == 0 && full) *full = 1;
        return;
    }
    __syncthreads();
    if (tid == 0) s_n = 0;
    __syncthreads();
    for (uint32_t i = tid; i < slots; i += GS_THREADS) {  // whole warps: slots >= 1024
        const bool used = T.cnt[i] != 0;
        const uint32_t m = __ballot_sync(QG_FULL_MASK, used);
        uint32_t at = 0;
        if (lane == 0 && m) at = atomicAdd(&s_n, (uint32_t)__popc(m));
        at = __shfl_sync(QG_FULL_MASK, at, 0);
        if (used) ord[at + __popc(m & qg_lanemask_lt())] = (unsigned long long)T.key[i] << 32 | i;
    }
    __syncthreads();
    const uint32_t g = s_n, top = T.cnt[slots] ? 1u : 0u;  // key 0xffffffff comes last
    qg_cta_sort(ord, whist, g);
    for (uint32_t r = tid; r < g + top && r < cap; r += GS_THREADS) {
        const uint32_t i = r < g ? (uint32_t)ord[r] : slots;
        gkey[r] = r < g ? (int32_t)(ord[r] >> 32) : -1;
        gsum[r] = (long long)T.lo[i] + ((long long)(int32_t)T.hi[i] << 16);
        gcnt[r] = T.cnt[i];
    }
    if (tid == 0) {
        *d_num = g + top;
        if (full) *full = 0;
    }
}

}  // namespace

// Launches the small form (1 <= n <= QG_GBS_MAX_ROWS) on the context's stream;
// after the stream is synchronised *full tells whether the table filled up
// (nothing valid was written; never below QG_GBS_SURE_ROWS rows, where full may
// be null), else *d_num holds the group count.
qg_status qg_gbs_launch(qg_ctx *ctx, const int32_t *key, const int32_t *val, const int32_t *val2, int32_t lo2,
                        int32_t hi2, int64_t n, int32_t *gkey, int64_t *gsum, int64_t *gcnt, int64_t cap,
                        volatile long long *d_num, volatile uint32_t *full) {
    static_assert(QG_GBS_MAX_ROWS <= 65536, "the sums' words");
    static_assert(QG_GBS_SURE_ROWS <= GS_SLOTS, "more slots than rows, and no checked round");
    uint32_t slots = 1024;
    while (slots < GS_SLOTS && slots < 2 * (uint32_t)n) slots <<= 1;
    auto bytes = [](uint32_t s) { return (size_t)s * 8 + 4 * (s + 4) * 4 + (size_t)GS_WARPS * 1024; };
    const size_t most = bytes(GS_SLOTS), smem = bytes(slots);
    static qg_per_device site[2];
    const bool pred = val2 != nullptr;
    auto kern = pred ? k_gb_small<true> : k_gb_small<false>;
    QG_TRY(qg_allow_smem(ctx, site[pred], kern, most));
    qg_pre_launch(ctx);
    kern<<<1, GS_THREADS, smem, ctx->stream>>>(key, val, val2, lo2, hi2, (int)n, slots, gkey, (long long *)gsum,
                                               (long long *)gcnt, cap, d_num, full);
    return qg_check_launch(ctx, "k_gb_small");
}
