// qg_join.cu -- hash join + filter + sort.
//
// Reference (kernel/hj_filter_sort/1/hj_filter_sort_op.cl):
//   buildHashTable (:25-60)  one 128-item work-group appends (key, val) into
//                            bucket key & (B-1) under a local spin lock,
//   probeHashTable (:62-109) scans every slot of the bucket and writes each
//                            match (S.val, R.val) into a per-work-item region,
//   then the filter (:117-349) and bitonic sort (:362-564) of the matches.
// The reference ships no host for this chain; the contract here is the one
// the operator list implies, with config 2's filter on S.payload applied
// before the join.
//
// GB300 design:
//   build  -- grid-wide open-addressing table of 64-bit slots
//             (key << 32 | payload) filled with atomicCAS; duplicate build
//             keys each take their own slot, so every match is found.  The
//             build also records min/max key for the sort and whether any
//             key occurs twice.
//   probe  -- persistent CTAs over tiles of S: the rows that pass the filter
//             are compacted in shared memory, look the table up by 32-byte
//             groups of slots, and the matches are collected per warp.  The
//             probe also counts the sort digits of its output.
//   sort   -- LSD radix passes over (key - min_key) on the three output
//             columns (qg_sort.cu), the last one into the caller's output; a
//             few thousand matches are sorted by one CTA.
#include <math.h>
#include <string.h>
#include <vector>
#include "qg_cta_sort.cuh"
#include "qg_internal.cuh"
#include "qg_join.cuh"
#include "qg_sort.cuh"

namespace {

constexpr unsigned long long EMPTY_SLOT = ~0ull;

struct JoinCtl {
    uint32_t kmin, kmax;
    unsigned long long n_special;  // build rows equal to EMPTY_SLOT (key -1, payload -1)
    unsigned long long cursor;     // output rows produced
    unsigned long long sortn;      // rows the device-planned sort orders (0 when over capacity)
    uint32_t crowded;              // 1: build keys repeat more than they may
    uint32_t twice;                // not 0: some build key occurs more than once
    qg_sort_range range;           // the device-planned sort's positions and key offset
    uint32_t hist[4][QG_RADIX];
};

// Reference-layout hash table (qg_hash_build_ref / qg_hash_probe_ref): this
// header, padded to 256 bytes, then `slots` 8-byte slots (key << 32 | value,
// EMPTY_SLOT = free).
struct RefHashHdr {
    JoinCtl jc;      // key range and the count of build rows equal to EMPTY_SLOT
    uint32_t slots;  // a power of two
    uint32_t magic;
};
constexpr uint32_t REF_HASH_MAGIC = 0x71684a31u;
constexpr size_t REF_HASH_HDR = (sizeof(RefHashHdr) + 255) / 256 * 256;

// A key's first slot: the table is walked from the start of a 32-byte group of
// four slots, so that one L2 sector answers most lookups (at load 1/2 one group
// in twenty overflows; walking slot by slot from a hashed slot, the slowest of a
// warp's lanes took ten dependent loads).
__device__ __forceinline__ uint32_t join_group(uint32_t k, uint32_t mask) { return qg_hash32(k) & mask & ~3u; }

__global__ void k_join_ctl_init(JoinCtl *jc) {
    qg_chain();
    int t = threadIdx.x;
    if (t == 0) {
        jc->kmin = 0xffffffffu;
        jc->kmax = 0;
        jc->n_special = 0;
        jc->cursor = 0;
        jc->sortn = 0;
        jc->crowded = 0;
        jc->twice = 0;
    }
    for (int i = t; i < 4 * QG_RADIX; i += blockDim.x) (&jc->hist[0][0])[i] = 0;
}

// Build: rows i of R at rkey[i * stride], rpay[i * stride].  LIMIT: the build is given
// up when its keys repeat more than the probe can bear, as far as a CTA sees: the squares
// of how many rows of its own key each row meets add up to more than `most`, a row has
// looked at JB_PROBES slots or met JB_SAME by itself, JB_SAME rows equal the free slots'
// mark.
// A CTA stops at what it has seen itself: one word that all of them add to or look at is
// a queue in L2 (0.3 % of 4M rows in pairs: 320 -> 540 us a call).
// Eight CTAs per SM: with six a build of 8M rows takes 50 us longer.
constexpr uint32_t JB_PROBES = 256;  // unique keys at load 1/2 need a few dozen
constexpr uint32_t JB_SAME = 16;
constexpr int JB_CTAS = 8;

template <bool LIMIT>
__global__ void __launch_bounds__(256, JB_CTAS)
k_join_build(const int32_t *__restrict__ rkey, const int32_t *__restrict__ rpay, uint32_t stride_el,
             uint32_t nR, unsigned long long *__restrict__ tab, uint32_t mask, JoinCtl *jc,
             qg_control *ctl, uint32_t most) {
    qg_chain();
    __shared__ uint32_t s_met;
    if (LIMIT) {
        if (threadIdx.x == 0) s_met = 0;
        __syncthreads();
    }
    uint32_t lmin = 0xffffffffu, lmax = 0, nspec = 0;
    bool twice = false;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nR; i += stride) {  // nR < 2^30
        if (LIMIT && *(volatile uint32_t *)&s_met > most) break;
        const uint32_t k = (uint32_t)__ldg(rkey + (size_t)i * stride_el);
        const uint32_t p = (uint32_t)__ldg(rpay + (size_t)i * stride_el);
        lmin = min(lmin, k);
        lmax = max(lmax, k);
        const unsigned long long packed = ((unsigned long long)k << 32) | p;
        if (packed == EMPTY_SLOT) { nspec++; continue; }
        uint32_t g = join_group(k, mask), probes = 0, same = 0;
        bool placed = false, over = false;
        while (!placed) {
            const ulonglong2 lo = __ldcg(reinterpret_cast<const ulonglong2 *>(tab + g)),
                             hi = __ldcg(reinterpret_cast<const ulonglong2 *>(tab + g + 2));
            const unsigned long long seen[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (placed) break;
                unsigned long long old = seen[j];
                if (old == EMPTY_SLOT) old = atomicCAS(&tab[g + j], EMPTY_SLOT, packed);
                // an equal key inserted before lies on this row's way to its slot
                if (old == EMPTY_SLOT) placed = true;
                else if ((uint32_t)(old >> 32) == k) same++;
            }
            if (placed) break;
            g = (g + 4) & mask;
            probes += 4;
            if (LIMIT && (probes > JB_PROBES || same > JB_SAME)) {
                over = true;
                break;
            }
            if (probes > mask) { qg_record_error(ctl, QG_ERR_TABLE_FULL, QG_SITE_JOIN_BUILD); break; }
        }
        if (same || over) {
            twice = true;
            if (LIMIT) atomicAdd(&s_met, over ? most + 1 : same * same);
        }
    }
    __syncwarp();
    lmin = __reduce_min_sync(QG_FULL_MASK, lmin);
    lmax = __reduce_max_sync(QG_FULL_MASK, lmax);
    if ((threadIdx.x & 31) == 0) {
        if (lmin != 0xffffffffu) atomicMin(&jc->kmin, lmin);
        if (lmax != 0) atomicMax(&jc->kmax, lmax);
    }
    if (twice) {
        jc->twice = 1;
        if (LIMIT && *(volatile uint32_t *)&s_met > most) jc->crowded = 1;
    }
    if (nspec && atomicAdd(&jc->n_special, (unsigned long long)nspec) + nspec > JB_SAME && LIMIT) jc->crowded = 1;
}

constexpr int PJ_THREADS = 256;
constexpr int PJ_WARPS = PJ_THREADS / 32;
constexpr int PJ_ROUNDS = 4;                         // int4 of keys + int4 of payloads per round and thread
constexpr int PJ_TILE = PJ_THREADS * PJ_ROUNDS * 4;  // 4096 S rows per tile
constexpr int PJ_STAGE = 128;  // matches a warp collects before it writes them

struct PjSmem {
    unsigned long long row[PJ_TILE];                // the tile's rows that pass the filter
    uint32_t ok[PJ_WARPS][PJ_STAGE], oa[PJ_WARPS][PJ_STAGE], ob[PJ_WARPS][PJ_STAGE];
    uint32_t hist[4][QG_RADIX];
    uint32_t cnt[2];  // rows of this tile, and the next one's counter
};

struct ProbeOut {
    uint32_t *k, *a, *b;
};

// Probe.  Persistent CTAs over tiles of 4096 S rows.  A tile's rows that pass the filter (and lie in R's key range) are
// compacted first, so that every lane of every lookup step has a row; matches are collected per warp and
// written 96 or more at a time, one reservation each.  When no build key occurs
// twice a row reads its slots by groups and stops at its match, two rows of a
// thread together; else every row walks to the end of its slots.  Looking rows up
// where they lay and emitting step by step left two thirds of the lanes idle
// behind votes, one row's slots at a time: 16M rows on a 1M-row table 494 us,
// 115 now; 190 with the slots walked one by one.
// The sort digits of key - (R's smallest key) are counted (npos positions).
// odd: where the matches go instead when that key range has an odd number of
// digits (unless null).
__global__ void __launch_bounds__(PJ_THREADS, 4)
k_join_probe(const int32_t *__restrict__ skey, const int32_t *__restrict__ spay, long long nS,
             int32_t slo, int32_t shi, const unsigned long long *__restrict__ tab, uint32_t mask,
             JoinCtl *jc, ProbeOut out, ProbeOut odd, long long cap, int npos, unsigned long long least) {
    qg_chain();
    extern __shared__ __align__(16) unsigned char pj_raw[];
    PjSmem &S = *reinterpret_cast<PjSmem *>(pj_raw);
    if (jc->crowded || (unsigned long long)(jc->kmax - jc->kmin) < least) return;  // the caller has another path
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t lt = qg_lanemask_lt();
    const long long ntiles = (nS + PJ_TILE - 1) / PJ_TILE;
    const unsigned long long nspec = jc->n_special;
    const uint32_t kmin = jc->kmin, kspan = jc->kmax - kmin;  // rows outside cannot match
    const uint32_t key_off = kmin;
    // a sort of an odd number of positions starts from the other columns
    if (odd.k && (qg_sort_npos(kmin, jc->kmax) & 1u)) out = odd;
    const bool once = jc->twice == 0 && nspec == 0;
    for (int i = tid; i < 4 * QG_RADIX; i += PJ_THREADS) (&S.hist[0][0])[i] = 0;
    if (tid < 2) S.cnt[tid] = 0;
    __syncthreads();
    uint32_t have = 0;  // matches in the warp's collection (warp-uniform)
    auto flush = [&]() {
        __syncwarp();
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(&jc->cursor, (unsigned long long)have);
        base = __shfl_sync(QG_FULL_MASK, base, 0);
        for (uint32_t q = lane; q < have; q += 32) {
            const uint32_t k = S.ok[warp][q];
            const long long g = (long long)base + q;
            if (g < cap) {
                out.k[g] = k;
                out.a[g] = S.oa[warp][q];
                out.b[g] = S.ob[warp][q];
            }
            const uint32_t kk = k - key_off;
            for (int p = 0; p < npos; p++) atomicAdd(&S.hist[p][(kk >> (8 * p)) & 255u], 1u);
        }
        __syncwarp();
        have = 0;
    };
    auto emit = [&](bool hit, uint32_t k, uint32_t a, uint32_t b) {  // all lanes
        const uint32_t bal = __ballot_sync(QG_FULL_MASK, hit);
        if (!bal) return;
        if (hit) {
            const uint32_t pos = have + __popc(bal & lt);
            S.ok[warp][pos] = k;
            S.oa[warp][pos] = a;
            S.ob[warp][pos] = b;
        }
        have += __popc(bal);
        if (have > PJ_STAGE - 32) flush();
    };
    int it = 0;
    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x, it ^= 1) {
        const long long gbase = t * PJ_TILE;
        int4 kv[PJ_ROUNDS], pv[PJ_ROUNDS];
#pragma unroll
        for (int r = 0; r < PJ_ROUNDS; r++) {
            const long long idx = gbase + (long long)(r * PJ_THREADS + tid) * 4;
            if (idx + 3 < nS) {
                kv[r] = qg_ldg_stream(reinterpret_cast<const int4 *>(skey + idx));
                pv[r] = qg_ldg_stream(reinterpret_cast<const int4 *>(spay + idx));
            } else {
                int tk[4] = {0, 0, 0, 0}, tp[4] = {0, 0, 0, 0};
                for (int j = 0; j < 4; j++)
                    if (idx + j < nS) { tk[j] = skey[idx + j]; tp[j] = spay[idx + j]; }
                kv[r] = make_int4(tk[0], tk[1], tk[2], tk[3]);
                pv[r] = make_int4(tp[0], tp[1], tp[2], tp[3]);
            }
        }
        uint32_t tot = 0, fl = 0;
        uint32_t at[PJ_ROUNDS];
#pragma unroll
        for (int r = 0; r < PJ_ROUNDS; r++) {
            const long long idx = gbase + (long long)(r * PJ_THREADS + tid) * 4;
            const int32_t kk[4] = {kv[r].x, kv[r].y, kv[r].z, kv[r].w}, pp[4] = {pv[r].x, pv[r].y, pv[r].z, pv[r].w};
            at[r] = tot;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const bool f = (idx + j < nS) & (pp[j] >= slo) & (pp[j] <= shi) & ((uint32_t)kk[j] - kmin <= kspan);
                const uint32_t b = __ballot_sync(QG_FULL_MASK, f);
                at[r] += __popc(b & lt);
                tot += __popc(b);
                fl |= (uint32_t)f << (4 * r + j);
            }
        }
        uint32_t base = 0;
        if (lane == 0 && tot) base = atomicAdd(&S.cnt[it], tot);
        base = __shfl_sync(QG_FULL_MASK, base, 0);
#pragma unroll
        for (int r = 0; r < PJ_ROUNDS; r++) {
            uint32_t pos = base + at[r];
            const int32_t kk[4] = {kv[r].x, kv[r].y, kv[r].z, kv[r].w}, pp[4] = {pv[r].x, pv[r].y, pv[r].z, pv[r].w};
#pragma unroll
            for (int j = 0; j < 4; j++)
                if ((fl >> (4 * r + j)) & 1u) S.row[pos++] = (unsigned long long)(uint32_t)kk[j] << 32 | (uint32_t)pp[j];
        }
        __syncthreads();
        const uint32_t n = S.cnt[it];
        if (tid == 0) S.cnt[it ^ 1] = 0;  // read by the last tile, added to after the next barrier
        if (once) {
            constexpr int U = 2;
            for (uint32_t i0 = warp * 32; i0 < n; i0 += U * PJ_THREADS) {  // whole warps
                uint32_t k[U], p[U], g[U], pay[U], go = 0, hit = 0;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const uint32_t i = i0 + u * PJ_THREADS + lane;
                    const unsigned long long v = i < n ? S.row[i] : 0ull;
                    k[u] = (uint32_t)(v >> 32);
                    p[u] = (uint32_t)v;
                    g[u] = join_group(k[u], mask);
                    pay[u] = 0;
                    go |= (uint32_t)(i < n) << u;
                }
                for (uint32_t probes = 0; go && probes <= mask; probes += 4) {
                    ulonglong2 lo[U], hi[U];
#pragma unroll
                    for (int u = 0; u < U; u++)
                        if ((go >> u) & 1u) {
                            lo[u] = __ldg(reinterpret_cast<const ulonglong2 *>(tab + g[u]));
                            hi[u] = __ldg(reinterpret_cast<const ulonglong2 *>(tab + g[u] + 2));
                        }
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        if (!((go >> u) & 1u)) continue;
                        const unsigned long long sl[4] = {lo[u].x, lo[u].y, hi[u].x, hi[u].y};
                        bool end = false;
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            // (a key of all ones never matches a free slot's: those rows take the other form)
                            if ((uint32_t)(sl[j] >> 32) == k[u] && sl[j] != EMPTY_SLOT) {
                                hit |= 1u << u;
                                pay[u] = (uint32_t)sl[j];
                                end = true;
                            }
                            end |= sl[j] == EMPTY_SLOT;
                        }
                        if (end) go &= ~(1u << u);
                        g[u] = (g[u] + 4) & mask;
                    }
                }
                __syncwarp();
#pragma unroll
                for (int u = 0; u < U; u++) emit((hit >> u) & 1u, k[u], pay[u], p[u]);
            }
        } else {
            for (uint32_t i0 = warp * 32; i0 < n; i0 += PJ_THREADS) {  // whole warps
                const uint32_t i = i0 + lane;
                const unsigned long long v = i < n ? S.row[i] : 0ull;
                const uint32_t k = (uint32_t)(v >> 32), p = (uint32_t)v;
                // Build rows equal to the empty-slot pattern (key -1, payload -1)
                // are counted, not stored; a probe key of -1 matches each of them.
                unsigned long long spec = i < n && k == 0xffffffffu ? nspec : 0ull;
                while (__any_sync(QG_FULL_MASK, spec != 0)) {
                    emit(spec != 0, k, 0xffffffffu, p);
                    if (spec) spec--;
                }
                uint32_t h = join_group(k, mask), probes = 0;
                unsigned long long sl = i < n ? __ldg(&tab[h]) : EMPTY_SLOT;
                bool a = sl != EMPTY_SLOT;
                while (__any_sync(QG_FULL_MASK, a)) {
                    const unsigned long long cur = sl;
                    const bool hit = a && (uint32_t)(cur >> 32) == k;
                    if (a) {
                        h = (h + 1) & mask;
                        sl = __ldg(&tab[h]);
                        if (sl == EMPTY_SLOT || ++probes > mask) a = false;
                    }
                    emit(hit, k, (uint32_t)cur, p);
                }
            }
        }
        __syncthreads();  // the rows are rewritten by the next tile
    }
    if (have) flush();
    __syncthreads();
    for (int i = tid; i < npos * QG_RADIX; i += PJ_THREADS) {
        uint32_t c = (&S.hist[0][0])[i];
        if (c) atomicAdd(&(&jc->hist[0][0])[i], c);
    }
}

// Reference-layout probe: interleaved (key, val) S pairs, output (S.val, R.val).  A step
// reads a group of four slots, one 32-byte sector, and reserves the places of all its
// matches at once.  8M rows on a table of 1M, all matching: 373 us a call; slot by slot
// 896, and 771 while rows did not start at a group's first slot.
__global__ void __launch_bounds__(256)
k_join_probe_ref(const uint32_t *__restrict__ s, long long nS, const unsigned long long *__restrict__ tab,
                 const RefHashHdr *__restrict__ hdr, unsigned long long *__restrict__ cursor,
                 uint32_t *__restrict__ out, long long cap) {
    const int lane = threadIdx.x & 31;
    const uint32_t lt = qg_lanemask_lt();
    const unsigned long long nspec = hdr->jc.n_special;
    const uint32_t mask = hdr->slots - 1;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long iters = (nS + stride - 1) / stride;
    for (long long it = 0; it < iters; it++) {
        const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x + it * stride;
        bool act = i < nS;
        uint32_t k = 0, v = 0;
        if (act) {
            uint2 kv = *reinterpret_cast<const uint2 *>(s + 2 * i);
            k = kv.x;
            v = kv.y;
        }
        uint32_t g = join_group(k, mask), probes = 0;
        unsigned long long spec_left = (act && k == 0xffffffffu) ? nspec : 0;
        while (__any_sync(QG_FULL_MASK, act || spec_left)) {
            uint32_t hits = 0;                      // slots of the group that match
            uint32_t rv[4] = {~0u, ~0u, ~0u, ~0u};  // (the mark's payload)
            if (spec_left) {
                hits = 1;
                spec_left--;
            } else if (act) {
                const ulonglong2 lo = __ldg(reinterpret_cast<const ulonglong2 *>(tab + g)),
                                 hi = __ldg(reinterpret_cast<const ulonglong2 *>(tab + g + 2));
                const unsigned long long sl[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if (sl[j] == EMPTY_SLOT) act = false;  // (slots fill in order: none is taken after a free one)
                    else if ((uint32_t)(sl[j] >> 32) == k) hits |= 1u << j;
                    rv[j] = (uint32_t)sl[j];
                }
                g = (g + 4) & mask;
                probes += 4;
                if (probes > mask) act = false;
            }
            uint32_t b[4], total = 0, pos = 0;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                b[j] = __ballot_sync(QG_FULL_MASK, (hits >> j) & 1u);
                total += __popc(b[j]);
                pos += __popc(b[j] & lt);
            }
            if (total == 0) continue;
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(cursor, (unsigned long long)total);
            base = __shfl_sync(QG_FULL_MASK, base, 0) + pos;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (!((hits >> j) & 1u)) continue;
                if ((long long)base < cap) *reinterpret_cast<uint2 *>(out + 2 * base) = make_uint2(v, rv[j]);
                base++;
            }
        }
    }
}

}  // namespace

static int grid_cap(qg_ctx *ctx, long long work, int per_block, int per_sm) {
    long long b = (work + per_block - 1) / per_block;
    long long c = (long long)ctx->sm_count * per_sm;
    if (b > c) b = c;
    if (b < 1) b = 1;
    return (int)b;
}

static int g_join_table_factor = 2;  // table slots >= factor * build rows (a power of two)

static uint32_t table_slots(long long nR) {
    uint64_t c = 1024;
    while (c < (uint64_t)nR * g_join_table_factor) c <<= 1;
    return (uint32_t)c;
}

void qg_join_set_table_factor(int factor) { g_join_table_factor = factor < 2 ? 2 : (factor > 8 ? 8 : factor); }

namespace {
// After the probe of the device-planned join: publish the count, and let the
// sort run only when the output fits.
__global__ void k_join_finish_async(JoinCtl *jc, long long cap, unsigned long long *d_count, qg_control *ctl) {
    const unsigned long long m = jc->cursor;
    jc->range = qg_sort_range{qg_sort_npos(jc->kmin, jc->kmax), jc->kmin};
    *d_count = m;
    if (m > (unsigned long long)cap) {
        jc->sortn = 0;
        qg_record_error(ctl, QG_ERR_CAPACITY, QG_SITE_JOIN_PROBE);
    } else {
        jc->sortn = m;
    }
}
}  // namespace

// Build the table in aux; returns the control block (in scratch) and mask.
static qg_status join_build(qg_ctx *ctx, const int32_t *rkey, const int32_t *rpay, long long stride,
                            long long nR, size_t extra_aux, bool limit, unsigned long long **tab_out,
                            uint32_t *mask_out, JoinCtl **jc_out, char **aux_tail) {
    if (nR >= (1LL << 30)) return QG_ERR_UNSUPPORTED;
    const uint32_t slots = table_slots(nR);
    const size_t tbytes = (size_t)slots * 8;
    char *aux;
    QG_TRY(qg_aux(ctx, tbytes + extra_aux + 256, &aux));
    char *scr;
    QG_TRY(qg_scratch(ctx, sizeof(JoinCtl), &scr));
    JoinCtl *jc = (JoinCtl *)scr;
    unsigned long long *tab = (unsigned long long *)aux;
    QG_TRY_CUDA(ctx, cudaMemsetAsync(tab, 0xff, tbytes, ctx->stream), "memset table");
    qg_pre_launch(ctx);
    k_join_ctl_init<<<1, 256, 0, ctx->stream>>>(jc);
    QG_TRY(qg_check_launch(ctx, "k_join_ctl_init"));
    if (nR > 0) {
        // What the probe bears (it then walks slot by slot, and clusters of equal keys
        // lengthen every row's way), hashed / partitioned: 4M build rows and 8M probe rows 430
        // / 500 us with unique keys, 490 / 500 with 25 % in pairs (an eighth of the rows), 520 /
        // 500 with 3 % in eights (half), 884 / 530 with 12 %; 200K and 100K rows all in pairs
        // (half) 145 / 217; 10K and 5K all in eights (17 times) 116 / 162, in thirty-twos 217 / 164.
        const int blocks = grid_cap(ctx, nR, 256, JB_CTAS);
        const float each = nR <= 16384 ? 30.f : nR <= (1 << 19) ? 1.f : 0.4f, share = each * (float)nR / (float)blocks;
        QG_TRY(qg_launch_chained(ctx, "k_join_build", limit ? k_join_build<true> : k_join_build<false>, blocks, 256, 0,
                                 rkey, rpay, (uint32_t)stride, (uint32_t)nR, tab, slots - 1, jc, ctx->ctl,
                                 (uint32_t)(share + 4.f * sqrtf(share) + 1.f)));
    }
    *tab_out = tab;
    *mask_out = slots - 1;
    *jc_out = jc;
    *aux_tail = aux + qg_align_up(tbytes, 256);
    return QG_OK;
}

namespace {
// A few matches: sorted by key by one CTA and written to the output columns.
__global__ void __launch_bounds__(QG_CS_THREADS, 1)
k_join_sort_small(qg_sort_bufs in, qg_sort_bufs out, uint32_t n) {
    qg_chain();
    extern __shared__ __align__(16) unsigned char js_raw[];
    uint32_t(*whist)[256] = reinterpret_cast<uint32_t(*)[256]>(js_raw);
    unsigned long long *ord = reinterpret_cast<unsigned long long *>(whist + 32);
    for (uint32_t i = threadIdx.x; i < n; i += QG_CS_THREADS) ord[i] = (unsigned long long)in.k[i] << 32 | i;
    __syncthreads();
    qg_cta_sort(ord, whist, n);
    for (uint32_t i = threadIdx.x; i < n; i += QG_CS_THREADS) {
        const uint32_t j = (uint32_t)ord[i];
        out.k[i] = (uint32_t)(ord[i] >> 32);
        out.a[i] = in.a[j];
        out.b[i] = in.b[j];
    }
}
}  // namespace

// Launch of k_join_probe.
static qg_status join_probe(qg_ctx *ctx, const int32_t *skey, const int32_t *spay, int64_t nS, int32_t slo, int32_t shi,
                            const unsigned long long *tab, uint32_t mask, JoinCtl *jc, const ProbeOut &po,
                            const ProbeOut &odd, int64_t cap, uint64_t least = 0) {
    const size_t smem = sizeof(PjSmem);
    static qg_per_device site;
    QG_TRY(qg_allow_smem(ctx, site, k_join_probe, smem));
    const long long ntiles = (nS + PJ_TILE - 1) / PJ_TILE;
    const int blocks = (int)(ntiles < (long long)ctx->sm_count * 4 ? ntiles : (long long)ctx->sm_count * 4);
    return qg_launch_chained(ctx, "k_join_probe", k_join_probe, blocks, PJ_THREADS, smem, skey, spay, nS, slo, shi,
                             tab, mask, jc, po, odd, cap, 4, (unsigned long long)least);
}

// Hash join + filter + radix sort of the output: the variant of
// qg_join_filter_sort selected by qg_join_set_knobs(3, ...), and its choice for
// R keys of no dense span.  One wait before the sort, for the match count.
qg_status qg_join_hash_sort(qg_ctx *ctx, const int32_t *rkey, const int32_t *rpay, int64_t nR,
                            const int32_t *skey, const int32_t *spay, int64_t nS, int32_t slo,
                            int32_t shi, int32_t *out_key, int32_t *out_rpay, int32_t *out_spay,
                            int64_t cap, int64_t *out_n, uint64_t least, qg_join_hash_end *end) {
    if (!ctx || nR < 0 || nS < 0 || cap < 0 || !out_n) return QG_ERR_INVALID;
    if ((nR > 0 && (!rkey || !rpay)) || (nS > 0 && (!skey || !spay)) ||
        (cap > 0 && (!out_key || !out_rpay || !out_spay)))
        return QG_ERR_INVALID;
    if ((((uintptr_t)skey) | ((uintptr_t)spay)) & 15) return QG_ERR_INVALID;
    if (cap >= (1LL << 30) || nS >= (1LL << 40)) return QG_ERR_UNSUPPORTED;
    *out_n = 0;
    if (nR == 0 || nS == 0) return QG_OK;
    unsigned long long *tab;
    uint32_t mask;
    JoinCtl *jc;
    char *tail;
    const size_t colbytes = qg_align_up((size_t)(cap > 0 ? cap : 1) * 4, 256);
    QG_TRY(join_build(ctx, rkey, rpay, 1, nR, 3 * colbytes, end != nullptr, &tab, &mask, &jc, &tail));
    qg_sort_bufs A{nullptr, (uint32_t *)tail, (uint32_t *)(tail + colbytes), (uint32_t *)(tail + 2 * colbytes)};
    const qg_sort_bufs B{nullptr, (uint32_t *)out_key, (uint32_t *)out_rpay, (uint32_t *)out_spay};
    QG_TRY(join_probe(ctx, skey, spay, nS, slo, shi, tab, mask, jc, ProbeOut{A.k, A.a, A.b}, ProbeOut{}, cap,
                      least));
    JoinCtl *hjc = reinterpret_cast<JoinCtl *>(ctx->pin_ctl);
    static_assert(sizeof(JoinCtl) <= sizeof(qg_control), "read back into the pinned control block");
    QG_TRY_CUDA(ctx, cudaMemcpyAsync(hjc, jc, sizeof(JoinCtl), cudaMemcpyDeviceToHost, ctx->stream), "ctl d2h");
    QG_TRY(qg_collect_error(ctx));
    const uint32_t range = hjc->kmax - hjc->kmin;
    if (end) {
        *end = hjc->crowded ? QG_JH_CROWDED : range < least ? QG_JH_CLOSE : QG_JH_DONE;
        if (*end != QG_JH_DONE) return QG_OK;
    }
    const long long m = (long long)hjc->cursor;
    *out_n = m;
    if (m > cap) return QG_ERR_CAPACITY;
    if (m == 0) return QG_OK;
    const int npos = range ? qg_sort_positions(32 - __builtin_clz(range)) : 0;
    // Up to 8192 matches: one launch (4 radix passes took 45 us for 4K of them)
    if (m <= QG_CS_MAX) {
        const size_t most = QG_CS_MAX * 8 + 32 * 1024, smem = (size_t)m * 8 + 32 * 1024;
        static qg_per_device site;
        QG_TRY(qg_allow_smem(ctx, site, k_join_sort_small, most));
        qg_pre_launch(ctx);
        k_join_sort_small<<<1, QG_CS_THREADS, smem, ctx->stream>>>(A, B, (uint32_t)m);
        QG_TRY(qg_check_launch(ctx, "k_join_sort_small"));
        return qg_ctx_check(ctx);
    }
    int passes[4];
    uint32_t bases[4 * QG_RADIX];
    const int np = npos ? qg_sort_plan(&hjc->hist[0][0], npos, m, passes, bases) : 0;
    const uint32_t key_off = hjc->kmin;
    auto copy_out = [&]() -> qg_status {
        QG_TRY_CUDA(ctx, cudaMemcpyAsync(out_key, A.k, (size_t)m * 4, cudaMemcpyDeviceToDevice, ctx->stream), "copy");
        QG_TRY_CUDA(ctx, cudaMemcpyAsync(out_rpay, A.a, (size_t)m * 4, cudaMemcpyDeviceToDevice, ctx->stream), "copy");
        QG_TRY_CUDA(ctx, cudaMemcpyAsync(out_spay, A.b, (size_t)m * 4, cudaMemcpyDeviceToDevice, ctx->stream), "copy");
        return QG_OK;
    };
    if (np == 0) {  // one key: in order as it is
        QG_TRY(copy_out());
        return qg_ctx_check(ctx);
    }
    // The last pass ends in the output: with an even number of them the first
    // goes to a third set of columns (the table is not needed any more), or, without
    // memory for one, the last ends where the first began and is copied.
    bool other = false;
    const size_t mb = qg_align_up((size_t)m * 4, 256);
    char *third = (char *)tab;
    if (!(np & 1) && 3 * mb > ((size_t)mask + 1) * 8) {
        const qg_status st = qg_spare(ctx, 3 * mb, &third);
        if (st == QG_ERR_OOM) third = nullptr;
        else QG_TRY(st);
    }
    if ((np & 1) || !third) {
        QG_TRY(qg_radix_passes(ctx, true, A, B, m, key_off, passes, np, bases, &other));
        if (!(np & 1)) QG_TRY(copy_out());
    } else {
        const qg_sort_bufs C{nullptr, (uint32_t *)third, (uint32_t *)(third + mb), (uint32_t *)(third + 2 * mb)};
        QG_TRY(qg_radix_passes(ctx, true, A, C, m, key_off, passes, 1, bases, &other));
        QG_TRY(qg_radix_passes(ctx, true, C, B, m, key_off, passes + 1, np - 1, bases, &other));
    }
    return qg_ctx_check(ctx);
}

// The hash join + filter + sort with no host round trip (for CUDA graph
// capture, e.g. by qg_batch): the sort is planned on the device from the build's
// key range and the probe's digit counts.  d_count (device
// int64) receives the match count; more matches than cap records
// QG_ERR_CAPACITY in the context's error word and leaves the output unsorted.
qg_status qg_join_hash_sort_async(qg_ctx *ctx, const int32_t *rkey, const int32_t *rpay, int64_t nR,
                                  const int32_t *skey, const int32_t *spay, int64_t nS, int32_t slo,
                                  int32_t shi, int32_t *out_key, int32_t *out_rpay, int32_t *out_spay,
                                  int64_t cap, int64_t *d_count) {
    if (!ctx || nR < 0 || nS < 0 || cap < 0 || !d_count) return QG_ERR_INVALID;
    if ((nR > 0 && (!rkey || !rpay)) || (nS > 0 && (!skey || !spay)) ||
        (cap > 0 && (!out_key || !out_rpay || !out_spay)))
        return QG_ERR_INVALID;
    if ((((uintptr_t)skey) | ((uintptr_t)spay)) & 15) return QG_ERR_INVALID;
    if (cap >= (1LL << 30) || nS >= (1LL << 40)) return QG_ERR_UNSUPPORTED;
    if (nR == 0 || nS == 0 || cap == 0) {
        QG_TRY_CUDA(ctx, cudaMemsetAsync(d_count, 0, 8, ctx->stream), "memset count");
        return QG_OK;
    }
    const size_t colbytes = qg_align_up((size_t)cap * 4, 256);
    const size_t work = qg_align_up(qg_radix_dev_work_bytes(cap), 256);
    unsigned long long *tab;
    uint32_t mask;
    JoinCtl *jc;
    char *tail;
    QG_TRY(join_build(ctx, rkey, rpay, 1, nR, 3 * colbytes + work, false, &tab, &mask, &jc, &tail));
    qg_sort_bufs A{nullptr, (uint32_t *)out_key, (uint32_t *)out_rpay, (uint32_t *)out_spay};
    qg_sort_bufs B{nullptr, (uint32_t *)tail, (uint32_t *)(tail + colbytes), (uint32_t *)(tail + 2 * colbytes)};
    // (with room for one row no sort follows, so it has to land in the output)
    QG_TRY(join_probe(ctx, skey, spay, nS, slo, shi, tab, mask, jc, ProbeOut{A.k, A.a, A.b},
                      cap > 1 ? ProbeOut{B.k, B.a, B.b} : ProbeOut{}, cap));
    qg_pre_launch(ctx);
    k_join_finish_async<<<1, 1, 0, ctx->stream>>>(jc, cap, (unsigned long long *)d_count, ctx->ctl);
    QG_TRY(qg_check_launch(ctx, "k_join_finish_async"));
    return qg_radix_passes_range(ctx, A, B, cap, &jc->sortn, &jc->hist[0][0], &jc->range, tail + 3 * colbytes);
}

// ---------------------------------------------------------------------------
// Reference layout: buildHashTable / probeHashTable
// (kernel/hj_filter_sort/1/hj_filter_sort_op.cl:25-60 and 62-109).  The
// reference's caller allocates the table (rHashTable, rHashCount) and may
// probe it with several S tables; here the caller allocates
// qg_hash_table_bytes(nR) bytes, qg_hash_build_ref fills them, and any number
// of qg_hash_probe_ref calls read them.
// ---------------------------------------------------------------------------
static uint32_t ref_table_slots(long long nR) {
    uint64_t c = 1024;
    while (c < (uint64_t)nR * 2) c <<= 1;
    return (uint32_t)c;
}

namespace {
__global__ void k_ref_hash_hdr_init(RefHashHdr *hdr, uint32_t slots) {
    if (threadIdx.x == 0) {
        hdr->slots = slots;
        hdr->magic = REF_HASH_MAGIC;
    }
}
}  // namespace

extern "C" QG_API int64_t qg_hash_table_bytes(int64_t nR) {
    if (nR < 0 || nR >= (1LL << 30)) return -1;
    return (int64_t)(REF_HASH_HDR + (size_t)ref_table_slots(nR) * 8);
}

extern "C" QG_API qg_status qg_hash_build_ref(qg_ctx *ctx, const uint32_t *r, int64_t nR, void *table,
                                              int64_t table_bytes) {
    if (!ctx || nR < 0 || !table || (nR > 0 && !r)) return QG_ERR_INVALID;
    if ((((uintptr_t)r) & 7) || (((uintptr_t)table) & 255)) return QG_ERR_INVALID;
    if (nR >= (1LL << 30)) return QG_ERR_UNSUPPORTED;
    if (table_bytes < qg_hash_table_bytes(nR)) return QG_ERR_CAPACITY;
    const uint32_t slots = ref_table_slots(nR);
    RefHashHdr *hdr = (RefHashHdr *)table;
    unsigned long long *tab = (unsigned long long *)((char *)table + REF_HASH_HDR);
    QG_TRY_CUDA(ctx, cudaMemsetAsync(tab, 0xff, (size_t)slots * 8, ctx->stream), "memset table");
    qg_pre_launch(ctx);
    k_join_ctl_init<<<1, 256, 0, ctx->stream>>>(&hdr->jc);
    QG_TRY(qg_check_launch(ctx, "k_join_ctl_init"));
    qg_pre_launch(ctx);
    k_ref_hash_hdr_init<<<1, 32, 0, ctx->stream>>>(hdr, slots);
    QG_TRY(qg_check_launch(ctx, "k_ref_hash_hdr_init"));
    if (nR > 0) {
        int blocks = grid_cap(ctx, nR, 256, JB_CTAS);
        QG_TRY(qg_launch_chained(ctx, "k_join_build", k_join_build<false>, blocks, 256, 0, (const int32_t *)r,
                                 (const int32_t *)r + 1, 2u, (uint32_t)nR, tab, slots - 1, &hdr->jc, ctx->ctl, 0u));
    }
    // a table that fills up (cannot happen at 2 slots per row) reports TABLE_FULL
    return qg_ctx_check(ctx);
}

extern "C" QG_API qg_status qg_hash_probe_ref(qg_ctx *ctx, const void *table, const uint32_t *s, int64_t nS,
                                              uint32_t *out, int64_t cap, int64_t *out_n) {
    if (!ctx || !table || nS < 0 || cap < 0 || !out_n) return QG_ERR_INVALID;
    if ((nS > 0 && !s) || (cap > 0 && !out)) return QG_ERR_INVALID;
    if ((((uintptr_t)s) | ((uintptr_t)out)) & 7 || (((uintptr_t)table) & 255)) return QG_ERR_INVALID;
    *out_n = 0;
    if (nS == 0) return QG_OK;
    const RefHashHdr *hdr = (const RefHashHdr *)table;
    const unsigned long long *tab = (const unsigned long long *)((const char *)table + REF_HASH_HDR);
    unsigned long long *cursor = &ctx->ctl->counter[0];
    QG_TRY_CUDA(ctx, cudaMemsetAsync(cursor, 0, 8, ctx->stream), "memset cursor");
    int blocks = grid_cap(ctx, nS, 256, 8);
    qg_pre_launch(ctx);
    k_join_probe_ref<<<blocks, 256, 0, ctx->stream>>>(s, nS, tab, hdr, cursor, out, cap);
    QG_TRY(qg_check_launch(ctx, "k_join_probe_ref"));
    long long m = 0;
    QG_TRY(qg_read_count(ctx, (const long long *)cursor, &m));
    *out_n = m;
    return m > cap ? QG_ERR_CAPACITY : QG_OK;
}

extern "C" QG_API qg_status qg_hash_join_ref(qg_ctx *ctx, const uint32_t *r, int64_t nR,
                                             const uint32_t *s, int64_t nS, uint32_t *out,
                                             int64_t cap, int64_t *out_n) {
    if (!ctx || nR < 0 || nS < 0 || cap < 0 || !out_n) return QG_ERR_INVALID;
    if ((nR > 0 && !r) || (nS > 0 && !s) || (cap > 0 && !out)) return QG_ERR_INVALID;
    if ((((uintptr_t)r) | ((uintptr_t)s) | ((uintptr_t)out)) & 7) return QG_ERR_INVALID;
    *out_n = 0;
    if (nR == 0 || nS == 0) return QG_OK;
    const int64_t tb = qg_hash_table_bytes(nR);
    if (tb < 0) return QG_ERR_UNSUPPORTED;
    char *aux;
    QG_TRY(qg_aux(ctx, (size_t)tb, &aux));  // the aux arena is 256-byte aligned
    QG_TRY(qg_hash_build_ref(ctx, r, nR, aux, tb));
    return qg_hash_probe_ref(ctx, aux, s, nS, out, cap, out_n);
}
