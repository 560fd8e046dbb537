// qg_cta_sort.cuh -- sort of a few thousand keys by one CTA in shared memory.
#pragma once
#include "qg_internal.cuh"

constexpr int QG_CS_THREADS = 1024;
constexpr int QG_CS_MAX = 8192;                           // entries, at most
constexpr int QG_CS_ITEMS = QG_CS_MAX / QG_CS_THREADS;    // per thread

constexpr uint32_t QG_CS_CROWD = 24;                      // entries of a bucket that are ranked pairwise

// Sort of ord[0 .. g) (shared memory, g <= QG_CS_MAX), distinct words, by the
// high words, entries with equal ones as they stand.  whist: [32][256] words,
// 16-byte aligned.  All QG_CS_THREADS threads call it; it ends with a barrier.
//
// One counting pass over the leading bits of the keys' range spreads the
// entries over up to 8192 buckets, about one in each unless the keys cluster,
// and an entry's place in its bucket is the number of smaller ones there.  A
// bucket of more than QG_CS_CROWD entries (clustered or repeated keys) leads to
// an LSD radix sort, 8 bits a pass, digits in which no two keys differ skipped.
// 4096 random keys take 4 us, 18 by the radix sort's four passes alone (a
// bitonic sort took 40, 78 dependent steps).
__device__ __forceinline__ void qg_cta_sort(unsigned long long *ord, uint32_t (*whist)[256], uint32_t g) {
    __shared__ uint32_t s_min, s_max, s_w[QG_CS_THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t per = (g + QG_CS_THREADS - 1) / QG_CS_THREADS;  // entries per thread
    const uint32_t warps = per ? (g + 32 * per - 1) / (32 * per) : 0, lt = qg_lanemask_lt();
    const uint32_t w0 = warp * 32 * per + lane;  // the lane's first entry
    uint32_t *cnt = &whist[0][0];                // [QG_CS_MAX] the buckets
    uint4 *cnt4 = reinterpret_cast<uint4 *>(cnt);
    static_assert(QG_CS_MAX == 8192 && QG_CS_ITEMS == 8, "two vectors of buckets per thread");
    unsigned long long it[QG_CS_ITEMS];
    uint32_t rank[QG_CS_ITEMS];
    uint32_t kmin = 0xffffffffu, kmax = 0;
#pragma unroll
    for (int i = 0; i < QG_CS_ITEMS; i++) {
        if (i >= (int)per) break;
        if (w0 + i * 32 < g) {
            it[i] = ord[w0 + i * 32];
            kmin = min(kmin, (uint32_t)(it[i] >> 32));
            kmax = max(kmax, (uint32_t)(it[i] >> 32));
        }
    }
    if (tid == 0) {
        s_min = 0xffffffffu;
        s_max = 0;
    }
    cnt4[2 * tid] = cnt4[2 * tid + 1] = make_uint4(0, 0, 0, 0);
    kmin = __reduce_min_sync(QG_FULL_MASK, kmin);
    kmax = __reduce_max_sync(QG_FULL_MASK, kmax);
    __syncthreads();
    if (lane == 0 && warp < (int)warps) {
        atomicMin(&s_min, kmin);
        atomicMax(&s_max, kmax);
    }
    __syncthreads();
    kmin = s_min;
    kmax = s_max;
    const int sh = max(0, 32 - 13 - __clz(kmax - kmin));  // buckets: (key - kmin) >> sh, below 8192
    bool crowd = false;
#pragma unroll
    for (int i = 0; i < QG_CS_ITEMS; i++) {
        if (i >= (int)per) break;
        if (w0 + i * 32 < g) {
            rank[i] = atomicAdd(&cnt[((uint32_t)(it[i] >> 32) - kmin) >> sh], 1u);
            crowd |= rank[i] >= QG_CS_CROWD;
        }
    }
    if (!__syncthreads_or(crowd)) {
        const uint4 c0 = cnt4[2 * tid], c1 = cnt4[2 * tid + 1];
        const uint32_t tot = c0.x + c0.y + c0.z + c0.w + c1.x + c1.y + c1.z + c1.w;
        uint32_t inc = tot;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t x = __shfl_up_sync(QG_FULL_MASK, inc, d);
            if (lane >= d) inc += x;
        }
        if (lane == 31) s_w[warp] = inc;
        __syncthreads();
        const uint32_t before = __reduce_add_sync(QG_FULL_MASK, lane < warp ? s_w[lane] : 0u) + inc - tot;
        uint4 p0, p1;
        p0.x = before;
        p0.y = p0.x + c0.x;
        p0.z = p0.y + c0.y;
        p0.w = p0.z + c0.z;
        p1.x = p0.w + c0.w;
        p1.y = p1.x + c1.x;
        p1.z = p1.y + c1.y;
        p1.w = p1.z + c1.z;
        cnt4[2 * tid] = p0;
        cnt4[2 * tid + 1] = p1;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < QG_CS_ITEMS; i++) {
            if (i >= (int)per) break;
            if (w0 + i * 32 < g) ord[cnt[((uint32_t)(it[i] >> 32) - kmin) >> sh] + rank[i]] = it[i];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < QG_CS_ITEMS; i++) {
            if (i >= (int)per) break;
            if (w0 + i * 32 < g) {
                const uint32_t b = ((uint32_t)(it[i] >> 32) - kmin) >> sh;
                const uint32_t lo = cnt[b], hi = b + 1 < QG_CS_MAX ? cnt[b + 1] : g;
                uint32_t r = lo;
                if (hi - lo > 1)
                    for (uint32_t j = lo; j < hi; j++) r += ord[j] < it[i] ? 1u : 0u;
                rank[i] = r;
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < QG_CS_ITEMS; i++) {
            if (i >= (int)per) break;
            if (w0 + i * 32 < g) ord[rank[i]] = it[i];
        }
        __syncthreads();
        return;
    }
    uint32_t diff = 0;
    for (uint32_t i = tid; i < g; i += QG_CS_THREADS) diff |= (uint32_t)(ord[i] >> 32) ^ (uint32_t)(ord[0] >> 32);
    diff = __reduce_or_sync(QG_FULL_MASK, diff);
    if (tid == 0) s_min = 0;
    __syncthreads();
    if (lane == 0 && diff) atomicOr(&s_min, diff);
    __syncthreads();
    diff = s_min;
    for (int shift = 32; shift < 64; shift += 8) {
        if (!((diff >> (shift - 32)) & 255u)) continue;
        if (warp < (int)warps) {
            for (int i = lane; i < 256; i += 32) whist[warp][i] = 0;
            __syncwarp();
#pragma unroll
            for (int i = 0; i < QG_CS_ITEMS; i++)
                if (i < (int)per) it[i] = w0 + i * 32 < g ? ord[w0 + i * 32] : ~0ull;
#pragma unroll
            for (int i = 0; i < QG_CS_ITEMS; i++) {
                if (i >= (int)per) break;
                const bool valid = w0 + i * 32 < g;
                const uint32_t d = (uint32_t)(it[i] >> shift) & 255u;
                uint32_t peers = __ballot_sync(QG_FULL_MASK, valid);
#pragma unroll
                for (int b = 0; b < 8; b++) {
                    const uint32_t bal = __ballot_sync(QG_FULL_MASK, (d >> b) & 1u);
                    peers &= ((d >> b) & 1u) ? bal : ~bal;
                }
                rank[i] = valid ? whist[warp][d] + __popc(peers & lt) : 0u;
                __syncwarp();
                if (valid && lane == 31 - __clz(peers)) whist[warp][d] = rank[i] + 1u;
                __syncwarp();
            }
        }
        __syncthreads();
        uint32_t tot = 0, inc = 0;
        if (tid < 256) {
            for (uint32_t w = 0; w < warps; w++) {  // to the digit's items before each warp's
                const uint32_t c = whist[w][tid];
                whist[w][tid] = tot;
                tot += c;
            }
            inc = tot;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t x = __shfl_up_sync(QG_FULL_MASK, inc, d);
                if (lane >= d) inc += x;
            }
            if (lane == 31) s_w[warp] = inc;
        }
        __syncthreads();
        if (tid < 256) {
            uint32_t run = inc - tot;
            for (int w = 0; w < warp; w++) run += s_w[w];
            for (uint32_t w = 0; w < warps; w++) whist[w][tid] += run;
        }
        __syncthreads();
        if (warp < (int)warps) {
#pragma unroll
            for (int i = 0; i < QG_CS_ITEMS; i++) {
                if (i >= (int)per) break;
                if (w0 + i * 32 < g) ord[whist[warp][(uint32_t)(it[i] >> shift) & 255u] + rank[i]] = it[i];
            }
        }
        __syncthreads();
    }
}
