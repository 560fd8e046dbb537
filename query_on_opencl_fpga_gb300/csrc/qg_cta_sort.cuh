// qg_cta_sort.cuh -- sort of a few thousand keys by one CTA in shared memory.
#pragma once
#include "qg_internal.cuh"

constexpr int QG_CS_THREADS = 1024;
constexpr int QG_CS_MAX = 8192;                           // entries, at most
constexpr int QG_CS_ITEMS = QG_CS_MAX / QG_CS_THREADS;    // per thread

// Stable sort of ord[0 .. g) (shared memory, g <= QG_CS_MAX) by the high words:
// LSD radix, 8 bits a pass, each warp 256 entries; a digit that all keys share
// is skipped.  whist: [ceil(g / 256)][256] words, dsum: 8 words of shared
// memory.  All QG_CS_THREADS threads call it; it ends with a barrier.  (A bitonic
// sort of 4096 entries took 40 us, 78 dependent steps; this takes 8.)
__device__ __forceinline__ void qg_cta_sort(unsigned long long *ord, uint32_t (*whist)[256], uint32_t *dsum,
                                            uint32_t g) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t warps = (g + 255) / 256, lt = qg_lanemask_lt();
    for (int shift = 32; shift < 64; shift += 8) {
        unsigned long long it[QG_CS_ITEMS];
        uint32_t rank[QG_CS_ITEMS];
        if (warp < (int)warps) {
            for (int i = lane; i < 256; i += 32) whist[warp][i] = 0;
            __syncwarp();
#pragma unroll
            for (int i = 0; i < QG_CS_ITEMS; i++) {
                const uint32_t at = warp * 256 + i * 32 + lane;
                it[i] = at < g ? ord[at] : ~0ull;
            }
#pragma unroll
            for (int i = 0; i < QG_CS_ITEMS; i++) {
                const bool valid = warp * 256 + i * 32 + lane < g;
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
            for (uint32_t w = 0; w < warps; w++) tot += whist[w][tid];
            inc = tot;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t x = __shfl_up_sync(QG_FULL_MASK, inc, d);
                if (lane >= d) inc += x;
            }
            if (lane == 31) dsum[warp] = inc;
        }
        if (__syncthreads_or(tid < 256 && tot == g)) continue;  // one digit value: in place already
        if (tid < 256) {
            uint32_t run = inc - tot;
            for (int w = 0; w < warp; w++) run += dsum[w];
            for (uint32_t w = 0; w < warps; w++) {
                const uint32_t c = whist[w][tid];
                whist[w][tid] = run;
                run += c;
            }
        }
        __syncthreads();
        if (warp < (int)warps) {
#pragma unroll
            for (int i = 0; i < QG_CS_ITEMS; i++)
                if (warp * 256 + i * 32 + lane < g) ord[whist[warp][(uint32_t)(it[i] >> shift) & 255u] + rank[i]] = it[i];
        }
        __syncthreads();
    }
}
