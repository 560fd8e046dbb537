// qg_keytable.cuh -- open-addressing key table in shared memory, walked by
// groups of four slots.
#pragma once
#include "qg_internal.cuh"

constexpr uint32_t QG_KT_FREE = 0xffffffffu;  // a free slot; a key of this value is kept apart by the caller

// First slot of key k's group in a table of mask + 1 slots (a power of two, at least 4).
__device__ __forceinline__ uint32_t qg_kt_group(uint32_t k, uint32_t mask) { return qg_hash32(k) & mask & ~3u; }

__device__ __forceinline__ uint4 qg_kt_read(const uint32_t *key, uint32_t group) {
    uint4 q;  // volatile: other threads insert meanwhile
    asm volatile("ld.volatile.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w)
                 : "r"(qg_smem_u32(key + group))
                 : "memory");
    return q;
}

// Match of k in a group (0 to 3, 4: none); the first free slot of a group.
__device__ __forceinline__ uint32_t qg_kt_match(const uint4 &q, uint32_t k) {
    return q.x == k ? 0u : q.y == k ? 1u : q.z == k ? 2u : q.w == k ? 3u : 4u;
}

// Slots h[u] of the keys k[u] of the rows in the bit mask `live`, inserted where
// new.  False: a key found no slot within `probes`.  Key QG_KT_FREE's slot is
// mask + 1, an entry behind the table.  fresh counts the keys this thread was
// the first to insert.
//
// One 16-byte read answers most rows: walking slot by slot, a warp's slowest
// lane took five dependent reads at load 1/2.  The rows that it does not answer
// (new keys, full groups) are walked together, a lane going on to its next row
// by itself: row after row, each row costs the warp its slowest lane's walk.
template <int U>
__device__ __forceinline__ bool qg_kt_find(uint32_t *key, uint32_t mask, const uint32_t (&k)[U], uint32_t live,
                                           uint32_t (&h)[U], uint32_t probes, uint32_t &fresh) {
    uint4 q[U];
#pragma unroll
    for (int u = 0; u < U; u++) q[u] = qg_kt_read(key, qg_kt_group(k[u], mask));
    uint32_t todo = 0;
#pragma unroll
    for (int u = 0; u < U; u++) {
        const uint32_t at = qg_kt_match(q[u], k[u]);
        h[u] = k[u] == QG_KT_FREE ? mask + 1 : qg_kt_group(k[u], mask) + at;
        if (((live >> u) & 1u) && k[u] != QG_KT_FREE && at == 4) todo |= 1u << u;
    }
    uint32_t p = 0, g = 0, kk = 0;
    while (todo) {
        if (p == 0) {
#pragma unroll
            for (int u = U - 1; u >= 0; u--)
                if ((todo >> u) & 1u) kk = k[u];
            g = qg_kt_group(kk, mask);
            p = 4;
        }
        const uint4 s = qg_kt_read(key, g);
        uint32_t at = qg_kt_match(s, kk);
        bool found = at < 4;
        if (!found) {
            at = qg_kt_match(s, QG_KT_FREE);
            if (at < 4) {  // slots fill in order, so the key is in none of the later ones
                const uint32_t old = atomicCAS(&key[g + at], QG_KT_FREE, kk);
                fresh += old == QG_KT_FREE;
                found = old == QG_KT_FREE || old == kk;  // else another key came first: read the group again
            } else {
                if (p >= probes) return false;
                p += 4;
                g = (g + 4) & mask;
            }
        }
        if (found) {
            const uint32_t low = todo & (0u - todo);
#pragma unroll
            for (int u = 0; u < U; u++)
                if (low == 1u << u) h[u] = g + at;
            todo ^= low;
            p = 0;
        }
    }
    return true;
}
