// qg_join.cuh -- the join paths that qg_join_filter_sort and batches share.
#pragma once
#include "qg_internal.cuh"

// Dense build side by counting (qg_jdirect.cu): six launches on the context's
// stream, no read back.  `work`: qg_jd_bytes(nR, nS) bytes, 256-byte aligned.
// Afterwards ctl->jd[QG_JD_OK] (also *result, when set) is QG_JD_DONE when the
// outputs hold the result, *d_count then the match count (the first cap rows
// are written); else what stood against it, and nothing was written.
enum { QG_JD_OK = 4 };
enum qg_jd_result : uint32_t {
    QG_JD_SPARSE = 0,  // R's keys spread over more than 2 nR values
    QG_JD_DONE = 1,
    QG_JD_TWICE = 2,   // dense span, but a build key twice
    QG_JD_HOT = 3,     // ... or a probe key with too many rows
};
size_t qg_jd_bytes(int64_t nR, int64_t nS);
qg_status qg_jd_launch(qg_ctx *ctx, char *work, const int32_t *rkey, const int32_t *rpay, int64_t nR,
                       const int32_t *skey, const int32_t *spay, int64_t nS, int32_t slo, int32_t shi, uint32_t *out_key,
                       uint32_t *out_rpay, uint32_t *out_spay, int64_t cap, long long *d_count, volatile uint32_t *result);

// Hash join + sort of the matches (qg_join.cu).  With `end` set it may be given up (*end
// says so, and nothing was written): build keys that repeat often, or that lie within
// fewer than `least` values.
enum qg_join_hash_end {
    QG_JH_DONE,
    QG_JH_CROWDED,  // build keys repeat too often
    QG_JH_CLOSE,    // too small a span
};
qg_status qg_join_hash_sort(qg_ctx *ctx, const int32_t *rkey, const int32_t *rpay, int64_t nR, const int32_t *skey,
                            const int32_t *spay, int64_t nS, int32_t slo, int32_t shi, int32_t *out_key,
                            int32_t *out_rpay, int32_t *out_spay, int64_t cap, int64_t *out_n,
                            uint64_t least = 0, qg_join_hash_end *end = nullptr);

// flags of the dense build side (u32 words): [1] dense span, [2..3] distinct
// keys (u64), [4] / [5] smallest / largest R payload (int32), [6] a sentinel
// payload exists, [7] the sentinel.
enum { PJ_F_DENSE = 1, PJ_F_DISTINCT = 2, PJ_F_PMIN = 4, PJ_F_PMAX = 5, PJ_F_SENT_OK = 6, PJ_F_SENT = 7, PJ_F_WORDS = 8 };

// Dense build side, large probe inputs (qg_jpart.cu): four launches, no read
// back.  r: R's payload table as k_pj_rtab leaves it.  rows: `room` rows of
// scratch, 16-byte aligned.  Afterwards *result is a qg_jp_result, and with QG_JP_DONE
// the outputs hold the result and *d_count the match count; qg_jp_done() is a word in
// device memory that is 1 then, for kernels that follow.  work: qg_jp_bytes(), 16-byte
// aligned.
enum qg_jp_result : uint32_t {
    QG_JP_REFUSED = 0,  // no dense build side, or the sample shows uneven rows
    QG_JP_DONE = 1,
    QG_JP_OVER = 2,     // a bucket outgrew its room while the rows were partitioned
};
struct qg_jp_r {
    const uint32_t *range;  // smallest and largest key
    const uint32_t *flags;  // PJ_F_*
    const uint32_t *bitmap, *T;
    int64_t nR;
};
size_t qg_jp_bytes();
const uint32_t *qg_jp_done(const char *work);
qg_status qg_jp_launch(qg_ctx *ctx, char *work, const qg_jp_r &r, const int32_t *skey, const int32_t *spay, int64_t nS,
                       int32_t slo, int32_t shi, unsigned long long *rows, int64_t room, uint32_t *out_key,
                       uint32_t *out_rpay, uint32_t *out_spay, int64_t cap, volatile long long *d_count,
                       volatile uint32_t *result);
