// segsort.cuh -- ascending sort of listed segments of distinct int32 values,
// one CTA per segment, for the large leaves / cells that the per-thread
// insertion sorts of the counting sorts leave alone.
#pragma once
#include <climits>

#include "pf_common.cuh"

namespace pf {

// Segments longer than this are sorted by seg_sort_listed; shorter ones by
// the callers' per-thread insertion sorts.
constexpr int SEG_SMALL = 64;

// Sort vals[start[id] .. start[id] + cnt[id]) for every id = list[k],
// k < *list_n (device count).  The values of a segment must be distinct.
// tmp: scratch with the same indexing as vals (only the listed segments'
// ranges are used).  max_segments bounds *list_n (grid size).
pf_status seg_sort_listed(const int32_t *list, const int32_t *list_n, const int32_t *start,
                          const int32_t *cnt, int32_t *vals, int32_t *tmp, int64_t max_segments,
                          cudaStream_t st);

}  // namespace pf

namespace {

constexpr int SEG_THREADS = 1024;
constexpr int SEG_CHUNK = 4096;  // values sorted in shared memory at a time

// number of values of the sorted run a[0 .. n) below x
__device__ __forceinline__ int count_below(const int32_t *__restrict__ a, int n, int32_t x) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (a[mid] < x)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

// One CTA of SEG_THREADS threads sorts v[0 .. c) (tmp: scratch of c values; s_v:
// SEG_CHUNK values of shared memory).
__device__ __forceinline__ void seg_sort_block(int32_t *__restrict__ v, int32_t *__restrict__ tmp,
                                               int c, int32_t *s_v) {
    // 1. sorted chunks
    for (int ch = 0; ch < c; ch += SEG_CHUNK) {
        const int len = min(SEG_CHUNK, c - ch);
        int p = 1;
        while (p < len) p <<= 1;
        for (int i = threadIdx.x; i < p; i += SEG_THREADS)
            s_v[i] = i < len ? v[ch + i] : INT_MAX;
        __syncthreads();
        for (int kk = 2; kk <= p; kk <<= 1) {
            for (int j = kk >> 1; j > 0; j >>= 1) {
                for (int i = threadIdx.x; i < p; i += SEG_THREADS) {
                    const int ij = i ^ j;
                    if (ij > i) {
                        const int32_t a = s_v[i], b = s_v[ij];
                        const bool up = (i & kk) == 0;
                        if ((a > b) == up) {
                            s_v[i] = b;
                            s_v[ij] = a;
                        }
                    }
                }
                __syncthreads();
            }
        }
        for (int i = threadIdx.x; i < len; i += SEG_THREADS) v[ch + i] = s_v[i];
        __syncthreads();
    }
    // 2. merge runs of width w, 2w, ... (vals and tmp alternate)
    int32_t *src = v, *dst = tmp;
    for (int w = SEG_CHUNK; w < c; w <<= 1) {
        for (int r0 = 0; r0 < c; r0 += 2 * w) {
            const int na = min(w, c - r0), nb = max(0, min(w, c - r0 - w));
            const int32_t *a = src + r0, *b = src + r0 + w;
            for (int i = threadIdx.x; i < na; i += SEG_THREADS)
                dst[r0 + i + count_below(b, nb, a[i])] = a[i];
            for (int j = threadIdx.x; j < nb; j += SEG_THREADS)
                dst[r0 + j + count_below(a, na, b[j])] = b[j];
        }
        __syncthreads();
        int32_t *t = src;
        src = dst;
        dst = t;
    }
    if (src != v) {
        for (int i = threadIdx.x; i < c; i += SEG_THREADS) v[i] = src[i];
    }
    __syncthreads();
}

}  // namespace
