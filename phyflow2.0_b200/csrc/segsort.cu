// segsort.cu -- one CTA per listed segment: chunks of SEG_CHUNK values sorted
// in shared memory (bitonic network), then runs merged pairwise, level by
// level, each value written straight to its place: its index in its own run
// plus the number of values of the other run below it (binary search; the
// values are distinct, so there are no ties).  O(c log^2 c) work for a
// segment of c values, no atomics, deterministic.
#include "segsort.cuh"

#include <algorithm>
#include <climits>

namespace {

__global__ void __launch_bounds__(SEG_THREADS)
k_seg_sort(const int32_t *__restrict__ list, const int32_t *__restrict__ list_n,
           const int32_t *__restrict__ start, const int32_t *__restrict__ cnt,
           int32_t *__restrict__ vals, int32_t *__restrict__ tmp) {
    __shared__ int32_t s_v[SEG_CHUNK];
    const int nlist = *list_n;
    for (int k = blockIdx.x; k < nlist; k += gridDim.x) {
        const int id = list[k];
        const int64_t s0 = start[id];
        seg_sort_block(vals + s0, tmp + s0, cnt[id], s_v);
    }
}

}  // namespace

namespace pf {

pf_status seg_sort_listed(const int32_t *list, const int32_t *list_n, const int32_t *start,
                          const int32_t *cnt, int32_t *vals, int32_t *tmp, int64_t max_segments,
                          cudaStream_t st) {
    if (max_segments <= 0) return PF_OK;
    // a few CTAs suffice (large segments are rare); each loops over the list
    const unsigned grid = (unsigned)std::min<int64_t>(max_segments, 64);
    k_seg_sort<<<grid, SEG_THREADS, 0, st>>>(list, list_n, start, cnt, vals, tmp);
    return launch_status("k_seg_sort");
}

}  // namespace pf
