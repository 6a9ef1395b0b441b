// hostcopy.h -- host memory copies split over a few threads: one thread copies at well
// under the host memory bandwidth, which would otherwise bound the transfers between
// caller memory and page-locked staging.
#pragma once

#include <algorithm>
#include <cstdint>
#include <cstring>

#include <sys/mman.h>

namespace xpr {

inline void par_memcpy(void *dst, const void *src, size_t n)
{
    constexpr size_t kTask = 4u << 20;
    const int64_t tasks = (int64_t)((n + kTask - 1) / kTask);
#pragma omp parallel for schedule(static) num_threads(8) if (tasks > 1)
    for (int64_t t = 0; t < tasks; ++t) {
        const size_t o = (size_t)t * kTask;
        std::memcpy((char *)dst + o, (const char *)src + o, std::min(kTask, n - o));
    }
}

// Maps the pages of [dst, dst + n), memory that is about to be overwritten, from several threads at
// once when the caller never touched most of them: a copy would map them one by one from its own
// thread.  Memory in use is left alone (64 pages are asked for; starting threads over it would
// add nothing but their jitter).
inline void par_map(void *dst, size_t n)
{
    constexpr size_t kPage = 4096;
    constexpr int kProbes = 64;
    const uintptr_t first = (uintptr_t)dst / kPage, last = ((uintptr_t)dst + n - 1) / kPage;
    int mapped = 0;
    for (int k = 0; k < kProbes; ++k) {
        unsigned char in = 1;
        if (mincore((void *)((first + (last - first) * k / kProbes) * kPage), 1, &in) != 0) return;
        mapped += in & 1;
    }
    if (mapped > kProbes / 2) return;
    volatile char *p = (volatile char *)dst;
    const int64_t pages = (int64_t)(n / kPage);
#pragma omp parallel for schedule(static) num_threads(8)
    for (int64_t i = 0; i < pages; ++i) p[(size_t)i * kPage] = 0;
    if (n) p[n - 1] = 0;
}

}  // namespace xpr
