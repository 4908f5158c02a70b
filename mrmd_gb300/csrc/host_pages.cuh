// Host pages made present ahead of a copy into them.
#pragma once

#include <sys/mman.h>
#include <unistd.h>

#include <cstddef>
#include <cstdint>

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23  // Linux 5.14
#endif

namespace mrmd_impl
{
// Makes the pages of [dst, dst + bytes) present and writable, by the host:
// left to a copy into fresh pages, the GPU faults them one by one (3 x 25 MB
// into new arrays 54 ms, 0.5 ms into pages that exist).  Then it reads each:
// the GPU's copy faults pages too that are present but that the host has not
// used for a while, pinned ones among them (3 x 96 MB: 3 to 10 ms in place of
// 2.0).  No byte is written, so that a copy that fails leaves the caller's data;
// memory that cannot be written (or a kernel without the call) is left to the
// copy to report.
inline void populate_pages(void* dst, std::size_t bytes)
{
    static const std::uintptr_t page = (std::uintptr_t)sysconf(_SC_PAGESIZE);
    if (dst == nullptr || bytes == 0) return;
    const std::uintptr_t begin = reinterpret_cast<std::uintptr_t>(dst) & ~(page - 1);
    const std::uintptr_t end = reinterpret_cast<std::uintptr_t>(dst) + bytes;
    if (madvise(reinterpret_cast<void*>(begin), (std::size_t)(end - begin), MADV_POPULATE_WRITE) != 0) return;
    for (std::uintptr_t p = begin; p < end; p += page) (void)*reinterpret_cast<const volatile char*>(p);
}
}  // namespace mrmd_impl
