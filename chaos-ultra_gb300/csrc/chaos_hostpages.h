// chaos_hostpages.h -- host pages brought in before a device-to-host copy.
#pragma once

#include <cstddef>
#include <cstdint>
#include <sys/mman.h>
#include <unistd.h>

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23
#endif

namespace chaos {

// Makes every page of [p, p + bytes) present and writable, as a write would,
// and changes no byte of it.  A range that is not mapped or may not be written,
// or a kernel before Linux 5.14, leaves the pages to the copy; so the copy's own
// answer stands.
inline void populate_pages(void *p, size_t bytes)
{
    if (!bytes) return;
    const long n = sysconf(_SC_PAGESIZE);
    const uintptr_t page = n > 0 ? (uintptr_t)n : 4096u;
    const uintptr_t from = (uintptr_t)p & ~(page - 1u), to = ((uintptr_t)p + bytes + page - 1u) & ~(page - 1u);
    (void)madvise(reinterpret_cast<void *>(from), to - from, MADV_POPULATE_WRITE);
}

}  // namespace chaos
