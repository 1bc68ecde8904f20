// host_pages.h -- the pages of a caller's host array (host calls only).
#pragma once

#include <stddef.h>
#include <stdint.h>
#include <sys/mman.h>
#include <unistd.h>

// madvise advice values of Linux 5.14+ (absent from older headers)
#ifndef MADV_POPULATE_READ
#define MADV_POPULATE_READ 22
#endif
#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23
#endif

namespace pg {

// Maps every page of [p, p + bytes) into the process, writable if `write`, without
// changing its contents.  False where that cannot be done: the range is not mapped to
// its end, may not be read (written), is a special mapping, or the kernel is older.
inline bool populate_pages(const void *p, size_t bytes, bool write)
{
    if (!p || !bytes) return true;
    static const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
    const uintptr_t lo = (uintptr_t)p & ~(page - 1);
    const uintptr_t hi = ((uintptr_t)p + bytes + page - 1) & ~(page - 1);
    return madvise((void *)lo, hi - lo, write ? MADV_POPULATE_WRITE : MADV_POPULATE_READ) == 0;
}

}  // namespace pg
