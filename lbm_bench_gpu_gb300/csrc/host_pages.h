// host_pages.h -- page tables of a host buffer (no CUDA).
#pragma once

#include <cerrno>
#include <cstddef>
#include <cstdint>

#include <sys/mman.h>
#include <unistd.h>

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23   // Linux 5.14
#endif

namespace lbm {

// Map the pages of a buffer for writing until done() says that they are needed
// no longer, without a change to what they hold.  Memory that cannot be written
// or is not there, and a kernel without the call, are left alone: the caller's
// own write then does what it would have done.
template <typename Done>
inline void populate_pages(void *buf, size_t bytes, Done &&done)
{
    const long sys = sysconf(_SC_PAGESIZE);
    const uintptr_t page = sys > 0 ? (uintptr_t)sys : 4096, begin = (uintptr_t)buf & ~(page - 1);
    const uintptr_t end = ((uintptr_t)buf + bytes + page - 1) & ~(page - 1);
    const int saved = errno;
    for (uintptr_t at = begin; at < end; at += 8 * page) {
        const uintptr_t left = end - at;
        if (done() || madvise((void *)at, left < 8 * page ? left : 8 * page, MADV_POPULATE_WRITE) != 0) break;
    }
    errno = saved;
}

}  // namespace lbm
