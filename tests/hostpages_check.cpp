// Host check of chaos::populate_pages (csrc/chaos_hostpages.h).  Prints "ok", "old kernel", or the failure.
#include <cerrno>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "chaos_hostpages.h"

#define CHECK(c)                                              \
    do {                                                      \
        if (!(c)) {                                           \
            std::printf("line %d: %s\n", __LINE__, #c);       \
            std::exit(1);                                     \
        }                                                     \
    } while (0)

int main()
{
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), n = 8 * page;
    auto map = [&](int prot) {
        void *p = mmap(nullptr, n, prot, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
        CHECK(p != MAP_FAILED);
        return static_cast<unsigned char *>(p);
    };
    auto resident = [&](unsigned char *p) {
        std::vector<unsigned char> in(n / page);
        CHECK(mincore(p, n, in.data()) == 0);
        size_t k = 0;
        for (unsigned char v : in) k += v & 1u;
        return k;
    };
    {  // contents stay
        unsigned char *p = map(PROT_READ | PROT_WRITE);
        for (size_t k = 0; k < n; k++) p[k] = (unsigned char)(k * 7 + 3);
        chaos::populate_pages(p + 5, n - 9);
        for (size_t k = 0; k < n; k++) CHECK(p[k] == (unsigned char)(k * 7 + 3));
        munmap(p, n);
        // an address that is not mapped, and one that may not be written: left to the caller's own access
        chaos::populate_pages(p, n);
        unsigned char *q = map(PROT_READ);
        chaos::populate_pages(q, n);
        CHECK(q[n - 1] == 0);
        chaos::populate_pages(nullptr, 0);
        chaos::populate_pages(nullptr, 100);
    }
    {  // a fresh buffer's pages are there afterwards, also for a range that starts and ends inside pages
        unsigned char *p = map(PROT_READ | PROT_WRITE);
        if (madvise(p, page, MADV_POPULATE_WRITE) != 0 && errno == EINVAL) return std::puts("old kernel"), 0;
        unsigned char *q = map(PROT_READ | PROT_WRITE);
        CHECK(resident(q) == 0);
        chaos::populate_pages(q + page + 1, n - 2 * page - 2);
        CHECK(resident(q) == n / page - 2);
    }
    std::puts("ok");
    return 0;
}
