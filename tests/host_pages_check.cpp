// populate_pages (csrc/host_pages.h): contents unchanged, pages resident.  Prints one line
// per size; exit status 1 on a mismatch.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../dugks-gpu_gb300/csrc/host_pages.h"

int main(int argc, char **argv)
{
    int bad = 0;
    const size_t page = size_t(sysconf(_SC_PAGESIZE));
    for (int i = 1; i + 1 < argc; i += 2) {
        const size_t off = std::strtoull(argv[i], nullptr, 0), n = std::strtoull(argv[i + 1], nullptr, 0);
        const size_t len = (off + n + 2 * page) / page * page;
        unsigned char *m = static_cast<unsigned char *>(
            mmap(nullptr, len, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
        if (m == MAP_FAILED) return 2;
        for (size_t o = 0; o < len; o += 7 * page) m[o] = (unsigned char)(o / page + 1);
        dg::populate_pages(m + off, n);
        std::vector<unsigned char> in(len / page);
        if (mincore(m, len, in.data())) return 2;
        const size_t lo = (off + page - 1) / page, hi = (off + n) / page;
        size_t res = 0;
        for (size_t q = lo; q < hi; ++q) res += in[q] & 1;
        for (size_t o = 0; o < len; o += page) {
            const unsigned char want = o % (7 * page) ? 0 : (unsigned char)(o / page + 1);
            if (m[o] != want) bad = 1;
        }
        std::printf("%zu %zu %zu %zu\n", n, hi > lo ? hi - lo : 0, res, page);
        munmap(m, len);
    }
    return bad;
}
