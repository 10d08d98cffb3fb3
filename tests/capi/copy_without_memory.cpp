// lfb_host_copy while allocations fail: the n-th operator new after arming
// throws, for every n that the copy reaches.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include "libfive_b200.h"

static long g_left = -1;   // allocations before one fails (-1: none does)
static long g_failed = 0;

void* operator new(std::size_t n)
{
    if (g_left == 0) {
        g_left = -1;
        ++g_failed;
        throw std::bad_alloc();
    }
    if (g_left > 0) --g_left;
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

int main()
{
    const std::size_t bytes = (std::size_t(33) << 20) + 5;   // eight threads
    std::vector<char> from(bytes), to(bytes);
    for (std::size_t i = 0; i < bytes; ++i) from[i] = static_cast<char>(i * 2654435761u >> 13);
    for (long n = 0; n < 30; ++n) {
        std::memset(to.data(), 0, bytes);
        g_left = n;
        lfb_host_copy(to.data(), from.data(), bytes);
        g_left = -1;
        if (std::memcmp(to.data(), from.data(), bytes) != 0) {
            std::printf("differs at %ld\n", n);
            return 1;
        }
    }
    std::printf("failed allocations: %ld\n", g_failed);
    return g_failed > 0 ? 0 : 2;
}
