// Host check of fr_hostcopy.h: copies of every part count, at odd addresses and odd
// lengths, leave the bytes around the destination alone; and with every allocation
// failing from the k-th on (a thread's state cannot be had) the copy is still whole and
// nothing is thrown. Exit status 0 = no difference.
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

#include "fr_hostcopy.h"

static long g_allow = -1;  // allocations that still succeed; < 0: all

void* operator new(size_t n)
{
    if (g_allow == 0) throw std::bad_alloc();
    if (g_allow > 0) --g_allow;
    void* p = std::malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

int main()
{
    const size_t MiB = 1 << 20;
    // one to four parts: one byte around each change of the part count, frames of odd
    // sizes (their bytes at three a pixel), and lengths whose last part is a few bytes
    const size_t sizes[] = {0, 1, 3, 2 * MiB - 1, 2 * MiB, 2 * MiB + 1, 3 * 1023 * 701, 3 * MiB - 1, 3 * MiB + 1,
                            3 * 1281 * 901, 4 * MiB - 1, 4 * MiB, 4 * MiB + 5, 3 * 1501 * 1001, 4 * 65536 * 17 - 1,
                            4 * 65536 * 17 + 1, 9 * MiB + 12345};
    const size_t most = 9 * MiB + 12345;
    std::vector<unsigned char> src(most + 16), dst(most + 64);
    for (size_t i = 0; i < src.size(); ++i) src[i] = (unsigned char)(i * 2654435761u >> 13);
    long bad = 0, copies = 0;
    for (size_t n : sizes)
        for (size_t off : {0, 1, 7})
            for (long allow = -1; allow <= 4; ++allow, ++copies)
            {
                std::fill(dst.begin(), dst.end(), (unsigned char)0xa5);
                g_allow = allow;
                fr::copy_bytes(dst.data() + 16 + off, src.data() + off, n);
                g_allow = -1;
                if (n && std::memcmp(dst.data() + 16 + off, src.data() + off, n)) ++bad;
                for (size_t i = 0; i < 16 + off; ++i) bad += dst[i] != 0xa5;
                for (size_t i = 16 + off + n; i < 16 + off + n + 16; ++i) bad += dst[i] != 0xa5;
            }
    std::printf("copies %ld differences %ld\n", copies, bad);
    return bad == 0 ? 0 : 1;
}
