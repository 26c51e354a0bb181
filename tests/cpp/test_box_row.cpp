// Host check of box_row (fr_exact.cuh) over every box that reaches it: widths to 16,384,
// pixels to 2^20 (a medium triangle's box), at the first, last and a middle pixel of every
// row; the host's form, and the device's written out (the pixel biased by 2^23 in the float
// format, the product rounded down to an integer by adding 2^23). Exit status 0 = no difference.
#include <cstdio>
#include <cstring>
#include <initializer_list>

#include "fr_exact.cuh"

namespace
{

// x + 2^23 rounded down, for 0 <= x < 2^22.
float add_rd(float x)
{
    float r = x + 8388608.f;
    if (r - 8388608.f > x) r -= 1.f;  // exact: both are integers below 2^24
    return r;
}

int device_row(int l, float rw)
{
    const unsigned biased = 0x4b000000u | (unsigned)l;
    float b;
    std::memcpy(&b, &biased, 4);
    const float f = b - 8388607.5f;
    const float r = add_rd(f * rw);
    int i;
    std::memcpy(&i, &r, 4);
    return i - 0x4b000000;
}

}  // namespace

int main()
{
    long bad = 0, checked = 0;
    for (int w = 1; w <= 16384; ++w)
    {
        const float rw = 1.f / (float)w;
        for (int row = 0; row * (long)w < (1 << 20); ++row)
            for (int x : {0, w / 2, w - 1})
            {
                const long l = (long)row * w + x;
                if (l >= (1 << 20)) continue;
                ++checked;
                if ((frx::box_row((int)l, rw) != row || device_row((int)l, rw) != row) && bad++ < 10)
                    std::printf("width %d pixel %ld: %d, %d\n", w, l, frx::box_row((int)l, rw), device_row((int)l, rw));
            }
    }
    std::printf("checked %ld mismatches %ld\n", checked, bad);
    return bad == 0 ? 0 : 1;
}
