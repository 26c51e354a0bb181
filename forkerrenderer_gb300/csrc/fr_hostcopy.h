// Host copies of downloaded frames (no CUDA).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <thread>

namespace fr
{

// dst = src, from 2 MiB by up to four threads (a fresh destination's page faults are
// most of its time). Never throws: what no thread can be had for is copied here.
inline void copy_bytes(unsigned char* dst, const unsigned char* src, size_t n)
{
    constexpr size_t kParts = 4;
    const size_t parts = std::min(kParts, n >> 20);
    if (parts < 2)
    {
        if (n) std::memcpy(dst, src, n);
        return;
    }
    const size_t step = ((n + parts - 1) / parts + 65535) & ~(size_t)65535;  // parts of them cover n
    std::thread ts[kParts - 1];
    size_t started = 0, at = step;
    try
    {
        for (; at < n; at += step, ++started)
            ts[started] = std::thread([=] { std::memcpy(dst + at, src + at, std::min(step, n - at)); });
    }
    catch (...)  // no thread, or no memory for its state
    {
        std::memcpy(dst + at, src + at, n - at);
    }
    std::memcpy(dst, src, step);
    for (size_t i = 0; i < started; ++i) ts[i].join();
}

}  // namespace fr
