// Host work of a table upload over a few threads of its own.
#pragma once
#include <algorithm>
#include <cstddef>
#include <thread>
#include <vector>

namespace esp {

// Parts for work of `items` steps of about 50 ns: a thread more for every 32 Ki
// of them (1.6 ms, against 20 us to start and join one), at most 4.
inline int work_parts(size_t items)
{
    return (int)std::min<size_t>(std::min(4u, std::max(1u, std::thread::hardware_concurrency())), 1 + (items >> 15));
}

// f(part) for every part, the first of them in the calling thread, and there
// too what finds no thread.
template <class F>
void for_parts(int parts, F &&f)
{
    std::vector<std::thread> th;
    int started = 1;
    try {
        th.reserve(parts);
        for (; started < parts; ++started) th.emplace_back([&f, started] { f(started); });
    } catch (...) {
    }
    f(0);
    for (int p = started; p < parts; ++p) f(p);
    for (std::thread &t : th) t.join();
}

}  // namespace esp
