// A few host threads beside the calling one, for the C entry points: nothing is thrown out of it.
#pragma once
#include <thread>

namespace q36 {

// work(0) on the calling thread and work(1) .. work(n - 1), n <= MAX, on threads of their own, until all are done.  A thread that
// cannot be had (no more of them: std::system_error; no memory for its state: std::bad_alloc) is left out with those after it:
// `work` hands out its items itself, so that whoever runs takes them all.
template <int MAX, typename F>
void run_on_threads(int n, F &work) {
    std::thread pool[MAX];
    int started = 1;
    try {
        for (; started < n; started++) pool[started] = std::thread([&work, w = started] { work(w); });
    } catch (...) {}
    work(0);
    for (int w = 1; w < started; w++) pool[w].join();
}

}  // namespace q36
