// Work shared out over host threads: every item is done once, also where the
// system grants no further thread (the address space is limited to less than a
// stack), and an exception reaches the caller after all threads have ended.
// Prints "0 failure(s)" on success.
#include "host/threads.hpp"

#include <sys/resource.h>

#include <atomic>
#include <cstdio>
#include <stdexcept>
#include <vector>

namespace {
int failures = 0;

void run(size_t threads, int items, int bad) {
    std::vector<std::atomic<int>> done(items);
    std::atomic<int> next{0};
    bool thrown = false;
    try {
        nsg::on_threads(threads, [&] {
            for (int i; (i = next.fetch_add(1)) < items;) {
                ++done[i];
                if (i == bad) throw std::runtime_error("item");
            }
        });
    } catch (const std::runtime_error&) {
        thrown = true;
    }
    if (thrown != (bad >= 0)) ++failures;
    if (bad < 0)
        for (auto& d : done) failures += d != 1;
}
}  // namespace

int main() {
    for (size_t threads : {0, 1, 2, 7, 64})
        for (int items : {0, 1, 5, 1000}) run(threads, items, -1);
    run(1, 10, 3);
    run(8, 1000, 500);
    rlimit lim{1 << 20, 1 << 20};  // below what the process maps already
    if (setrlimit(RLIMIT_AS, &lim) != 0) ++failures;
    for (size_t threads : {2, 16}) run(threads, 100, -1);
    std::printf("%d failure(s)\n", failures);
    return failures == 0 ? 0 : 1;
}
