// The hand-off between two groups of a walk's warps (tcq_handoff.cuh) with host threads in their place, built with the thread sanitizer and run by
// test_handoff.py: the leader publishes what it has written; a follower that reads it without having it would be reported as a race.
#include <thread>
#include <vector>

#include "../trellis-everywhere_b200/csrc/tcq_handoff.cuh"

constexpr int kThreads = 2;            // followers

static int order() {
    static int path[512], word = 0;
    long long sums[kThreads] = {};
    std::vector<std::thread> threads;
    for (int k = 0; k < kThreads; ++k)
        threads.emplace_back([&, k] {
            for (int n = 1; n <= 512; ++n) {
                while (tcq::handoff_count(word) < n) std::this_thread::yield();
                sums[k] += path[n - 1];
            }
        });
    for (int n = 0; n < 512; ++n) {
        path[n] = n;
        tcq::handoff_publish(word, n + 1);
        if (n % 16 == 0) std::this_thread::yield();
    }
    for (std::thread& t : threads) t.join();
    return sums[0] == 512 * 511 / 2 && sums[1] == sums[0] ? 0 : 1;
}

int main() { return order(); }
