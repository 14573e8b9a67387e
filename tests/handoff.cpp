// The hand-off between two groups of a walk's warps (tcq_handoff.cuh) with host threads in their place, built with the thread sanitizer and run by
// test_handoff.py.  Arguments: "order" (the leader publishes what it has written; a follower that reads it without having it would
// be reported as a race), or "limit" (one follower's clock runs out, another's does not).
#include <atomic>
#include <barrier>
#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>

#include "../trellis-everywhere_b200/csrc/tcq_handoff.cuh"

constexpr int kThreads = 2;            // followers: a thread for each of the two warps at K = 3

struct Shared {
    std::barrier<> barrier{kThreads};
    std::atomic<int> no[2] = {0, 0};
};
struct Group {
    Shared& sh;
    long long ticks = 0, step = 1;     // of this thread's clock
    int turn = 0;
    long long clock() { return ticks += step; }
    void pause() { std::this_thread::yield(); }
    bool all(bool x) {                 // (two words by turns, so that one barrier is enough)
        std::atomic<int>& no = sh.no[turn];
        if (!x) no = 1;
        sh.barrier.arrive_and_wait();
        const bool every = no == 0;
        sh.barrier.arrive_and_wait();
        no = 0;
        turn ^= 1;
        return every;
    }
};

static int order() {
    static int path[512], word = 0;
    Shared sh;
    long long sums[kThreads] = {};
    std::vector<std::thread> threads;
    for (int k = 0; k < kThreads; ++k)
        threads.emplace_back([&, k] {
            Group g{sh};
            for (int n = 1; n <= 512; ++n)
                if (tcq::handoff_wait(g, word, n, 1LL << 40)) sums[k] += path[n - 1];
        });
    for (int n = 0; n < 512; ++n) {
        path[n] = n;
        tcq::handoff_publish(word, n + 1);
        if (n % 16 == 0) std::this_thread::yield();
    }
    for (std::thread& t : threads) t.join();
    return sums[0] == 512 * 511 / 2 && sums[1] == sums[0] ? 0 : 1;
}

// The second follower's clock runs out, and only then does the leader publish, for which the first one still waits.
static int limit() {
    int word = 0;
    bool got[kThreads];
    std::atomic<bool> gave_up = false;
    Shared sh;
    std::vector<std::thread> threads;
    for (int k = 0; k < kThreads; ++k)
        threads.emplace_back([&, k] {
            struct Timed : Group {
                std::atomic<bool>& gave_up;
                Timed(Shared& s, std::atomic<bool>& u) : Group{s}, gave_up(u) {}
                bool all(bool x) {
                    if (!x) gave_up = true;
                    return Group::all(x);
                }
            } g(sh, gave_up);
            g.step = k == 0 ? 0 : 50;
            got[k] = tcq::handoff_wait(g, word, 1, 100);
            if (!got[k]) gave_up = true;
        });
    while (!gave_up) std::this_thread::yield();
    tcq::handoff_publish(word, 1);
    for (std::thread& t : threads) t.join();
    std::printf("outcomes %d %d\n", int(got[0]), int(got[1]));
    return got[0] || got[1];
}

int main(int, char** argv) { return std::strcmp(argv[1], "order") == 0 ? order() : limit(); }
