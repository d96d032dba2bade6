// Two threads' first calls that need different amounts: the limit must end at the larger one.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>

#include "../../singe_b200/csrc/raised_limit.cuh"

int main() {
    int done = 0;
    std::mutex mutex;
    std::atomic<int> limit{0};
    std::atomic<bool> small_inside{false};
    // the smaller call is interrupted just ahead of setting the limit
    std::thread small([&] {
        singe::raise_limit(60, done, mutex, [&](int needed) {
            small_inside = true;
            std::this_thread::sleep_for(std::chrono::milliseconds(300));
            limit = needed;
            return 0;
        });
    });
    while (!small_inside) std::this_thread::yield();
    auto set = [&](int needed) {
        limit = needed;
        return 0;
    };
    singe::raise_limit(100, done, mutex, set);
    small.join();
    if (limit != 100 || done != 100) {
        std::printf("limit %d, known %d\n", limit.load(), done);
        return 1;
    }
    // a smaller amount changes nothing, a refused one is asked for again
    int asked = 0;
    singe::raise_limit(80, done, mutex, [&](int) { return ++asked; });
    if (asked != 0) return 2;
    auto refuse = [&](int) {
        ++asked;
        return 7;
    };
    if (singe::raise_limit(200, done, mutex, refuse) != 7 || singe::raise_limit(200, done, mutex, refuse) != 7 || asked != 2 || done != 100) return 3;
    std::printf("raised limit ok\n");
    return 0;
}
