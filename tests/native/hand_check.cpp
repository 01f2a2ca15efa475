/* Host check of the hand-over list's slots (pt_hand.h): threads in the place of
 * warps add 1..32 to the count of one list until several in a row found it
 * full, round after round.  Every slot below the written ones' number must have
 * been given out or marked as empty exactly once, and none above it.
 * Usage: hand_check <rounds> <threads>; exits 1 on a violation. */
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>

#include "pt_hand.h"

int main(int argc, char **argv)
{
    const int rounds = argc > 1 ? std::atoi(argv[1]) : 200, nt = argc > 2 ? std::atoi(argv[2]) : 8;
    const unsigned cap = 257;
    long long given = 0, marked = 0, partial = 0;
    for (int r = 0; r < rounds; ++r) {
        std::atomic<unsigned long long> count{ 0 };
        std::vector<std::atomic<int>> owner(cap);
        for (auto &o : owner) o = 0;
        std::atomic<long long> g{ 0 }, k{ 0 }, part{ 0 };
        std::atomic<bool> go{ false };
        auto work = [&](unsigned seed) {
            while (!go) {}
            for (int full = 0; full < 8;) {
                seed = seed * 1664525u + 1013904223u;
                const unsigned n = 1 + (seed >> 16) % 32;
                const unsigned long long at = count.fetch_add(n);
                if (pt_hand_fits(at, n, cap)) {
                    for (unsigned i = 0; i < n; ++i) ++owner[at + i];
                    g += n;
                    continue;
                }
                ++full;
                if (pt_hand_marks(at, cap)) ++part;
                for (unsigned i = 0; i < n; ++i)
                    if (pt_hand_marks(at + i, cap)) { ++owner[at + i]; ++k; }
            }
        };
        std::vector<std::thread> th;
        for (int t = 0; t < nt; ++t) th.emplace_back(work, 77u * r + t);
        go = true;
        for (auto &t : th) t.join();
        bool bad = false;
        const unsigned long long written = pt_hand_written(count.load(), cap);
        for (unsigned i = 0; i < cap; ++i)
            if (owner[i] != (i < written ? 1 : 0)) bad = true;
        if (bad || part > 1 || g + k != (long long)written) {
            std::printf("round %d: written %llu, given %lld\n", r, written, (long long)g);
            return 1;
        }
        given += g;
        marked += k;
        partial += part;
    }
    std::printf("given %lld marked %lld partial %lld\n", given, marked, partial);
    return 0;
}
