/* Host check of pt_hand_reserve: threads reserve ranges of 1..32 slots of one
 * list until several in a row found it full, round after round with the list
 * almost full from the start.  Every slot below the final count must have been
 * given out exactly once and none above it.
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
    const unsigned long long cap = 257;
    long long given = 0, refused = 0;
    for (int r = 0; r < rounds; ++r) {
        std::atomic<unsigned long long> count{ 0 };
        std::vector<std::atomic<int>> owner(cap);
        for (auto &o : owner) o = 0;
        std::atomic<long long> g{ 0 }, f{ 0 };
        std::atomic<bool> bad{ false }, go{ false };
        auto work = [&](unsigned seed) {
            while (!go) {}
            for (int full = 0; full < 8;) {
                seed = seed * 1664525u + 1013904223u;
                const unsigned long long n = 1 + (seed >> 16) % 32;
                auto cas = [&](unsigned long long expected, unsigned long long wanted) {
                    count.compare_exchange_strong(expected, wanted);
                    return expected;
                };
                const unsigned long long at = pt_hand_reserve(count.load(), n, cap, cas);
                if (at >= cap) { ++full; ++f; continue; }
                if (at + n > cap) { bad = true; return; }
                for (unsigned long long i = at; i < at + n; ++i) ++owner[i];
                g += (long long)n;
            }
        };
        std::vector<std::thread> th;
        for (int t = 0; t < nt; ++t) th.emplace_back(work, 77u * r + t);
        go = true;
        for (auto &t : th) t.join();
        for (unsigned long long i = 0; i < cap; ++i)
            if (owner[i] != (i < count.load() ? 1 : 0)) bad = true;
        if (bad || count.load() > cap || g != (long long)count.load()) {
            std::printf("round %d: count %llu, given %lld\n", r, count.load(), (long long)g);
            return 1;
        }
        given += g;
        refused += f;
    }
    std::printf("given %lld refused %lld\n", given, refused);
    return 0;
}
