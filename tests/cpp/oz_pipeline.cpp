// The emulated-FP64 update's book-keeping (cuda/oz_pipeline.hpp) against a model of mbarriers:
//  * after any sequence of copies, ended at any point, the waits that PhaseLog asks for end when
//    and only when nothing is in flight (waiting with a fixed parity does not: counted);
//  * join() and leave(): of threads that run down a list of tiles, some of them late or without
//    patience, all or none come to a tile's barrier, and one that may not leave finds its tile.
// Prints one JSON line; exit status 0 when all checks hold.
#include <atomic>
#include <cstdio>
#include <random>
#include <thread>
#include <vector>

#include "cuda/oz_pipeline.hpp"

using sankhya::dev::join;
using sankhya::dev::leave;
using sankhya::dev::PhaseLog;

namespace {

long failed = 0, checks = 0;
void check(bool ok) {
    ++checks;
    if (!ok) ++failed;
}

// one phase at a time: started, then completed by its copy
struct Barrier {
    int phase = 0;
    bool in_flight = false;
    bool done(unsigned parity) const { return (static_cast<unsigned>(phase) & 1u) != parity; }   // try_wait.parity
    void complete() {
        ++phase;
        in_flight = false;
    }
};

// The copying warp's order of work: tile t fills B's buffer t & 1 (two halves) once the tile
// t - 2 is multiplied, and A's halves, where its rows are new, once the tile t - 1 is.
long copies(std::mt19937& rng) {
    Barrier bar[6];
    PhaseLog log;
    const int tiles = static_cast<int>(rng() % 12), stop = static_cast<int>(rng() % 25);
    int issued = 0;
    auto start = [&](int b) {
        if (bar[b].in_flight) bar[b].complete();       // its phase was waited for
        bar[b].in_flight = true;
        log.start(b);
    };
    for (int t = 0; t < tiles && issued < stop; ++t) {
        const bool fresh = t == 0 || rng() % 2;
        for (int h = 0; h < 2; ++h) start(2 + 2 * (t & 1) + h);
        if (++issued >= stop) break;                   // gives up between B's and A's copies
        if (fresh)
            for (int h = 0; h < 2; ++h) start(h);
    }
    for (auto& b : bar)
        if (b.in_flight && rng() % 2) b.complete();
    long fixed_parity_leaves = 0;
    for (int b = 0; b < 6; ++b) {
        check(log.any(b) || !bar[b].in_flight);
        if (!log.any(b)) continue;
        check(bar[b].done(log.last_parity(b)) == !bar[b].in_flight);
        if (bar[b].in_flight && bar[b].done(0)) ++fixed_parity_leaves;
        if (bar[b].in_flight) bar[b].complete();
        check(bar[b].done(log.last_parity(b)));
    }
    return fixed_parity_leaves;
}

// Eight warps take tiles from a ring: tile t is there once all of them are done with tile t - 3.
// A warp's wait ends without its tile when its patience does; a publisher that stops (trouble 2)
// lets every wait run out.
void tiles(std::mt19937& rng, long& together, long& apart, long& kept) {
    constexpr int W = 8, T = 12;
    const int trouble = static_cast<int>(rng() % 3), stop = trouble == 2 ? static_cast<int>(rng() % T) : T;
    bool first[T];
    for (bool& f : first) f = rng() % 2 != 0;
    std::atomic<int> state{0}, published{0}, stuck{0}, stays{0}, over{0};
    std::atomic<int> done[T] = {}, at_barrier[T] = {};
    int went[W][T] = {};
    std::vector<std::thread> th;
    for (int w = 0; w < W; ++w) {
        const unsigned seed = rng();
        th.emplace_back([&, w, seed] {
            std::mt19937 r(seed);
            auto cas = [&](int e, int d) {
                state.compare_exchange_strong(e, d);
                return e;
            };
            auto nap = [&](unsigned n) {
                for (unsigned k = n; k > 0; --k) std::this_thread::yield();
            };
            for (int t = 0, tri = 0; t < T; ++t) {
                for (bool there = false; !there;) {
                    const unsigned patience = trouble == 0 ? ~0u : r() % 8 == 0 ? r() % 20 : 20000;
                    for (unsigned k = 0; !there && k < patience; ++k) {
                        there = published.load() > t;
                        if (!there) std::this_thread::yield();
                    }
                    if (there) break;
                    if (leave(tri, cas)) {
                        over.fetch_add(1);
                        return;
                    }
                    stays.fetch_add(1);
                    if (published.load() <= t) stuck.fetch_add(1);     // must not be
                }
                if (trouble > 0 && r() % 4 == 0) nap(r() % 300);
                if (first[t] && join(tri++, cas)) {
                    went[w][t] = 1;
                    at_barrier[t].fetch_add(1);
                    long k = 0;
                    for (; at_barrier[t].load() < W && k < 20000000; ++k) std::this_thread::yield();
                    if (at_barrier[t].load() < W) stuck.fetch_add(1);  // a barrier without a limit
                }
                done[t].fetch_add(1);
            }
            over.fetch_add(1);
        });
    }
    for (int t = 0; t < stop && over.load() < W;) {
        if (t >= 3 && done[t - 3].load() < W) {
            std::this_thread::yield();
            continue;
        }
        published.store(++t);
    }
    for (auto& t : th) t.join();
    check(stuck.load() == 0);
    for (int t = 0; t < T; ++t) {
        int in = 0;
        for (int w = 0; w < W; ++w) in += went[w][t];
        check(in == 0 || in == W);                     // together or not at all
        if (!first[t]) check(in == 0);
        else if (trouble == 0) check(in == W);         // and together when nobody gives up
        if (in) ++together; else if (first[t]) ++apart;
    }
    kept += stays.load();
}

}  // namespace

int main() {
    std::mt19937 rng(7);
    long leaves = 0, together = 0, apart = 0, kept = 0;
    for (int k = 0; k < 20000; ++k) leaves += copies(rng);
    for (int k = 0; k < 1000; ++k) tiles(rng, together, apart, kept);
    std::printf("{\"failed\": %ld, \"checks\": %ld, \"fixed_parity_leaves\": %ld, \"together\": %ld, "
                "\"apart\": %ld, \"kept\": %ld}\n", failed, checks, leaves, together, apart, kept);
    return failed == 0 ? 0 : 1;
}
