// The emulated-FP64 update's book-keeping (cuda/oz_pipeline.hpp) against a model of mbarriers:
// after any sequence of copies, ended at any point, the waits that PhaseLog asks for end when
// and only when nothing is in flight (waiting with a fixed parity does not: counted).
// Prints one JSON line; exit status 0 when all checks hold.
#include <cstdio>
#include <random>

#include "cuda/oz_pipeline.hpp"

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

}  // namespace

int main() {
    std::mt19937 rng(7);
    long leaves = 0;
    for (int k = 0; k < 20000; ++k) leaves += copies(rng);
    std::printf("{\"failed\": %ld, \"checks\": %ld, \"fixed_parity_leaves\": %ld}\n", failed, checks, leaves);
    return failed == 0 ? 0 : 1;
}
