// The pool behind page-locked host memory (cuda/block_pool.hpp) on a counting backend: a block
// has one owner at a time, is used again, leaves when the pool is full, when it is dead or when
// memory runs out; from several threads too. Exit status 0 when all checks hold.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <random>
#include <set>
#include <thread>
#include <vector>

#include "cuda/block_pool.hpp"

namespace {

std::atomic<long> failed{0}, checks{0};
void check(bool ok, const char* what) {
    ++checks;
    if (!ok && failed++ < 10) std::fprintf(stderr, "failed: %s\n", what);
}

struct Backend {
    static std::mutex m;
    static std::set<void*> live, dead;
    static size_t limit;            // blocks at a time
    static long gets, puts;
    static void* get(size_t bytes) {
        std::lock_guard<std::mutex> lock(m);
        if (live.size() >= limit) return nullptr;
        void* p = std::malloc(bytes);
        live.insert(p);
        ++gets;
        return p;
    }
    static void put(void* p) {
        std::lock_guard<std::mutex> lock(m);
        check(live.erase(p) == 1, "put of a block that is not live");
        ++puts;
        std::free(p);
    }
    static bool alive(void* p) {
        std::lock_guard<std::mutex> lock(m);
        return dead.count(p) == 0;
    }
};
std::mutex Backend::m;
std::set<void*> Backend::live, Backend::dead;
size_t Backend::limit = ~size_t(0);
long Backend::gets = 0, Backend::puts = 0;

using Pool = sankhya::dev::BlockPool<Backend>;

void one_thread() {
    Pool pool;
    size_t a = 0, b = 0;
    void* p = pool.take(16, a);
    check(p && a == Pool::kMinBlock, "smallest size");
    pool.give(p, a);
    const long gets = Backend::gets;
    check(pool.take(a, b) == p && b == a && Backend::gets == gets, "used again");
    void* q = pool.take(a + 1, b);
    check(q && q != p && b == 2 * a, "next size");
    pool.give(p, a);
    pool.give(q, b);
    check(pool.kept() == a + b, "kept");
    // larger blocks are neither rounded nor kept
    void* big = pool.take(Pool::kMaxBlock + 8, b);
    check(big && b == Pool::kMaxBlock + 8, "large block");
    const long puts = Backend::puts;
    pool.give(big, b);
    check(Backend::puts == puts + 1, "large block leaves");
    // the bound
    std::vector<void*> all;
    for (int k = 0; k < 9; ++k) all.push_back(pool.take(Pool::kMaxBlock, b));
    for (void* x : all) pool.give(x, b);
    check(pool.kept() <= Pool::kMaxKept, "bound");
    // a dead block is dropped, not handed out and not put back
    pool.trim();
    check(pool.kept() == 0, "trim");
    p = pool.take(100, a);
    pool.give(p, a);
    Backend::dead.insert(p);
    Backend::live.erase(p);
    q = pool.take(100, a);
    check(q && q != p, "dead block");
    pool.give(q, a);
    Backend::dead.clear();
    // out of memory: what is kept is given back first
    Backend::limit = Backend::live.size();
    void* r = pool.take(2 * Pool::kMinBlock, b);
    check(r && b == 2 * Pool::kMinBlock && pool.kept() == 0, "kept blocks make room");
    check(pool.take(4 * Pool::kMinBlock, a) == nullptr, "none left");
    Backend::limit = ~size_t(0);
    pool.give(r, b);
    pool.trim();
    check(Backend::live.empty(), "all given back");
}

void many_threads() {
    Pool pool;
    std::vector<std::thread> th;
    for (int t = 0; t < 8; ++t)
        th.emplace_back([&, t] {
            std::mt19937 rng(static_cast<unsigned>(t));
            std::vector<std::pair<void*, size_t>> mine;
            for (int k = 0; k < 4000; ++k) {
                if (mine.size() < 4 && rng() % 2) {
                    size_t size = 0;
                    void* p = pool.take(1 + rng() % 20000, size);
                    std::memset(p, t, size);                       // an owner of its own
                    mine.push_back({p, size});
                } else if (!mine.empty()) {
                    const auto b = mine.back();
                    mine.pop_back();
                    const unsigned char* c = static_cast<const unsigned char*>(b.first);
                    check(c[0] == t && c[b.second - 1] == t, "block of another owner");
                    pool.give(b.first, b.second);
                }
            }
            for (const auto& b : mine) pool.give(b.first, b.second);
        });
    for (auto& t : th) t.join();
    check(pool.kept() <= Pool::kMaxKept, "bound after threads");
    pool.trim();
    check(Backend::live.empty(), "all given back after threads");
}

}  // namespace

int main() {
    one_thread();
    many_threads();
    std::printf("{\"failed\": %ld, \"checks\": %ld}\n", failed.load(), checks.load());
    return failed.load() == 0 ? 0 : 1;
}
