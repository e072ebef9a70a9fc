// Book-keeping of the persistent emulated-FP64 update's asynchronous work (k_update_oz), apart
// from its memory traffic, so that the host tests can run it against a model of the barriers.
#pragma once

#ifdef __CUDACC__
#define SK_HD __host__ __device__ __forceinline__
#else
#define SK_HD inline
#endif

namespace sankhya {
namespace dev {

// The phases that one warp has started on its mbarriers (a copy or a batch of MMAs each, one
// outstanding per barrier), as bits: barriers used, and whether their phases are an odd number.
struct PhaseLog {
    unsigned used = 0, odd = 0;
    SK_HD void start(int bar) {
        used |= 1u << bar;
        odd ^= 1u << bar;
    }
    SK_HD bool any(int bar) const { return (used >> bar) & 1u; }
    // parity to wait with for the last phase started: the n-th has parity (n - 1) & 1
    SK_HD unsigned last_parity(int bar) const { return ((odd >> bar) & 1u) ^ 1u; }
};

// Several warps run down a list of tiles, some of which end in code with unbounded barriers. A
// warp whose bounded wait for its next tile ran out may leave only if none of the others has
// joined the barriers that come next for it, and none joins them once it has left: the first to
// swap `state` decides. It holds the number of such tiles that were joined, or kApart for good;
// n: those that this warp has seen. compare_and_swap(expected, desired) works on `state` and
// returns its old value.
constexpr int kApart = -1;
// With the tile in hand: true if this warp takes part, as then all the others do.
template <class Cas>
SK_HD bool join(int n, Cas&& compare_and_swap) {
    const int old = compare_and_swap(n, n + 1);
    return old == n || old == n + 1;
}
// After a time-out: true if this warp may leave. If not, another warp is further on, so that
// the tile waited for is there.
template <class Cas>
SK_HD bool leave(int n, Cas&& compare_and_swap) {
    const int old = compare_and_swap(n, kApart);
    return old == n || old == kApart;
}

}  // namespace dev
}  // namespace sankhya
