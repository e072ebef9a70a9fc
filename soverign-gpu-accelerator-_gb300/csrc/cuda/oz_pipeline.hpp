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

}  // namespace dev
}  // namespace sankhya
