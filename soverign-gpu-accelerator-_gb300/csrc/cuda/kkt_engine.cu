// Device normal-equation engine (see kkt_engine.hpp).
//
// Kernels, in the order one factorisation + solve runs them:
//   assembly    k_asm_*          D (A Theta A^T) D + delta I into the fronts
//   factor      k_potrf          Cholesky and inverse of a level's first 64x64 diagonal tiles; later
//                                ones are factored by the update before them (potrf_tile)
//               panel rows below the tile, X = B Linv^T:
//               k_trsm           FP32
//               k_trsm_rows      FP64 on the FP64 pipe
//               k_panel_oz       FP64 with BF16 digits on the tensor cores
//               trailing update C -= X_i X_j^T:
//               k_tc_split, k_update_tcs  FP32 on the tensor cores (TF32 x3); k_update without
//               k_update_split   FP64 on the FP64 pipe
//               k_update_oz      FP64 with BF16 digits on the tensor cores
//               k_extend_add     child update matrix into the parent front
//   solve       k_fwd_gather     frontal right-hand sides of one level
//               k_fwd_tasks      L z = r, dependency-driven 64-row block tasks
//               k_bwd_tasks      L^T x = z, same scheme in reverse
//   products    k_row_sums       A Theta A^T x and residuals
// Factorisation grids are lists of (front, tile) work items of one level / step, decoded by a
// warp-wide search over a prefix of per-front tile counts (find_item).
#include "cuda/kkt_engine.hpp"

#include "cuda/oz_pipeline.hpp"

#include <algorithm>
#include <cmath>
#include <stdexcept>
#include <type_traits>

namespace sankhya {
namespace dev {

struct PlanDev {
    const int* sn_first;
    const int* sn_ncols;
    const int* sn_nrows;
    const int* sn_lda;
    const int64_t* F_off;
    const int64_t* f_off;
    const int64_t* rows_off;
    const int* rows;
    const int64_t* ea_off;
    const int* ea_map;
    const int* ch_ptr;
    const int* ch_list;
    const int* sn_parent;
    const int* sn_lp;      // LP of each front (fronts never span LPs)
    const int* lp_on;      // 1 while an LP of the batch is still being solved; 0 skips its fronts
    int* lp_fail;          // per LP: set to 1 when one of its pivots was not positive
};

namespace {

constexpr int T64 = ipm::kTile;   // 64
constexpr int LDS = T64 + 1;      // padded leading dimension of shared tiles

struct StepArgs {
    int k;
    int item_off;
    int nitems;
    int tp_off;   // trsm prefix offset
    int up_off;   // update prefix offset (64x64 tiles)
    int up2_off;  // update prefix offset (128x128 blocks, tensor-core path)
    int up3_off;  // update prefix offset (128x64 blocks, emulated FP64 path)
    int dr_off;   // digit-row offsets of the items (emulated FP64 path)
};


// Largest i in [0, n) with prefix[i] <= b (prefix ascending, prefix[0] = 0 <= b). The
// whole warp searches (every lane must call it, converged, with the same arguments):
// each round probes 32 evenly spaced entries and keeps the segment after the last
// one <= b, so n <= 32 takes one dependent load and n <= 1024 two, where a binary
// search takes log2(n) (this sits at the head of every tile of a factorisation step).
__device__ __forceinline__ int find_item(const int* prefix, int n, int b) {
    const int lane = threadIdx.x & 31;
    int lo = 0, len = n;      // the answer lies in [lo, lo + len)
    while (len > 1) {
        const int step = (len + 31) >> 5;
        const int idx = lo + lane * step;
        const bool le = idx < lo + len && prefix[idx] <= b;
        const unsigned m = __ballot_sync(0xffffffffu, le);   // lane 0 probes lo: always set
        const int nlo = lo + (31 - __clz(m)) * step;
        len = min(step, lo + len - nlo);
        lo = nlo;
    }
    return lo;
}

// Item i and tile of update unit u in a grid of nitems + prefix[nitems] units: the first
// tile of every item comes first, because the block that finishes it goes on to factor the
// next diagonal tile, which takes longer than a whole tile of update; in the list's order
// the last front's factorisation was the kernel's tail. Result -1: nothing to do.
__device__ __forceinline__ int update_unit(const int* prefix, int nitems, int u, int& i) {
    const bool first = u < nitems;
    i = first ? u : find_item(prefix, nitems, u - nitems);
    const int lt = first ? 0 : u - nitems - prefix[i];
    return first ? (prefix[i + 1] > prefix[i] ? 0 : -1) : (lt > 0 ? lt : -1);
}

__device__ __forceinline__ void tri_index(int lt, int& ti, int& tj) {
    int t = static_cast<int>((sqrtf(8.0f * static_cast<float>(lt) + 1.0f) - 1.0f) * 0.5f);
    while ((t + 1) * (t + 2) / 2 <= lt) ++t;
    while (t > 0 && t * (t + 1) / 2 > lt) --t;
    ti = t;
    tj = lt - t * (t + 1) / 2;
}

// ------------------------------------------------------------------ assembly

// Diagonal of A Theta A^T and the equilibration D = 1/sqrt(max(|m_ii|, 1e-12))
// (reference src/cuda/kkt.cu:65-94). Row i of W holds a_ik^2 for the entries of
// row i of A, so the rows have A's row lengths: G lanes share a row, G being the
// width the SpMV autotuner chose for A.
template <int G>
__global__ void __launch_bounds__(256) k_asm_diag_sparse(int M, const int64_t* __restrict__ w_ptr,
                                                         const int* __restrict__ w_col,
                                                         const double* __restrict__ w_val,
                                                         const double* __restrict__ theta,
                                                         double* __restrict__ Mdiag, double* __restrict__ D) {
    const int64_t gid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int i = static_cast<int>(gid / G), lane = static_cast<int>(gid % G);
    const bool valid = i < M;
    double acc = 0.0;
    if (valid) {
        int64_t t = w_ptr[i] + lane;
        const int64_t t1 = w_ptr[i + 1];
        for (; t + 3 * G < t1; t += 4 * G) {   // four entries' loads in flight; same summation order
            const int c0 = w_col[t], c1 = w_col[t + G], c2 = w_col[t + 2 * G], c3 = w_col[t + 3 * G];
            const double v0 = w_val[t], v1 = w_val[t + G], v2 = w_val[t + 2 * G], v3 = w_val[t + 3 * G];
            const double h0 = theta[c0], h1 = theta[c1], h2 = theta[c2], h3 = theta[c3];
            acc += v0 * h0;
            acc += v1 * h1;
            acc += v2 * h2;
            acc += v3 * h3;
        }
        for (; t < t1; t += G) acc += w_val[t] * theta[w_col[t]];
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, G);
    if (valid && lane == 0) {
        Mdiag[i] = acc;
        D[i] = 1.0 / sqrt(fmax(fabs(acc), 1e-12));
    }
}

// Slots of LPs whose fronts are not being factored (lp_on 0) are left alone.
template <class T>
__global__ void k_asm_slots_sparse(int64_t nslots, int M, const int64_t* __restrict__ w_ptr,
                                   const int* __restrict__ w_col, const double* __restrict__ w_val,
                                   const double* __restrict__ theta, const int* __restrict__ si,
                                   const int* __restrict__ sj, const int64_t* __restrict__ pos,
                                   const double* __restrict__ Mdiag, const double* __restrict__ D,
                                   const double* __restrict__ params, const int* __restrict__ q_lp,
                                   const int* __restrict__ lp_on, T* __restrict__ F) {
    const int64_t s = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (s >= nslots) return;
    // every load that depends only on s first, then the ones they index, so a slot
    // waits for three rounds of loads rather than one per link of the chain
    const bool diag = s < M;
    const int i = diag ? static_cast<int>(s) : si[s];
    const int j = diag ? static_cast<int>(s) : sj[s];
    const int64_t p = pos[s];
    const int64_t t0 = diag ? 0 : w_ptr[s], t1 = diag ? 0 : w_ptr[s + 1];
    const double di = D[i], dj = D[j];
    const int on = lp_on[q_lp[i]];
    double acc = 0.0;
    for (int64_t t = t0; t < t1; ++t) acc += w_val[t] * theta[w_col[t]];
    if (!on) return;
    const double v = diag ? Mdiag[s] * di * di + params[0] : acc * di * dj;
    F[p] = static_cast<T>(v);
}

template <int G>
__global__ void __launch_bounds__(256) k_asm_diag_dense(int M, const int* __restrict__ rp, const int* __restrict__ ci,
                                                        const double* __restrict__ av,
                                                        const double* __restrict__ theta,
                                                        double* __restrict__ Mdiag, double* __restrict__ D) {
    const int64_t gid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int i = static_cast<int>(gid / G), lane = static_cast<int>(gid % G);
    const bool valid = i < M;
    double acc = 0.0;
    if (valid)
        for (int q = rp[i] + lane; q < rp[i + 1]; q += G) acc += av[q] * av[q] * theta[ci[q]];
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, G);
    if (valid && lane == 0) {
        Mdiag[i] = acc;
        D[i] = 1.0 / sqrt(fmax(fabs(acc), 1e-12));
    }
}

// Launches a diagonal kernel K<G> with G lanes per row (2, 4, 8, 16; else 32).
template <template <int> class K, class... Args>
void launch_diag(int M, int group, cudaStream_t st, Args... args) {
    if (M <= 0) return;
    const int64_t threads = static_cast<int64_t>(M) * group;
    const int blocks = static_cast<int>((threads + 255) / 256);
    switch (group) {
    case 2: K<2>::launch(blocks, st, M, args...); break;
    case 4: K<4>::launch(blocks, st, M, args...); break;
    case 8: K<8>::launch(blocks, st, M, args...); break;
    case 16: K<16>::launch(blocks, st, M, args...); break;
    default: K<32>::launch(blocks, st, M, args...); break;
    }
}
template <int G>
struct DiagSparse {
    template <class... A>
    static void launch(int blocks, cudaStream_t st, A... a) { k_asm_diag_sparse<G><<<blocks, 256, 0, st>>>(a...); }
};
template <int G>
struct DiagDense {
    template <class... A>
    static void launch(int blocks, cudaStream_t st, A... a) { k_asm_diag_dense<G><<<blocks, 256, 0, st>>>(a...); }
};

// One warp per column j of M (dense mode: one front per LP, natural order).
// Column j below the diagonal is sum_k a_jk theta_k A(:,k); the k loop is
// sequential so every entry is summed in a fixed order. The column ranges and
// coefficients of 32 k at a time are loaded by the lanes together and broadcast,
// and the rows, values and D of the next k are loaded before the current k's
// read-modify-write, so the loop carries one dependent memory round trip per k
// (the update of the front column) instead of four.
template <class T>
__global__ void k_asm_cols_dense(int M, const int* __restrict__ rp, const int* __restrict__ ci,
                                 const double* __restrict__ av, const int* __restrict__ tp,
                                 const int* __restrict__ ti, const double* __restrict__ tv,
                                 const double* __restrict__ theta, const double* __restrict__ Mdiag,
                                 const double* __restrict__ D, const int* __restrict__ row_lp, PlanDev pd,
                                 const double* __restrict__ params, T* __restrict__ F) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= M) return;
    const int j = warp;
    const int s = row_lp[j];
    if (!pd.lp_on[s]) return;            // dense mode: front s is LP s
    const int first = pd.sn_first[s];
    T* col = F + pd.F_off[s] + static_cast<int64_t>(j - first) * pd.sn_lda[s] - first;
    const double dj = D[j];
    const int q0 = rp[j], q1 = rp[j + 1];
    for (int qb = q0; qb < q1; qb += 32) {
        int ts = 0, te = 0;
        double cf = 0.0;
        if (qb + lane < q1) {
            const int k = ci[qb + lane];
            ts = tp[k];
            te = tp[k + 1];
            cf = av[qb + lane] * theta[k] * dj;
        }
        const int nq = min(32, q1 - qb);
        // first chunk (32 rows) of k = qb: loaded ahead
        int s0 = __shfl_sync(0xffffffffu, ts, 0), e0 = __shfl_sync(0xffffffffu, te, 0);
        int i0 = -1;
        double v0 = 0.0, d0 = 0.0;
        if (s0 + lane < e0) {
            i0 = ti[s0 + lane];
            v0 = tv[s0 + lane];
            d0 = D[i0];
        }
        for (int u = 0; u < nq; ++u) {              // nq is the same for every lane
            const double coef = __shfl_sync(0xffffffffu, cf, u);
            const int s1 = s0, e1 = e0, i1 = i0;
            const double v1 = v0, d1 = d0;
            if (u + 1 < nq) {                        // next k's first chunk
                s0 = __shfl_sync(0xffffffffu, ts, u + 1);
                e0 = __shfl_sync(0xffffffffu, te, u + 1);
                i0 = -1;
                if (s0 + lane < e0) {
                    i0 = ti[s0 + lane];
                    v0 = tv[s0 + lane];
                    d0 = D[i0];
                }
            }
            if (i1 > j) col[i1] = static_cast<T>(static_cast<double>(col[i1]) + coef * v1 * d1);
            for (int t = s1 + 32 + lane; t < e1; t += 32) {   // columns longer than 32 rows
                const int i = ti[t];
                if (i > j) col[i] = static_cast<T>(static_cast<double>(col[i]) + coef * tv[t] * D[i]);
            }
            __syncwarp();
        }
    }
    if (lane == 0) col[j] = static_cast<T>(Mdiag[j] * dj * dj + params[0]);
}

// ------------------------------------------------------------------- factor

// Cholesky of the 64x64 diagonal tile of step k of one front, in the front's precision T,
// plus the explicit inverse of the factored tile (used by the panel solve and by both
// triangular solves), stored column-major in Linv. A partial tile is padded with the
// identity. This runs in one block on the critical path of every 64-column step, by blocks
// of 16 columns: the 16x16 diagonal block, the rows below it, the trailing update. Every
// entry keeps its own ascending sequence of fused multiply-adds, roots and reciprocals, so the
// result does not depend on how the work is dealt out:
//  * FP32 is bound by the latency of the pivot chain, FP64 also by the SM's FP64 pipe: a
//    warp's FP64 instruction takes 64 cycles of its SM quarter whatever its active lanes, a
//    dependent one follows at once, and shuffles and shared loads queue with it (measured:
//    sqrt 600 cycles, a division 355, a 64-bit shuffle 16).
//  * So warp 0 alone factors the diagonal block, from registers (shuffles, no barrier),
//    while the warps of the other three quarters (helpers) apply the previous block's
//    update to the rows below (two of them first) and form the inverse's block rows that
//    are already known (four of them, in the last block all). Warp 0 joins them when its
//    block is done; warp 4 shares its quarter and stays out.
//  * The root and the reciprocal of an FP64 pivot take five dependent FP64 instructions
//    instead of a sqrt and a division.
// One tile: FP64 116 -> 53 us, FP32 38 -> 15 us.
constexpr int kPB = 16;
constexpr int kPBTri = kPB * (kPB + 1) / 2;

// These barriers count whole warps, which therefore meet first: a thread that reported a bad
// pivot, or left a loop early, may still be on its own.
// The barrier of the warps that extend the inverse, and the one on which the others wait for
// its block row.
__device__ __forceinline__ void inverse_sync(int threads) {
    __syncwarp();
    asm volatile("bar.sync 1, %0;" :: "r"(threads) : "memory");
}
__device__ __forceinline__ void inverse_arrive() {
    __syncwarp();
    asm volatile("bar.arrive 2, 224;" ::: "memory");
}
__device__ __forceinline__ void inverse_wait() {
    __syncwarp();
    asm volatile("bar.sync 2, 224;" ::: "memory");
}

// The 256 threads of a diagonal tile (the emulated update's block has two more warps).
__device__ __forceinline__ void tile_sync() {
    __syncwarp();
    asm volatile("bar.sync 3, 256;" ::: "memory");
}

__device__ __noinline__ void report_pivot(int s, const PlanDev& pd, int* err) {
    if ((threadIdx.x & 31) != 0) return;
    if (atomicCAS(err, 0, 1) == 0) err[1] = s;
    pd.lp_fail[pd.sn_lp[s]] = 1;
}

// Pivots that pivot_root() takes: positive, in FP64 also finite and so large that the
// residual p - d^2 is a normal number (tested without the FP64 pipe).
__device__ __forceinline__ bool plain_pivot(float p) { return p > 0.f; }
__device__ __forceinline__ bool plain_pivot(double p) {
    return static_cast<unsigned>(__double2hiint(p)) - 0x08000000u < 0x7ff00000u - 0x08000000u;
}

__device__ __forceinline__ float fma_ordered(float x, float y, float z) { return fmaf(x, y, z); }
// FP64: in program order with the other ordered ones.
__device__ __forceinline__ double fma_ordered(double x, double y, double z) {
    double r;
    asm volatile("fma.rn.f64 %0, %1, %2, %3;" : "=d"(r) : "d"(x), "d"(y), "d"(z));
    return r;
}

// d = sqrt(p) and rd = 1 / d, correctly rounded (p > 0). `fill(n)` is called between the
// parts, n = 0, 1, ..: independent work for the time they leave idle.
template <class Fill>
__device__ __forceinline__ void pivot_root(float p, float& d, float& rd, Fill fill) {
    d = sqrtf(p);
    rd = 1.f / d;
    for (int n = 0; n < 4; ++n) fill(n);
}
// FP64: y ~ p^(-1/2) to about 2^-45 without the FP64 pipe: the mantissa m in [1, 4) as two
// floats, the approximate unit's seed y0, e = 1 - m y0^2 with the square's low part, and one
// third-order step, whose correction is added to y0's bits as an integer. Then d0 = p y, the
// residual corrections d = d0 + (p - d0^2) y / 2 and rd = y + (1 - d y) y (Markstein 1990).
// Their last rounding is the correct one unless the exact value lies within about 2^-90 of a
// rounding boundary, where it may be the other neighbour: the reciprocal of 1 - j 2^-53, j odd
// and small, lies j^2 2^-106 from one and comes out a place low.
template <class Fill>
__device__ __forceinline__ void pivot_root(double p, double& d, double& rd, Fill fill) {
    const int hi = __double2hiint(p), lo = __double2loint(p);
    const unsigned ex = static_cast<unsigned>(hi) >> 20;
    const int odd = (static_cast<int>(ex) - 1023) & 1, half = (static_cast<int>(ex) - 1023 - odd) >> 1;
    const float mh = __int_as_float(((127 + odd) << 23) | ((hi & 0xfffff) << 3) |
                                    static_cast<int>(static_cast<unsigned>(lo) >> 29));
    const float ml = static_cast<float>(lo & 0x1fffffff) * (odd ? 0x1p-51f : 0x1p-52f);
    float y0;
    asm volatile("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(mh));
    fill(0);
    y0 = fminf(fmaxf(y0, 0.5f), 0x1.fffffep-1f);
    const float q = y0 * y0, ql = fmaf(y0, y0, -q);
    const float e = fmaf(-ml, q, fmaf(-mh, ql, fmaf(-mh, q, 1.f)));
    const float f = y0 * e * fmaf(0.375f, e, 0.5f) * 0x1p53f;       // in units of y0's last FP64 bit
    int c;
    asm volatile("cvt.rni.s32.f32 %0, %1;" : "=r"(c) : "f"(f));
    fill(1);
    long long bits = (static_cast<long long>(__float_as_int(y0)) << 29) + (896LL << 52) + c;
    bits -= static_cast<long long>(half) << 52;
    const double y = __longlong_as_double(bits), yh = __longlong_as_double(bits - (1LL << 52));
    const double d0 = fma_ordered(p, y, 0.0);
    fill(2);
    const double res = fma_ordered(__longlong_as_double(__double_as_longlong(d0) ^ (1LL << 63)), d0, p);
    d = fma_ordered(res, yh, d0);
    const double t = fma_ordered(__longlong_as_double(__double_as_longlong(d) ^ (1LL << 63)), y, 1.0);
    rd = fma_ordered(t, y, y);
    fill(3);
}

// The diagonal block at c0 from its column j on, for any pivot: one that is not positive
// counts as 1 (result true). Warp 0.
template <class T>
__device__ __noinline__ bool factor_rest(T* A, T* rdiag, int c0, int j) {
    const int lane = threadIdx.x & 31, r = c0 + (lane & 15);
    bool bad = false;
    for (; j < kPB; ++j) {
        const int c = c0 + j;
        T p = A[c * LDS + c];
        if (!(p > T(0))) {
            bad = true;
            p = T(1);
        }
        const T d = sqrt(p), rd = T(1) / d;
        __syncwarp();
        if (lane < kPB && r > c) A[r * LDS + c] *= rd;
        if (lane == 0) {
            A[c * LDS + c] = d;
            rdiag[c] = rd;
        }
        __syncwarp();
        if (r > c)
            for (int q = c + 1 + (lane >> 4); q <= r; q += 2) A[r * LDS + q] -= A[r * LDS + c] * A[q * LDS + c];
        __syncwarp();
    }
    return bad;
}

// Warp 0: the diagonal block at c0. Leaves L in A and 1 / L(c, c) in rdiag. Result: a pivot was
// not positive (it counts as 1). FP32: lane (r, h) holds the columns 2k + h of row r. Column j
// updates column j + 1 at once and the others while the next pivot's root forms.
__device__ __forceinline__ bool factor_block(float* A, float* rdiag, int c0) {
    const int lane = threadIdx.x & 31, r = lane & 15, h = lane >> 4;
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int c = 2 * k + h;
        v[k] = r >= c ? A[(c0 + r) * LDS + c0 + c] : 0.f;
    }
    float l = 0.f;
#pragma unroll
    for (int j = 0; j < kPB; ++j) {
        const float a = __shfl_sync(0xffffffffu, v[j >> 1], r + 16 * (j & 1));    // column j of every row
        const float p = __shfl_sync(0xffffffffu, v[j >> 1], j + 16 * (j & 1));
        auto update = [&](int k, int from) {           // columns 2k, 2k + 1 by column `from`
            const float lc = __shfl_sync(0xffffffffu, l, 2 * k + h);
            const float t = fmaf(-l, lc, v[k]);
            v[k] = 2 * k + h > from ? t : v[k];
        };
        float d, rd;
        const int rest = (j >> 1) + 1;                 // column j - 1's columns still to update: 2 rest ..
        if (!plain_pivot(p)) {
#pragma unroll
            for (int k = rest; k < 8; ++k)
                if (j > 0) update(k, j - 1);
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (2 * k + h >= j && r >= 2 * k + h) A[(c0 + r) * LDS + c0 + 2 * k + h] = v[k];
            __syncwarp();
            return factor_rest(A, rdiag, c0, j);
        }
        pivot_root(p, d, rd, [&](int n) {
            if (j == 0) return;
            if (rest + n < 8) update(rest + n, j - 1);
            if (n == 3)
#pragma unroll
                for (int k = rest + 4; k < 8; ++k) update(k, j - 1);
        });
        l = a * rd;
        if (j + 1 < kPB) update((j + 1) >> 1, j);
        if (h == 0 && r >= j) A[(c0 + r) * LDS + c0 + j] = r == j ? d : l;
        if (lane == 0) rdiag[c0 + j] = rd;
    }
    return false;
}

// FP64: lane r (and r + 16) holds row r of the column that is to be factored; the columns
// after it are packed into four registers a lane, the last column first, so that the entries
// still to be updated fill whole warps: a column costs its 7 dependent FP64 instructions and
// 1.7 for the others (as two columns a register 4.5: 1240 cycles a column, now 810). Column
// j - 1 updates them while column j's root forms, then column j + 1 leaves them.
__device__ __forceinline__ bool factor_block(double* A, double* rdiag, int c0) {
    const int lane = threadIdx.x & 31, r = lane & 15;
    constexpr int kSlots = 4;
    auto live = [](int j) { return (15 - j) * (16 - j) / 2; };       // entries in the columns after j
    double v[kSlots];
    double* at[kSlots];                                 // the entry's place
    int ri[kSlots], rq[kSlots];                         // its row and column of A, as offsets of their rows
    double* Ac = A + c0 * LDS + c0;
#pragma unroll
    for (int k = 0; k < kSlots; ++k) {
        int n, i;                                       // entry i of the n-th column from the last
        tri_index(min(lane + 32 * k, 119), n, i);
        const int q = 15 - n;
        ri[k] = (q + i) * LDS;
        rq[k] = q * LDS;
        at[k] = Ac + ri[k] + q;
        v[k] = *at[k];
    }
    double a = Ac[r * LDS], l = 0.0;
#pragma unroll
    for (int j = 0; j < kPB; ++j) {
        const double p = __shfl_sync(0xffffffffu, a, j);
        auto update = [&](int k) {                      // slot k by column j - 1
            v[k] = fma_ordered(-Ac[ri[k] + j - 1], Ac[rq[k] + j - 1], v[k]);
        };
        const int slots = (live(j) + 31) / 32;          // with columns after j
        if (!plain_pivot(p)) {
#pragma unroll
            for (int k = 0; k < kSlots; ++k)
                if (k < slots && j > 0) update(k);
            __syncwarp();
#pragma unroll
            for (int k = 0; k < kSlots; ++k)
                if (lane + 32 * k < live(j)) *at[k] = v[k];
            if (lane < kPB && r >= j) Ac[r * LDS + j] = a;
            __syncwarp();
            return factor_rest(A, rdiag, c0, j);
        }
        double d, rd, b = 0.0;
        pivot_root(p, d, rd, [&](int n) {
            if (j > 0 && n < slots) update(n);
            if (n == 3 && j + 1 < kPB) {                // column j + 1 leaves the slots
#pragma unroll
                for (int k = 0; k < kSlots; ++k)
                    if (32 * k < live(j) && 32 * k + 32 > live(j + 1) && lane + 32 * k >= live(j + 1) &&
                        lane + 32 * k < live(j))
                        *at[k] = v[k];
            }
        });
        __syncwarp();
        if (j + 1 < kPB) b = Ac[r * LDS + j + 1];       // rows above it are not used
        l = a * rd;
        if (lane < kPB && r >= j) Ac[r * LDS + j] = r == j ? d : l;
        if (lane == 0) rdiag[c0 + j] = rd;
        if (j + 1 < kPB) a = fma_ordered(-l, __shfl_sync(0xffffffffu, l, j + 1), b);
        __syncwarp();
    }
    return false;
}

// Rows below block c0 (nt of them): the block's columns of L. FP32: one thread per row.
__device__ __forceinline__ void panel_rows(float* A, const float* rdiag, int c0, int nt) {
    if (static_cast<int>(threadIdx.x) >= nt) return;
    float* row = A + (c0 + kPB + threadIdx.x) * LDS + c0;
    float x[kPB];
#pragma unroll
    for (int c = 0; c < kPB; ++c) x[c] = row[c];
#pragma unroll
    for (int q = 0; q < kPB; ++q) {
        x[q] = x[q] * rdiag[c0 + q];
#pragma unroll
        for (int c = q + 1; c < kPB; ++c) x[c] = fmaf(-x[q], A[(c0 + c) * LDS + c0 + q], x[c]);
    }
#pragma unroll
    for (int c = 0; c < kPB; ++c) row[c] = x[c];
}
// FP64: a warp takes 8 rows, lane (r, g) their columns 4k + g.
__device__ __forceinline__ void panel_rows(double* A, const double* rdiag, int c0, int nt) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (8 * wid >= nt) return;
    const int r = c0 + kPB + 8 * wid + (lane & 7), g = lane >> 3;
    double v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = A[r * LDS + c0 + 4 * k + g];
#pragma unroll
    for (int q = 0; q < kPB; ++q) {
        const double t = v[q >> 2] * rdiag[c0 + q];
        if (g == (q & 3)) v[q >> 2] = t;
        if (q == kPB - 1) break;
        const double x = __shfl_sync(0xffffffffu, t, (lane & 7) + 8 * (q & 3));
#pragma unroll
        for (int k = (q + 1) >> 2; k < 4; ++k)
            if (4 * k + g > q) v[k] = fma(-x, A[(c0 + 4 * k + g) * LDS + c0 + q], v[k]);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) A[r * LDS + c0 + 4 * k + g] = v[k];
}

// Entry e of the lower triangle that starts at c0 + 16, less the 16 columns at c0.
template <class T>
__device__ __forceinline__ void trail_entry(T* A, int c0, int e) {
    int i, j;
    tri_index(e, i, j);
    const T* a = A + (c0 + kPB + i) * LDS + c0;
    const T* b = A + (c0 + kPB + j) * LDS + c0;
    T v = a[kPB + j];
#pragma unroll
    for (int q = 0; q < kPB; ++q) v -= a[q] * b[q];
    A[(c0 + kPB + i) * LDS + c0 + kPB + j] = v;
}

// The same for a square of two rows and two columns (e: row by row).
template <class T>
__device__ __forceinline__ void trail_square(T* A, int c0, int e) {
    int i, j;
    tri_index(e, i, j);
    const T* a = A + (c0 + kPB + 2 * i) * LDS + c0;
    const T* b = A + (c0 + kPB + 2 * j) * LDS + c0;
    T* out = A + (c0 + kPB + 2 * i) * LDS + c0 + kPB + 2 * j;
    T v00 = out[0], v01 = i == j ? T(0) : out[1], v10 = out[LDS], v11 = out[LDS + 1];
#pragma unroll
    for (int q = 0; q < kPB; ++q) {
        const T a0 = a[q], a1 = a[LDS + q], b0 = b[q], b1 = b[LDS + q];
        v00 -= a0 * b0;
        v01 -= a0 * b1;
        v10 -= a1 * b0;
        v11 -= a1 * b1;
    }
    out[0] = v00;
    if (i != j) out[1] = v01;
    out[LDS] = v10;
    out[LDS + 1] = v11;
}

// The inverse's diagonal block at c0. FP32: thread j < 16 forms column j.
__device__ __forceinline__ void inverse_block(const float* A, float* X, const float* rdiag, int c0, int j) {
    if (j >= kPB) return;
    float x[kPB];
#pragma unroll
    for (int i = 0; i < kPB; ++i) x[i] = i == j ? 1.f : 0.f;
#pragma unroll
    for (int q = 0; q < kPB; ++q) {
        x[q] = x[q] * rdiag[c0 + q];
#pragma unroll
        for (int i = q + 1; i < kPB; ++i) x[i] = fmaf(-A[(c0 + i) * LDS + c0 + q], x[q], x[i]);
    }
#pragma unroll
    for (int i = 0; i < kPB; ++i)
        if (i >= j) X[(c0 + i) * LDS + c0 + j] = x[i];
}
// FP64: warps t / 32 < 4 take four columns each, lane (c, g) the rows 8k + g of column c.
__device__ __forceinline__ void inverse_block(const double* A, double* X, const double* rdiag, int c0, int t) {
    if (t >= 128) return;
    const int lane = t & 31, c = lane & 3, g = lane >> 2, j = (t >> 5) * 4 + c;
    double x[2] = {g == j ? 1.0 : 0.0, g + 8 == j ? 1.0 : 0.0};
#pragma unroll
    for (int q = 0; q < kPB; ++q) {
        const double t1 = x[q >> 3] * rdiag[c0 + q];
        if (g == (q & 7)) x[q >> 3] = t1;
        if (q == kPB - 1) break;
        const double xq = __shfl_sync(0xffffffffu, t1, c + 4 * (q & 7));
#pragma unroll
        for (int k = (q + 1) >> 3; k < 2; ++k)
            if (8 * k + g > q) x[k] = fma(-A[(c0 + 8 * k + g) * LDS + c0 + q], xq, x[k]);
    }
#pragma unroll
    for (int k = 0; k < 2; ++k)
        if (8 * k + g >= j) X[(c0 + 8 * k + g) * LDS + c0 + j] = x[k];
}

// Block row at r0 of the inverse: T(i, j) = sum_{j <= q < r0} L(i, q) X(q, j) for the
// columns j < r0, kept transposed in X's upper triangle (e: rows i, i + 8 of kCols columns),
// then X(i, j) = -sum_q X(i, r0 + q) T(r0 + q, j) (e: row i of kCols columns). FP32 is bound
// by its shared loads here and takes two columns at a time, FP64 by how evenly the
// warps' instructions are dealt out (with two columns 134k cycles a tile, with one 130k); a
// warp takes eight rows of four neighbouring columns, whose sums are about equally long (as two
// rows of sixteen columns 23% of its instructions had idle lanes).
template <class T> constexpr int kCols = sizeof(T) == 4 ? 2 : 1;

template <class T>
__device__ __forceinline__ void inverse_sums(const T* A, T* X, int r0, int e) {
    constexpr int C = kCols<T>;
    const int i = r0 + (e & 7), j = C * (e >> 3);
    const T* a = A + i * LDS;
    T u[C], v[C];
#pragma unroll
    for (int c = 0; c < C; ++c) u[c] = v[c] = T(0);
    if (C == 2) {
        u[0] = a[j] * X[j * LDS + j];
        v[0] = a[8 * LDS + j] * X[j * LDS + j];
    }
#pragma unroll 2
    for (int q = j + C - 1; q < r0; ++q) {
        const T a0 = a[q], a1 = a[8 * LDS + q];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const T x = X[q * LDS + j + c];
            u[c] += a0 * x;
            v[c] += a1 * x;
        }
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
        X[(j + c) * LDS + i] = u[c];
        X[(j + c) * LDS + i + 8] = v[c];
    }
}
template <class T>
__device__ __forceinline__ void inverse_rows(T* X, int r0, int e) {
    constexpr int C = kCols<T>;
    const int nj = r0 / C, i = r0 + e / nj, j = C * (e % nj);
    T u[C];
#pragma unroll
    for (int c = 0; c < C; ++c) u[c] = T(0);
    for (int q = r0; q <= i; ++q) {
        const T x = X[i * LDS + q];
#pragma unroll
        for (int c = 0; c < C; ++c) u[c] += x * X[(j + c) * LDS + q];
    }
#pragma unroll
    for (int c = 0; c < C; ++c) X[i * LDS + j + c] = -u[c];
}

template <class T>
__device__ __noinline__ void potrf_tile(int s, int kstep, PlanDev pd, T* F, T* __restrict__ Linv,
                                        const int64_t* __restrict__ inv_off, int* err, unsigned char* smraw) {
    T* A = reinterpret_cast<T*>(smraw);   // A[r * LDS + c], lower triangle
    T* X = A + T64 * LDS;                 // L^{-1}, same layout
    T* rdiag = X + T64 * LDS;             // 1 / L(c, c)
    int* next = reinterpret_cast<int*>(rdiag + T64);   // per block: the next 32 of its helpers' entries
    const int LD = pd.sn_lda[s];
    const int k0 = kstep * T64;
    const int w = min(T64, pd.sn_ncols[s] - k0);
    T* Fs = F + pd.F_off[s];
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
    {
        T x[16];                          // all of a thread's entries in flight together
#pragma unroll
        for (int it = 0; it < 16; ++it) {
            const int r = tid & 63, c = (tid >> 6) + 4 * it;
            x[it] = c <= r && r < w ? Fs[(k0 + r) + static_cast<int64_t>(k0 + c) * LD] : r == c ? T(1) : T(0);
        }
#pragma unroll
        for (int it = 0; it < 16; ++it) {
            const int r = tid & 63, c = (tid >> 6) + 4 * it;
            if (c <= r) A[r * LDS + c] = x[it];
        }
    }
    if (tid < 12) next[tid] = 0;
    tile_sync();
    const int ht = (wid < 4 ? wid - 1 : wid - 2) * 32 + lane;   // helpers: warps 1-3 and 5-7
    // 32 entries of [0, n) at a time, to whichever helper is free
    auto share = [&](int* counter, int n, auto&& work) {
        for (;;) {
            int e = 0;
            if (lane == 0) e = atomicAdd(counter, 32);
            e = __shfl_sync(0xffffffffu, e, 0);
            if (e >= n) break;
            if (e + lane < n) work(e + lane);
            __syncwarp();
        }
    };
    for (int c0 = 0; c0 < T64; c0 += kPB) {
        const int nt = T64 - kPB - c0;
        int* counter = next + (c0 / kPB) * 3;
        const bool helper = (wid & 3) != 0;
        if (wid == 0 && factor_block(A, rdiag, c0)) report_pivot(s, pd, err);
        if (c0 > 0) {
            if (wid != 4) {
                auto sums = [&] {
                    share(counter + 1, c0 * kPB / (2 * kCols<T>), [&](int e) { inverse_sums(A, X, c0, e); });
                };
                auto trail = [&] {                     // less the diagonal block's entries or squares
                    constexpr int C = kCols<T>, kDone = kPB / C * (kPB / C + 1) / 2;
                    share(counter + 2, (nt + kPB) / C * ((nt + kPB) / C + 1) / 2 - kDone, [&](int e) {
                        if constexpr (C == 2) trail_square(A, c0 - kPB, kDone + e);
                        else trail_entry(A, c0 - kPB, kDone + e);
                    });
                };
                // the inverse's block row: by four warps while the others update, by all six in the
                // last block, where there is nothing else
                const int ni = nt > 0 ? 128 : 192;
                if (helper && ht < ni) {
                    inverse_block(A, X, rdiag, c0 - kPB, ht);
                    inverse_sync(ni);
                    if (c0 > kPB)
                        share(counter, (c0 - kPB) * kPB / kCols<T>, [&](int e) { inverse_rows(X, c0 - kPB, e); });
                    inverse_sync(ni);
                    inverse_arrive();
                    sums();
                    trail();
                } else {
                    trail();
                    inverse_wait();
                    sums();
                }
            }
        }
        tile_sync();
        if (nt == 0) break;
        panel_rows(A, rdiag, c0, nt);
        tile_sync();
        if (tid < kPBTri) trail_entry(A, c0, tid);   // the next diagonal block
        tile_sync();
    }
    inverse_block(A, X, rdiag, T64 - kPB, tid);
    tile_sync();
    for (int e = tid; e < (T64 - kPB) * kPB / kCols<T>; e += 256) inverse_rows(X, T64 - kPB, e);
    tile_sync();
    T* Li = Linv + inv_off[s] + static_cast<int64_t>(kstep) * T64 * T64;
#pragma unroll
    for (int it = 0; it < 16; ++it) {
        const int idx = tid + it * 256;
        const int r = idx & 63, c = idx >> 6;
        const bool in = r < w && c <= r;
        if (in) Fs[(k0 + r) + static_cast<int64_t>(k0 + c) * LD] = A[r * LDS + c];
        Li[r + c * T64] = in ? X[r * LDS + c] : T(0);
    }
}

constexpr size_t potrf_smem(size_t elem) { return (2 * T64 * LDS + T64) * elem + 12 * sizeof(int); }

// Diagonal-tile Cholesky of the first step of each front of a level (later steps
// are factored at the end of the previous step's update, see k_update).
template <class T>
__global__ void __launch_bounds__(256) k_potrf(StepArgs a, const int* __restrict__ items, PlanDev pd, T* F,
                                               T* __restrict__ Linv, const int64_t* __restrict__ inv_off,
                                               int* err) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const int s = items[a.item_off + blockIdx.x];
    if (!pd.lp_on[pd.sn_lp[s]]) return;
    potrf_tile(s, a.k, pd, F, Linv, inv_off, err, smraw);
}

// FP32 panel rows below the diagonal tile: X = B L_kk^{-T} = B Linv^T (a small GEMM).
__global__ void __launch_bounds__(256) k_trsm(StepArgs a, const int* __restrict__ items,
                                              const int* __restrict__ prefix, PlanDev pd, float* F,
                                              const float* __restrict__ Linv, const int64_t* __restrict__ inv_off) {
    extern __shared__ __align__(16) unsigned char smraw[];
    float* Iv = reinterpret_cast<float*>(smraw);    // Linv column-major [q + c*64]
    float* B = Iv + T64 * T64;                   // B[c][r] (column-major)
    const int i = find_item(prefix + a.tp_off, a.nitems, blockIdx.x);
    const int s = items[a.item_off + i];
    if (!pd.lp_on[pd.sn_lp[s]]) return;
    const int lt = blockIdx.x - prefix[a.tp_off + i];
    const int N = pd.sn_nrows[s], K = pd.sn_ncols[s];
    const int LD = pd.sn_lda[s];
    const int k0 = a.k * T64;
    const int w = min(T64, K - k0);
    const int r0 = k0 + w + lt * T64;
    const int nr = min(T64, N - r0);
    float* Fs = F + pd.F_off[s];
    const float* Li = Linv + inv_off[s] + static_cast<int64_t>(a.k) * T64 * T64;
    const int tid = threadIdx.x;
    for (int idx = tid; idx < T64 * T64; idx += blockDim.x) Iv[idx] = Li[idx];
    for (int idx = tid; idx < T64 * T64; idx += blockDim.x) {
        const int r = idx & 63, c = idx >> 6;
        B[c * T64 + r] = (r < nr && c < w) ? Fs[(r0 + r) + static_cast<int64_t>(k0 + c) * LD] : 0.f;
    }
    __syncthreads();
    // X[r][c] = sum_{q <= c} B[r][q] Linv[c][q]; thread: row r, 16 columns
    const int r = tid & 63, cg = tid >> 6;
    float acc[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) acc[t] = 0.f;
    for (int q = 0; q < w; ++q) {
        const float bq = B[q * T64 + r];
#pragma unroll
        for (int t = 0; t < 16; ++t) acc[t] += bq * Iv[(cg * 16 + t) + q * T64];   // Linv[c][q], 0 when q > c
    }
    if (r < nr)
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            const int c = cg * 16 + t;
            if (c < w) Fs[(r0 + r) + static_cast<int64_t>(k0 + c) * LD] = acc[t];
        }
}

// FP64 panel rows below the diagonal tile, X = B Linv^T. Bound by the FP64 pipe (2560
// multiply-adds a row, 2 a cycle and SM), so a block takes only 2 W rows: two per warp, lane
// (row, c) their columns 16 b + c, each an ascending sum over the columns up to its own
// block's end (the inverse is 0 beyond its diagonal). With 64-row tiles a step took 69 us at
// any size up to 9700 rows; now 10 us up to 1200 rows and 26 us at 4700.
constexpr int kTrLd = T64 + 2;              // 16-byte aligned rows, no bank conflicts
constexpr size_t tr_smem(int warps) { return (T64 + 2 * warps) * kTrLd * sizeof(double); }

template <int W>
__global__ void __launch_bounds__(32 * W) k_trsm_rows(StepArgs a, const int* __restrict__ items,
                                                      const int* __restrict__ prefix, PlanDev pd, double* F,
                                                      const double* __restrict__ Linv,
                                                      const int64_t* __restrict__ inv_off) {
    constexpr int kRows = 2 * W, kParts = T64 / kRows, kT = 32 * W;
    extern __shared__ __align__(16) unsigned char smraw[];
    double* L = reinterpret_cast<double*>(smraw);   // the tile's inverse, L[c * kTrLd + q]
    double* X = L + T64 * kTrLd;                    // the block's rows, X[r * kTrLd + c]
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int sub = blockIdx.x % kParts, unit = blockIdx.x / kParts;
    const int i = find_item(prefix + a.tp_off, a.nitems, unit);
    const int s = items[a.item_off + i];
    if (!pd.lp_on[pd.sn_lp[s]]) return;
    const int N = pd.sn_nrows[s], LD = pd.sn_lda[s];
    const int k0 = a.k * T64;
    const int w = min(T64, pd.sn_ncols[s] - k0);
    const int r0 = k0 + w + (unit - prefix[a.tp_off + i]) * T64 + sub * kRows;
    const int nr = min(kRows, N - r0);
    if (nr <= 0) return;
    double* Fs = F + pd.F_off[s];
    const double* Li = Linv + inv_off[s] + static_cast<int64_t>(a.k) * T64 * T64;
    double l[T64 * T64 / kT], x[4];
#pragma unroll
    for (int it = 0; it < T64 * T64 / kT; ++it) l[it] = Li[tid + it * kT];
#pragma unroll
    for (int it = 0; it < 4; ++it) {
        const int idx = tid + it * kT, r = idx % kRows, c = idx / kRows;
        x[it] = r < nr && c < w ? Fs[(r0 + r) + static_cast<int64_t>(k0 + c) * LD] : 0.0;
    }
#pragma unroll
    for (int it = 0; it < T64 * T64 / kT; ++it) {
        const int idx = tid + it * kT;
        L[(idx & 63) * kTrLd + (idx >> 6)] = l[it];
    }
#pragma unroll
    for (int it = 0; it < 4; ++it) {
        const int idx = tid + it * kT;
        X[(idx % kRows) * kTrLd + idx / kRows] = x[it];
    }
    __syncthreads();
    const int c = lane & 15;
    double* xr = X + (2 * wid + (lane >> 4)) * kTrLd;
    double out[T64 / 16];
#pragma unroll
    for (int b = 0; b < T64 / 16; ++b) {
        const double* lc = L + (16 * b + c) * kTrLd;
        double v = 0.0;
#pragma unroll 2
        for (int q = 0; q < 16 * (b + 1); q += 4) {
            const double2 x0 = *reinterpret_cast<const double2*>(xr + q);
            const double2 x1 = *reinterpret_cast<const double2*>(xr + q + 2);
            const double2 l0 = *reinterpret_cast<const double2*>(lc + q);
            const double2 l1 = *reinterpret_cast<const double2*>(lc + q + 2);
            v = fma(x0.x, l0.x, v);
            v = fma(x0.y, l0.y, v);
            v = fma(x1.x, l1.x, v);
            v = fma(x1.y, l1.y, v);
        }
        out[b] = v;
    }
    __syncwarp();
#pragma unroll
    for (int b = 0; b < T64 / 16; ++b) xr[16 * b + c] = out[b];
    __syncthreads();
#pragma unroll
    for (int it = 0; it < 4; ++it) {
        const int idx = tid + it * kT, r = idx % kRows, q = idx / kRows;
        if (r < nr && q < w) Fs[(r0 + r) + static_cast<int64_t>(k0 + q) * LD] = X[r * kTrLd + q];
    }
}

// FP32 update without the tensor cores, C(64x64) -= A_i (64 x w) A_j^T; 256 threads, 4x4 outputs each. The C tile is
// read into registers and both panel tiles are staged with fully unrolled loads
// before any arithmetic, so every global load of a thread is in flight at once.
__global__ void __launch_bounds__(256) k_update(StepArgs a, const int* __restrict__ items,
                                                const int* __restrict__ prefix, PlanDev pd, float* F,
                                                float* __restrict__ Linv, const int64_t* __restrict__ inv_off,
                                                int* err) {
    extern __shared__ __align__(16) unsigned char smraw[];
    float* As = reinterpret_cast<float*>(smraw);     // [kk][r]
    float* Bs = As + T64 * T64;                  // [kk][c]
    int i;
    const int lt = update_unit(prefix + a.up_off, a.nitems, blockIdx.x, i);
    if (lt < 0) return;
    const int s = items[a.item_off + i];
    if (!pd.lp_on[pd.sn_lp[s]]) return;
    int ti, tj;
    tri_index(lt, ti, tj);
    const int N = pd.sn_nrows[s], K = pd.sn_ncols[s];
    const int LD = pd.sn_lda[s];
    const int k0 = a.k * T64;
    const int w = min(T64, K - k0);
    const int t0 = k0 + w;
    const int ri0 = t0 + ti * T64, cj0 = t0 + tj * T64;
    const int nri = min(T64, N - ri0), ncj = min(T64, N - cj0);
    float* Fs = F + pd.F_off[s];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    float cv[4][4];
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = ty * 4 + q, c = tx * 4 + p;
            const bool in = r < nri && c < ncj && (ti != tj || r >= c);
            cv[q][p] = in ? Fs[(ri0 + r) + static_cast<int64_t>(cj0 + c) * LD] : 0.f;
        }
    float va[16], vb[16];
#pragma unroll
    for (int it = 0; it < 16; ++it) {
        const int idx = tid + it * 256;
        const int r = idx & (T64 - 1), kk = idx >> 6;
        const int64_t cofs = static_cast<int64_t>(k0 + kk) * LD;
        va[it] = (kk < w && r < nri) ? Fs[ri0 + r + cofs] : 0.f;
        vb[it] = (kk < w && r < ncj) ? Fs[cj0 + r + cofs] : 0.f;
    }
#pragma unroll
    for (int it = 0; it < 16; ++it) {
        const int idx = tid + it * 256;
        As[idx] = va[it];
        Bs[idx] = vb[it];
    }
    __syncthreads();
    float acc[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int p = 0; p < 4; ++p) acc[q][p] = 0.f;
#pragma unroll 4
    for (int kk = 0; kk < w; ++kk) {
        float av[4], bv[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) { av[q] = As[kk * T64 + ty * 4 + q]; bv[q] = Bs[kk * T64 + tx * 4 + q]; }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int p = 0; p < 4; ++p) acc[q][p] += av[q] * bv[p];
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int r = ty * 4 + q, c = tx * 4 + p;
            if (r < nri && c < ncj && (ti != tj || r >= c))
                Fs[(ri0 + r) + static_cast<int64_t>(cj0 + c) * LD] = cv[q][p] - acc[q][p];
        }
    // The block that finished the first trailing diagonal tile factors it right away
    // (step k + 1's diagonal tile), overlapping the rest of this step's update.
    if (lt == 0 && t0 < K) {
        __syncthreads();
        potrf_tile(s, a.k + 1, pd, F, Linv, inv_off, err, smraw);
    }
}

// FP64 update on the FP64 pipe, in TS x TS parts of the 64x64 tiles. Bound by the pipe (two
// multiply-adds a cycle and SM): a 64x64 tile takes 65 us of one SM, a 32x32 part 16 us
// and a 16x16 part 4 us (plus its shared loads, two per product instead of one), so small
// trailing parts need the small parts to fill the chip, and large ones lose less in their
// last wave (m = 4001: update 23.2 ms with 64x64 tiles, 18.5 ms with 32x32 parts). The next
// diagonal tile is spread over several blocks: the last of them to finish (cnt, per front)
// factors it. Its FP64 work shares the pipe with the SM's other blocks, so while that tile
// decides the step's time a block asks for more than half of the SM's shared memory.
template <int TS>
__global__ void __launch_bounds__(256) k_update_split(StepArgs a, const int* __restrict__ items,
                                                      const int* __restrict__ prefix, PlanDev pd, double* F,
                                                      double* __restrict__ Linv, const int64_t* __restrict__ inv_off,
                                                      int* __restrict__ cnt, int* err) {
    constexpr int P = T64 / TS, E = TS / 16;        // parts per tile side, entries per thread and side
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ int last;
    double* As = reinterpret_cast<double*>(smraw);  // [kk][r]
    double* Bs = As + T64 * TS;                      // [kk][c]
    const int part = blockIdx.x % (P * P);
    int i;
    const int lt = update_unit(prefix + a.up_off, a.nitems, blockIdx.x / (P * P), i);
    if (lt < 0) return;
    const int s = items[a.item_off + i];
    if (!pd.lp_on[pd.sn_lp[s]]) return;
    int ti, tj;
    tri_index(lt, ti, tj);
    const int N = pd.sn_nrows[s], K = pd.sn_ncols[s];
    const int LD = pd.sn_lda[s];
    const int k0 = a.k * T64;
    const int w = min(T64, K - k0);
    const int t0 = k0 + w;
    const int si = part / P, sj = part % P;
    const int ri0 = t0 + ti * T64 + si * TS, cj0 = t0 + tj * T64 + sj * TS;
    const bool diag = ri0 == cj0;
    if (ri0 >= N || cj0 >= N || ri0 < cj0) return;
    const int nri = min(TS, N - ri0), ncj = min(TS, N - cj0);
    double* Fs = F + pd.F_off[s];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;          // rows E * tx .., columns E * ty ..
    double cv[E][E];
#pragma unroll
    for (int p = 0; p < E; ++p)
#pragma unroll
        for (int q = 0; q < E; ++q) {
            const int r = tx * E + q, c = ty * E + p;
            const bool in = r < nri && c < ncj && (!diag || r >= c);
            cv[q][p] = in ? Fs[(ri0 + r) + static_cast<int64_t>(cj0 + c) * LD] : 0.0;
        }
    double va[TS / 4], vb[TS / 4];
#pragma unroll
    for (int it = 0; it < TS / 4; ++it) {
        const int idx = tid + it * 256;
        const int r = idx & (TS - 1), kk = idx / TS;
        const int64_t cofs = static_cast<int64_t>(k0 + kk) * LD;
        va[it] = (kk < w && r < nri) ? Fs[ri0 + r + cofs] : 0.0;
        vb[it] = (kk < w && r < ncj) ? Fs[cj0 + r + cofs] : 0.0;
    }
#pragma unroll
    for (int it = 0; it < TS / 4; ++it) {
        const int idx = tid + it * 256;
        As[idx] = va[it];
        Bs[idx] = vb[it];
    }
    __syncthreads();
    double acc[E][E];
#pragma unroll
    for (int q = 0; q < E; ++q)
#pragma unroll
        for (int p = 0; p < E; ++p) acc[q][p] = 0.0;
#pragma unroll 4
    for (int kk = 0; kk < w; ++kk) {
        double av[E], bv[E];
#pragma unroll
        for (int q = 0; q < E; ++q) { av[q] = As[kk * TS + tx * E + q]; bv[q] = Bs[kk * TS + ty * E + q]; }
#pragma unroll
        for (int q = 0; q < E; ++q)
#pragma unroll
            for (int p = 0; p < E; ++p) acc[q][p] += av[q] * bv[p];
    }
#pragma unroll
    for (int p = 0; p < E; ++p)
#pragma unroll
        for (int q = 0; q < E; ++q) {
            const int r = tx * E + q, c = ty * E + p;
            if (r < nri && c < ncj && (!diag || r >= c))
                Fs[(ri0 + r) + static_cast<int64_t>(cj0 + c) * LD] = cv[q][p] - acc[q][p];
        }
    if (lt == 0 && t0 < K) {
        __threadfence();                             // this block's C writes, before the counter
        __syncthreads();
        if (tid == 0) {
            const int nb = (min(T64, N - t0) + TS - 1) / TS, parts = nb * (nb + 1) / 2;
            const int prev = atomicAdd(cnt + s, 1);
            last = prev == parts - 1;
            if (last) atomicExch(cnt + s, 0);
            __threadfence();
        }
        __syncthreads();
        if (last) potrf_tile(s, a.k + 1, pd, F, Linv, inv_off, err, smraw);
    }
}
constexpr size_t kSplitAlone = 120 * 1024;          // leaves room for one block per SM
template <int TS>
constexpr size_t split_smem() {
    return 2 * T64 * TS * sizeof(double) > potrf_smem(sizeof(double)) ? 2 * T64 * TS * sizeof(double)
                                                                      : potrf_smem(sizeof(double));
}

// ---- shared helpers of the tensor-core kernels (tcgen05) --------------------
// Shared-memory descriptors of the canonical K-major no-swizzle layout: 8-row x
// 16-byte core matrices, K-adjacent core matrices 128 B apart, 8-row groups 2048 B
// apart (64 four-byte elements per row).
constexpr uint32_t kTcLbo = 128;                     // bytes between K-adjacent core matrices
constexpr uint32_t kTcSbo = 2048;                    // bytes between 8-row groups (64 fp32 per row)

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint64_t tc_sdesc(uint32_t saddr) {
    uint64_t d = static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(kTcLbo >> 4) << 16;
    d |= static_cast<uint64_t>(kTcSbo >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;             // descriptor version bits 46-48 = 0b001
    return d;                                        // base offset 0, no swizzle
}
__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}

// ---- emulated FP64 trailing update on the tensor cores (BF16 digits) --------
// FP64 fronts of the late iterations of a mixed-precision solve. Each trailing
// row of the step's panel (its 64 L entries a_k) is written as
//     a_k = sum_{i=0..6} d_ik 2^(E - 7 - 8 i),   E = floor(log2 max_k |a_k|),
// with balanced base-256 digits (d_0 in [-256, 256], d_i in [-128, 127] for
// i >= 1): 56 bits, the row to 2^-56 of its largest entry. Every digit is an
// integer of at most 8 significant bits, exact in BF16 (k_panel_oz, once per
// panel row). C -= A B^T is then the sum over digit pairs (i, j); the pairs of
// one level L = i + j share the scale 2^(E_a + E_b - 14 - 8 L) and accumulate in
// one FP32 TMEM accumulator. With K <= 64 each level sum is an integer below
// 9 * 2^20 in magnitude (|d_0 e_0| <= 2^16, |d_0 e_j| <= 2^15, |d_i e_j| <= 2^14,
// at most L + 1 pairs of 64 products), so the tensor cores add it exactly. Levels
// 0..6 (28 pairs; the pairs beyond level 6 weigh below 2^-56 and are left out)
// are combined in 64-bit integers, hi = levels 0..2 and lo = levels 3..6, folded
// into u = hi 2^22 + round(lo 2^-10) (below 2^62 in magnitude) and applied with
// one FP64 subtraction per entry: C - u 2^(Ea+Eb-52) (GB300's FP64 pipe
// is the scarce resource of this epilogue).
// This is the error-free splitting of Ozaki, Ogita, Oishi and Rump (2012) with
// BF16 digits, exact FP32 tensor-core sums and an integer epilogue; the result
// agrees with an FP64 product to about 2^-53 of sum_k |a_k| |b_k|.
//
// Digit layout (global and shared alike): per digit plane i, K half h = k >> 5, row q
// and column k at byte i * plane + h * (plane / 2) + (q >> 3) * 512 + ((k & 31) >> 3) * 128
// + (q & 7) * 16 + (k & 7) * 2: within one half the canonical K-major no-swizzle layout
// of 8-row x 16-byte core matrices, so a block's 128 (32, 64) consecutive rows of one
// plane and half are one contiguous 8 KB (2 KB, 4 KB) bulk copy, and a block streams
// the two K halves through one buffer.

constexpr int kOzDigits = 7;
constexpr uint32_t kOzLbo = 128;                       // bytes between K-adjacent core matrices
constexpr uint32_t kOzSbo = 512;                       // bytes between 8-row groups (32 bf16 per row and half)
constexpr size_t kOzA = 128 * 64;                      // 128 rows of one plane and half: 8 KB
constexpr size_t kOzB = 64 * 64;                       // 64 rows: 4 KB
constexpr long long kOzCycles = 1LL << 31;             // how long a copy or an MMA batch may take: a second
// instruction descriptors (kind::f16): D = F32 (bits 4-5 = 1), A = B = BF16 (bits 7-9, 10-12 = 1),
// both K-major, N >> 3 at bits 17-22 (added per product), M >> 4 at bits 24-28 (M = 128)
constexpr uint32_t kOzIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 4) << 24);

__device__ __forceinline__ uint64_t oz_sdesc(uint32_t saddr) {
    uint64_t d = static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(kOzLbo >> 4) << 16;
    d |= static_cast<uint64_t>(kOzSbo >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    return d;
}
__device__ __forceinline__ double oz_pow2(int p) {       // 2^p, 0 below the normal range
    if (p < -1022) return 0.0;
    return __longlong_as_double(static_cast<long long>(p + 1023) << 52);
}
__device__ __forceinline__ bool oz_wait(uint32_t bar, uint32_t parity = 0, long long limit = kOzCycles,
                                        int polls = 4096) {
    uint32_t done = 0;
    const long long start = clock64();
    for (int spin = 0; !done; ++spin) {
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                     " selp.u32 %0, 1, 0, p;\n}\n" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        // back-to-back polls first: a copy or an MMA batch of one tile completes within
        // microseconds, and a sleep per poll adds its own latency to every tile
        if (!done && spin >= polls) __nanosleep(polls ? 32 : 1000);
        if (!done && (spin & 15) == 15 && clock64() - start > limit) break;
    }
    return done != 0;
}

// v 2^(55 - E) rounded to an integer (to nearest, ties to even; |v| < 2^(E + 1)), and u 2^e
// with u rounded to FP64, on the integer pipe: an FP64 instruction takes 64 cycles of its SM
// quarter here, and these conversions were most of the FP64 work of the digit kernels.
__device__ __forceinline__ long long oz_fixed(double v, int E) {
    const long long b = __double_as_longlong(v);
    const int ex = static_cast<int>(b >> 52) & 0x7ff;
    const long long m = ((b & 0xfffffffffffffLL) | (ex ? 1LL << 52 : 0LL)) << 3;
    const int n = min(max(E + 1023 - max(ex, 1), 0), 60);           // |v| = m 2^-n 2^(E - 55)
    const long long half = (1LL << n) >> 1, odd = n > 0 ? (m >> n) & 1 : 1;
    const long long f = (m + half - 1 + odd) >> n;
    return b < 0 ? -f : f;
}
__device__ __noinline__ double oz_value_any(long long u, int e) {
    return u == 0 ? 0.0 : static_cast<double>(u) * oz_pow2(e);
}
// e for which every u below 2^62 gives zero or a normal number
__device__ __forceinline__ bool oz_plain(int e) { return e >= -1000 && e <= 900; }
// The same for |u| of 2^32 or more (else `small` is set and the result is nothing) and plain e, without a
// branch.
__device__ __forceinline__ double oz_value(long long u, int e, bool& small) {
    const int s = static_cast<int>(u >> 32) >> 31;
    const unsigned long long a = (u ^ s) - s;                        // |u|, below 2^62
    const unsigned ah = static_cast<unsigned>(a >> 32);
    small |= ah == 0;
    const int n = __clz(static_cast<int>(ah)) - 1;
    const unsigned tl = static_cast<unsigned>(a) << n;               // its highest bit at 62
    const unsigned th = __funnelshift_l(static_cast<unsigned>(a), ah, n);
    const unsigned long long t = (static_cast<unsigned long long>(th) << 32) | tl;
    // 53 bits, ties to even; 2^53 carries over into the exponent
    const unsigned long long m = (t + 511 + ((tl >> 10) & 1)) >> 10;
    const unsigned hi = static_cast<unsigned>(m >> 32) + (static_cast<unsigned>(1084 - n + e) << 20);
    return __hiloint2double(static_cast<int>(hi | (static_cast<unsigned>(s) & 0x80000000u)), static_cast<int>(m));
}
// |v| for an integer maximum (a NaN counts as 0), and the exponent E of a row's largest one:
// at -968 or above, so that 2^(55 - E) stays a normal double (rows whose largest entry is
// below 2^-967 keep fewer digits; they do not matter next to 1); 0 for a row of zeros.
__device__ __forceinline__ long long oz_abs(double v) {
    const long long b = __double_as_longlong(v) & 0x7fffffffffffffffLL;
    return b <= 0x7ff0000000000000LL ? b : 0;
}
__device__ __forceinline__ int oz_exponent(long long mx) {
    return mx > 0 ? max(static_cast<int>(mx >> 52) - 1023, -968) : 0;
}

// The 7 balanced base-256 digits of NV entries v of row q (columns NV cg .., NV = 8 or 16)
// with row exponent E, as BF16 into the digit planes (layout above). With 128 added to each
// digit below the first they are the bytes of one integer; a byte in the last mantissa bits
// of 2^23 less 2^23 + 128 is the digit as a float, whose upper half is its BF16.
template <int NV>
__device__ __forceinline__ void oz_store_digits(const double* v, int E, int q, int cg, unsigned char* dig,
                                                int64_t plane, int64_t half) {
    uint32_t pk[kOzDigits][NV / 2];                 // BF16 digits per plane, packed in pairs
#pragma unroll
    for (int t = 0; t < NV; t += 2) {
        uint32_t w[2][kOzDigits];                   // the digits as float bits
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const long long f = oz_fixed(v[t + x], E) + 0x808080808080LL;
            const uint32_t lo = static_cast<uint32_t>(f), hi = static_cast<uint32_t>(f >> 32);
            w[x][0] = __float_as_uint(__uint_as_float(0x4B000000u + ((static_cast<int>(hi) >> 16) + 512)) - 8389120.f);
#pragma unroll
            for (int j = 1; j < kOzDigits; ++j) {
                const uint32_t word = j < 3 ? hi : lo;
                const int byte = j < 3 ? 2 - j : 6 - j;
                const uint32_t m = __byte_perm(word, 0x4B000000u, 0x7440u | byte);   // 2^23 + that byte
                w[x][j] = __float_as_uint(__uint_as_float(m) - 8388736.f);
            }
        }
#pragma unroll
        for (int j = 0; j < kOzDigits; ++j) pk[j][t >> 1] = __byte_perm(w[0][j], w[1][j], 0x7632u);
    }
    constexpr int G = 32 / NV;                      // column groups of a K half
    unsigned char* base = dig + (cg / G) * half + static_cast<int64_t>(q >> 3) * kOzSbo + (q & 7) * 16;
#pragma unroll
    for (int j = 0; j < kOzDigits; ++j)
#pragma unroll
        for (int h = 0; h < NV / 8; ++h)
            *reinterpret_cast<uint4*>(base + j * plane + ((cg % G) * (NV / 8) + h) * kOzLbo) =
                make_uint4(pk[j][4 * h], pk[j][4 * h + 1], pk[j][4 * h + 2], pk[j][4 * h + 3]);
}

// Lanes 0..6 of a warp: bulk copies of K half h of the 7 planes of `rows` digit rows from
// row q on into dst (plane after plane), completing on the mbarrier at bar.
__device__ __forceinline__ void oz_copy_rows(int h, uint32_t bar, unsigned char* dst, const unsigned char* dig,
                                             int64_t plane, int q, int rows) {
    const int lane = threadIdx.x & 31;
    const uint32_t bytes = static_cast<uint32_t>(rows) * 64;
    if (lane == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                     :: "r"(bar), "r"(kOzDigits * bytes) : "memory");
    __syncwarp();
    if (lane < kOzDigits) {
        const unsigned char* src = dig + lane * plane + h * (plane >> 1) + static_cast<int64_t>(q >> 3) * kOzSbo;
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     :: "r"(smem_addr(dst + lane * bytes)), "l"(src), "r"(bytes), "r"(bar) : "memory");
    }
    __syncwarp();
}

// One thread: the products of levels l0..l1-1 (at most four) over K half h, whose planes are
// at sa and sb; level L into TMEM columns 64 L .. 64 L + 63. Plane da of A meets the planes
// db of B with da + db in l0..l1-1; these follow one another in shared memory and their
// levels in TMEM, so that they are one product with N = 64 per plane: 20 instead of 56 MMAs
// a half, and A is read once for up to four planes (pair by pair a tile took 7,700 cycles,
// twice what its multiplications need).
__device__ __forceinline__ void oz_products(uint32_t tmem, uint32_t sa, uint32_t sb, int h, int l0, int l1) {
#pragma unroll
    for (int ks = 0; ks < 2; ++ks)
        for (int da = 0; da < l1; ++da) {
            const int L = max(l0, da);
            const uint32_t acc = (h > 0 || da > 0 || ks > 0) ? 1u : 0u;
            const uint32_t idesc = kOzIdesc | (static_cast<uint32_t>((l1 - L) * 64) >> 3 << 17);
            const uint64_t adesc = oz_sdesc(sa + da * static_cast<uint32_t>(kOzA) + ks * 2 * kOzLbo);
            const uint64_t bdesc = oz_sdesc(sb + (L - da) * static_cast<uint32_t>(kOzB) + ks * 2 * kOzLbo);
            asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                         " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                         :: "r"(tmem + static_cast<uint32_t>(64 * L)), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc));
        }
}
__device__ __forceinline__ void oz_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(bar) : "memory");
}

// One entry's sum from its level accumulators, in units of 2^(Ea+Eb-52): hi 2^(E-30) from the
// levels 0..2 plus lo 2^(E-62) from 3..6, lo rounded to 2^(E-53) (hi below 2^39.2, lo below
// 2^47.2). The multiply-adds are 32-bit as long as the levels' bounds (4, 4, 5, 6, 7, 8 and
// 9 * 2^20) allow it: every integer instruction takes two cycles here, a conversion eight.
__device__ __forceinline__ long long mad_wide(int x, int y, long long z) {
    long long d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(x), "r"(y), "l"(z));
    return d;
}
__device__ __forceinline__ int oz_int(uint32_t v) {           // in program order with sub_ordered
    int i;
    asm volatile("cvt.rni.s32.f32 %0, %1;" : "=r"(i) : "f"(__uint_as_float(v)));
    return i;
}
__device__ __forceinline__ double sub_ordered(double x, double y) {
    double d;
    asm volatile("sub.rn.f64 %0, %1, %2;" : "=d"(d) : "d"(x), "d"(y));
    return d;
}
// |v| <= 2^22: the last bits of 1.5 * 2^23 + v, less 0x4B400000
__device__ __forceinline__ uint32_t oz_int_biased(uint32_t v) {
    return __float_as_uint(__uint_as_float(v) + 12582912.f);
}
__device__ __forceinline__ long long oz_lower(const uint32_t* v, int stride) {
    const int b = oz_int(v[0]) * 256 + oz_int(v[stride]);
    const long long c = mad_wide(oz_int(v[2 * stride]), 256, static_cast<long long>(oz_int(v[3 * stride]) + 512));
    return mad_wide(b, 65536, c) >> 10;
}
__device__ __forceinline__ long long oz_sum(const uint32_t* v, int stride, long long lower) {
    const uint32_t a = oz_int_biased(v[stride]) * 256u + (static_cast<uint32_t>(oz_int(v[2 * stride])) - 0x40000000u);
    const long long u = mad_wide(static_cast<int>(a), 4194304, lower);
    const uint32_t hi = static_cast<uint32_t>(u >> 32) + (oz_int_biased(v[0]) << 6) - 0xD0000000u;
    return (static_cast<long long>(hi) << 32) | static_cast<uint32_t>(u);
}

__device__ __forceinline__ void tmem_load8(uint32_t* v, uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(addr));
}
__device__ __forceinline__ void tmem_load16(uint32_t* v, uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                   "=r"(v[15])
                 : "r"(addr));
}

// The integers u (sum = u 2^(Ea+Eb-52), below 2^62) of 8 columns from TMEM column c on, for
// this thread's lane.
__device__ __forceinline__ void oz_read8(uint32_t taddr, long long* u) {
    uint32_t v[kOzDigits * 8];
#pragma unroll
    for (int L = 0; L < kOzDigits; ++L) tmem_load8(v + 8 * L, taddr + static_cast<uint32_t>(64 * L));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int q = 0; q < 8; ++q) u[q] = oz_sum(v + q, 8, oz_lower(v + 24 + q, 8));
}

// Row block bi of block lb in a list where row block bi holds 2 bi + 2 blocks
// (bi (bi + 1) <= lb < (bi + 1)(bi + 2)); FP32 estimate corrected in integers (the
// FP64 pipe is kept for the epilogues).
__device__ __forceinline__ int block_row_of(int lb) {
    int bi = static_cast<int>((sqrtf(4.0f * static_cast<float>(lb) + 1.0f) - 1.0f) * 0.5f);
    while ((bi + 1) * (bi + 2) <= lb) ++bi;
    while (bi > 0 && bi * (bi + 1) > lb) --bi;
    return bi;
}

// C(128 x 64) -= A B^T from the digit planes, over the 128 x 64 blocks of the trailing lower
// part (row block bi holds column blocks 0..2bi+1). One block per SM stays for the whole step
// and takes runs of tiles from a counter, long ones first, so that the next tiles of a run find
// their 128 rows of A in shared memory (7 planes, 112 KB) and load only 64 rows of B (56 KB,
// two buffers). Warp 9 fetches tiles and copies, warp 8 issues the MMAs, warps 0..7 take the
// sums from TMEM (448 columns) to C, 32 columns a thread. The lower levels are multiplied
// first: their accumulators are free for the next tile as soon as they are in registers, while
// the upper levels' products run. Bound by the epilogue: of the 16,000 cycles that a tile takes
// at 3,260 rows an SM quarter's FP64 subtractions need 4,100 (64 cycles an instruction), its integer
// instructions 4,700 and its conversions 2,600, one after the other in each warp, so these are kept
// apart in neighbouring groups of columns and have no branch between them; the tensor pipe is busy
// for 22% of the time. The block
// with a front's first tile factors the next diagonal tile and waits for it without polling.
// As 128 x 32 tiles of blocks that copied, multiplied and subtracted in turn, two on an SM, a
// tile's half took 29,000 cycles: mean step at m = 4740 85 -> 69 us (there the diagonal tile is
// the limit), of 40 LPs (54,000 rows) 161 -> 110 us. Waits are bounded: on a
// time-out the block records err[2] and takes no further tile; at its end it waits, again with a
// limit, for the copies and MMAs that it has in flight, and frees its TMEM. The barriers of the
// diagonal tile have no limit, so the eight warps go there together or not at all (join()).
constexpr size_t kOzSmemU = kOzDigits * (2 * kOzA + 4 * kOzB) + 512;

struct OzTile {
    int s, r0, c0, qa, qb, N, LD;             // s < 0: no more tiles
    bool first, fresh;                        // factors the next diagonal tile; its rows of A are copied
    int64_t F;
};

__global__ void __launch_bounds__(320, 1) k_update_oz(StepArgs a, const int* __restrict__ items,
                                                      const int* __restrict__ prefix, PlanDev pd, double* F,
                                                      double* __restrict__ Linv, const int64_t* __restrict__ inv_off,
                                                      const unsigned char* __restrict__ dig,
                                                      const int* __restrict__ dexp, int64_t plane,
                                                      int* __restrict__ next, int* err) {
    extern __shared__ __align__(1024) unsigned char smraw[];
    constexpr int kA = kOzDigits * static_cast<int>(kOzA), kB = kOzDigits * static_cast<int>(kOzB);   // a K half
    unsigned char* As = smraw;                        // [half][plane]
    unsigned char* Bs = smraw + 2 * kA;               // [buffer][half][plane]
    uint64_t* bars = reinterpret_cast<uint64_t*>(Bs + 4 * kB);
    OzTile* slot = reinterpret_cast<OzTile*>(bars + 16);              // [4]
    uint32_t* tslot = reinterpret_cast<uint32_t*>(slot + 4);
    volatile int* fail = reinterpret_cast<volatile int*>(tslot + 1);
    int* joined = reinterpret_cast<int*>(tslot + 2);
    static_assert(16 * 8 + 4 * sizeof(OzTile) + 12 <= 512, "kOzSmemU");
    // A's halves, B's buffers and halves, the slots' descriptions; a tile's lower sums done, an
    // even and an odd tile's upper ones (the copying warp may look after the next is done too),
    // their accumulators free again, the diagonal tile factored
    const uint32_t bA = smem_addr(bars), bB = bA + 16, bTile = bA + 48, bLo = bA + 80, bHi = bA + 88,
                   bLoFree = bA + 104, bHiFree = bA + 112, bTri = bA + 120;
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int b = 0; b < 16; ++b)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bA + 8 * b), "r"(b < 13 ? 1 : 8));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *fail = *reinterpret_cast<volatile int*>(err + 2);   // an earlier step's time-out: no more tiles
        *joined = 0;
    }
    if (wid == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" :: "r"(smem_addr(tslot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot;
    // for another warp, whose own waits end before
    auto wait_warp = [&](uint32_t bar, int n, int code, int polls = 4096) {
        bool done = oz_wait(bar, n & 1, 2 * kOzCycles, polls);
        done = __all_sync(0xffffffffu, done);         // the warp goes on together
        if (!done && lane == 0) {
            *fail = 1;
            atomicExch(err + 2, code);
        }
        __syncwarp();
        return done;
    };
    // a copy or an MMA batch that does not complete
    auto wait_async = [&](uint32_t bar, int n) {      // the n-th phase of a barrier
        bool done = *fail == 0 && oz_wait(bar, n & 1);
        done = __all_sync(0xffffffffu, done);
        if (!done && lane == 0) {
            *fail = 1;
            atomicExch(err + 2, 1);
        }
        __syncwarp();
        return done;
    };
    PhaseLog issued;      // by warp 9: copies, on A's (0, 1) and B's (2 .. 5) barriers; by warp 8: batches, on bLo, bHi
    if (wid == 9) {
        const int* up = prefix + a.up3_off;
        const int grid = gridDim.x, total = a.nitems + up[a.nitems];
        int u = blockIdx.x, end = u + 1, last = grid;
        int item = -1, rows = -1;                     // whose rows are in As
        int tri = 0;
        bool first = false;                           // the tile before was a first one
        for (int t = 0;; ++t) {
            // the diagonal tile needs the SM's issue slots: no polling beside it
            if (first) wait_warp(bTri, tri++, 2, 0);
            OzTile w;
            w.s = -1;
            while (u < total && w.s < 0) {
                if (u >= end) {
                    // runs of half the block's share of what is left; first tiles one by one
                    const int run = last < a.nitems ? 1 : max(1, min(8, (total - last) / (2 * grid)));
                    if (lane == 0) u = grid + atomicAdd(next, run);
                    u = __shfl_sync(0xffffffffu, u, 0);
                    end = min(u + run, total);
                    last = u;
                    continue;
                }
                int i;
                const int lb = update_unit(up, a.nitems, u++, i);
                if (lb < 0) continue;
                const int s = items[a.item_off + i];
                if (!pd.lp_on[pd.sn_lp[s]]) continue;
                const int bi = block_row_of(lb), bj = lb - bi * (bi + 1);
                const int K = pd.sn_ncols[s], t0 = min(K, (a.k + 1) * T64);
                w.N = pd.sn_nrows[s];
                w.r0 = t0 + bi * 128;
                w.c0 = t0 + bj * T64;
                if (w.c0 >= w.N) continue;            // a column block past the front
                w.s = s;
                w.LD = pd.sn_lda[s];
                w.F = pd.F_off[s];
                w.qa = prefix[a.dr_off + i] + bi * 128;
                w.qb = prefix[a.dr_off + i] + bj * T64;
                w.first = lb == 0 && t0 < K;
                w.fresh = first || i != item || bi != rows;
                item = i;
                rows = bi;
            }
            const int buf = t & 1;
            bool ok = w.s >= 0 && *fail == 0;
            if (ok && t > 1) ok = wait_async(bHi + 8 * buf, (t - 2) >> 1);              // B's buffer is no longer read
            if (ok)
                for (int h = 0; h < 2; ++h) {
                    oz_copy_rows(h, bB + 16 * buf + 8 * h, Bs + (2 * buf + h) * kB, dig, plane, w.qb, 64);
                    issued.start(2 + 2 * buf + h);
                }
            if (ok && w.fresh) {
                if (t > 0) ok = wait_async(bHi + 8 * (buf ^ 1), (t - 1) >> 1);                // nor are A's rows
                if (ok)
                    for (int h = 0; h < 2; ++h) {
                        oz_copy_rows(h, bA + 8 * h, As + h * kA, dig, plane, w.qa, 128);
                        issued.start(h);
                    }
            }
            if (!ok) w.s = -1;
            first = w.first;
            if (lane == 0) {
                slot[t & 3] = w;
                mbar_arrive(bTile + 8 * (t & 3));
            }
            if (!ok) break;
        }
    } else if (wid == 8) {
        const uint32_t sa = smem_addr(As);
        int na = 0;
        for (int t = 0;; ++t) {
            if (!wait_warp(bTile + 8 * (t & 3), t >> 2, 3, t > 0 && slot[(t - 1) & 3].first ? 0 : 4096) ||
                slot[t & 3].s < 0) break;
            na += slot[t & 3].fresh;
            if (t > 0) wait_warp(bLoFree, t - 1, 4);
            const uint32_t sb = smem_addr(Bs) + (t & 1) * 2 * kB;
            bool ok = true;
            for (int h = 0; h < 2; ++h) {
                ok = ok && wait_async(bA + 8 * h, na - 1) && wait_async(bB + 16 * (t & 1) + 8 * h, t >> 1);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (ok && lane == 0) oz_products(tmem, sa + h * kA, sb + h * kB, h, 3, kOzDigits);
            }
            if (lane == 0) oz_commit(bLo);
            issued.start(0);
            if (t > 0) wait_warp(bHiFree, t - 1, 5);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (lane == 0) {
                if (ok)
                    for (int h = 0; h < 2; ++h) oz_products(tmem, sa + h * kA, sb + h * kB, h, 0, 3);
                oz_commit(bHi + 8 * (t & 1));
            }
            issued.start(1 + (t & 1));
            __syncwarp();
        }
    } else {
        const int row = 32 * (wid & 3) + lane, ch = 32 * (wid >> 2);      // this thread's row and columns
        const uint32_t tl = tmem + (static_cast<uint32_t>(32 * (wid & 3)) << 16) + static_cast<uint32_t>(ch);
        auto swap_joined = [&](int n, int v) {        // by lane 0, for the warp
            int old = 0;
            if (lane == 0) old = atomicCAS(joined, n, v);
            return __shfl_sync(0xffffffffu, old, 0);
        };
        bool left = false;
        for (int t = 0, tri = 0;; ++t) {
            while (!left && !wait_warp(bTile + 8 * (t & 3), t >> 2, 6)) left = leave(tri, swap_joined);
            if (left) break;
            const OzTile w = slot[t & 3];
            if (w.s < 0) break;
            const int r = w.r0 + row;
            // columns c0 + ch + j of row r for j < nj
            const int nj = r < w.N ? min(32, min(w.N, r + 1) - (w.c0 + ch)) : 0;
            double* C = F + w.F + r + static_cast<int64_t>(w.c0 + ch) * w.LD;
            const int ea = dexp[w.qa + row] - 52, eb = dexp[w.qb + ch + lane];
            const int elo = __reduce_min_sync(0xffffffffu, eb), ehi = __reduce_max_sync(0xffffffffu, eb);
            const bool plain = oz_plain(ea + elo) && oz_plain(ea + ehi);
            double cv[2][16];
            auto load_c = [&](int h) {
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    cv[h][j] = 16 * h + j < nj ? C[static_cast<int64_t>(16 * h + j) * w.LD] : 0.0;
            };
            load_c(0);
            wait_warp(bLo, t, 7);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            long long lo[32];
            {
                uint32_t v[4 * 32];
#pragma unroll
                for (int L = 0; L < 4; ++L) {
                    tmem_load16(v + 32 * L, tl + static_cast<uint32_t>(64 * (3 + L)));
                    tmem_load16(v + 32 * L + 16, tl + static_cast<uint32_t>(64 * (3 + L) + 16));
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(bLoFree);
#pragma unroll
                for (int j = 0; j < 32; ++j) lo[j] = oz_lower(v + j, 32);
            }
            wait_warp(bHi + 8 * (t & 1), t >> 1, 8);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int last = *fail == 0 ? nj : 0;
            // Eight columns at a time; their subtractions are issued between the integer work of
            // the next eight, which they would otherwise wait for and hold up. The vote at the end
            // of each comes after every access that is not the same for all lanes: it brings the
            // warp together for the next TMEM loads, which take a converged one (a __syncwarp before
            // them instead cost the 512-LP batch 0.8 %).
            double x[2][8];
            auto store = [&](int g) {
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (8 * g + q < last) C[static_cast<int64_t>(8 * g + q) * w.LD] = x[g & 1][q];
            };
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                uint32_t v[3 * 8];
#pragma unroll
                for (int L = 0; L < 3; ++L) tmem_load8(v + 8 * L, tl + static_cast<uint32_t>(64 * L + 8 * g));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (g == 1) load_c(1);
                if (g == 3) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bHiFree);
                }
                long long u[8];
                bool any = !plain;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    u[q] = oz_sum(v + q, 8, lo[8 * g + q]);
                    if (g > 0)
                        x[(g - 1) & 1][q] = sub_ordered(cv[(g - 1) >> 1][(8 * (g - 1) + q) & 15], x[(g - 1) & 1][q]);
                    x[g & 1][q] = oz_value(u[q], ea + __shfl_sync(0xffffffffu, eb, 8 * g + q), any);
                }
                if (g > 0) store(g - 1);
                if (__any_sync(0xffffffffu, any)) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const int e = ea + __shfl_sync(0xffffffffu, eb, 8 * g + q);
                        if (any) x[g & 1][q] = oz_value_any(u[q], e);
                    }
                    __syncwarp();
                }
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) x[1][q] = cv[1][8 + q] - x[1][q];
            store(3);
            if (w.first) {
                int in = 0;
                if (lane == 0) in = join(tri, [&](int n, int v) { return atomicCAS(joined, n, v); });
                ++tri;
                __threadfence();                      // C, before the other warps read it
                if (__shfl_sync(0xffffffffu, in, 0)) {
                    tile_sync();
                    potrf_tile(w.s, a.k + 1, pd, F, Linv, inv_off, err, smraw);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // before A is copied there again
                __syncwarp();
                if (lane == 0) mbar_arrive(bTri);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*fail != 0 && wid >= 8) {                     // what may still be in flight (else all was waited for)
        const uint32_t base = wid == 9 ? bA : bLo;
#pragma unroll 1
        for (int b = 0; b < 6; ++b)
            if (issued.any(b)) oz_wait(base + 8 * b, issued.last_parity(b));
    }
    if (wid == 8) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" :: "r"(tmem));
    }
}

// ---- FP64 panel solve on the tensor cores (the same digit products) ----------
// X = B Linv^T for 128 of the step's panel rows below the diagonal tile (B = their current
// values, Linv = the inverse of the factored diagonal tile), and the digits of X for the
// update. One block forms the digits of its rows of B and of the 64 rows of Linv in shared
// memory, runs the 28 digit pairs of both K halves as MMAs with M = 128, N = 64 (level L in
// TMEM columns 64 L ..), and takes X = u 2^(Ea+Eb-52) from the accumulators through the
// registers to the front and to the digit planes. Bound by the integer work of the digits
// and of the 64-bit sums (half of its 45,000 cycles; the MMAs take 4,000). As separate
// kernels (digits of B, of Linv, MMAs, digits of X, each through memory) a step took 33 us
// at m = 4740 and 112 us at 54,000 rows; now 24 and 90 us. Every wait is bounded: on a
// time-out the block records err[2], waits once more for what it issued and frees its TMEM.
constexpr size_t kOzPanelSmem = 2 * kOzDigits * (kOzA + kOzB) + 8 * 128 * sizeof(long long) +
                                (128 + 64) * sizeof(int) + 64;

__global__ void __launch_bounds__(512, 1) k_panel_oz(StepArgs a, const int* __restrict__ items,
                                                     const int* __restrict__ prefix, PlanDev pd, double* F,
                                                     const double* __restrict__ Linv,
                                                     const int64_t* __restrict__ inv_off,
                                                     unsigned char* __restrict__ dig, int* __restrict__ dexp,
                                                     int64_t plane, int* __restrict__ next, int* err) {
    extern __shared__ __align__(1024) unsigned char smraw[];
    if (blockIdx.x == 0 && threadIdx.x == 0) *next = 0;        // the update's tile counter
    unsigned char* As = smraw;
    unsigned char* Bs = As + 2 * kOzDigits * kOzA;                               // both [half][plane]
    long long* rmax = reinterpret_cast<long long*>(Bs + 2 * kOzDigits * kOzB);   // [4][128], then [8][64]
    int* ea = reinterpret_cast<int*>(rmax + 8 * 128);
    int* eb = ea + 128;
    uint64_t* bar = reinterpret_cast<uint64_t*>(eb + 64);                         // MMAs done
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);
    int* fail = reinterpret_cast<int*>(tslot + 1);
    const int i = find_item(prefix + a.dr_off, a.nitems, blockIdx.x * 128);
    const int s = items[a.item_off + i];
    if (!pd.lp_on[pd.sn_lp[s]]) return;
    const int blk = blockIdx.x - prefix[a.dr_off + i] / 128;
    const int N = pd.sn_nrows[s], K = pd.sn_ncols[s], LD = pd.sn_lda[s];
    const int k0 = a.k * T64;
    const int w = min(T64, K - k0);
    const int r0 = k0 + w + blk * 128;
    if (r0 >= N) return;                               // a padded block of the digit rows
    const int nra = min(128, N - r0);
    const int qa = prefix[a.dr_off + i] + blk * 128;
    double* Fs = F + pd.F_off[s];
    const double* Li = Linv + inv_off[s] + static_cast<int64_t>(a.k) * T64 * T64;   // column-major 64 x 64
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
    if (wid == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" :: "r"(smem_addr(tslot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_addr(bar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *fail = 0;
    }
    // B: row `brow`, columns 16 bg ..; Linv: row `lrow`, columns 8 lg ..
    const int brow = tid & 127, bg = tid >> 7, lrow = tid & 63, lg = tid >> 6;
    double v[16];
    {
        double l[8];
        long long ml = 0, mb = 0;
#pragma unroll
        for (int t = 0; t < 8; ++t) l[t] = Li[lrow + (lg * 8 + t) * T64];
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            const int k = 16 * bg + t;
            v[t] = brow < nra && k < w ? Fs[(r0 + brow) + static_cast<int64_t>(k0 + k) * LD] : 0.0;
        }
#pragma unroll
        for (int t = 0; t < 8; ++t) ml = max(ml, oz_abs(l[t]));
#pragma unroll
        for (int t = 0; t < 16; ++t) mb = max(mb, oz_abs(v[t]));
        rmax[bg * 128 + brow] = mb;
        rmax[512 + lg * 64 + lrow] = ml;
        __syncthreads();
        mb = max(max(rmax[brow], rmax[128 + brow]), max(rmax[256 + brow], rmax[384 + brow]));
#pragma unroll
        for (int g = 0; g < 8; ++g) ml = max(ml, rmax[512 + g * 64 + lrow]);
        const int eB = oz_exponent(mb), eL = oz_exponent(ml);
        if (bg == 0) ea[brow] = eB;
        if (lg == 0) eb[lrow] = eL;
        oz_store_digits<8>(l, eL, lrow, lg, Bs, kOzB, kOzDigits * kOzB);
        oz_store_digits<16>(v, eB, brow, bg, As, kOzA, kOzDigits * kOzA);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot;
    if (tid == 0) {
        const uint32_t sa = smem_addr(As), sb = smem_addr(Bs), b0 = smem_addr(bar);
        for (int h = 0; h < 2; ++h) {
            const uint32_t ah = sa + h * static_cast<uint32_t>(kOzDigits * kOzA);
            const uint32_t bh = sb + h * static_cast<uint32_t>(kOzDigits * kOzB);
            oz_products(tmem, ah, bh, h, 0, 3);
            oz_products(tmem, ah, bh, h, 3, kOzDigits);
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                     :: "r"(b0) : "memory");
        if (!oz_wait(b0)) {
            oz_wait(b0);                               // a second bounded wait before TMEM is freed
            *fail = 1;
            atomicExch(err + 2, 1);
        }
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const bool ok = *fail == 0;
    // X: row `row` (TMEM lane), columns ch ..
    const int row = 32 * (wid & 3) + lane, ch = 16 * (wid >> 2);
    long long mx = 0;
    if (ok) {
        const int er = ea[row];
#pragma unroll
        for (int c8 = 0; c8 < 2; ++c8) {
            __syncwarp();                              // the TMEM loads take a converged warp
            long long u[8];
            oz_read8(tmem + (static_cast<uint32_t>(32 * (wid & 3)) << 16) + static_cast<uint32_t>(ch + 8 * c8), u);
            bool any = false;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int e = er + eb[ch + 8 * c8 + q] - 52;
                any |= !oz_plain(e);
                v[8 * c8 + q] = oz_value(u[q], e, any);
            }
            if (__any_sync(0xffffffffu, any)) {
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (any) v[8 * c8 + q] = oz_value_any(u[q], er + eb[ch + 8 * c8 + q] - 52);
                __syncwarp();
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int j = 8 * c8 + q, col = ch + j;
                v[j] = row < nra && col < w ? v[j] : 0.0;
                if (row < nra && col < w) Fs[(r0 + row) + static_cast<int64_t>(k0 + col) * LD] = v[j];
                mx = max(mx, oz_abs(v[j]));
            }
        }
        rmax[(wid >> 2) * 128 + row] = mx;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (wid == 0) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" :: "r"(tmem));
    }
    if (!ok) return;
    const int E = oz_exponent(max(max(rmax[row], rmax[128 + row]), max(rmax[256 + row], rmax[384 + row])));
    oz_store_digits<16>(v, E, qa + row, ch / 16, dig, plane, plane >> 1);
    if (ch == 0) dexp[qa + row] = E;
}

// ---- FP32 trailing update on the tensor cores from pre-split panels -----------
// The step's trailing panel rows (64 FP32 entries each) are split once per step
// into TF32 parts hi = tf32(x), lo = tf32(x - hi) (k_tc_split, one block per 64-row
// trsm tile) and written to the digit buffer in the canonical K-major no-swizzle
// layout of 8-row x 16-byte core matrices (K-adjacent core matrices 128 B apart,
// 8-row groups 2048 B apart): a block's 128 (A) or 64 (B) consecutive rows are one
// contiguous 32 KB / 16 KB bulk copy per part. k_update_tcs then computes C(128 x 64)
// -= A B^T as lo_A hi_B + hi_A lo_B + hi_A hi_B (TF32 x3, close to FP32 accuracy):
// one thread copies the four parts with cp.async.bulk and issues the 24 MMAs (M=128,
// N=64, K=8) into 64 TMEM columns while every thread loads its 32 C values; 96 KB of
// shared memory and at most 128 registers per thread leave room for two blocks per
// SM. Blocks follow the 128-row x 64-column lower-part list of the emulated FP64
// update (row block bi holds column blocks 0..2bi+1). Every wait is bounded: on a
// time-out the block records err[2], waits once more for what it issued, frees its
// TMEM and leaves C untouched.
constexpr uint32_t kTsLbo = 128;                       // bytes between K-adjacent core matrices
constexpr uint32_t kTsSbo = 2048;                      // bytes between 8-row groups (64 FP32 per row)
constexpr size_t kTsA = 128 * 256;                     // 128 rows x 64 FP32: 32 KB per part
constexpr size_t kTsB = 64 * 256;                      // 64 rows: 16 KB per part
constexpr size_t kTsSmem = 2 * (kTsA + kTsB) + 64;
// instruction descriptor: D = F32 (bits 4-5 = 1), A = B = TF32 (bits 7-9, 10-12 = 2), both
// K-major, N >> 3 at bits 17-22 (N = 64), M >> 4 at bits 24-28 (M = 128)
constexpr uint32_t kTsIdesc = (1u << 4) | (2u << 7) | (2u << 10) | ((64u >> 3) << 17) | ((128u >> 4) << 24);

__global__ void __launch_bounds__(256) k_tc_split(StepArgs a, const int* __restrict__ items,
                                                  const int* __restrict__ prefix, PlanDev pd,
                                                  const float* __restrict__ F, unsigned char* __restrict__ dig,
                                                  int64_t plane) {
    const int i = find_item(prefix + a.tp_off, a.nitems, blockIdx.x);
    const int s = items[a.item_off + i];
    if (!pd.lp_on[pd.sn_lp[s]]) return;
    const int lt = blockIdx.x - prefix[a.tp_off + i];
    const int N = pd.sn_nrows[s], K = pd.sn_ncols[s], LD = pd.sn_lda[s];
    const int k0 = a.k * T64;
    const int w = min(T64, K - k0);
    const int t0 = k0 + w;
    const int r = threadIdx.x & 63, cg = threadIdx.x >> 6;
    const int row = t0 + lt * T64 + r;
    const bool rin = row < N;
    const float* Fs = F + pd.F_off[s];
    const int q = prefix[a.dr_off + i] + lt * T64 + r;
    unsigned char* base = dig + static_cast<int64_t>(q >> 3) * kTsSbo + (q & 7) * 16;
#pragma unroll
    for (int h = 0; h < 4; ++h) {                      // one core matrix (4 columns) per pass
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = cg * 16 + h * 4 + u;
            const float v = (rin && k < w) ? Fs[row + static_cast<int64_t>(k0 + k) * LD] : 0.f;
            hi[u] = to_tf32(v);
            lo[u] = to_tf32(v - __uint_as_float(hi[u]));
        }
        const int kc = cg * 4 + h;
        *reinterpret_cast<uint4*>(base + kc * kTsLbo) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(base + plane + kc * kTsLbo) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
}

__global__ void __launch_bounds__(256, 2) k_update_tcs(StepArgs a, const int* __restrict__ items,
                                                       const int* __restrict__ prefix, PlanDev pd, float* F,
                                                       float* __restrict__ Linv, const int64_t* __restrict__ inv_off,
                                                       const unsigned char* __restrict__ dig, int64_t plane,
                                                       int* err) {
    extern __shared__ __align__(1024) unsigned char smraw[];
    unsigned char* Ah = smraw;
    unsigned char* Al = Ah + kTsA;
    unsigned char* Bh = Al + kTsA;
    unsigned char* Bl = Bh + kTsB;
    uint64_t* bar = reinterpret_cast<uint64_t*>(Bl + kTsB);   // [0] parts loaded, [1] MMAs done
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 2);
    int* fail = reinterpret_cast<int*>(bar + 3);
    int i;
    const int lb = update_unit(prefix + a.up3_off, a.nitems, blockIdx.x, i);
    if (lb < 0) return;
    const int s = items[a.item_off + i];
    if (!pd.lp_on[pd.sn_lp[s]]) return;
    int bi = block_row_of(lb);
    const int bj = lb - bi * (bi + 1);
    const int N = pd.sn_nrows[s], K = pd.sn_ncols[s], LD = pd.sn_lda[s];
    const int k0 = a.k * T64;
    const int w = min(T64, K - k0);
    const int t0 = k0 + w;
    const int r0 = t0 + bi * 128, c0 = t0 + bj * T64;
    if (c0 >= N) return;                              // the whole block: column block past the front
    const int nra = min(128, N - r0), ncb = min(T64, N - c0);
    const int qa = prefix[a.dr_off + i] + bi * 128, qb = prefix[a.dr_off + i] + bj * T64;
    float* Fs = F + pd.F_off[s];
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
    // thread 0 starts the copies first; TMEM allocation and every thread's C loads
    // then overlap them
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_addr(bar)));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_addr(bar + 1)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *fail = 0;
        const uint32_t b0 = smem_addr(bar);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                     :: "r"(b0), "r"(static_cast<uint32_t>(2 * (kTsA + kTsB))) : "memory");
        const unsigned char* ga = dig + static_cast<int64_t>(qa >> 3) * kTsSbo;
        const unsigned char* gb = dig + static_cast<int64_t>(qb >> 3) * kTsSbo;
        const unsigned char* src[4] = {ga, ga + plane, gb, gb + plane};
        unsigned char* dst[4] = {Ah, Al, Bh, Bl};
        const uint32_t len[4] = {static_cast<uint32_t>(kTsA), static_cast<uint32_t>(kTsA),
                                 static_cast<uint32_t>(kTsB), static_cast<uint32_t>(kTsB)};
        for (int c = 0; c < 4; ++c)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         :: "r"(smem_addr(dst[c])), "l"(src[c]), "r"(len[c]), "r"(b0) : "memory");
    }
    if (wid == 0) {
        __syncwarp();                                  // thread 0 has been on its own
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 64;" :: "r"(smem_addr(tslot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    // this thread's row (TMEM lane) and 32 columns, and its C values
    const int row = 32 * (wid & 3) + lane, ch = 32 * (wid >> 2);
    const bool rok = row < nra;
    float cv[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        const int col = ch + j;
        const bool in = rok && col < ncb && r0 + row >= c0 + col;
        cv[j] = in ? Fs[(r0 + row) + static_cast<int64_t>(c0 + col) * LD] : 0.f;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot;
    if (tid == 0) {
        const uint32_t b0 = smem_addr(bar);
        bool ok = oz_wait(b0);
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t ah = smem_addr(Ah), al = smem_addr(Al), bh = smem_addr(Bh), bl = smem_addr(Bl);
            uint32_t acc = 0;
            for (int ks = 0; ks < T64 / 8; ++ks) {
                const uint32_t ko = static_cast<uint32_t>(ks) * 2 * kTsLbo;
                const uint64_t da[3] = {tc_sdesc(al + ko), tc_sdesc(ah + ko), tc_sdesc(ah + ko)};
                const uint64_t db[3] = {tc_sdesc(bh + ko), tc_sdesc(bl + ko), tc_sdesc(bh + ko)};
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                                 " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n"
                                 :: "r"(tmem), "l"(da[q]), "l"(db[q]), "r"(kTsIdesc), "r"(acc));
                    acc = 1;
                }
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         :: "r"(smem_addr(bar + 1)) : "memory");
            ok = oz_wait(smem_addr(bar + 1));
            if (!ok) oz_wait(smem_addr(bar + 1));     // a second bounded wait before TMEM is freed
        } else {
            oz_wait(b0);                               // copies still in flight: a second bounded wait
        }
        if (!ok) {
            *fail = 1;
            atomicExch(err + 2, 1);
        }
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const bool ok = *fail == 0;
    if (ok) {
#pragma unroll
        for (int c16 = 0; c16 < 2; ++c16) {
            __syncwarp();                              // the TMEM loads take a converged warp
            uint32_t v[16];
            const uint32_t taddr = tmem + (static_cast<uint32_t>(32 * (wid & 3)) << 16) +
                                   static_cast<uint32_t>(ch + 16 * c16);
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                         : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                           "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                           "=r"(v[14]), "=r"(v[15])
                         : "r"(taddr));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const int j = 16 * c16 + q, col = ch + j;
                if (rok && col < ncb && r0 + row >= c0 + col)
                    Fs[(r0 + row) + static_cast<int64_t>(c0 + col) * LD] = cv[j] - __uint_as_float(v[q]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (wid == 0) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 64;" :: "r"(tmem));
    }
    if (!ok) return;
    // the block holding the first trailing diagonal tile factors it (as in k_update)
    if (lb == 0 && t0 < K) {
        __syncthreads();
        potrf_tile(s, a.k + 1, pd, F, Linv, inv_off, err, smraw);
    }
}

template <class T>
__global__ void k_extend_add(int item_off, int nitems, int prefix_off, const int* __restrict__ items,
                             const int* __restrict__ prefix, PlanDev pd, T* F) {
    const int i = find_item(prefix + prefix_off, nitems, blockIdx.x);
    const int c = items[item_off + i];
    if (!pd.lp_on[pd.sn_lp[c]]) return;
    const int lt = blockIdx.x - prefix[prefix_off + i];
    int ti, tj;
    tri_index(lt, ti, tj);
    const int Kc = pd.sn_ncols[c], Nc = pd.sn_nrows[c];
    const int u = Nc - Kc;
    const int p = pd.sn_parent[c];
    const T* Fc = F + pd.F_off[c];
    T* Fp = F + pd.F_off[p];
    const int* map = pd.ea_map + pd.ea_off[c];
    const int rr = ti * 32 + threadIdx.x;
    if (rr >= u) return;
    const int mr = map[rr];
    for (int cc = tj * 32 + threadIdx.y; cc < tj * 32 + 32 && cc < u; cc += blockDim.y) {
        if (rr < cc) continue;
        const T v = Fc[(Kc + rr) + static_cast<int64_t>(Kc + cc) * pd.sn_lda[c]];
        T* dst = Fp + mr + static_cast<int64_t>(map[cc]) * pd.sn_lda[p];
        *dst = *dst + v;
    }
}

// -------------------------------------------------------------------- solve
// Vectors of the solve are in the front precision T; the caller's vectors are FP64.

// A solution entry that is not there yet: an all-ones NaN, which no arithmetic result is
// (publish() stores the canonical NaN instead).
template <class T> struct Pending;
template <> struct Pending<float> {
    __device__ static float value() { return __uint_as_float(0xffffffffu); }
    __device__ static bool is(float v) { return __float_as_uint(v) == 0xffffffffu; }
};
template <> struct Pending<double> {
    __device__ static double value() { return __longlong_as_double(-1LL); }
    __device__ static bool is(double v) { return __double_as_longlong(v) == -1LL; }
};

// zp = D src in elimination order; both solution vectors pending.
template <class T>
__global__ void k_permute_scale(int M, const int* __restrict__ perm, const double* __restrict__ D,
                                const double* __restrict__ src, T* __restrict__ zp, T* __restrict__ zsol,
                                T* __restrict__ xp) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= M) return;
    zp[q] = static_cast<T>(D[q] * src[perm[q]]);
    zsol[q] = Pending<T>::value();
    xp[q] = Pending<T>::value();
}

// Rows of the LPs in `own` receive D xp; rows of the LPs in `other` (the set the
// other precision's pass serves; may be null) are left as they are; all other
// rows get 0.
template <class T>
__global__ void k_unpermute_scale(int M, const int* __restrict__ perm, const double* __restrict__ D,
                                  const T* __restrict__ xp, const int* __restrict__ row_lp,
                                  const int* __restrict__ own, const int* __restrict__ other,
                                  double* __restrict__ dst) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < M) {
        const int r = perm[q];
        const int k = row_lp[r];
        if (own[k]) dst[r] = D[q] * static_cast<double>(xp[q]);
        else if (!other || !other[k]) dst[r] = 0.0;
    }
}

// Zeroes the fronts of the LPs being factored, one chunk of a front per block
// (the fronts of other LPs keep their factors).
constexpr int kZeroChunk = 8192;
template <class T>
__global__ void __launch_bounds__(256) k_zero_fronts(const int* __restrict__ zc_sn, const int* __restrict__ zc_len,
                                                     const int64_t* __restrict__ zc_off, PlanDev pd,
                                                     T* __restrict__ F) {
    const int s = zc_sn[blockIdx.x];
    if (!pd.lp_on[pd.sn_lp[s]]) return;
    T* p = F + zc_off[blockIdx.x];
    const int len = zc_len[blockIdx.x];
    for (int i = threadIdx.x; i < len; i += blockDim.x) p[i] = T(0);
}

// Frontal right-hand sides of one level: one thread per front row, the row's own
// entry of the permuted rhs (or 0 outside the front's columns) plus the children's
// update-vector entries that map to it, added in child order.
template <class T>
__global__ void k_fwd_gather(int n, const int* __restrict__ dst, const int* __restrict__ zpi,
                             const int* __restrict__ ptr, const int* __restrict__ src, const T* __restrict__ zp,
                             T* __restrict__ fv) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int z = zpi[t];
    T acc = z >= 0 ? zp[z] : T(0);
    for (int q = ptr[t]; q < ptr[t + 1]; ++q) acc += fv[src[q]];
    fv[dst[t]] = acc;
}

// ---- dependency-driven triangular solves -------------------------------------
// Each front's rows are split into 64-row blocks; block i of front s is one task.
// Tasks of a level are handed out in dependency order by an atomic counter, so a
// task only ever waits for tasks that have already started. The chain from block to
// block bounds these kernels, so a block's solution is its own signal: the entries are
// pending (k_permute_scale) until their value is stored, and a waiting task polls the
// values themselves. One trip through the L2 then links two blocks, where a flag took
// four (values, fence, flag; flag, then values). Every wait is bounded: on time-out the
// task sets *err and returns (the host checks *err and reports an error).
// Chain of one front, per 64-row block: FP32 forward 2.2 -> 1.0 us, backward 3.2 -> 1.0
// us; FP64 forward 4.4 -> 2.6 us, backward 8.2 -> 3.2 us (m = 1447 .. 4740). In a batch a
// task starts behind its chain and is bound by how fast it takes in the blocks that are
// there: with two of them in registers the FP32 solves of 40 LPs take 206 -> 110 us forward
// and 133 -> 93 us backward.

constexpr long long kAwaitCycles = 1LL << 32;      // two seconds
constexpr int kReadyBlocks = 16;   // column blocks taken per pass once they are there

__device__ __forceinline__ float peek(const float* p) {
    float v;
    asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ double peek(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void publish(float* p, float v) {
    if (Pending<float>::is(v)) v = __uint_as_float(0x7fffffffu);
    asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" :: "l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void publish(double* p, double v) {
    if (Pending<double>::is(v)) v = __longlong_as_double(0x7ff8000000000000LL);
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" :: "l"(p), "d"(v) : "memory");
}

// *p once it is there; false on time-out or when another task gave up.
template <class T>
__device__ __forceinline__ bool await(const T* p, T& v, int* err) {
    const long long start = clock64();
    for (int spins = 0;; ++spins) {
        v = peek(p);
        if (!Pending<T>::is(v)) return true;
        if ((spins & 255) == 255 &&
            (clock64() - start > kAwaitCycles || *reinterpret_cast<volatile int*>(err) != 0)) {
            atomicExch(err, 1);
            return false;
        }
        // back to back first (the last dependency usually comes within microseconds: this wait is
        // on the solve's critical path), then back off
        if (spins > 512) __nanosleep(64);
    }
}

struct TakeSync {
    unsigned char ready[8];   // per warp: its four 32-entry parts that are there
    int abort;
};

// Solution blocks j, j + dir, ... (n of them at most; rows 64 b .. of the front's own K)
// into out, 64 entries each: those that are there already, at least block j, which is
// waited for. Returns how many (0: given up). Called by all 256 threads.
template <class T>
__device__ __forceinline__ int take_blocks(const T* sol, int j, int dir, int n, int K, T* out, TakeSync* sh,
                                           int* err) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    n = min(n, kReadyBlocks);
    unsigned mine = 0;
#pragma unroll
    for (int u = 0; u < kReadyBlocks / 4; ++u) {
        const int b = 4 * u + (tid >> 6);            // the same for a warp
        if (b >= n) break;
        const int row = (j + dir * b) * T64 + (tid & 63);
        const T v = row < K ? peek(sol + row) : T(0);
        out[b * T64 + (tid & 63)] = v;
        if (__all_sync(0xffffffffu, !Pending<T>::is(v))) mine |= 1u << u;
    }
    if (lane == 0) sh->ready[wid] = static_cast<unsigned char>(mine);
    if (tid == 0) sh->abort = 0;
    __syncthreads();
    int got = 0;
    while (got < n && (sh->ready[(2 * got) & 7] & sh->ready[(2 * got + 1) & 7] & (1u << (got >> 2)))) ++got;
    if (got > 0) return got;
    if (tid < T64) {
        const int row = j * T64 + tid;
        T v = T(0);
        if (row < K && !await(sol + row, v, err)) sh->abort = 1;
        out[tid] = v;
    }
    __syncthreads();
    return sh->abort ? 0 : 1;
}

// Rows of a 64x64 triangular product dealt to a thread quad: warp w takes the eight rows
// of group w or 11 - w, so that the two warps of each SM quarter share the work of a
// triangle evenly.
__device__ __forceinline__ int tri_group(int wid) { return wid < 4 ? wid : 11 - wid; }

// Forward: task (s, i). Own block i < nb covers rows [64 i, min(64 i + 64, K));
// external block i >= nb covers rows [K + 64 (i - nb), ...) < N. The task forms
// f_rows - sum_{j < min(i, nb)} L(rows, block j) z_j; an own block then publishes
// z_i = Linv_i (..) in zsol, an external block stores the parent's update vector in f.
// Column blocks that are there already are taken together (up to kReadyBlocks per
// pass); the first block of each pass has its L values loaded before the wait, so the
// latency-critical last dependency only waits for its z values.
template <class T>
__global__ void __launch_bounds__(256, 1) k_fwd_tasks(const int2* __restrict__ tasks, int ntasks, int* counter,
                                                   PlanDev pd, const T* __restrict__ F, const T* __restrict__ Linv,
                                                   const int64_t* __restrict__ inv_off, T* fv, T* zsol, int* err) {
    __shared__ int task_sh;
    __shared__ TakeSync take;
    __shared__ T zs[kReadyBlocks * T64];
    __shared__ T red[4][T64];
    __shared__ T fb[T64];
    const int tid = threadIdx.x;
    if (tid == 0) task_sh = atomicAdd(counter, 1);
    __syncthreads();
    const int t = task_sh;
    if (t >= ntasks) return;
    const int s = tasks[t].x, i = tasks[t].y;
    if (!pd.lp_on[pd.sn_lp[s]]) return;   // every task of the front's LP is skipped alike
    const int N = pd.sn_nrows[s], K = pd.sn_ncols[s], first = pd.sn_first[s];
    const int LD = pd.sn_lda[s];
    const int nb = (K + T64 - 1) / T64;
    const T* Fs = F + pd.F_off[s];
    T* f = fv + pd.f_off[s];
    const int r = tid & 63, cg = tid >> 6;
    const bool own = i < nb;
    const int row0 = own ? i * T64 : K + (i - nb) * T64;
    const int rend = own ? K : N;
    const int row = row0 + r;
    const bool rv = row < rend;
    // this thread's entries of the diagonal-tile inverse (own blocks), loaded up front
    const int w = own ? min(T64, K - i * T64) : 0;
    const int grp = tri_group(tid >> 5), zc = 8 * grp + ((tid & 31) >> 2), zpart = tid & 3;
    T li[16];
    if (own) {
        const T* Li = Linv + inv_off[s] + static_cast<int64_t>(i) * T64 * T64;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int q = zpart + 4 * k;
            li[k] = (zc < w && q <= zc) ? Li[zc + q * T64] : T(0);
        }
    }
    // this block's right-hand side (written by the gather before this kernel), loaded up front
    const T fown = (tid < T64 && row0 + tid < rend) ? f[row0 + tid] : T(0);
    T acc = T(0);
    const int jmax = own ? i : nb;
    for (int j = 0; j < jmax;) {
        T pre[16];
        const int colp = j * T64 + cg * 16;
#pragma unroll
        for (int c = 0; c < 16; ++c)
            pre[c] = (rv && colp + c < K) ? Fs[row + static_cast<int64_t>(colp + c) * LD] : T(0);
        const int got = take_blocks(zsol + first, j, 1, jmax - j, K, zs, &take, err);
        if (got == 0) return;
        const int e = j + got;
#pragma unroll
        for (int c = 0; c < 16; ++c) acc += pre[c] * zs[cg * 16 + c];
        if (rv && got > 1) {              // behind: the next block's L is loaded while one is summed
            auto load = [&](T* l, int jj) {
                const T* Lc = Fs + row + static_cast<int64_t>(jj * T64 + cg * 16) * LD;
#pragma unroll
                for (int c = 0; c < 16; ++c)
                    l[c] = jj * T64 + cg * 16 + c < K ? Lc[static_cast<int64_t>(c) * LD] : T(0);
            };
            T cur[16];
            load(cur, j + 1);
            for (int jj = j + 1; jj < e; ++jj) {
                T nxt[16];
                if (jj + 1 < e) load(nxt, jj + 1);
                const T* zz = zs + (jj - j) * T64 + cg * 16;
#pragma unroll
                for (int c = 0; c < 16; ++c) acc += cur[c] * zz[c];
#pragma unroll
                for (int c = 0; c < 16; ++c) cur[c] = nxt[c];
            }
        }
        j = e;
        if (j < jmax) __syncthreads();    // zs is refilled
    }
    red[cg][r] = acc;
    __syncthreads();
    if (tid < T64) {
        const int rw = row0 + tid;
        fb[tid] = rw < rend ? fown - ((red[0][tid] + red[1][tid]) + (red[2][tid] + red[3][tid])) : T(0);
    }
    __syncthreads();
    if (own) {
        T z = T(0);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int q = zpart + 4 * k;
            if (k > 2 * grp + 1) break;       // beyond the diagonal for the whole warp
            if (q <= zc) z += li[k] * fb[q];
        }
        z += __shfl_xor_sync(0xffffffffu, z, 1);
        z += __shfl_xor_sync(0xffffffffu, z, 2);
        if (zpart == 0 && zc < w) publish(zsol + first + i * T64 + zc, z);
    } else {
        if (tid < T64 && row0 + tid < N) f[row0 + tid] = fb[tid];
    }
}

// Backward: task (s, i), i descending: x_i = Linv_i^T (z_i - sum_{rows r below
// block i} L(r, block i)^T x_r); rows of own later blocks are waited for, rows outside
// the front's columns come from ancestors (earlier levels). Later blocks are taken
// oldest first (nb - 1 downwards), those that are there together, and the L values of
// the first block of each pass are loaded before its wait. Each lane sums its rows for
// eight columns; the lanes' sums are added by shuffles in FP32 and through shared memory
// in FP64, where the shuffles' forty additions per warp on the FP64 pipe (64 cycles
// each) were a third of the chain.
template <class T>
__global__ void __launch_bounds__(256, 2) k_bwd_tasks(const int2* __restrict__ tasks, int ntasks, int* counter,
                                                   PlanDev pd, const T* __restrict__ F, const T* __restrict__ Linv,
                                                   const int64_t* __restrict__ inv_off, T* xp,
                                                   const T* __restrict__ zsol, int* err) {
    constexpr bool kWide = std::is_same<T, double>::value;
    __shared__ int task_sh;
    __shared__ TakeSync take;
    __shared__ T xb[kReadyBlocks * T64];   // x of ready own blocks, or of a chunk of outside rows
    __shared__ T tb[T64];
    __shared__ T lanes[kWide ? T64 * 33 : 1];
    const int tid = threadIdx.x;
    if (tid == 0) task_sh = atomicAdd(counter, 1);
    __syncthreads();
    const int t = task_sh;
    if (t >= ntasks) return;
    const int s = tasks[t].x, i = tasks[t].y;
    if (!pd.lp_on[pd.sn_lp[s]]) return;   // every task of the front's LP is skipped alike
    const int N = pd.sn_nrows[s], K = pd.sn_ncols[s], first = pd.sn_first[s];
    const int LD = pd.sn_lda[s];
    const int nb = (K + T64 - 1) / T64;
    const int w = min(T64, K - i * T64);
    const T* Fs = F + pd.F_off[s];
    const int* R = pd.rows + pd.rows_off[s];
    const int lane = tid & 31, wid = tid >> 5;
    T part[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) part[q] = T(0);
    const int c0 = i * T64 + wid * 8;
    // rows outside the front's own columns (solved by ancestors): their x values are
    // gathered into shared memory a chunk at a time, then each warp runs down the rows
    constexpr int kOut = kReadyBlocks * T64;
    for (int r0 = K; r0 < N; r0 += kOut) {
        const int nr = min(kOut, N - r0);
        for (int q = tid; q < nr; q += 256) xb[q] = xp[R[r0 + q]];
        __syncthreads();
        // four rows per lane per pass: 32 independent loads in flight
        int q = lane;
        for (; q + 96 < nr; q += 128) {
            T fr[4][8];
#pragma unroll
            for (int h = 0; h < 4; ++h)
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    fr[h][u] = c0 + u < K ? Fs[(r0 + q + 32 * h) + static_cast<int64_t>(c0 + u) * LD] : T(0);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const T xr = xb[q + 32 * h];
#pragma unroll
                for (int u = 0; u < 8; ++u) part[u] += fr[h][u] * xr;
            }
        }
        for (; q < nr; q += 32) {
            const T xr = xb[q];
            const T* Fr = Fs + (r0 + q);
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (c0 + u < K) part[u] += Fr[static_cast<int64_t>(c0 + u) * LD] * xr;
        }
        __syncthreads();
    }
    // this thread's entries of the diagonal-tile inverse and of z
    const int grp = tri_group(wid), xc = 8 * grp + (lane >> 2), xpq = lane & 3;
    T li[16];
    {
        const T* Li = Linv + inv_off[s] + static_cast<int64_t>(i) * T64 * T64;
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int q = xc + xpq + 4 * k;
            li[k] = (xc < w && q < w) ? Li[q + xc * T64] : T(0);
        }
    }
    const int zq = kWide ? tid >> 2 : wid * 8 + (lane & 7);      // the column of tb this thread may form
    const T zown = zq < w ? zsol[first + i * T64 + zq] : T(0);
    // rows of own later blocks
    for (int j = nb - 1; j > i;) {
        T pre[16];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int rr = j * T64 + lane + 32 * h;
#pragma unroll
            for (int q = 0; q < 8; ++q)
                pre[h * 8 + q] = (rr < K && c0 + q < K) ? Fs[rr + static_cast<int64_t>(c0 + q) * LD] : T(0);
        }
        const int got = take_blocks(static_cast<const T*>(xp + first), j, -1, j - i, K, xb, &take, err);
        if (got == 0) return;
        const int e = j - got;   // blocks j, j - 1, ..., e + 1 are there
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const T xr = xb[lane + 32 * h];
#pragma unroll
            for (int q = 0; q < 8; ++q) part[q] += pre[h * 8 + q] * xr;
        }
        if constexpr (kWide) {            // a second block of L in registers would not leave room for two
            for (int blk = j - 1; blk > e; --blk) {                  // blocks on an SM (77 -> 93 us at m = 1447)
                const T* xx = xb + (j - blk) * T64;
                for (int rr = lane; rr < T64; rr += 32) {
                    const T xr = xx[rr];
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        if (c0 + q < K) part[q] += Fs[blk * T64 + rr + static_cast<int64_t>(c0 + q) * LD] * xr;
                }
            }
        } else if (got > 1) {             // behind: the next block's L is loaded while one is summed
            auto load = [&](T* l, int blk) {         // a block before the last: all its rows are there
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        l[h * 8 + q] = c0 + q < K ? Fs[blk * T64 + lane + 32 * h + static_cast<int64_t>(c0 + q) * LD]
                                                  : T(0);
            };
            T cur[16];
            load(cur, j - 1);
            for (int blk = j - 1; blk > e; --blk) {
                T nxt[16];
                if (blk - 1 > e) load(nxt, blk - 1);
                const T* xx = xb + (j - blk) * T64;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const T xr = xx[lane + 32 * h];
#pragma unroll
                    for (int q = 0; q < 8; ++q) part[q] += cur[h * 8 + q] * xr;
                }
#pragma unroll
                for (int q = 0; q < 16; ++q) cur[q] = nxt[q];
            }
        }
        j = e;
        if (j > i) __syncthreads();       // xb is refilled
    }
    if constexpr (kWide) {
#pragma unroll
        for (int q = 0; q < 8; ++q) lanes[(wid * 8 + q) * 33 + lane] = part[q];
        __syncthreads();
        // the sum tree of the shuffles below: lanes 16, 8, 4, 2, 1 apart
        const T* v4 = lanes + (tid >> 2) * 33 + (tid & 3);
        T v = ((v4[0] + v4[16]) + (v4[8] + v4[24])) + ((v4[4] + v4[20]) + (v4[12] + v4[28]));
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        if ((tid & 3) == 0) tb[zq] = zq < w ? zown - v : T(0);
    } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            T v = part[q];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == q) tb[zq] = zq < w ? zown - v : T(0);
        }
    }
    __syncthreads();
    {
        T x = T(0);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const int q = xc + xpq + 4 * k;
            if (k > 15 - 2 * grp) break;      // past the tile for the whole warp
            if (q < w) x += li[k] * tb[q];
        }
        x += __shfl_xor_sync(0xffffffffu, x, 1);
        x += __shfl_xor_sync(0xffffffffu, x, 2);
        if (xpq == 0 && xc < w) publish(xp + first + i * T64 + xc, x);
    }
}

// ------------------------------------------------------- normal-matrix apply

// What a row's product becomes: y = scale .* (A x), and r = b - A x with its largest entry.
// |r| orders like its bits, with a NaN above every number: one NaN makes the largest entry one.
__device__ __forceinline__ void absmax_add(double v, unsigned long long* mx) {
    unsigned long long m = static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7fffffffffffffffULL;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(mx, m);
}
struct RowScaled {
    const double* scale;               // may be null
    double* y;
    unsigned long long* clear;         // may be null: the next product's maximum
    __device__ void operator()(int r, bool valid, double acc) const {
        if (valid) y[r] = scale ? acc * scale[r] : acc;
        if (clear && r == 0) *clear = 0;
    }
};
struct RowResidual {
    const double* b;
    double* res;
    unsigned long long* mx;
    __device__ void operator()(int r, bool valid, double acc) const {
        const double d = valid ? b[r] - acc : 0.0;
        if (valid) res[r] = d;
        absmax_add(d, mx);
    }
};

// A x, each row summed by one lane in its entries' order. The sums are as long as the longest
// row (64 cycles an entry), so a block takes only 32 rows; their entries come through shared
// memory, 32 of every row at a time: four warps load whole row segments of the next tile
// while warp 0 sums one (a lane's own loads, one row each, made the product latency bound: A^T y,
// A x, residual and its maximum 70 us at m = 4740 with 47 and 120 entries a row, now 24).
// Rows of fewer than kRowSegment entries on average would leave most lanes of a segment idle,
// and a lane loads its own: A^T y with 6 entries a row 3.1 us, by segments 3.7.
constexpr int kRowSegment = 8;
template <bool Staged, class Epi>
__global__ void __launch_bounds__(Staged ? 160 : 256) k_row_sums(int rows, const int* __restrict__ rp,
                                                                 const int* __restrict__ ci,
                                                                 const double* __restrict__ v,
                                                                 const double* __restrict__ x, Epi epi) {
    const int row = Staged ? blockIdx.x * 32 + (threadIdx.x & 31) : blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = row < rows;
    const int q0 = valid ? rp[row] : 0, n = valid ? rp[row + 1] - q0 : 0;
    double acc = 0.0;
    if constexpr (Staged) {
        constexpr int S = 33;
        __shared__ double vs[2][32 * S], xs[2][32 * S];
        const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
        const int len = __reduce_max_sync(0xffffffffu, n), tiles = (len + 31) / 32;   // the same in every warp
        for (int t = 0; t <= tiles; ++t) {
            if (wid > 0 && t < tiles) {               // tile t: eight rows a warp
                const int k = 32 * t + lane, r0 = 8 * (wid - 1);
                int c[8];
                double a[8], g[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const bool in = k < __shfl_sync(0xffffffffu, n, r0 + i);
                    const int q = __shfl_sync(0xffffffffu, q0, r0 + i) + k;
                    c[i] = in ? ci[q] : -1;
                    a[i] = in ? v[q] : 0.0;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) g[i] = c[i] >= 0 ? x[c[i]] : 0.0;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    vs[t & 1][(r0 + i) * S + lane] = a[i];
                    xs[t & 1][(r0 + i) * S + lane] = g[i];
                }
            }
            if (wid == 0 && t > 0) {
                const double* va = vs[(t - 1) & 1] + lane * S;
                const double* xa = xs[(t - 1) & 1] + lane * S;
                const int m = min(32, n - 32 * (t - 1));
#pragma unroll 8
                for (int k = 0; k < 32; ++k)
                    if (k < m) acc += va[k] * xa[k];
            }
            __syncthreads();
        }
        if (wid > 0) return;
    } else {
        for (int q = q0; q < q0 + n; ++q) acc += v[q] * x[ci[q]];
    }
    epi(row, valid, acc);
}

inline int blocks_for(int64_t n, int t) { return static_cast<int>((n + t - 1) / t); }

}  // namespace

// ------------------------------------------------------------------ engine

// FP64 updates of fewer 64x64 tiles than this take 16x16 parts (about two waves of the 152
// SMs): m = 500 LP 16.5 ms, with 32x32 parts from 12 tiles on 16.8 ms; one front of 130 rows 257 us
// with 32x32 parts, 232 with these. It counts the tiles of all fronts together, and several fronts
// with that few would rather have 32x32 parts (ten fronts of 100 rows 198 us, 181 with those; 16
// of 512 rows 1157, 1101).
constexpr int kSplit16Tiles = 24;
// Fewer tiles than this run one block per SM, so that the next diagonal tile has an SM to
// itself: m = 1447 3.12 -> 2.89 ms; with 800 here m = 4001 loses 1 %. With many fronts, too: 40 of
// 100 rows 232 -> 194 us, 100 of 192 rows 558 -> 508, 60 of 320 rows 1031 -> 992, the same from
// 150 fronts of 100 rows on.
constexpr int kAloneTiles = 300;
// Panel solves of fewer 64-row units than this take 8 rows a block instead of 16: m = 500
// LP 17.5 -> 16.0 ms, one front of 130 rows 243 -> 232 us, one warp then has an SM quarter to
// itself; more blocks than SMs only load the diagonal tile more often (10 to 400 fronts of 100 to
// 700 rows: the same either way, within 2 %).
constexpr int kTr4Tiles = 76;

struct KktEngine::Prof {
    cudaStream_t st;
    std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> ev;
    double upd_flops = 0.0, upd_bytes = 0.0;
    double mma_flops = 0.0;   // flops the tensor cores execute in the update launches
    template <class F>
    void timed(int cls, F&& launch) {
        cudaEvent_t a, b;
        SK_CUDA(cudaEventCreate(&a));
        SK_CUDA(cudaEventCreate(&b));
        SK_CUDA(cudaEventRecord(a, st));
        launch();
        SK_CUDA(cudaEventRecord(b, st));
        ev.push_back({cls, {a, b}});
    }
};

template <class T>
static void set_smem_attrs() {
    if (std::is_same<T, float>::value)
        SK_CUDA(cudaFuncSetAttribute(k_update_tcs, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(kTsSmem)));
    SK_CUDA(cudaFuncSetAttribute(k_potrf<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(potrf_smem(sizeof(T)))));
    if (std::is_same<T, double>::value)
        SK_CUDA(cudaFuncSetAttribute(k_update_oz, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(kOzSmemU)));
    if (std::is_same<T, double>::value) {
        SK_CUDA(cudaFuncSetAttribute(k_update_split<16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(split_smem<16>())));
        SK_CUDA(cudaFuncSetAttribute(k_update_split<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(kSplitAlone)));
    }
    if (std::is_same<T, double>::value)
        SK_CUDA(cudaFuncSetAttribute(k_panel_oz, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(kOzPanelSmem)));
}

KktEngine::KktEngine(const ipm::FrontPlan& plan, const DeviceLP& lp, cudaStream_t stream)
    : plan_(plan), lp_(lp), st_(stream) {
    const auto& p = plan_;
    int dev = 0;
    SK_CUDA(cudaGetDevice(&dev));
    SK_CUDA(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, dev));
    host_flags_.alloc(4);
    // tile-inverse offsets and per-level column-block prefixes of the backward pass
    std::vector<int64_t> inv_off(static_cast<size_t>(p.ns), 0);
    inv_size_ = 0;
    for (int s = 0; s < p.ns; ++s) {
        inv_off[s] = inv_size_;
        inv_size_ += static_cast<int64_t>((p.sn_ncols[s] + T64 - 1) / T64) * T64 * T64;
    }
    // solve task lists per level (forward: row blocks ascending; backward: own
    // column blocks descending)
    // Within a level the tasks are ordered by their position in their front's chain
    // (forward: block index; backward: distance from the last own block), fronts
    // interleaved: blocks take tasks in list order, so the first tasks of every
    // front of a level (e.g. all LPs of a dense batch) run side by side instead of
    // a few fronts' chains at a time. A task only waits on tasks of smaller position
    // in its own front, which come earlier in the list, so the earliest unfinished
    // task can always proceed.
    std::vector<int2> ftask, btask;
    fwd_task_off_.assign(static_cast<size_t>(p.nlevels) + 1, 0);
    bwd_task_off_.assign(static_cast<size_t>(p.nlevels) + 1, 0);
    for (int l = 0; l < p.nlevels; ++l) {
        fwd_task_off_[l] = static_cast<int>(ftask.size());
        bwd_task_off_[l] = static_cast<int>(btask.size());
        std::vector<std::pair<int, int2>> fl, bl;   // (position, task)
        for (int q = p.level_ptr[l]; q < p.level_ptr[l + 1]; ++q) {
            const int s = p.level_sn[q];
            const int nb = (p.sn_ncols[s] + T64 - 1) / T64;
            const int neb = (p.sn_nrows[s] - p.sn_ncols[s] + T64 - 1) / T64;
            for (int i = 0; i < nb + neb; ++i) fl.push_back({i, make_int2(s, i)});
            for (int i = nb - 1; i >= 0; --i) bl.push_back({nb - 1 - i, make_int2(s, i)});
        }
        auto by_pos = [](const std::pair<int, int2>& a, const std::pair<int, int2>& b) { return a.first < b.first; };
        std::stable_sort(fl.begin(), fl.end(), by_pos);
        std::stable_sort(bl.begin(), bl.end(), by_pos);
        for (const auto& t : fl) ftask.push_back(t.second);
        for (const auto& t : bl) btask.push_back(t.second);
    }
    fwd_task_off_[p.nlevels] = static_cast<int>(ftask.size());
    bwd_task_off_[p.nlevels] = static_cast<int>(btask.size());
    // forward right-hand-side gather lists (one item per front row, level by level)
    if (p.f_size >= (int64_t(1) << 31)) throw std::runtime_error("front vectors exceed 2^31 entries");
    std::vector<int> g_dst, g_zp, g_ptr(1, 0), g_src;
    gather_off_.assign(static_cast<size_t>(p.nlevels) + 1, 0);
    for (int l = 0; l < p.nlevels; ++l) {
        gather_off_[l] = static_cast<int>(g_dst.size());
        for (int q = p.level_ptr[l]; q < p.level_ptr[l + 1]; ++q) {
            const int s = p.level_sn[q];
            const int N = p.sn_nrows[s], K = p.sn_ncols[s];
            std::vector<int> cnt(static_cast<size_t>(N) + 1, 0);
            for (int e = p.ch_ptr[s]; e < p.ch_ptr[s + 1]; ++e) {
                const int c = p.ch_list[e], u = p.sn_nrows[c] - p.sn_ncols[c];
                for (int r = 0; r < u; ++r) cnt[p.ea_map[p.ea_off[c] + r] + 1]++;
            }
            for (int r = 0; r < N; ++r) cnt[r + 1] += cnt[r];
            std::vector<int> src(static_cast<size_t>(cnt[N])), pos(cnt.begin(), cnt.end() - 1);
            for (int e = p.ch_ptr[s]; e < p.ch_ptr[s + 1]; ++e) {
                const int c = p.ch_list[e], Kc = p.sn_ncols[c], u = p.sn_nrows[c] - Kc;
                for (int r = 0; r < u; ++r)
                    src[pos[p.ea_map[p.ea_off[c] + r]]++] = static_cast<int>(p.sn_f_off[c] + Kc + r);
            }
            for (int r = 0; r < N; ++r) {
                g_dst.push_back(static_cast<int>(p.sn_f_off[s] + r));
                g_zp.push_back(r < K ? p.sn_first[s] + r : -1);
                g_ptr.push_back(g_ptr.back() + cnt[r + 1] - cnt[r]);
            }
            g_src.insert(g_src.end(), src.begin(), src.end());
        }
    }
    gather_off_[p.nlevels] = static_cast<int>(g_dst.size());
    // LP of each front (from the batch row of its first column) and the all-on LP mask
    const std::vector<int> sn_lp = ipm::supernode_lps(p);
    sn_lp_h_ = sn_lp;
    on32_h_.assign(static_cast<size_t>(std::max(1, p.nlp)), 1);
    on64_h_ = on32_h_;
    // LP of each permuted row
    std::vector<int> q_lp(static_cast<size_t>(std::max<Index>(1, p.M)), 0);
    for (Index q = 0; q < p.M; ++q)
        q_lp[q] = static_cast<int>(std::upper_bound(p.row_off.begin(), p.row_off.end(), p.perm[q]) -
                                   p.row_off.begin()) - 1;
    // front-zeroing chunks (front, start, length), kZeroChunk entries at most
    std::vector<int> zc_sn, zc_len;
    std::vector<int64_t> zc_off;
    for (int s = 0; s < p.ns; ++s) {
        const int64_t size = static_cast<int64_t>(p.sn_lda[s]) * p.sn_nrows[s];
        for (int64_t o = 0; o < size; o += kZeroChunk) {
            zc_sn.push_back(s);
            zc_off.push_back(p.sn_F_off[s] + o);
            zc_len.push_back(static_cast<int>(std::min<int64_t>(kZeroChunk, size - o)));
        }
    }
    nzc_ = static_cast<int64_t>(zc_sn.size());
    if (zc_sn.empty()) { zc_sn.push_back(0); zc_off.push_back(0); zc_len.push_back(0); }
    auto rsv = [&](auto& slot, const auto& vec) { reserve(arena_, slot, vec.size()); };
    rsv(sn_first_, p.sn_first); rsv(sn_ncols_, p.sn_ncols); rsv(sn_nrows_, p.sn_nrows); rsv(sn_lda_, p.sn_lda); rsv(sn_parent_, p.sn_parent);
    rsv(rows_, p.rows); rsv(ea_map_, p.ea_map); rsv(ch_ptr_, p.ch_ptr); rsv(ch_list_, p.ch_list);
    rsv(perm_, p.perm); rsv(sn_F_off_, p.sn_F_off); rsv(sn_f_off_, p.sn_f_off); rsv(sn_rows_off_, p.sn_rows_off);
    rsv(ea_off_, p.ea_off); rsv(step_items_, p.step_items); rsv(step_prefix_, p.step_prefix);
    rsv(round_items_, p.round_items); rsv(round_prefix_, p.round_prefix); rsv(level_sn_, p.level_sn);
    rsv(slot_pos_, p.slot_pos); rsv(w_ptr_, p.w_ptr); rsv(slot_i_, p.slot_i); rsv(slot_j_, p.slot_j);
    rsv(w_col_, p.w_col); rsv(w_val_, p.w_val); rsv(inv_off_, inv_off);
    rsv(fwd_tasks_, ftask); rsv(bwd_tasks_, btask);
    rsv(g_dst_, g_dst); rsv(g_zp_, g_zp); rsv(g_ptr_, g_ptr); rsv(g_src_, g_src);
    rsv(sn_lp_, sn_lp); rsv(on32_, on32_h_); rsv(on64_, on64_h_); rsv(q_lp_, q_lp);
    rsv(zc_sn_, zc_sn); rsv(zc_len_, zc_len); rsv(zc_off_, zc_off);
    reserve(arena_, counters_, static_cast<size_t>(2 * std::max(1, p.nlevels)));
    reserve(arena_, solve_err_, 1);
    reserve(arena_, D_, static_cast<size_t>(p.M));
    reserve(arena_, Mdiag_, static_cast<size_t>(p.M));
    reserve(arena_, zp_, static_cast<size_t>(p.M));
    reserve(arena_, xp_, static_cast<size_t>(p.M));
    reserve(arena_, zsol_, static_cast<size_t>(p.M));
    reserve(arena_, fvec_, static_cast<size_t>(p.f_size));
    reserve(arena_, tn_, static_cast<size_t>(std::max(1, p.N)));
    reserve(arena_, params_, 4);
    reserve(arena_, err_, 4);
    reserve(arena_, oz_cnt_, p.sn_ncols.size() + 1);
    reserve(arena_, lp_fail_, std::max<size_t>(1, static_cast<size_t>(p.nlp)));
    for (auto& sb : sub_) {
        reserve(arena_, sb.d_items, std::max<size_t>(1, p.step_items.size()));
        reserve(arena_, sb.d_prefix, std::max<size_t>(1, p.step_prefix.size()));
    }
    arena_.commit();
    auto bnd = [&](auto& slot) { bind(arena_, slot); };
    bnd(sn_first_); bnd(sn_ncols_); bnd(sn_nrows_); bnd(sn_lda_); bnd(sn_parent_); bnd(rows_); bnd(ea_map_); bnd(ch_ptr_);
    bnd(ch_list_); bnd(perm_); bnd(sn_F_off_); bnd(sn_f_off_); bnd(sn_rows_off_); bnd(ea_off_); bnd(step_items_);
    bnd(step_prefix_); bnd(round_items_); bnd(round_prefix_); bnd(level_sn_); bnd(slot_pos_); bnd(w_ptr_);
    bnd(slot_i_); bnd(slot_j_); bnd(w_col_); bnd(w_val_); bnd(inv_off_); bnd(fwd_tasks_);
    bnd(bwd_tasks_); bnd(g_dst_); bnd(g_zp_); bnd(g_ptr_); bnd(g_src_); bnd(sn_lp_); bnd(on32_);
    bnd(on64_); bnd(q_lp_); bnd(zc_sn_); bnd(zc_len_); bnd(zc_off_); bnd(counters_); bnd(solve_err_); bnd(D_);
    bnd(Mdiag_);
    bnd(zp_); bnd(xp_); bnd(zsol_); bnd(fvec_); bnd(tn_); bnd(params_); bnd(err_); bnd(lp_fail_); bnd(oz_cnt_);
    for (auto& sb : sub_) { bnd(sb.d_items); bnd(sb.d_prefix); }
    upload(sn_first_, p.sn_first, st_); upload(sn_ncols_, p.sn_ncols, st_); upload(sn_nrows_, p.sn_nrows, st_);
    upload(sn_lda_, p.sn_lda, st_);
    upload(sn_parent_, p.sn_parent, st_); upload(rows_, p.rows, st_); upload(ea_map_, p.ea_map, st_);
    upload(ch_ptr_, p.ch_ptr, st_); upload(ch_list_, p.ch_list, st_); upload(perm_, p.perm, st_);
    upload(sn_F_off_, p.sn_F_off, st_); upload(sn_f_off_, p.sn_f_off, st_); upload(sn_rows_off_, p.sn_rows_off, st_);
    upload(ea_off_, p.ea_off, st_); upload(step_items_, p.step_items, st_); upload(step_prefix_, p.step_prefix, st_);
    upload(round_items_, p.round_items, st_); upload(round_prefix_, p.round_prefix, st_);
    upload(level_sn_, p.level_sn, st_); upload(slot_pos_, p.slot_pos, st_); upload(w_ptr_, p.w_ptr, st_);
    upload(slot_i_, p.slot_i, st_); upload(slot_j_, p.slot_j, st_); upload(w_col_, p.w_col, st_);
    upload(w_val_, p.w_val, st_); upload(inv_off_, inv_off, st_);
    upload(fwd_tasks_, ftask, st_); upload(bwd_tasks_, btask, st_);
    upload(g_dst_, g_dst, st_); upload(g_zp_, g_zp, st_); upload(g_ptr_, g_ptr, st_); upload(g_src_, g_src, st_);
    upload(sn_lp_, sn_lp, st_); upload(on32_, on32_h_, st_); upload(on64_, on64_h_, st_); upload(q_lp_, q_lp, st_);
    upload(zc_sn_, zc_sn, st_); upload(zc_len_, zc_len, st_); upload(zc_off_, zc_off, st_);
    SK_CUDA(cudaMemsetAsync(solve_err_.ptr, 0, sizeof(int), st_));
    SK_CUDA(cudaStreamSynchronize(st_));
    set_smem_attrs<float>();
    set_smem_attrs<double>();
    // per LP: the update blocks (plus the panel tiles) of one factorisation
    lp_work_.assign(sn_lp.empty() ? 0 : static_cast<size_t>(*std::max_element(sn_lp.begin(), sn_lp.end())) + 1, 0.0);
    for (const auto& st : p.steps)
        for (int i = 0; i < st.nitems; ++i) {
            const int s = p.step_items[st.item_off + i];
            const double w = p.step_prefix[st.upd3_prefix_off + i + 1] - p.step_prefix[st.upd3_prefix_off + i] +
                             p.step_prefix[st.trsm_prefix_off + i + 1] - p.step_prefix[st.trsm_prefix_off + i] + 1;
            lp_work_[sn_lp[s]] += w;
            total_work_ += w;
        }
}

KktEngine::~KktEngine() {
    cudaStreamSynchronize(st_);                  // nothing uses host_flags_ any more
    for (int q = 0; q < 2; ++q)
        if (fev_[q]) cudaEventDestroy(fev_[q]);
    for (int q = 0; q < 4; ++q)
        if (gfac_[q]) cudaGraphExecDestroy(gfac_[q]);
    for (int q = 0; q < 2; ++q)
        if (gsol_[q]) cudaGraphExecDestroy(gsol_[q]);
}

PlanDev KktEngine::pd(bool fp32) const {
    return PlanDev{sn_first_.ptr, sn_ncols_.ptr, sn_nrows_.ptr, sn_lda_.ptr, sn_F_off_.ptr, sn_f_off_.ptr, sn_rows_off_.ptr,
                   rows_.ptr, ea_off_.ptr, ea_map_.ptr, ch_ptr_.ptr, ch_list_.ptr, sn_parent_.ptr, sn_lp_.ptr,
                   fp32 ? on32_.ptr : on64_.ptr, lp_fail_.ptr};
}

template <class T>
void KktEngine::launch_factor(T* F, T* Linv, Prof* prof, const SubSteps* sub) {
    auto run = [&](int cls, auto&& f) {
        if (prof) prof->timed(cls, f); else f();
    };
    const auto& p = plan_;
    const PlanDev pdv = pd(std::is_same<T, float>::value);
    if (nzc_ > 0)
        k_zero_fronts<T><<<static_cast<int>(nzc_), 256, 0, st_>>>(zc_sn_.ptr, zc_len_.ptr, zc_off_.ptr, pdv, F);
    SK_CUDA(cudaMemsetAsync(err_.ptr, 0, 4 * sizeof(int), st_));
    SK_CUDA(cudaMemsetAsync(lp_fail_.ptr, 0, lp_fail_.count * sizeof(int), st_));
    if (std::is_same<T, double>::value)   // blocks of the first update tile that have finished
        SK_CUDA(cudaMemsetAsync(oz_cnt_.ptr, 0, oz_cnt_.count * sizeof(int), st_));
    const double* theta = theta_bound_;
    run(0, [&] {
        if (p.dense_mode) {
            launch_diag<DiagDense>(p.M, lp_.spmv_group_A, st_, lp_.a_rp, lp_.a_ci, lp_.a_v, theta, Mdiag_.ptr,
                                   D_.ptr);
            k_asm_cols_dense<T><<<blocks_for(static_cast<int64_t>(p.M) * 32, 256), 256, 0, st_>>>(
                p.M, lp_.a_rp, lp_.a_ci, lp_.a_v, lp_.t_rp, lp_.t_ci, lp_.t_v, theta, Mdiag_.ptr, D_.ptr, lp_.row_lp,
                pdv, params_.ptr, F);
        } else {
            launch_diag<DiagSparse>(p.M, lp_.spmv_group_A, st_, w_ptr_.ptr, w_col_.ptr, w_val_.ptr, theta,
                                    Mdiag_.ptr, D_.ptr);
            k_asm_slots_sparse<T><<<blocks_for(p.nslots, 256), 256, 0, st_>>>(
                p.nslots, p.M, w_ptr_.ptr, w_col_.ptr, w_val_.ptr, theta, slot_i_.ptr, slot_j_.ptr, slot_pos_.ptr,
                Mdiag_.ptr, D_.ptr, params_.ptr, q_lp_.ptr, pdv.lp_on, F);
        }
    });
    const std::vector<ipm::PlanStep>& steps = sub ? sub->rs.steps : p.steps;
    const std::vector<int>& level_ptr = sub ? sub->rs.level_ptr : p.step_level_ptr;
    const int* items = sub ? sub->d_items.ptr : step_items_.ptr;
    const int* prefix = sub ? sub->d_prefix.ptr : step_prefix_.ptr;
    for (int l = 0; l < p.nlevels; ++l) {
        for (int q = level_ptr[l]; q < level_ptr[l + 1]; ++q) {
            const auto& st = steps[q];
            StepArgs a{st.k,           st.item_off,         st.nitems,           st.trsm_prefix_off,
                       st.upd_prefix_off, st.upd2_prefix_off, st.upd3_prefix_off, st.digit_row_off};
            if (st.k == 0)   // later diagonal tiles are factored by the previous step's update
                run(1, [&] {
                    k_potrf<T><<<st.nitems, 256, potrf_smem(sizeof(T)), st_>>>(a, items, pdv, F, Linv,
                                                                               inv_off_.ptr, err_.ptr);
                });
            if (st.trsm_tiles > 0)
                run(2, [&] {
                    const int tiles = static_cast<int>(st.trsm_tiles);
                    if constexpr (std::is_same<T, float>::value) {
                        k_trsm<<<tiles, 256, 2 * T64 * T64 * sizeof(T), st_>>>(a, items, prefix, pdv, F, Linv,
                                                                              inv_off_.ptr);
                    } else if (emulate64_) {   // FP64-accurate panel solve on the tensor cores
                        k_panel_oz<<<static_cast<int>(st.digit_rows / 128), 512, kOzPanelSmem, st_>>>(
                            a, items, prefix, pdv, F, Linv, inv_off_.ptr, dig_.ptr, dexp_.ptr,
                            plan_.max_digit_rows * 128, oz_cnt_.ptr + plan_.ns, err_.ptr);
                    } else if (tiles < kTr4Tiles) {
                        k_trsm_rows<4><<<8 * tiles, 128, tr_smem(4), st_>>>(a, items, prefix, pdv, F, Linv,
                                                                            inv_off_.ptr);
                    } else {
                        k_trsm_rows<8><<<4 * tiles, 256, tr_smem(8), st_>>>(a, items, prefix, pdv, F, Linv,
                                                                            inv_off_.ptr);
                    }
                });
            if (st.upd_tiles > 0) {
                run(3, [&] {
                    bool tc = false;
                    if constexpr (std::is_same<T, float>::value) {
                        if (tensor_) {
                            tc = true;
                            const int64_t plane = plan_.max_digit_rows * 256;
                            k_tc_split<<<static_cast<int>(st.trsm_tiles), 256, 0, st_>>>(
                                a, items, prefix, pdv, F, dig_.ptr, plane);
                            k_update_tcs<<<st.nitems + static_cast<int>(st.upd3_blocks), 256, kTsSmem, st_>>>(
                                a, items, prefix, pdv, F, Linv, inv_off_.ptr, dig_.ptr, plane,
                                err_.ptr);
                        }
                    } else {
                        if (emulate64_) {
                            tc = true;
                            const int64_t plane = plan_.max_digit_rows * 128;
                            const int64_t units = st.nitems + st.upd3_blocks;
                            k_update_oz<<<static_cast<int>(std::min<int64_t>(units, sms_)), 320, kOzSmemU, st_>>>(
                                a, items, prefix, pdv, F, Linv, inv_off_.ptr, dig_.ptr,
                                dexp_.ptr, plane, oz_cnt_.ptr + plan_.ns, err_.ptr);
                        }
                    }
                    if (tc) return;
                    const int tiles = static_cast<int>(st.upd_tiles);
                    if constexpr (std::is_same<T, float>::value)
                        k_update<<<st.nitems + tiles, 256, potrf_smem(sizeof(T)), st_>>>(
                            a, items, prefix, pdv, F, Linv, inv_off_.ptr, err_.ptr);
                    else if (tiles < kSplit16Tiles)
                        k_update_split<16><<<(st.nitems + tiles) * 16, 256, split_smem<16>(), st_>>>(
                            a, items, prefix, pdv, F, Linv, inv_off_.ptr, oz_cnt_.ptr, err_.ptr);
                    else
                        k_update_split<32><<<(st.nitems + tiles) * 4, 256,
                                             tiles < kAloneTiles ? kSplitAlone : split_smem<32>(), st_>>>(
                            a, items, prefix, pdv, F, Linv, inv_off_.ptr, oz_cnt_.ptr, err_.ptr);
                });
                if (prof) {
                    for (int it = 0; it < st.nitems; ++it) {
                        const int s2 = (sub ? sub->rs.items : p.step_items)[st.item_off + it];
                        const double w = std::min<int64_t>(T64, p.sn_ncols[s2] - static_cast<int64_t>(st.k) * T64);
                        const double t = p.sn_nrows[s2] - static_cast<double>(st.k) * T64 - w;
                        prof->upd_flops += 2.0 * w * t * (t + 1.0) / 2.0;
                        prof->upd_bytes += sizeof(T) * (t * w + 2.0 * t * (t + 1.0) / 2.0);
                    }
                    // per 128 x 64 block of the lower part, K padded to 64: TF32 x3 runs
                    // three products, the emulated FP64 update 28 BF16 digit-pair products
                    const double blk = 2.0 * 128 * 64 * 64 * static_cast<double>(st.upd3_blocks);
                    if (std::is_same<T, float>::value && tensor_) prof->mma_flops += 3.0 * blk;
                    if (std::is_same<T, double>::value && emulate64_) prof->mma_flops += 28.0 * blk;
                }
            }
        }
        for (int q = p.round_level_ptr[l]; q < p.round_level_ptr[l + 1]; ++q) {
            const auto& rd = p.rounds[q];
            run(4, [&] {
                k_extend_add<T><<<static_cast<int>(rd.tiles), dim3(32, 8), 0, st_>>>(
                    rd.item_off, rd.nitems, rd.prefix_off, round_items_.ptr, round_prefix_.ptr, pdv, F);
            });
        }
    }
    SK_CUDA(cudaGetLastError());
}

template <class T>
void KktEngine::launch_solve(const T* F, const T* Linv, Prof* prof) {
    auto run = [&](int cls, auto&& f) {
        if (prof) prof->timed(cls, f); else f();
    };
    const auto& p = plan_;
    const PlanDev pdv = pd(std::is_same<T, float>::value);
    T* zp = reinterpret_cast<T*>(zp_.ptr);
    T* xp = reinterpret_cast<T*>(xp_.ptr);
    T* zs = reinterpret_cast<T*>(zsol_.ptr);
    T* fv = reinterpret_cast<T*>(fvec_.ptr);
    SK_CUDA(cudaMemsetAsync(counters_.ptr, 0, sizeof(int) * 2 * static_cast<size_t>(std::max(1, p.nlevels)), st_));
    for (int l = 0; l < p.nlevels; ++l) {
        const int nt = fwd_task_off_[l + 1] - fwd_task_off_[l];
        const int g0 = gather_off_[l], ng = gather_off_[l + 1] - g0;
        run(5, [&] {
            if (ng > 0)
                k_fwd_gather<T><<<blocks_for(ng, 256), 256, 0, st_>>>(ng, g_dst_.ptr + g0, g_zp_.ptr + g0,
                                                                      g_ptr_.ptr + g0, g_src_.ptr, zp, fv);
            k_fwd_tasks<T><<<nt, 256, 0, st_>>>(fwd_tasks_.ptr + fwd_task_off_[l], nt, counters_.ptr + l, pdv, F,
                                                Linv, inv_off_.ptr, fv, zs,
                                                solve_err_.ptr);
        });
    }
    for (int l = p.nlevels - 1; l >= 0; --l) {
        const int nt = bwd_task_off_[l + 1] - bwd_task_off_[l];
        run(6, [&] {
            k_bwd_tasks<T><<<nt, 256, 0, st_>>>(bwd_tasks_.ptr + bwd_task_off_[l], nt, counters_.ptr + p.nlevels + l,
                                                pdv, F, Linv, inv_off_.ptr, xp, zs,
                                                solve_err_.ptr);
        });
    }
    SK_CUDA(cudaGetLastError());
}

int KktEngine::solve_error() {
    read_solve_error(host_flags_.ptr + 3);
    SK_CUDA(cudaStreamSynchronize(st_));
    return host_flags_.ptr[3];
}

void KktEngine::read_solve_error(int* host) {
    SK_CUDA(cudaMemcpyAsync(host, solve_err_.ptr, sizeof(int), cudaMemcpyDeviceToHost, st_));
}

void KktEngine::ensure_fronts(bool fp32) {
    if (fp32 && !F32_.ptr) {
        f32_arena_.reset();
        reserve(f32_arena_, F32_, static_cast<size_t>(plan_.F_size));
        reserve(f32_arena_, Linv32_, static_cast<size_t>(std::max<int64_t>(1, inv_size_)));
        f32_arena_.commit();
        bind(f32_arena_, F32_);
        bind(f32_arena_, Linv32_);
    }
    if (!fp32 && !F64_.ptr) {
        f64_arena_.reset();
        reserve(f64_arena_, F64_, static_cast<size_t>(plan_.F_size));
        reserve(f64_arena_, Linv64_, static_cast<size_t>(std::max<int64_t>(1, inv_size_)));
        f64_arena_.commit();
        bind(f64_arena_, F64_);
        bind(f64_arena_, Linv64_);
    }
}

void KktEngine::ensure_digits() {
    if (dig_.ptr || plan_.max_digit_rows <= 0) return;
    dig_arena_.reset();
    reserve(dig_arena_, dig_, static_cast<size_t>(kOzDigits) * static_cast<size_t>(plan_.max_digit_rows) * 128);
    reserve(dig_arena_, dexp_, static_cast<size_t>(plan_.max_digit_rows));
    dig_arena_.commit();
    bind(dig_arena_, dig_);
    bind(dig_arena_, dexp_);
}

// The step lists for a factorisation of the LPs of this precision's mask: the
// plan's own (and its captured graph) while the LPs that are on hold at least 3/4
// of the batch's update blocks, else lists restricted to them (rebuilt and
// uploaded when the mask has changed since the last call).
const KktEngine::SubSteps* KktEngine::pick_steps(bool fp32) {
    const std::vector<int>& mask = fp32 ? on32_h_ : on64_h_;
    double on_work = 0.0;
    for (size_t k = 0; k < mask.size() && k < lp_work_.size(); ++k)
        if (mask[k]) on_work += lp_work_[k];
    if (on_work >= 0.75 * total_work_) return nullptr;
    SubSteps& sb = sub_[fp32 ? 0 : 1];
    if (sb.mask == mask && !sb.rs.level_ptr.empty()) return &sb;
    sb.mask = mask;
    ipm::restrict_steps(plan_, sn_lp_h_, mask, sb.rs);
    if (!sb.rs.items.empty())
        SK_CUDA(cudaMemcpyAsync(sb.d_items.ptr, sb.rs.items.data(), sizeof(int) * sb.rs.items.size(),
                                cudaMemcpyHostToDevice, st_));
    if (!sb.rs.prefix.empty())
        SK_CUDA(cudaMemcpyAsync(sb.d_prefix.ptr, sb.rs.prefix.data(), sizeof(int) * sb.rs.prefix.size(),
                                cudaMemcpyHostToDevice, st_));
    return &sb;
}

bool KktEngine::factor(const double* d_theta, double delta, bool fp32) {
    const int q = fp32 ? (tensor_ ? 2 : 1) : (emulate64_ ? 3 : 0);
    ensure_fronts(fp32);
    if ((!fp32 && emulate64_) || (fp32 && tensor_)) ensure_digits();
    fp32_ = fp32;
    double hp[4] = {delta, 0, 0, 0};
    SK_CUDA(cudaMemcpyAsync(params_.ptr, hp, sizeof(hp), cudaMemcpyHostToDevice, st_));
    if (!fev_[0]) {
        SK_CUDA(cudaEventCreate(&fev_[0]));
        SK_CUDA(cudaEventCreate(&fev_[1]));
    }
    const SubSteps* sub = pick_steps(fp32);
    if (sub) {   // a few LPs of the batch: their blocks only, launched directly
        theta_bound_ = d_theta;
        SK_CUDA(cudaEventRecord(fev_[0], st_));
        if (fp32) launch_factor<float>(F32_.ptr, Linv32_.ptr, nullptr, sub);
        else launch_factor<double>(F64_.ptr, Linv64_.ptr, nullptr, sub);
        SK_CUDA(cudaEventRecord(fev_[1], st_));
    } else {
        if (!gfac_[q] || gfac_theta_[q] != d_theta) {
            if (gfac_[q]) { cudaGraphExecDestroy(gfac_[q]); gfac_[q] = nullptr; }
            theta_bound_ = d_theta;
            cudaGraph_t g;
            SK_CUDA(cudaStreamBeginCapture(st_, cudaStreamCaptureModeThreadLocal));
            if (fp32) launch_factor<float>(F32_.ptr, Linv32_.ptr); else launch_factor<double>(F64_.ptr, Linv64_.ptr);
            SK_CUDA(cudaStreamEndCapture(st_, &g));
            SK_CUDA(cudaGraphInstantiate(&gfac_[q], g, 0));
            cudaGraphDestroy(g);
            gfac_theta_[q] = d_theta;
        }
        SK_CUDA(cudaEventRecord(fev_[0], st_));
        SK_CUDA(cudaGraphLaunch(gfac_[q], st_));
        SK_CUDA(cudaEventRecord(fev_[1], st_));
    }
    const int* herr = host_flags_.ptr;
    SK_CUDA(cudaMemcpyAsync(host_flags_.ptr, err_.ptr, 3 * sizeof(int), cudaMemcpyDeviceToHost, st_));
    SK_CUDA(cudaStreamSynchronize(st_));
    float fms = 0.f;
    SK_CUDA(cudaEventElapsedTime(&fms, fev_[0], fev_[1]));
    fact_ms_[fp32 ? 0 : 1] += fms;
    if (herr[2]) throw std::runtime_error("tensor-core update: a copy or an MMA did not complete in time");
    failed_sn_ = herr[0] ? herr[1] : -1;
    failed_lps_.clear();
    if (herr[0]) {
        std::vector<int> f(lp_fail_.count, 0);
        SK_CUDA(cudaMemcpy(f.data(), lp_fail_.ptr, sizeof(int) * f.size(), cudaMemcpyDeviceToHost));
        for (size_t k = 0; k < f.size(); ++k)
            if (f[k]) failed_lps_.push_back(static_cast<int>(k));
    }
    return herr[0] == 0;
}

// One precision's solve: permute and scale src, the level-scheduled triangular
// solves of that precision's fronts (graph `graph`), unscale and unpermute into
// dst. Rows of LPs in `other` keep their dst values (see k_unpermute_scale).
template <class T>
void KktEngine::solve_pass(const T* F, const T* Linv, const int* mask, bool keep, const double* d_src,
                           double* d_dst, int graph) {
    const auto& p = plan_;
    k_permute_scale<T><<<blocks_for(p.M, 256), 256, 0, st_>>>(
        p.M, perm_.ptr, D_.ptr, d_src, reinterpret_cast<T*>(zp_.ptr), reinterpret_cast<T*>(zsol_.ptr),
        reinterpret_cast<T*>(xp_.ptr));
    if (!gsol_[graph]) {
        cudaGraph_t g;
        SK_CUDA(cudaStreamBeginCapture(st_, cudaStreamCaptureModeThreadLocal));
        launch_solve<T>(F, Linv);
        SK_CUDA(cudaStreamEndCapture(st_, &g));
        SK_CUDA(cudaGraphInstantiate(&gsol_[graph], g, 0));
        cudaGraphDestroy(g);
    }
    SK_CUDA(cudaGraphLaunch(gsol_[graph], st_));
    const int* other = keep ? (std::is_same<T, float>::value ? on64_.ptr : on32_.ptr) : nullptr;
    k_unpermute_scale<T><<<blocks_for(p.M, 256), 256, 0, st_>>>(
        p.M, perm_.ptr, D_.ptr, reinterpret_cast<const T*>(xp_.ptr), lp_.row_lp, mask, other, d_dst);
    SK_CUDA(cudaGetLastError());
}

void KktEngine::apply_inverse(const double* d_src, double* d_dst) {
    if (!mixed_) {
        if (fp32_) solve_pass<float>(F32_.ptr, Linv32_.ptr, on32_.ptr, false, d_src, d_dst, 1);
        else solve_pass<double>(F64_.ptr, Linv64_.ptr, on64_.ptr, false, d_src, d_dst, 0);
        return;
    }
    bool any32 = false, any64 = false;
    for (size_t k = 0; k < on32_h_.size(); ++k) { any32 |= on32_h_[k] != 0; any64 |= on64_h_[k] != 0; }
    // The FP32 pass writes only the rows of on32 (and zeroes the inactive ones); the FP64
    // pass then reads the rows of on64 from src, which the first pass left alone, so src
    // and dst may still alias.
    if (!any32 && !any64) {          // no LP left: every row is 0
        SK_CUDA(cudaMemsetAsync(d_dst, 0, sizeof(double) * static_cast<size_t>(plan_.M), st_));
        return;
    }
    if (any32) {
        ensure_fronts(true);
        solve_pass<float>(F32_.ptr, Linv32_.ptr, on32_.ptr, true, d_src, d_dst, 1);
    }
    if (any64) {
        ensure_fronts(false);
        solve_pass<double>(F64_.ptr, Linv64_.ptr, on64_.ptr, true, d_src, d_dst, 0);
    }
}

void KktEngine::upload_mask(Slot<int>& dev, std::vector<int>& host, const std::vector<char>& on) {
    if (on.size() != host.size()) throw std::invalid_argument("set_active: one flag per LP");
    bool same = true;
    for (size_t k = 0; same && k < on.size(); ++k) same = (on[k] != 0) == (host[k] != 0);
    if (same) return;
    for (size_t k = 0; k < on.size(); ++k) host[k] = on[k] ? 1 : 0;
    SK_CUDA(cudaMemcpyAsync(dev.ptr, host.data(), sizeof(int) * host.size(), cudaMemcpyHostToDevice, st_));
}

void KktEngine::set_active(const std::vector<char>& on) {
    restricted_ = false;
    mixed_ = false;
    upload_mask(on32_, on32_h_, on);
    upload_mask(on64_, on64_h_, on);
}

void KktEngine::set_masks(const std::vector<char>& on32, const std::vector<char>& on64) {
    for (size_t k = 0; k < on32.size() && k < on64.size(); ++k)
        if (on32[k] && on64[k]) throw std::invalid_argument("set_masks: an LP in both precisions");
    restricted_ = false;
    mixed_ = true;
    upload_mask(on32_, on32_h_, on32);
    upload_mask(on64_, on64_h_, on64);
}

void KktEngine::restrict_solves(const std::vector<char>& sub) {
    if (!restricted_) {
        full32_h_ = on32_h_;
        full64_h_ = on64_h_;
        restricted_ = true;
    }
    if (sub.size() != full32_h_.size()) throw std::invalid_argument("restrict_solves: one flag per LP");
    std::vector<char> a(sub.size()), b(sub.size());
    for (size_t k = 0; k < sub.size(); ++k) {
        a[k] = full32_h_[k] && sub[k];
        b[k] = full64_h_[k] && sub[k];
    }
    upload_mask(on32_, on32_h_, a);
    upload_mask(on64_, on64_h_, b);
}

void KktEngine::unrestrict_solves() {
    if (!restricted_) return;
    restricted_ = false;
    const std::vector<char> a(full32_h_.begin(), full32_h_.end()), b(full64_h_.begin(), full64_h_.end());
    upload_mask(on32_, on32_h_, a);
    upload_mask(on64_, on64_h_, b);
}

int KktEngine::failed_lp() const {
    return failed_sn_ >= 0 && failed_sn_ < static_cast<int>(sn_lp_h_.size()) ? sn_lp_h_[failed_sn_] : -1;
}

namespace {
template <class Epi>
void row_sums(int rows, int64_t nnz, const int* rp, const int* ci, const double* v, const double* x, Epi epi,
              cudaStream_t st) {
    if (rows <= 0) return;
    if (nnz >= static_cast<int64_t>(kRowSegment) * rows)
        k_row_sums<true><<<blocks_for(rows, 32), 160, 0, st>>>(rows, rp, ci, v, x, epi);
    else
        k_row_sums<false><<<blocks_for(rows, 256), 256, 0, st>>>(rows, rp, ci, v, x, epi);
    SK_CUDA(cudaGetLastError());
}
}  // namespace

void KktEngine::apply_normal(const double* d_theta, const double* d_src, double* d_dst) {
    // t = theta .* (A^T src); dst = A t
    row_sums(lp_.N, lp_.nnz, lp_.t_rp, lp_.t_ci, lp_.t_v, d_src, RowScaled{d_theta, tn_.ptr, nullptr}, st_);
    row_sums(lp_.M, lp_.nnz, lp_.a_rp, lp_.a_ci, lp_.a_v, tn_.ptr, RowScaled{nullptr, d_dst, nullptr}, st_);
}

void KktEngine::residual(const double* d_theta, const double* d_b, const double* d_x, double* d_res, double* d_max) {
    unsigned long long* mx = reinterpret_cast<unsigned long long*>(d_max);
    if (lp_.N <= 0) SK_CUDA(cudaMemsetAsync(d_max, 0, sizeof(double), st_));
    row_sums(lp_.N, lp_.nnz, lp_.t_rp, lp_.t_ci, lp_.t_v, d_x, RowScaled{d_theta, tn_.ptr, mx}, st_);
    row_sums(lp_.M, lp_.nnz, lp_.a_rp, lp_.a_ci, lp_.a_v, tn_.ptr, RowResidual{d_b, d_res, mx}, st_);
}

void KktEngine::profile(const double* d_theta, double delta, bool fp32, const double* d_rhs, double* d_out,
                        double* out) {
    factor(d_theta, delta, fp32);   // allocates the fronts and sets D
    Prof pr;
    pr.st = st_;
    double hp[4] = {delta, 0, 0, 0};
    SK_CUDA(cudaMemcpyAsync(params_.ptr, hp, sizeof(hp), cudaMemcpyHostToDevice, st_));
    theta_bound_ = d_theta;
    if (fp32) launch_factor<float>(F32_.ptr, Linv32_.ptr, &pr);
    else launch_factor<double>(F64_.ptr, Linv64_.ptr, &pr);
    if (fp32) {
        k_permute_scale<float><<<blocks_for(plan_.M, 256), 256, 0, st_>>>(
            plan_.M, perm_.ptr, D_.ptr, d_rhs, reinterpret_cast<float*>(zp_.ptr), reinterpret_cast<float*>(zsol_.ptr),
            reinterpret_cast<float*>(xp_.ptr));
        launch_solve<float>(F32_.ptr, Linv32_.ptr, &pr);
        k_unpermute_scale<float><<<blocks_for(plan_.M, 256), 256, 0, st_>>>(
            plan_.M, perm_.ptr, D_.ptr, reinterpret_cast<const float*>(xp_.ptr), lp_.row_lp, on32_.ptr, nullptr,
            d_out);
    } else {
        k_permute_scale<double><<<blocks_for(plan_.M, 256), 256, 0, st_>>>(plan_.M, perm_.ptr, D_.ptr, d_rhs, zp_.ptr,
                                                                           zsol_.ptr, xp_.ptr);
        launch_solve<double>(F64_.ptr, Linv64_.ptr, &pr);
        k_unpermute_scale<double><<<blocks_for(plan_.M, 256), 256, 0, st_>>>(plan_.M, perm_.ptr, D_.ptr, xp_.ptr,
                                                                             lp_.row_lp, on64_.ptr, nullptr, d_out);
    }
    SK_CUDA(cudaStreamSynchronize(st_));
    for (int q = 0; q < 16; ++q) out[q] = 0.0;
    for (auto& e : pr.ev) {
        float ms = 0.f;
        SK_CUDA(cudaEventElapsedTime(&ms, e.second.first, e.second.second));
        out[2 * e.first] += ms;
        out[2 * e.first + 1] += 1.0;
        cudaEventDestroy(e.second.first);
        cudaEventDestroy(e.second.second);
    }
    out[14] = pr.upd_flops;
    out[15] = pr.upd_bytes;
    out[16] = assembly_bytes(fp32 ? sizeof(float) : sizeof(double));
    out[17] = pr.mma_flops;
}

double KktEngine::assembly_bytes(size_t elem) const {
    const auto& p = plan_;
    const double M = p.M, N = p.N;
    const double diag_out = 16.0 * M;               // Mdiag and D
    if (p.dense_mode) {
        // A as CSR for the diagonal and as CSR + CSC for the columns (12 bytes per entry
        // and 4 per pointer each), Theta, and the lower triangle of every front written once
        double tri = 0.0;
        for (int s = 0; s < p.ns; ++s) tri += 0.5 * double(p.sn_nrows[s]) * (p.sn_nrows[s] + 1.0);
        return 3.0 * 12.0 * lp_.nnz + 8.0 * (M + 1) + 4.0 * (N + 1) + 8.0 * N + diag_out + elem * tri;
    }
    // Khatri-Rao map: 12 bytes per entry, 8 per row pointer; per off-diagonal slot its
    // two row indices (8), front position (8) and the front entry written; Theta once
    const double w = static_cast<double>(p.w_ptr.empty() ? 0 : p.w_ptr.back());
    const double offd = static_cast<double>(p.nslots) - M;
    return 12.0 * w + 8.0 * (p.nslots + 1.0) + 8.0 * N + diag_out + (16.0 + elem) * offd + elem * M;
}

namespace {
// L's diagonal entries of every front (one block per front, a thread per own column).
__global__ void k_pivots(const int* __restrict__ sn_first, const int* __restrict__ sn_ncols,
                         const int* __restrict__ sn_lda, const int64_t* __restrict__ F_off,
                         const double* __restrict__ F, double* __restrict__ out) {
    const int s = blockIdx.x;
    const int K = sn_ncols[s], LD = sn_lda[s], f = sn_first[s];
    for (int c = threadIdx.x; c < K; c += blockDim.x) out[f + c] = F[F_off[s] + c + static_cast<int64_t>(c) * LD];
}
}  // namespace

std::vector<double> KktEngine::pivots_host() {
    if (fp32_ || !F64_.ptr) throw std::logic_error("pivots_host: no FP64 factor");
    std::vector<double> out(static_cast<size_t>(plan_.M));
    Arena tmp;
    Slot<double> d;
    reserve(tmp, d, static_cast<size_t>(std::max<int64_t>(1, plan_.M)));
    tmp.commit();
    bind(tmp, d);
    if (plan_.ns > 0)
        k_pivots<<<plan_.ns, 128, 0, st_>>>(sn_first_.ptr, sn_ncols_.ptr, sn_lda_.ptr, sn_F_off_.ptr, F64_.ptr, d.ptr);
    SK_CUDA(cudaGetLastError());
    SK_CUDA(cudaMemcpyAsync(out.data(), d.ptr, sizeof(double) * out.size(), cudaMemcpyDeviceToHost, st_));
    SK_CUDA(cudaStreamSynchronize(st_));
    return out;
}

std::vector<double> KktEngine::fronts_host() {
    std::vector<double> out(static_cast<size_t>(plan_.F_size));
    if (fp32_) {
        std::vector<float> tmp(out.size());
        SK_CUDA(cudaMemcpyAsync(tmp.data(), F32_.ptr, sizeof(float) * tmp.size(), cudaMemcpyDeviceToHost, st_));
        SK_CUDA(cudaStreamSynchronize(st_));
        for (size_t q = 0; q < out.size(); ++q) out[q] = tmp[q];
    } else {
        SK_CUDA(cudaMemcpyAsync(out.data(), F64_.ptr, sizeof(double) * out.size(), cudaMemcpyDeviceToHost, st_));
        SK_CUDA(cudaStreamSynchronize(st_));
    }
    return out;
}

}  // namespace dev
}  // namespace sankhya

namespace sankhya {
namespace dev {

namespace {
__global__ void k_absmax_partial(int n, const double* __restrict__ a, double* __restrict__ part) {
    double m = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) m = fmax(m, fabs(a[i]));
    m = warp_max(m);
    __shared__ double sh[8];
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        double r = 0.0;
        for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) r = fmax(r, sh[w]);
        part[blockIdx.x] = r;
    }
}
__global__ void k_sum(int n, const double* __restrict__ a, const double* __restrict__ b, double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = a[i] + b[i];
}
}  // namespace

void absmax_partials(int n, const double* a, double* part64, cudaStream_t st) {
    k_absmax_partial<<<64, 256, 0, st>>>(n, a, part64);
    SK_CUDA(cudaGetLastError());
}

void vec_sum(int n, const double* a, const double* b, double* out, cudaStream_t st) {
    k_sum<<<(n + 255) / 256, 256, 0, st>>>(n, a, b, out);
    SK_CUDA(cudaGetLastError());
}

}  // namespace dev
}  // namespace sankhya
