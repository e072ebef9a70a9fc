// Learned warm start network: hand-written BF16-weight forward / backward
// kernels and Adam (see gnn.hpp for the model).
#include "cuda/gnn.hpp"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace sankhya {
namespace dev {

namespace {

constexpr int H = kGnnHidden;
constexpr int L = kGnnLayers;

// parameter layout (floats)
struct Layout {
    size_t Ec, ec, Er, er;
    size_t Wrr[L], Wrm[L], br[L], Wcc[L], Wcm[L], bc[L];
    size_t Hc, oc, Hr, orr;
    size_t total;
};

Layout make_layout() {
    Layout y{};
    size_t o = 0;
    y.Ec = o; o += H * 3; y.ec = o; o += H;
    y.Er = o; o += H * 3; y.er = o; o += H;
    for (int l = 0; l < L; ++l) {
        y.Wrr[l] = o; o += H * H; y.Wrm[l] = o; o += H * H; y.br[l] = o; o += H;
        y.Wcc[l] = o; o += H * H; y.Wcm[l] = o; o += H * H; y.bc[l] = o; o += H;
    }
    y.Hc = o; o += 2 * H; y.oc = o; o += 2;
    y.Hr = o; o += H; y.orr = o; o += 1;
    y.total = o;
    return y;
}

const Layout kLay = make_layout();

__device__ __forceinline__ float bf(uint16_t w) { return __uint_as_float(static_cast<uint32_t>(w) << 16); }

__host__ __device__ inline uint16_t to_bf16(float f) {   // round to nearest even
    uint32_t u;
    std::memcpy(&u, &f, 4);
    if ((u & 0x7f800000u) == 0x7f800000u) return static_cast<uint16_t>(u >> 16);   // inf / nan
    u += 0x7fffu + ((u >> 16) & 1u);
    return static_cast<uint16_t>(u >> 16);
}

__global__ void k_to_bf16(int n, const float* __restrict__ w, uint16_t* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        uint32_t u = __float_as_uint(w[i]);
        if ((u & 0x7f800000u) != 0x7f800000u) u += 0x7fffu + ((u >> 16) & 1u);
        out[i] = static_cast<uint16_t>(u >> 16);
    }
}

// One side (columns or rows) of the graph: its entries (CSR of the side), its right-hand
// side, and its node count.
struct Side {
    int nodes;
    const int* rp;
    const int* ci;
    const double* v;
    const double* rhs;
};

// Features, inverse degree and embedding of every node, columns in the first blocks, then
// rows: f = (rhs, log(1 + degree), 2-norm), h0[o] = relu(E[o] . f + e[o]). A thread per node
// forms the features (an FP64 instruction costs the same for one lane as for 32, so the
// norms and roots are taken 32 nodes at a time), then the block's threads the embeddings.
struct EmbedSide {
    Side side;
    const uint16_t* W;
    const uint16_t* b;
    float* f;
    float* inv_deg;
    float* h;
};
constexpr int kEmbedThreads = 128;
__global__ void __launch_bounds__(kEmbedThreads) k_embed(EmbedSide cols, EmbedSide rows, int col_blocks) {
    __shared__ float fs[kEmbedThreads][3];
    const bool col = static_cast<int>(blockIdx.x) < col_blocks;
    const EmbedSide& e = col ? cols : rows;
    const int n0 = (col ? blockIdx.x : blockIdx.x - col_blocks) * kEmbedThreads, tid = threadIdx.x;
    const int node = n0 + tid;
    if (node < e.side.nodes) {
        const int q0 = e.side.rp[node], q1 = e.side.rp[node + 1];
        double s2 = 0.0;
#pragma unroll 8
        for (int q = q0; q < q1; ++q) s2 += e.side.v[q] * e.side.v[q];
        const int d = q1 - q0;
        fs[tid][0] = static_cast<float>(e.side.rhs[node]);
        fs[tid][1] = logf(1.0f + static_cast<float>(d));
        fs[tid][2] = static_cast<float>(sqrt(s2));
        for (int k = 0; k < 3; ++k) e.f[node * 3 + k] = fs[tid][k];
        e.inv_deg[node] = 1.0f / static_cast<float>(d > 0 ? d : 1);
    }
    __syncthreads();
    const int o = tid & (H - 1);
    const float w0 = bf(e.W[o * 3 + 0]), w1 = bf(e.W[o * 3 + 1]), w2 = bf(e.W[o * 3 + 2]), b0 = bf(e.b[o]);
    const int n1 = min(e.side.nodes, n0 + kEmbedThreads);
    for (int n = n0 + tid / H; n < n1; n += kEmbedThreads / H) {
        const float* f = fs[n - n0];
        float acc = b0;
        acc += w0 * f[0];
        acc += w1 * f[1];
        acc += w2 * f[2];
        e.h[static_cast<size_t>(n) * H + o] = acc > 0.f ? acc : 0.f;
    }
}

// sum_q v[q] scale_in[ci[q]] in[ci[q]][:] over q0 <= q < q1, in that order, for the row of
// each half warp (an empty range where it has none); a lane holds four features. Bound by
// the L2's rate of gathered rows (256 bytes an entry): a half warp reads 16 entries' indices
// and values at a time and keeps U rows in flight: four,
// with more warps per SM, on large graphs (layer 47 -> 39 us), eight where few warps run (16
// -> 13 us at 5000 nodes).
template <int U>
__device__ __forceinline__ float4 gather_row(int q0, int q1, const int* __restrict__ ci, const double* __restrict__ v,
                                             const float* __restrict__ scale_in, const float* __restrict__ in) {
    const int l16 = threadIdx.x & 15;
    const float4* in4 = reinterpret_cast<const float4*>(in);
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int q = q0; __any_sync(0xffffffffu, q < q1); q += 16) {
        const int cnt = min(16, max(0, q1 - q));
        int c = 0;
        float w = 0.f;
        if (l16 < cnt) {
            c = ci[q + l16];
            w = static_cast<float>(v[q + l16]) * (scale_in ? scale_in[c] : 1.f);
        }
        const int most = max(cnt, __shfl_xor_sync(0xffffffffu, cnt, 16));
        for (int t = 0; t < most; t += U) {
            float4 x[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int cu = __shfl_sync(0xffffffffu, c, t + u, 16);
                if (t + u < cnt) x[u] = in4[static_cast<size_t>(cu) * (H / 4) + l16];
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const float wu = __shfl_sync(0xffffffffu, w, t + u, 16);
                if (t + u < cnt) {
                    a.x += wu * x[u].x;
                    a.y += wu * x[u].y;
                    a.z += wu * x[u].z;
                    a.w += wu * x[u].w;
                }
            }
        }
    }
    return a;
}
__device__ __forceinline__ float4 mask_positive(float4 g, float4 y) {
    if (!(y.x > 0.f)) g.x = 0.f;
    if (!(y.y > 0.f)) g.y = 0.f;
    if (!(y.z > 0.f)) g.z = 0.f;
    if (!(y.w > 0.f)) g.w = 0.f;
    return g;
}

// Two 64x64 BF16 matrices into shared memory as FP32, W[o][k]; transposed: at [k][o].
template <bool Transposed>
__device__ __forceinline__ void stage_weights(const uint16_t* __restrict__ W1, const uint16_t* __restrict__ W2,
                                              float* s1, float* s2) {
    const int o = threadIdx.x & 63, k0 = (threadIdx.x >> 6) * 16;
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const uint4* src = reinterpret_cast<const uint4*>((m ? W2 : W1) + o * H + k0);
        float* dst = m ? s2 : s1;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint4 u = src[h];
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const uint32_t bits = t & 1 ? w[t >> 1] & 0xffff0000u : w[t >> 1] << 16;
                const int k = k0 + 8 * h + t;
                dst[Transposed ? k * H + o : o * H + k] = __uint_as_float(bits);
            }
        }
    }
}

constexpr int kLd = H + 4;      // staged node rows: 16-byte aligned, two rows in different banks
constexpr size_t layer_smem(int nodes, int arrays) { return (2 * H * H + arrays * nodes * kLd) * sizeof(float); }

// One side of a layer: m = inv_deg sum_q v h_other (kept in mout when the gradient needs it),
// out[o] = relu(W1[o] . x1 + W2[o] . m + b[o]). A block gathers the messages of 16 * NPT
// nodes (half a warp per node) into shared memory next to their own features and then forms a
// 4-output x NPT-node tile per thread from 16-byte shared loads. Gather and product as two
// kernels, one output per thread and step, took 11 + 23 us a side at 2000 / 5000 nodes and
// 41 + 90 us at 19,000 / 48,000; now 13 and 39 us.
template <int NPT>
__global__ void __launch_bounds__(256, NPT == 1 ? 3 : 4) k_layer(Side side, const float* __restrict__ inv_deg,
                                                  const float* __restrict__ other, const float* __restrict__ x1,
                                                  const uint16_t* __restrict__ W1, const uint16_t* __restrict__ W2,
                                                  const uint16_t* __restrict__ b, float* __restrict__ mout,
                                                  float* __restrict__ out) {
    constexpr int TN = 16 * NPT;
    extern __shared__ __align__(16) float sm[];
    float *Wa = sm, *Wb = Wa + H * H, *xs1 = Wb + H * H, *xs2 = xs1 + TN * kLd;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int og = tid & 15, ng = tid >> 4;
    stage_weights<true>(W1, W2, Wa, Wb);
    float bo[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) bo[c] = bf(b[4 * og + c]);
    for (int n0 = blockIdx.x * TN; n0 < side.nodes; n0 += gridDim.x * TN) {
        for (int nn = 2 * wid + (lane >> 4); nn < TN; nn += 16) {      // half a warp per node
            const int node = n0 + nn;
            const bool on = node < side.nodes;
            const size_t at = static_cast<size_t>(node) * (H / 4) + (lane & 15);
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (on) x = reinterpret_cast<const float4*>(x1)[at];
            float4 m = gather_row<NPT == 1 ? 8 : 4>(on ? side.rp[node] : 0, on ? side.rp[node + 1] : 0, side.ci,
                                                    side.v, nullptr, other);
            const float so = on ? inv_deg[node] : 0.f;
            m = make_float4(so * m.x, so * m.y, so * m.z, so * m.w);
            if (on && mout) reinterpret_cast<float4*>(mout)[at] = m;
            *reinterpret_cast<float4*>(xs1 + nn * kLd + 4 * (lane & 15)) = x;
            *reinterpret_cast<float4*>(xs2 + nn * kLd + 4 * (lane & 15)) = m;
        }
        __syncthreads();
        float acc[NPT][4];
#pragma unroll
        for (int p = 0; p < NPT; ++p)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[p][c] = bo[c];
#pragma unroll 2
        for (int k = 0; k < H; k += 4) {
            float a1[NPT][4], a2[NPT][4];
#pragma unroll
            for (int p = 0; p < NPT; ++p) {
                *reinterpret_cast<float4*>(a1[p]) = *reinterpret_cast<const float4*>(xs1 + (ng + 16 * p) * kLd + k);
                *reinterpret_cast<float4*>(a2[p]) = *reinterpret_cast<const float4*>(xs2 + (ng + 16 * p) * kLd + k);
            }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                float w1[4], w2[4];
                *reinterpret_cast<float4*>(w1) = *reinterpret_cast<const float4*>(Wa + (k + kk) * H + 4 * og);
                *reinterpret_cast<float4*>(w2) = *reinterpret_cast<const float4*>(Wb + (k + kk) * H + 4 * og);
#pragma unroll
                for (int p = 0; p < NPT; ++p)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[p][c] += w1[c] * a1[p][kk] + w2[c] * a2[p][kk];
            }
        }
#pragma unroll
        for (int p = 0; p < NPT; ++p) {
            const int node = n0 + ng + 16 * p;
            if (node < side.nodes) {
                float r[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) r[c] = acc[p][c] > 0.f ? acc[p][c] : 0.f;
                *reinterpret_cast<float4*>(out + static_cast<size_t>(node) * H + 4 * og) =
                    *reinterpret_cast<const float4*>(r);
            }
        }
        __syncthreads();
    }
}

// Outputs of every node, a warp per node: columns (log x, log s) into oc (N x 2), rows y into
// orr (M); as FP64 into the given arrays (may be null).
__global__ void __launch_bounds__(256) k_heads(int N, int M, const float* __restrict__ hc,
                                               const float* __restrict__ hr, const uint16_t* __restrict__ Wc,
                                               const uint16_t* __restrict__ bc, const uint16_t* __restrict__ Wr,
                                               const uint16_t* __restrict__ br, float* __restrict__ oc,
                                               float* __restrict__ orr, double* __restrict__ lx,
                                               double* __restrict__ ls, double* __restrict__ ly) {
    const int node = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (node >= N + M) return;
    const bool col = node < N;
    const int i = col ? node : node - N, OUT = col ? 2 : 1;
    const float* x = (col ? hc : hr) + static_cast<size_t>(i) * H;
    const uint16_t* W = col ? Wc : Wr;
    const uint16_t* b = col ? bc : br;
    const float x0 = x[lane], x1 = x[lane + 32];
    for (int o = 0; o < OUT; ++o) {
        float acc = 0.f;
        acc += bf(W[o * H + lane]) * x0;
        acc += bf(W[o * H + lane + 32]) * x1;
        for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
        if (lane == 0) {
            const float r = acc + bf(b[o]);
            (col ? oc : orr)[i * OUT + o] = r;
            double* out = col ? (o ? ls : lx) : ly;
            if (out) out[i] = static_cast<double>(r);
        }
    }
}

// loss: columns (log x, log s) vs targets, rows y vs target; writes d_out and adds the loss
__global__ void k_loss(int N, int M, const float* __restrict__ oc, const float* __restrict__ orr,
                       const double* __restrict__ tx, const double* __restrict__ ts, const double* __restrict__ ty,
                       float* __restrict__ doc, float* __restrict__ dor, double* loss) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    double l = 0.0;
    const float wc = 1.0f / (2.0f * N), wr = 1.0f / M;
    if (t < N) {
        const float ex = oc[2 * t] - static_cast<float>(fmin(fmax(tx[t], -30.0), 30.0));
        const float es = oc[2 * t + 1] - static_cast<float>(fmin(fmax(ts[t], -30.0), 30.0));
        doc[2 * t] = 2.f * wc * ex;
        doc[2 * t + 1] = 2.f * wc * es;
        l += wc * (ex * ex + es * es);
    } else if (t < N + M) {
        const int i = t - N;
        const float ey = orr[i] - static_cast<float>(ty[i]);
        dor[i] = 2.f * wr * ey;
        l += wr * ey * ey;
    }
    l = warp_sum(l);
    if ((threadIdx.x & 31) == 0 && l != 0.0) atomicAdd(loss, l);
}

// Heads backward, columns (OUT = 2) in the first `col_blocks` blocks, then rows (OUT = 1):
// dx[node][k] = sum_o d[node][o] W[o][k]; dW, db accumulated. Thread (k, g) runs down every
// fourth node of the block's kHeadNodes with its sums in registers.
constexpr int kHeadNodes = 256;
__global__ void __launch_bounds__(256) k_heads_bwd(int N, int M, int col_blocks, const float* __restrict__ hc,
                                                   const float* __restrict__ hr, const float* __restrict__ doc,
                                                   const float* __restrict__ dor, const uint16_t* __restrict__ Wc,
                                                   const uint16_t* __restrict__ Wr, float* __restrict__ dhc,
                                                   float* __restrict__ dhr, float* __restrict__ gWc,
                                                   float* __restrict__ gbc, float* __restrict__ gWr,
                                                   float* __restrict__ gbr) {
    __shared__ float red[4][4][H];
    const bool col = static_cast<int>(blockIdx.x) < col_blocks;
    const int nodes = col ? N : M, OUT = col ? 2 : 1;
    const float* x = col ? hc : hr;
    const float* d = col ? doc : dor;
    const uint16_t* W = col ? Wc : Wr;
    float* dx = col ? dhc : dhr;
    const int k = threadIdx.x & 63, g = threadIdx.x >> 6;
    const int n0 = (col ? blockIdx.x : blockIdx.x - col_blocks) * kHeadNodes, n1 = min(nodes, n0 + kHeadNodes);
    const float w0 = bf(W[k]), w1 = col ? bf(W[H + k]) : 0.f;
    float s0 = 0.f, s1 = 0.f, b0 = 0.f, b1 = 0.f;
#pragma unroll 4
    for (int node = n0 + g; node < n1; node += 4) {
        const float d0 = d[node * OUT], d1 = col ? d[node * OUT + 1] : 0.f;
        const float xv = x[static_cast<size_t>(node) * H + k];
        dx[static_cast<size_t>(node) * H + k] = d0 * w0 + d1 * w1;
        s0 += d0 * xv;
        s1 += d1 * xv;
        b0 += d0;
        b1 += d1;
    }
    red[g][0][k] = s0;
    red[g][1][k] = s1;
    red[g][2][k] = b0;
    red[g][3][k] = b1;
    __syncthreads();
    if (g == 0) {
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            if (o >= OUT) break;
            atomicAdd((col ? gWc : gWr) + o * H + k, (red[0][o][k] + red[1][o][k]) + (red[2][o][k] + red[3][o][k]));
            if (k == 0)
                atomicAdd((col ? gbc : gbr) + o,
                          (red[0][2 + o][0] + red[1][2 + o][0]) + (red[2][2 + o][0] + red[3][2 + o][0]));
        }
    }
}

// One side of a layer backward. The gradient of the layer's output, d plus (Gather) the
// messages sum_q v scale_in src of the other side's, is masked with y > 0 into g (kept in d),
// and dx1 = g W1, dx2 = g W2. Blocks and threads as in k_layer.
template <bool Gather, int NPT>
__global__ void __launch_bounds__(256, NPT == 1 ? 3 : 4) k_layer_bwd(Side side, const float* __restrict__ scale_in,
                                                      const float* __restrict__ src, float* __restrict__ d,
                                                      const float* __restrict__ y, const uint16_t* __restrict__ W1,
                                                      const uint16_t* __restrict__ W2, float* __restrict__ dx1,
                                                      float* __restrict__ dx2) {
    constexpr int TN = 16 * NPT;
    extern __shared__ __align__(16) float sm[];
    float *Wa = sm, *Wb = Wa + H * H, *gs = Wb + H * H;      // W[o][k]
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int kg = tid & 15, ng = tid >> 4;
    stage_weights<false>(W1, W2, Wa, Wb);
    for (int n0 = blockIdx.x * TN; n0 < side.nodes; n0 += gridDim.x * TN) {
        for (int nn = 2 * wid + (lane >> 4); nn < TN; nn += 16) {      // half a warp per node
            const int node = n0 + nn;
            const bool on = node < side.nodes;
            const size_t at = static_cast<size_t>(node) * (H / 4) + (lane & 15);
            float4 g = make_float4(0.f, 0.f, 0.f, 0.f), yv = g;
            if (on) {
                g = reinterpret_cast<float4*>(d)[at];
                yv = reinterpret_cast<const float4*>(y)[at];
            }
            if (Gather) {
                const float4 m = gather_row<NPT == 1 ? 8 : 4>(on ? side.rp[node] : 0, on ? side.rp[node + 1] : 0,
                                                              side.ci, side.v, scale_in, src);
                g = make_float4(g.x + m.x, g.y + m.y, g.z + m.z, g.w + m.w);
            }
            g = mask_positive(g, yv);
            if (on) reinterpret_cast<float4*>(d)[at] = g;
            *reinterpret_cast<float4*>(gs + nn * kLd + 4 * (lane & 15)) = g;
        }
        __syncthreads();
        float a1[NPT][4] = {}, a2[NPT][4] = {};
#pragma unroll 2
        for (int o = 0; o < H; o += 4) {
            float g[NPT][4];
#pragma unroll
            for (int p = 0; p < NPT; ++p)
                *reinterpret_cast<float4*>(g[p]) = *reinterpret_cast<const float4*>(gs + (ng + 16 * p) * kLd + o);
#pragma unroll
            for (int oo = 0; oo < 4; ++oo) {
                float w1[4], w2[4];
                *reinterpret_cast<float4*>(w1) = *reinterpret_cast<const float4*>(Wa + (o + oo) * H + 4 * kg);
                *reinterpret_cast<float4*>(w2) = *reinterpret_cast<const float4*>(Wb + (o + oo) * H + 4 * kg);
#pragma unroll
                for (int p = 0; p < NPT; ++p)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        a1[p][c] += g[p][oo] * w1[c];
                        a2[p][c] += g[p][oo] * w2[c];
                    }
            }
        }
#pragma unroll
        for (int p = 0; p < NPT; ++p) {
            const int node = n0 + ng + 16 * p;
            if (node < side.nodes) {
                const size_t at = static_cast<size_t>(node) * H + 4 * kg;
                *reinterpret_cast<float4*>(dx1 + at) = *reinterpret_cast<const float4*>(a1[p]);
                *reinterpret_cast<float4*>(dx2 + at) = *reinterpret_cast<const float4*>(a2[p]);
            }
        }
        __syncthreads();
    }
}

// k_grad_w's sums over the nodes n0 .. n1 - 1, with a choice at each product (any values).
__device__ __noinline__ void grad_w_masked(int n0, int n1, const float* __restrict__ g, const float* __restrict__ x1,
                                           const float* __restrict__ x2, float* __restrict__ dW1,
                                           float* __restrict__ dW2, float* __restrict__ db) {
    const int o = threadIdx.x & 63, k0 = (threadIdx.x >> 6) * 32;       // output o, 32 of the 128 columns
    const float* x = k0 < H ? x1 + k0 : x2 + k0 - H;
    float sum[32] = {}, sumb = 0.f;
    for (int n = n0; n < n1; ++n) {
        const float gv = g[static_cast<size_t>(n) * H + o];
        sumb += gv;
#pragma unroll
        for (int c = 0; c < 32; ++c)
            if (gv != 0.f) sum[c] += gv * x[static_cast<size_t>(n) * H + c];
    }
    float* dW = (k0 < H ? dW1 + k0 : dW2 + k0 - H) + o * H;
#pragma unroll
    for (int c = 0; c < 32; ++c) atomicAdd(dW + c, sum[c]);
    if (k0 == 0) atomicAdd(db + o, sumb);
}

// dW1[o][k] += sum_node g[node][o] x1[node][k], dW2 with x2, db[o] += sum_node g[node][o] over
// `chunk` nodes a block: a 64 x 128 product with the nodes as its inner dimension. Thread
// (og, kg) keeps 4 outputs x 8 of the 128 columns in registers (32 multiply-adds per three
// 16-byte shared loads); the next 32 nodes are loaded while the present ones are summed. One
// output column group per thread with the operands from the L1 took 182 us a matrix at
// 19,000 / 48,000 nodes; now 20 us for both. Sums of 32 nodes are added up separately. A
// masked gradient (0) leaves its node's features out whatever they are: a block with a sum that
// is not finite, where 0 may have met an infinity or a NaN, adds up once more by grad_w_masked().
__global__ void __launch_bounds__(256) k_grad_w(int nodes, int chunk, const float* __restrict__ g,
                                                const float* __restrict__ x1, const float* __restrict__ x2,
                                                float* __restrict__ dW1, float* __restrict__ dW2,
                                                float* __restrict__ db) {
    constexpr int S = 32;
    __shared__ __align__(16) float gs[S * H], xs[S * 2 * H];
    const int tid = threadIdx.x, og = tid & 15, kg = tid >> 4;
    const int n0 = blockIdx.x * chunk, n1 = min(nodes, n0 + chunk);
    float sum[4][8] = {}, sumb[4] = {};            // of the stages' own sums
    float4 pg[2], px[4];
    auto load = [&](int n) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int e = tid + 256 * u, node = n + (e >> 4);
            pg[u] = node < n1 ? reinterpret_cast<const float4*>(g)[static_cast<size_t>(node) * 16 + (e & 15)]
                              : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = tid + 256 * (u & 1), node = n + (e >> 4);
            const float4* x = reinterpret_cast<const float4*>(u < 2 ? x1 : x2);
            px[u] = node < n1 ? x[static_cast<size_t>(node) * 16 + (e & 15)] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    load(n0);
    for (int n = n0; n < n1; n += S) {
#pragma unroll
        for (int u = 0; u < 2; ++u) reinterpret_cast<float4*>(gs)[tid + 256 * u] = pg[u];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int e = tid + 256 * (u & 1);
            reinterpret_cast<float4*>(xs)[(e >> 4) * 32 + (u < 2 ? 0 : 16) + (e & 15)] = px[u];
        }
        __syncthreads();
        if (n + S < n1) load(n + S);
        float acc[4][8] = {}, accb[4] = {};
#pragma unroll 4
        for (int nn = 0; nn < S; ++nn) {
            float gv[4], xv[8];
            *reinterpret_cast<float4*>(gv) = *reinterpret_cast<const float4*>(gs + nn * H + 4 * og);
            *reinterpret_cast<float4*>(xv) = *reinterpret_cast<const float4*>(xs + nn * 2 * H + 8 * kg);
            *reinterpret_cast<float4*>(xv + 4) = *reinterpret_cast<const float4*>(xs + nn * 2 * H + 8 * kg + 4);
#pragma unroll
            for (int o = 0; o < 4; ++o) {
                accb[o] += gv[o];
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[o][c] += gv[o] * xv[c];
            }
        }
#pragma unroll
        for (int o = 0; o < 4; ++o) {
            sumb[o] += accb[o];
#pragma unroll
            for (int c = 0; c < 8; ++c) sum[o][c] += acc[o][c];
        }
        __syncthreads();
    }
    float none = 0.f;                              // stays 0 over finite sums
#pragma unroll
    for (int o = 0; o < 4; ++o)
#pragma unroll
        for (int c = 0; c < 8; ++c) none += 0.f * sum[o][c];
    if (__syncthreads_or(none != 0.f)) {
        grad_w_masked(n0, n1, g, x1, x2, dW1, dW2, db);
        return;
    }
    float* dW = (kg < 8 ? dW1 : dW2) + 8 * (kg & 7);
#pragma unroll
    for (int o = 0; o < 4; ++o) {
        float4* dst = reinterpret_cast<float4*>(dW + (4 * og + o) * H);
        atomicAdd(dst, make_float4(sum[o][0], sum[o][1], sum[o][2], sum[o][3]));
        atomicAdd(dst + 1, make_float4(sum[o][4], sum[o][5], sum[o][6], sum[o][7]));
        if (kg == 0) atomicAdd(db + 4 * og + o, sumb[o]);
    }
}

// Embeddings backward, columns in the first `col_blocks` blocks (their gradient d plus the
// messages of the first layer's rows), then rows: g = d masked with h0 > 0, dE[o][k] += g[o]
// f[k], de[o] += g[o]; a masked gradient (0) leaves its node's features out, which may be
// infinite or no numbers. Half a warp takes every sixteenth node of the block's kEmbedNodes.
struct EmbedGrad {
    int nodes;
    const float *d, *h, *f;
    float *dW, *db;
};
constexpr int kEmbedNodes = 256;
__global__ void __launch_bounds__(256) k_embed_bwd(EmbedGrad cols, EmbedGrad rows, int col_blocks, Side side,
                                                   const float* __restrict__ scale_in,
                                                   const float* __restrict__ src) {
    __shared__ float red[16][16][17];
    const int l16 = threadIdx.x & 15, hw = threadIdx.x >> 4;
    const bool col = static_cast<int>(blockIdx.x) < col_blocks;
    const EmbedGrad& e = col ? cols : rows;
    const int n0 = (col ? blockIdx.x : blockIdx.x - col_blocks) * kEmbedNodes;
    float s[4][4] = {};
    for (int nn = hw; nn < kEmbedNodes; nn += 16) {
        const int node = n0 + nn;
        const bool on = node < e.nodes;
        const size_t at = static_cast<size_t>(node) * (H / 4) + l16;
        float4 g = make_float4(0.f, 0.f, 0.f, 0.f), y = g;
        float f[4] = {0.f, 0.f, 0.f, 1.f};
        if (on) {
            g = reinterpret_cast<const float4*>(e.d)[at];
            y = reinterpret_cast<const float4*>(e.h)[at];
            for (int k = 0; k < 3; ++k) f[k] = e.f[node * 3 + k];
        }
        if (col) {
            const float4 m = gather_row<4>(on ? side.rp[node] : 0, on ? side.rp[node + 1] : 0, side.ci, side.v,
                                           scale_in, src);
            g = make_float4(g.x + m.x, g.y + m.y, g.z + m.z, g.w + m.w);
        }
        g = mask_positive(g, y);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (g.x != 0.f) s[0][k] += g.x * f[k];
            if (g.y != 0.f) s[1][k] += g.y * f[k];
            if (g.z != 0.f) s[2][k] += g.z * f[k];
            if (g.w != 0.f) s[3][k] += g.w * f[k];
        }
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) red[hw][q][l16] = s[q >> 2][q & 3];
    __syncthreads();
    float t = 0.f;
    for (int w = 0; w < 16; ++w) t += red[w][hw][l16];           // sum q = hw of every half warp
    const int o = 4 * l16 + (hw >> 2), k = hw & 3;
    atomicAdd(k < 3 ? e.dW + o * 3 + k : e.db + o, t);
}

__global__ void k_adam(int n, float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, float lr, float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = isfinite(g[i]) ? fminf(fmaxf(g[i], -10.f), 10.f) : 0.f;
    m[i] = 0.9f * m[i] + 0.1f * gi;
    v[i] = 0.999f * v[i] + 0.001f * gi * gi;
    w[i] -= lr * (m[i] / c1) / (sqrtf(v[i] / c2) + 1e-8f);
}

// Launches of the layer kernels: 16 nodes a block while that leaves at most four blocks per
// SM, then 32 (half the weight loads per node). 5000 nodes on 152 SMs: 16 a block.
inline bool wide_layer(int nodes, int sms) { return nodes > sms * 4 * 16; }
inline int layer_blocks(int nodes, int per, int sms) { return std::min((nodes + per - 1) / per, sms * 4); }

void layer_forward(const Side& side, const float* inv_deg, const float* other, const float* x1, const uint16_t* W1,
                   const uint16_t* W2, const uint16_t* b, float* mout, float* out, int sms, cudaStream_t st) {
    if (wide_layer(side.nodes, sms))
        k_layer<2><<<layer_blocks(side.nodes, 32, sms), 256, layer_smem(32, 2), st>>>(side, inv_deg, other, x1, W1,
                                                                                      W2, b, mout, out);
    else
        k_layer<1><<<layer_blocks(side.nodes, 16, sms), 256, layer_smem(16, 2), st>>>(side, inv_deg, other, x1, W1,
                                                                                      W2, b, mout, out);
}

template <bool Gather>
void layer_backward(const Side& side, const float* scale_in, const float* src, float* d, const float* y,
                    const uint16_t* W1, const uint16_t* W2, float* dx1, float* dx2, int sms, cudaStream_t st) {
    if (wide_layer(side.nodes, sms))
        k_layer_bwd<Gather, 2><<<layer_blocks(side.nodes, 32, sms), 256, layer_smem(32, 1), st>>>(
            side, scale_in, src, d, y, W1, W2, dx1, dx2);
    else
        k_layer_bwd<Gather, 1><<<layer_blocks(side.nodes, 16, sms), 256, layer_smem(16, 1), st>>>(
            side, scale_in, src, d, y, W1, W2, dx1, dx2);
}

void grad_weights(int nodes, const float* g, const float* x1, const float* x2, float* dW1, float* dW2, float* db,
                  int sms, cudaStream_t st) {
    const int chunk = std::max(64, ((nodes + sms - 1) / sms + 31) / 32 * 32);
    k_grad_w<<<(nodes + chunk - 1) / chunk, 256, 0, st>>>(nodes, chunk, g, x1, x2, dW1, dW2, db);
}

inline int nb(int64_t n, int t = 256) { return static_cast<int>((n + t - 1) / t); }

}  // namespace

Gnn::Gnn(unsigned long long seed) {
    nparams_ = kLay.total;
    int device = 0;
    SK_CUDA(cudaGetDevice(&device));
    SK_CUDA(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, device));
    SK_CUDA(cudaMalloc(&master_, sizeof(float) * nparams_));
    SK_CUDA(cudaMalloc(&wbf_, sizeof(uint16_t) * nparams_));
    SK_CUDA(cudaMalloc(&grad_, sizeof(float) * nparams_));
    SK_CUDA(cudaMalloc(&adam_m_, sizeof(float) * nparams_));
    SK_CUDA(cudaMalloc(&adam_v_, sizeof(float) * nparams_));
    SK_CUDA(cudaMalloc(&loss_, sizeof(double)));
    loss_host_.alloc(1);
    SK_CUDA(cudaEventCreateWithFlags(&loss_ready_, cudaEventDisableTiming));
    for (auto* f : {k_layer<1>, k_layer<2>})
        SK_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(layer_smem(32, 2))));
    SK_CUDA(cudaMemset(adam_m_, 0, sizeof(float) * nparams_));
    SK_CUDA(cudaMemset(adam_v_, 0, sizeof(float) * nparams_));
    // Glorot-uniform weights, zero biases (portable splitmix64 stream)
    std::vector<float> w(nparams_, 0.f);
    uint64_t st = seed ? seed : 0x5eedULL;
    auto next = [&]() {
        uint64_t z = (st += 0x9E3779B97F4A7C15ull);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return static_cast<double>(z >> 11) * (1.0 / 9007199254740992.0);
    };
    auto fill = [&](size_t off, int fo, int fi) {
        const double lim = std::sqrt(6.0 / (fo + fi));
        for (int q = 0; q < fo * fi; ++q) w[off + q] = static_cast<float>((2.0 * next() - 1.0) * lim);
    };
    fill(kLay.Ec, H, 3);
    fill(kLay.Er, H, 3);
    for (int l = 0; l < L; ++l) {
        fill(kLay.Wrr[l], H, H); fill(kLay.Wrm[l], H, H); fill(kLay.Wcc[l], H, H); fill(kLay.Wcm[l], H, H);
    }
    fill(kLay.Hc, 2, H);
    fill(kLay.Hr, 1, H);
    for (size_t q = 0; q < H; ++q) { w[kLay.ec + q] = 0.01f; w[kLay.er + q] = 0.01f; }
    set_params(w.data());
}

Gnn::~Gnn() {
    for (void* p : {static_cast<void*>(master_), static_cast<void*>(wbf_), static_cast<void*>(grad_),
                    static_cast<void*>(adam_m_), static_cast<void*>(adam_v_), static_cast<void*>(loss_),
                    static_cast<void*>(fc_), static_cast<void*>(fr_), static_cast<void*>(hc_),
                    static_cast<void*>(hr_), static_cast<void*>(mc_), static_cast<void*>(mr_),
                    static_cast<void*>(oc_), static_cast<void*>(or_), static_cast<void*>(dc_),
                    static_cast<void*>(dr_), static_cast<void*>(dm_), static_cast<void*>(dt_),
                    static_cast<void*>(inv_deg_r_), static_cast<void*>(inv_deg_c_)})
        if (p) cudaFree(p);
    if (loss_ready_) {
        cudaEventSynchronize(loss_ready_);                    // nothing uses loss_host_ any more
        cudaEventDestroy(loss_ready_);
    }
}

void Gnn::get_params(float* out) const {
    SK_CUDA(cudaMemcpy(out, master_, sizeof(float) * nparams_, cudaMemcpyDeviceToHost));
}

void Gnn::set_params(const float* in) {
    SK_CUDA(cudaMemcpy(master_, in, sizeof(float) * nparams_, cudaMemcpyHostToDevice));
    k_to_bf16<<<nb(static_cast<int64_t>(nparams_)), 256>>>(static_cast<int>(nparams_), master_, wbf_);
    SK_CUDA(cudaGetLastError());
    SK_CUDA(cudaDeviceSynchronize());
}

void Gnn::ensure(const DeviceLP& lp) {
    if (lp.N <= capN_ && lp.M <= capM_) return;
    for (float** p : {&fc_, &fr_, &hc_, &hr_, &mc_, &mr_, &oc_, &or_, &dc_, &dr_, &dm_, &dt_, &inv_deg_r_, &inv_deg_c_})
        if (*p) { cudaFree(*p); *p = nullptr; }
    capN_ = lp.N;
    capM_ = lp.M;
    const size_t N = capN_, M = capM_, X = std::max(N, M);
    SK_CUDA(cudaMalloc(&fc_, sizeof(float) * N * 3));
    SK_CUDA(cudaMalloc(&fr_, sizeof(float) * M * 3));
    SK_CUDA(cudaMalloc(&hc_, sizeof(float) * (L + 1) * N * H));
    SK_CUDA(cudaMalloc(&hr_, sizeof(float) * (L + 1) * M * H));
    SK_CUDA(cudaMalloc(&mc_, sizeof(float) * L * N * H));
    SK_CUDA(cudaMalloc(&mr_, sizeof(float) * L * M * H));
    SK_CUDA(cudaMalloc(&oc_, sizeof(float) * N * 2));
    SK_CUDA(cudaMalloc(&or_, sizeof(float) * M));
    SK_CUDA(cudaMalloc(&dc_, sizeof(float) * 2 * N * H));
    SK_CUDA(cudaMalloc(&dr_, sizeof(float) * 2 * M * H));
    SK_CUDA(cudaMalloc(&dm_, sizeof(float) * X * H));
    SK_CUDA(cudaMalloc(&dt_, sizeof(float) * X * H));
    SK_CUDA(cudaMalloc(&inv_deg_r_, sizeof(float) * M));
    SK_CUDA(cudaMalloc(&inv_deg_c_, sizeof(float) * N));
}

void Gnn::forward(const DeviceLP& lp, cudaStream_t st, double* out_logx, double* out_logs, double* out_y,
                  const double* t_logx, const double* t_logs, const double* t_y) {
    ensure(lp);
    const int N = lp.N, M = lp.M;
    const size_t NH = static_cast<size_t>(N) * H, MH = static_cast<size_t>(M) * H;
    const uint16_t* w = wbf_;
    const Side cols{N, lp.t_rp, lp.t_ci, lp.t_v, lp.c}, rows{M, lp.a_rp, lp.a_ci, lp.a_v, lp.b};
    const int all = nb((static_cast<int64_t>(N) + M) * 32);
    const int cb = nb(N, kEmbedThreads);
    k_embed<<<cb + nb(M, kEmbedThreads), kEmbedThreads, 0, st>>>(
        EmbedSide{cols, w + kLay.Ec, w + kLay.ec, fc_, inv_deg_c_, hc_},
        EmbedSide{rows, w + kLay.Er, w + kLay.er, fr_, inv_deg_r_, hr_}, cb);
    const bool keep = t_logx != nullptr;               // backward() needs the messages
    for (int l = 0; l < L; ++l) {
        float* hcl = hc_ + l * NH;
        float* hrl = hr_ + l * MH;
        layer_forward(rows, inv_deg_r_, hcl, hrl, w + kLay.Wrr[l], w + kLay.Wrm[l], w + kLay.br[l],
                      keep ? mr_ + l * MH : nullptr, hrl + MH, sms_, st);
        layer_forward(cols, inv_deg_c_, hrl + MH, hcl, w + kLay.Wcc[l], w + kLay.Wcm[l], w + kLay.bc[l],
                      keep ? mc_ + l * NH : nullptr, hcl + NH, sms_, st);
    }
    k_heads<<<all, 256, 0, st>>>(N, M, hc_ + L * NH, hr_ + L * MH, w + kLay.Hc, w + kLay.oc, w + kLay.Hr,
                                 w + kLay.orr, oc_, or_, out_logx, out_logs, out_y);
    SK_CUDA(cudaGetLastError());
    if (!t_logx) return;
    SK_CUDA(cudaMemsetAsync(loss_, 0, sizeof(double), st));
    // d_oc -> dm_ (N x 2), d_or -> dt_ (M)
    k_loss<<<nb(static_cast<int64_t>(N) + M), 256, 0, st>>>(N, M, oc_, or_, t_logx, t_logs, t_y, dm_, dt_, loss_);
    SK_CUDA(cudaMemcpyAsync(loss_host_.ptr, loss_, sizeof(double), cudaMemcpyDeviceToHost, st));
    SK_CUDA(cudaEventRecord(loss_ready_, st));
}

double Gnn::loss() const {
    SK_CUDA(cudaEventSynchronize(loss_ready_));
    return *loss_host_.ptr;
}

void Gnn::backward(const DeviceLP& lp, cudaStream_t st, float* grad_host) {
    const int N = lp.N, M = lp.M;
    const size_t NH = static_cast<size_t>(N) * H, MH = static_cast<size_t>(M) * H;
    const uint16_t* w = wbf_;
    float* gr = grad_;
    const Side cols{N, lp.t_rp, lp.t_ci, lp.t_v, lp.c}, rows{M, lp.a_rp, lp.a_ci, lp.a_v, lp.b};
    SK_CUDA(cudaMemsetAsync(gr, 0, sizeof(float) * nparams_, st));
    float* dhc = dc_;          // gradient w.r.t. hc[l] (current)
    float* dhc2 = dc_ + NH;    // next buffer
    float* dhr = dr_;
    float* dhr2 = dr_ + MH;
    // heads: dm_ holds d_oc (N x 2), dt_ holds d_or (M)
    const int hb = nb(N, kHeadNodes);
    k_heads_bwd<<<hb + nb(M, kHeadNodes), 256, 0, st>>>(N, M, hb, hc_ + L * NH, hr_ + L * MH, dm_, dt_, w + kLay.Hc,
                                                        w + kLay.Hr, dhc, dhr, gr + kLay.Hc, gr + kLay.oc,
                                                        gr + kLay.Hr, gr + kLay.orr);
    for (int l = L - 1; l >= 0; --l) {
        float* hcl = hc_ + l * NH;
        float* hrl = hr_ + l * MH;
        // hc[l+1] = relu(Wcc hc[l] + Wcm mc[l] + bc), with the messages of the layer above
        // (mr[l+1] = diag(inv_deg_r) A hc[l+1]); d mc[l] -> dm_
        if (l == L - 1)
            layer_backward<false>(cols, nullptr, nullptr, dhc, hcl + NH, w + kLay.Wcc[l], w + kLay.Wcm[l], dhc2, dm_,
                                  sms_, st);
        else
            layer_backward<true>(cols, inv_deg_r_, dt_, dhc, hcl + NH, w + kLay.Wcc[l], w + kLay.Wcm[l], dhc2, dm_,
                                 sms_, st);
        grad_weights(N, dhc, hcl, mc_ + l * NH, gr + kLay.Wcc[l], gr + kLay.Wcm[l], gr + kLay.bc[l], sms_, st);
        // hr[l+1] = relu(Wrr hr[l] + Wrm mr[l] + br), and mc[l] = diag(inv_deg_c) A^T hr[l+1];
        // d mr[l] -> dt_
        layer_backward<true>(rows, inv_deg_c_, dm_, dhr, hrl + MH, w + kLay.Wrr[l], w + kLay.Wrm[l], dhr2, dt_,
                             sms_, st);
        grad_weights(M, dhr, hrl, mr_ + l * MH, gr + kLay.Wrr[l], gr + kLay.Wrm[l], gr + kLay.br[l], sms_, st);
        std::swap(dhc, dhc2);
        std::swap(dhr, dhr2);
    }
    const int eb = nb(N, kEmbedNodes);
    k_embed_bwd<<<eb + nb(M, kEmbedNodes), 256, 0, st>>>(
        EmbedGrad{N, dhc, hc_, fc_, gr + kLay.Ec, gr + kLay.ec},
        EmbedGrad{M, dhr, hr_, fr_, gr + kLay.Er, gr + kLay.er}, eb, cols, inv_deg_r_, dt_);
    SK_CUDA(cudaGetLastError());
    if (grad_host) {
        SK_CUDA(cudaMemcpyAsync(grad_host, gr, sizeof(float) * nparams_, cudaMemcpyDeviceToHost, st));
        SK_CUDA(cudaStreamSynchronize(st));
    }
}

void Gnn::adam_step(cudaStream_t st, float lr) {
    ++adam_t_;
    const float c1 = 1.f - std::pow(0.9f, static_cast<float>(adam_t_));
    const float c2 = 1.f - std::pow(0.999f, static_cast<float>(adam_t_));
    k_adam<<<nb(static_cast<int64_t>(nparams_)), 256, 0, st>>>(static_cast<int>(nparams_), master_, grad_, adam_m_,
                                                                 adam_v_, lr, c1, c2);
    k_to_bf16<<<nb(static_cast<int64_t>(nparams_)), 256, 0, st>>>(static_cast<int>(nparams_), master_, wbf_);
    SK_CUDA(cudaGetLastError());
}

}  // namespace dev
}  // namespace sankhya
