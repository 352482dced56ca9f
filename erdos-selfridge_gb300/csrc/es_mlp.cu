// Learned cost model of the planner: a 3-layer FP32 MLP (in -> H -> H -> out, ReLU), trained and
// evaluated on the GPU by these kernels.  Sizes are tiny (in <= 64, H 32 or 64, out <= 8, samples in
// the thousands): plain FP32 FMAs, every sum in FP32 in index order; tensor cores would not pay for
// themselves at this size, and would change the rounding.
//
// Parameters, flat FP32: W1[H][D], b1[H], W2[H][H], b2[H], W3[O][H], b3[O].
// Loss: mean squared error over samples x outputs.  Gradients are reduced deterministically: one
// partial gradient per tile of 32 samples, the tiles summed in order.  Optimiser: Adam (Kingma & Ba),
// bias-corrected.
//
// One CTA works on one tile with the parameters in shared memory: lanes along the units of a layer,
// warps along the samples, rows padded to odd strides so that a weight matrix reads without bank
// conflicts in both directions.  Training is one launch per stretch of whole epochs, a cluster of
// eight CTAs that keeps parameters, moments and gradients on chip: each CTA differentiates its
// tiles, the cluster sums them through distributed shared memory (each CTA owns an eighth of the
// parameters and their Adam moments, in registers), and every owner writes its new parameters to
// all eight CTAs.  Two hardware cluster barriers per step are the only synchronisation.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/es_gb300.h"

namespace {

constexpr int kTile = 32;        // samples per tile
constexpr int kMaxD = 64, kMaxH = 64, kMaxO = 8;
constexpr int kThreads = 256;    // 8 warps x 4 samples
constexpr int kRow = 68;         // activation row stride: 16-byte aligned, rows on shifted banks
constexpr int kCluster = 8;

thread_local std::string g_mlp_err;
int mlp_fail(int code, const std::string& m) {
    g_mlp_err = m;
    return code;
}

struct Dims {
    int D, H, O;
    __host__ __device__ int nW1() const { return H * D; }
    __host__ __device__ int oB1() const { return nW1(); }
    __host__ __device__ int oW2() const { return oB1() + H; }
    __host__ __device__ int oB2() const { return oW2() + H * H; }
    __host__ __device__ int oW3() const { return oB2() + H; }
    __host__ __device__ int oB3() const { return oW3() + O * H; }
    __host__ __device__ int n() const { return oB3() + O; }
    // the same in shared memory, with padded rows: W1 rows of sD (odd, zeros past D), W2 of H + 1
    __host__ __device__ int D4() const { return (D + 3) / 4 * 4; }
    __host__ __device__ int sD() const { return D4() + 1; }
    __host__ __device__ int pB1() const { return H * sD(); }
    __host__ __device__ int pW2() const { return pB1() + H; }
    __host__ __device__ int pB2() const { return pW2() + H * (H + 1); }
    __host__ __device__ int pW3() const { return pB2() + H; }
    __host__ __device__ int pB3() const { return pW3() + O * H; }
    __host__ __device__ int pn() const { return (pB3() + O + 3) / 4 * 4; }
    // padded place of flat parameter p
    __host__ __device__ int place(int p) const {
        if (p < nW1()) return p / D * sD() + p % D;
        if (p < oW2()) return pB1() + (p - oB1());
        if (p < oB2()) return pW2() + (p - oW2()) / H * (H + 1) + (p - oW2()) % H;
        return pB2() + (p - oB2());   // b2, W3 and b3 keep their order
    }
};

__device__ __forceinline__ float at4(const float4 v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// Copies the flat parameters to their padded places (the padding is zeroed first).
__device__ __forceinline__ void load_params(const Dims& d, const float* __restrict__ P, float* sp) {
    for (int i = threadIdx.x; i < d.pn(); i += kThreads) sp[i] = 0.f;
    __syncthreads();
    for (int p = threadIdx.x; p < d.n(); p += kThreads) sp[d.place(p)] = P[p];
}

// out[t][j] = relu(b[j] + sum_i W[j][i] in[t][i]) for the tile; W rows of `stride`, K inputs (a
// multiple of 4, zero-padded).  A thread sums its units j = lane (and lane + 32) for four samples.
template <int H>
__device__ __forceinline__ void layer(const float* W, int stride, const float* b, const float* in, int K, float* out) {
    constexpr int NJ = H / 32;
    const int lane = threadIdx.x & 31, t0 = (threadIdx.x >> 5) * 4;
    float acc[NJ][4];
#pragma unroll
    for (int u = 0; u < NJ; ++u)
#pragma unroll
        for (int t = 0; t < 4; ++t) acc[u][t] = b[lane + 32 * u];
#pragma unroll 2
    for (int i = 0; i < K; i += 4) {
        float4 x[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) x[t] = *reinterpret_cast<const float4*>(in + (t0 + t) * kRow + i);
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int u = 0; u < NJ; ++u) {
                const float w = W[(lane + 32 * u) * stride + i + c];
#pragma unroll
                for (int t = 0; t < 4; ++t) acc[u][t] = fmaf(w, at4(x[t], c), acc[u][t]);
            }
    }
#pragma unroll
    for (int u = 0; u < NJ; ++u)
#pragma unroll
        for (int t = 0; t < 4; ++t) out[(t0 + t) * kRow + lane + 32 * u] = fmaxf(acc[u][t], 0.f);
}

// y of sample t, output o: b3[o] + sum_i W3[o][i] a2[t][i]
template <int H>
__device__ __forceinline__ float output(const Dims& d, const float* sp, const float* a2, int t, int o) {
    const float* w = sp + d.pW3() + o * H;
    float acc = sp[d.pB3() + o];
#pragma unroll 4
    for (int i = 0; i < H; i += 4) {
        const float4 a = *reinterpret_cast<const float4*>(a2 + t * kRow + i);
        acc = fmaf(w[i], a.x, acc);
        acc = fmaf(w[i + 1], a.y, acc);
        acc = fmaf(w[i + 2], a.z, acc);
        acc = fmaf(w[i + 3], a.w, acc);
    }
    return acc;
}

// dW[j][i] = sum_t g[t][j] x[t][i] for i < D, into rows of `stride`; db[j] = sum_t g[t][j]
template <int H>
__device__ __forceinline__ void weight_grad(const float* g, const float* x, int D, float* dW, int stride, float* db) {
    constexpr int NJ = H / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = 4 * warp; i < D; i += 4 * (kThreads / 32)) {
        float acc[NJ][4];
#pragma unroll
        for (int u = 0; u < NJ; ++u)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[u][c] = 0.f;
#pragma unroll 8
        for (int t = 0; t < kTile; ++t) {
            const float4 v = *reinterpret_cast<const float4*>(x + t * kRow + i);
#pragma unroll
            for (int u = 0; u < NJ; ++u) {
                const float gv = g[t * kRow + lane + 32 * u];
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[u][c] = fmaf(gv, at4(v, c), acc[u][c]);
            }
        }
#pragma unroll
        for (int u = 0; u < NJ; ++u)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (i + c < D) dW[(lane + 32 * u) * stride + i + c] = acc[u][c];
    }
    if (warp == (kThreads / 32) - 1) {
#pragma unroll
        for (int u = 0; u < NJ; ++u) {
            float acc = 0.f;
#pragma unroll 8
            for (int t = 0; t < kTile; ++t) acc += g[t * kRow + lane + 32 * u];
            db[lane + 32 * u] = acc;
        }
    }
}

// Shared memory of one tile's forward and backward pass, after the parameters.
struct TileMem {
    float *xs, *ts, *a1, *a2, *g2, *g1, *go, *G;
};
constexpr int kAct = kTile * kRow;

// Gradient of one tile of nt samples (rows past nt are zero) into G, in the parameters' padded
// places, of the loss sum (y - t)^2 * scale over all tiles.  err (or null): y - t of sample t, output o
// at [32 o + t].
template <int H>
__device__ __forceinline__ void tile_grad(const Dims& d, const float* sp, const TileMem& m, int nt, float scale, float* err) {
    constexpr int NJ = H / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, t0 = warp * 4;
    layer<H>(sp, d.sD(), sp + d.pB1(), m.xs, d.D4(), m.a1);
    __syncthreads();
    layer<H>(sp + d.pW2(), H + 1, sp + d.pB2(), m.a1, H, m.a2);
    __syncthreads();
    // d loss / d out of sample t (a lane) and output o (a warp)
    if (warp < d.O) {
        const int t = lane, o = warp;
        float e = 0.f;
        if (t < nt) {
            e = output<H>(d, sp, m.a2, t, o) - m.ts[t * kMaxO + o];
        }
        if (err) err[32 * o + t] = e;
        m.go[t * kMaxO + o] = 2.f * e * scale;
    }
    __syncthreads();
    // back through layer 3: g2 = (W3^T go) * [a2 > 0]
#pragma unroll
    for (int t = t0; t < t0 + 4; ++t)
#pragma unroll
        for (int u = 0; u < NJ; ++u) {
            const int j = lane + 32 * u;
            float acc = 0.f;
            for (int o = 0; o < d.O; ++o) acc = fmaf(sp[d.pW3() + o * H + j], m.go[t * kMaxO + o], acc);
            m.g2[t * kRow + j] = m.a2[t * kRow + j] > 0.f ? acc : 0.f;
        }
    __syncthreads();
    // g1 = (W2^T g2) * [a1 > 0]
    {
        float acc[NJ][4];
#pragma unroll
        for (int u = 0; u < NJ; ++u)
#pragma unroll
            for (int t = 0; t < 4; ++t) acc[u][t] = 0.f;
        const float* W2 = sp + d.pW2();
#pragma unroll 2
        for (int i = 0; i < H; i += 4) {
            float4 x[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) x[t] = *reinterpret_cast<const float4*>(m.g2 + (t0 + t) * kRow + i);
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int u = 0; u < NJ; ++u) {
                    const float w = W2[(i + c) * (H + 1) + lane + 32 * u];
#pragma unroll
                    for (int t = 0; t < 4; ++t) acc[u][t] = fmaf(w, at4(x[t], c), acc[u][t]);
                }
        }
#pragma unroll
        for (int u = 0; u < NJ; ++u)
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int at = (t0 + t) * kRow + lane + 32 * u;
                m.g1[at] = m.a1[at] > 0.f ? acc[u][t] : 0.f;
            }
    }
    weight_grad<H>(m.g2, m.a1, H, m.G + d.pW2(), H + 1, m.G + d.pB2());
    // dW3[o][j], db3[o]
    for (int x = threadIdx.x; x < d.O * H; x += kThreads) {
        const int o = x / H, j = x % H;
        float acc = 0.f;
#pragma unroll 8
        for (int t = 0; t < kTile; ++t) acc = fmaf(m.go[t * kMaxO + o], m.a2[t * kRow + j], acc);
        m.G[d.pW3() + x] = acc;
    }
    if (threadIdx.x < d.O) {
        float acc = 0.f;
        for (int t = 0; t < kTile; ++t) acc += m.go[t * kMaxO + threadIdx.x];
        m.G[d.pB3() + threadIdx.x] = acc;
    }
    __syncthreads();
    weight_grad<H>(m.g1, m.xs, d.D, m.G, d.sD(), m.G + d.pB1());
}

// The tile memory carved out of `at` (16-byte aligned).
__device__ __forceinline__ TileMem carve(float* at, float* G) {
    TileMem m;
    m.xs = at;
    m.a1 = m.xs + kAct;
    m.a2 = m.a1 + kAct;
    m.g2 = m.a2 + kAct;
    m.g1 = m.g2 + kAct;
    m.ts = m.g1 + kAct;
    m.go = m.ts + kTile * kMaxO;
    m.G = G;
    return m;
}
constexpr int kTileFloats = 5 * kAct + 2 * kTile * kMaxO;

// Forward of one tile per CTA.  Shared memory: parameters, x and two activations.
template <int H>
__global__ void __launch_bounds__(kThreads) mlp_forward_kernel(Dims d, const float* __restrict__ P,
                                                               const float* __restrict__ X, uint64_t n,
                                                               float* __restrict__ Y) {
    extern __shared__ __align__(16) float sm[];
    float* sp = sm;
    float* xs = sm + d.pn();
    float *a1 = xs + kAct, *a2 = xs;   // layer 2 writes over x, which nothing reads any more
    const uint64_t n0 = (uint64_t)blockIdx.x * kTile;
    load_params(d, P, sp);
    for (int i = threadIdx.x; i < kTile * d.D4(); i += kThreads) {
        const int t = i / d.D4(), c = i % d.D4();
        xs[t * kRow + c] = (n0 + t < n && c < d.D) ? X[(n0 + t) * d.D + c] : 0.f;
    }
    __syncthreads();
    layer<H>(sp, d.sD(), sp + d.pB1(), xs, d.D4(), a1);
    __syncthreads();
    layer<H>(sp + d.pW2(), H + 1, sp + d.pB2(), a1, H, a2);
    __syncthreads();
    const int t = threadIdx.x & 31, o = threadIdx.x >> 5;
    if (o < d.O && n0 + t < n) Y[(n0 + t) * d.O + o] = output<H>(d, sp, a2, t, o);
}

// Gradient of one tile per CTA to Gout[blockIdx.x][n_params] and its squared error to L[blockIdx.x].
template <int H>
__global__ void __launch_bounds__(kThreads) mlp_grad_kernel(Dims d, const float* __restrict__ P,
                                                            const float* __restrict__ X, const float* __restrict__ T,
                                                            uint64_t n, float scale, float* __restrict__ Gout,
                                                            float* __restrict__ L) {
    extern __shared__ __align__(16) float sm[];
    float* sp = sm;
    const TileMem m = carve(sm + d.pn(), sm + d.pn() + kTileFloats);
    __shared__ float red[kThreads];
    const uint64_t n0 = (uint64_t)blockIdx.x * kTile;
    const int nt = (int)((n - n0) < (uint64_t)kTile ? (n - n0) : (uint64_t)kTile);
    load_params(d, P, sp);
    for (int i = threadIdx.x; i < kTile * d.D4(); i += kThreads) {
        const int t = i / d.D4(), c = i % d.D4();
        m.xs[t * kRow + c] = (t < nt && c < d.D) ? X[(n0 + t) * d.D + c] : 0.f;
    }
    for (int i = threadIdx.x; i < kTile * d.O; i += kThreads)
        m.ts[i / d.O * kMaxO + i % d.O] = i / d.O < nt ? T[(n0 + i / d.O) * d.O + i % d.O] : 0.f;
    __syncthreads();
    tile_grad<H>(d, sp, m, nt, scale, red);
    __syncthreads();
    float* g = Gout + (uint64_t)blockIdx.x * d.n();
    for (int p = threadIdx.x; p < d.n(); p += kThreads) g[p] = m.G[d.place(p)];
    if (threadIdx.x < 32) {   // a lane per output sums its samples in order, lane 0 the outputs
        float s = 0.f;
        if (threadIdx.x < d.O)
            for (int t = 0; t < kTile; ++t) s = fmaf(red[32 * threadIdx.x + t], red[32 * threadIdx.x + t], s);
        float all = 0.f;
        for (int o = 0; o < d.O; ++o) all += __shfl_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) L[blockIdx.x] = all;
    }
}

// Deterministic sum of the tiles' partial gradients (and losses) in tile order.
__global__ void mlp_reduce_kernel(const float* __restrict__ G, int tiles, int np, float* __restrict__ out,
                                  const float* __restrict__ L, float* __restrict__ loss) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < np) {
        float acc = 0.f;
#pragma unroll 8
        for (int t = 0; t < tiles; ++t) acc += G[(uint64_t)t * np + p];
        out[p] = acc;
    }
    if (p == 0 && loss) {
        float s = 0.f;
        for (int t = 0; t < tiles; ++t) s += L[t];
        *loss = s;
    }
}

// ---- training ----------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of `saddr` (a shared address of this CTA) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t peer_addr(uint32_t saddr, uint32_t rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
    return a;
}
__device__ __forceinline__ float4 peer_load(uint32_t a) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void peer_store(uint32_t a, const float4 v) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}

struct TrainArgs {
    Dims d;
    float *P, *m, *v;
    const float *X, *T;
    const uint32_t* idx;      // [epochs][n] sample order
    const float2* bias;       // per step: 1 - b1^s, 1 - b2^s
    uint32_t n, batch, steps_per_epoch, steps;
    float lr, b1, b2, eps;
};

// One Adam step of one parameter (m, v updated in place); c = bias corrections.
__device__ __forceinline__ float adam(float w, float gi, float& m, float& v, const TrainArgs& A, const float2 c) {
    const float mi = A.b1 * m + (1.f - A.b1) * gi;
    const float vi = A.b2 * v + (1.f - A.b2) * gi * gi;
    m = mi;
    v = vi;
    return w - A.lr * (mi / c.x) / (sqrtf(vi / c.y) + A.eps);
}

// One cluster trains `steps` minibatches.  An iteration is one tile per CTA; a step has `rounds` of
// them (batches above 256 samples), whose tiles the owners add in order.  The samples of the next
// iteration are fetched into registers during this one, their indices one iteration earlier still.
template <int H>
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kThreads) mlp_train_kernel(const TrainArgs A) {
    extern __shared__ __align__(16) float sm[];
    const Dims d = A.d;
    float* sp = sm;
    float* G = sm + d.pn();
    TileMem m = carve(G + d.pn(), G);
    uint32_t* rows = reinterpret_cast<uint32_t*>(G + d.pn() + kTileFloats);   // [2][32] sample indices
    const uint32_t rank = cluster_rank();
    const int tid = threadIdx.x;
    // CTA `rank` owns a contiguous eighth of the padded parameters, float4 by float4; the padding has
    // zero gradients and stays zero
    constexpr int kMaxPadded = kMaxH * (kMaxD + 1) + kMaxH + kMaxH * (kMaxH + 1) + kMaxH + kMaxO * kMaxH + kMaxO + 4;
    constexpr int kOwn = (kMaxPadded / 4 + kCluster * kThreads) / (kCluster * kThreads);
    constexpr int kFetch = kTile * kMaxD / kThreads;
    const int np = d.n(), n4 = d.pn() / 4, slice = (n4 + kCluster - 1) / kCluster;
    load_params(d, A.P, sp);
    for (int i = tid; i < kAct; i += kThreads) m.xs[i] = 0.f;
    int own[kOwn];      // this thread's float4s, or -1
    float4 mo[kOwn], ve[kOwn];
#pragma unroll
    for (int k = 0; k < kOwn; ++k) {
        const int i = tid + kThreads * k, at = (int)rank * slice + i;
        own[k] = i < slice && at < n4 ? at : -1;
    }
    float4* G4 = reinterpret_cast<float4*>(G);
    auto moments = [&](const float* src, float4 (&dst)[kOwn]) {   // flat global -> padded, own part
        for (int i = tid; i < d.pn(); i += kThreads) G[i] = 0.f;
        __syncthreads();
        for (int p = tid; p < np; p += kThreads) G[d.place(p)] = src[p];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kOwn; ++k) dst[k] = own[k] >= 0 ? G4[own[k]] : make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
    };
    moments(A.m, mo);
    moments(A.v, ve);
    for (int i = tid; i < d.pn(); i += kThreads) G[i] = 0.f;
    const uint32_t rounds = ((A.batch + kTile - 1) / kTile + kCluster - 1) / kCluster;
    const uint32_t iters = A.steps * rounds;
    // samples of iteration `it` for this CTA: first position in the epoch's order, and how many
    auto tile_of = [&](uint32_t it, uint32_t& base, int& nt) {
        const uint32_t step = it / rounds, q = (it % rounds) * kCluster + rank;
        const uint32_t ep = step / A.steps_per_epoch, b0 = (step % A.steps_per_epoch) * A.batch;
        const uint32_t nb = min(A.batch, A.n - b0);
        nt = it < iters && q * kTile < nb ? (int)min(nb - q * kTile, (uint32_t)kTile) : 0;
        base = ep * A.n + b0 + q * kTile;
    };
    float fx[kFetch];
    float ft = 0.f;
    const int nx = kTile * d.D, nty = kTile * d.O;   // values of a tile's x and targets
    auto fetch_rows = [&](uint32_t it) -> uint32_t {   // lanes of warp 0: one sample index each
        uint32_t base, v = 0;
        int nt;
        tile_of(it, base, nt);
        if (tid < nt) v = __ldg(A.idx + base + tid);
        return v;
    };
    auto fetch = [&](uint32_t it) {
        uint32_t base;
        int nt;
        tile_of(it, base, nt);
        const uint32_t* r = rows + (it & 1u) * kTile;
#pragma unroll
        for (int k = 0; k < kFetch; ++k) {
            const int e = tid + kThreads * k, t = e / d.D;
            fx[k] = e < nx && t < nt ? __ldg(A.X + (uint64_t)r[t] * d.D + (e - t * d.D)) : 0.f;
        }
        const int t = tid / d.O;
        ft = tid < nty && t < nt ? __ldg(A.T + (uint64_t)r[t] * d.O + (tid - t * d.O)) : 0.f;
    };
    auto put = [&]() {
#pragma unroll
        for (int k = 0; k < kFetch; ++k) {
            const int e = tid + kThreads * k, t = e / d.D;
            if (e < nx) m.xs[t * kRow + (e - t * d.D)] = fx[k];
        }
        if (tid < nty) m.ts[tid / d.O * kMaxO + tid % d.O] = ft;
    };
    if (tid < kTile) {
        rows[tid] = fetch_rows(0);
        rows[kTile + tid] = fetch_rows(1);
    }
    __syncthreads();
    fetch(0);
    put();
    cluster_sync();   // every CTA of the cluster runs before its shared memory is written
    const uint32_t g_addr = (uint32_t)__cvta_generic_to_shared(G), p_addr = (uint32_t)__cvta_generic_to_shared(sp);
    float4 acc[kOwn];
#pragma unroll
    for (int k = 0; k < kOwn; ++k) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t it = 0; it < iters; ++it) {
        uint32_t base;
        int nt;
        tile_of(it, base, nt);
        const uint32_t step = it / rounds, round = it % rounds;
        const uint32_t b0 = (step % A.steps_per_epoch) * A.batch, nb = min(A.batch, A.n - b0);
        fetch(it + 1);
        const uint32_t next_row = tid < kTile ? fetch_rows(it + 2) : 0u;
        if (nt > 0) tile_grad<H>(d, sp, m, nt, 1.f / (float)((uint64_t)nb * d.O), nullptr);
        cluster_sync();   // all tiles' gradients are there
        const uint32_t tiles = (nb + kTile - 1) / kTile;
        const uint32_t here = tiles > round * kCluster ? min(tiles - round * kCluster, (uint32_t)kCluster) : 0u;
        float4 part[kOwn][kCluster];
#pragma unroll
        for (int k = 0; k < kOwn; ++k)
#pragma unroll
            for (uint32_t r = 0; r < kCluster; ++r)
                if (own[k] >= 0 && r < here) part[k][r] = peer_load(peer_addr(g_addr + 16u * own[k], r));
#pragma unroll
        for (int k = 0; k < kOwn; ++k)
#pragma unroll
            for (uint32_t r = 0; r < kCluster; ++r)
                if (own[k] >= 0 && r < here) {
                    acc[k].x += part[k][r].x;
                    acc[k].y += part[k][r].y;
                    acc[k].z += part[k][r].z;
                    acc[k].w += part[k][r].w;
                }
        if (round + 1 == rounds) {
            const float2 c = __ldg(A.bias + step);
#pragma unroll
            for (int k = 0; k < kOwn; ++k) {
                if (own[k] < 0) continue;
                float4 w = reinterpret_cast<const float4*>(sp)[own[k]];
                w.x = adam(w.x, acc[k].x, mo[k].x, ve[k].x, A, c);
                w.y = adam(w.y, acc[k].y, mo[k].y, ve[k].y, A, c);
                w.z = adam(w.z, acc[k].z, mo[k].z, ve[k].z, A, c);
                w.w = adam(w.w, acc[k].w, mo[k].w, ve[k].w, A, c);
                acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (uint32_t r = 0; r < kCluster; ++r) peer_store(peer_addr(p_addr + 16u * own[k], r), w);
            }
        }
        put();
        if (tid < kTile) rows[(it & 1u) * kTile + tid] = next_row;
        cluster_sync();   // the new parameters are everywhere; gradients may be overwritten
    }
    // this CTA's part of the parameters and moments back to the flat arrays
    const int lo = 4 * (int)rank * slice, hi = lo + 4 * slice;
    auto store = [&](const float* padded, float* dst) {
        for (int p = tid; p < np; p += kThreads) {
            const int at = d.place(p);
            if (at >= lo && at < hi) dst[p] = padded[at];
        }
    };
    store(sp, A.P);
    auto flat = [&](const float4 (&src)[kOwn], float* dst) {
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kOwn; ++k)
            if (own[k] >= 0) G4[own[k]] = src[k];
        __syncthreads();
        store(G, dst);
    };
    flat(mo, A.m);
    flat(ve, A.v);
}

size_t fwd_smem(const Dims& d) { return sizeof(float) * (size_t)(d.pn() + 2 * kAct); }
size_t grad_smem(const Dims& d) { return sizeof(float) * (size_t)(2 * d.pn() + kTileFloats); }
size_t train_smem(const Dims& d) { return grad_smem(d) + 2 * kTile * sizeof(uint32_t); }

uint64_t splitmix(uint64_t& s) {
    uint64_t z = (s += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

}  // namespace

namespace {

// Device memory that grows to the largest request and is kept by its owner; requests above kKeep
// bytes are given back at the end of the call that made them.
struct Buffer {
    static constexpr size_t kKeep = 64u << 20;
    void* p = nullptr;
    size_t cap = 0;
    cudaError_t need(size_t bytes) {
        if (bytes <= cap) return cudaSuccess;
        release();
        const cudaError_t e = cudaMalloc(&p, bytes);
        if (e == cudaSuccess) cap = bytes;
        else p = nullptr;
        return e;
    }
    void release() {
        cudaFree(p);
        p = nullptr;
        cap = 0;
    }
    void trim() {
        if (cap > kKeep) release();
    }
    template <class T> T* as() const { return static_cast<T*>(p); }
};

}  // namespace

struct es_mlp {
    Dims d{};
    float* P = nullptr;      // parameters (one allocation with the four below)
    float* m = nullptr;      // Adam moments
    float* v = nullptr;
    float* g = nullptr;      // reduced gradient
    float* loss = nullptr;   // device scalar
    uint64_t steps = 0;
    Buffer X, T, Y, G, L, idx, bias;   // workspaces of the calls below
    cudaStream_t copy = nullptr;       // uploads of sample orders beside the training launches
    cudaEvent_t up = nullptr;
    void trim() {
        for (Buffer* b : {&X, &T, &Y, &G, &L, &idx, &bias}) b->trim();
    }
};

namespace {

// Every instance may use the shared memory it needs (above 48 KB on request), once per device.
cudaError_t allow_smem() {
    static bool done[64] = {false};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || (dev >= 0 && dev < 64 && done[dev])) return e;
    const Dims big{kMaxD, kMaxH, kMaxO};
    const void* fns[] = {(const void*)mlp_forward_kernel<32>, (const void*)mlp_forward_kernel<64>,
                         (const void*)mlp_grad_kernel<32>, (const void*)mlp_grad_kernel<64>,
                         (const void*)mlp_train_kernel<32>, (const void*)mlp_train_kernel<64>};
    for (const void* f : fns)
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)train_smem(big));
    if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev] = true;
    return e;
}

}  // namespace

extern "C" {

const char* es_mlp_last_error(void) { return g_mlp_err.c_str(); }

int es_mlp_destroy(es_mlp* M) {
    if (!M) return ES_OK;
    if (M->copy) cudaStreamSynchronize(M->copy);
    cudaFree(M->P);
    for (Buffer* b : {&M->X, &M->T, &M->Y, &M->G, &M->L, &M->idx, &M->bias}) b->release();
    if (M->up) cudaEventDestroy(M->up);
    if (M->copy) cudaStreamDestroy(M->copy);
    delete M;
    return ES_OK;
}

int es_mlp_create(uint32_t in_dim, uint32_t hidden, uint32_t out_dim, uint64_t seed, es_mlp** out) {
    if (!out) return mlp_fail(ES_ERR_ARG, "null output");
    *out = nullptr;
    if (in_dim < 1 || in_dim > kMaxD || hidden < 8 || hidden > kMaxH || hidden % 32 || out_dim < 1 ||
        out_dim > kMaxO || out_dim > hidden)
        return mlp_fail(ES_ERR_RANGE, "MLP dims must be in <= 64, hidden 32 or 64, out <= 8");
    es_mlp* M = new es_mlp();
    M->d = Dims{(int)in_dim, (int)hidden, (int)out_dim};
    const int np = M->d.n();
    std::vector<float> h(3 * np, 0.f);   // parameters, then the moments' zeros
    // He-uniform init for the ReLU layers, Glorot-uniform for the output, zero biases
    uint64_t s = seed;
    auto uni = [&](float a) { return (float)(((splitmix(s) >> 11) * (1.0 / 9007199254740992.0)) * 2.0 - 1.0) * a; };
    for (int i = 0; i < M->d.nW1(); ++i) h[i] = uni(std::sqrt(6.f / in_dim));
    for (int i = 0; i < (int)(hidden * hidden); ++i) h[M->d.oW2() + i] = uni(std::sqrt(6.f / hidden));
    for (int i = 0; i < (int)out_dim * (int)hidden; ++i) h[M->d.oW3() + i] = uni(std::sqrt(6.f / (hidden + out_dim)));
    cudaError_t e = allow_smem();
    if (e == cudaSuccess) e = cudaMalloc(&M->P, 4ull * (4 * np + 1));
    if (e == cudaSuccess) e = cudaMemcpy(M->P, h.data(), 12ull * np, cudaMemcpyHostToDevice);
    M->m = M->P + np;
    M->v = M->m + np;
    M->g = M->v + np;
    M->loss = M->g + np;
    if (e != cudaSuccess) {
        es_mlp_destroy(M);
        return mlp_fail(ES_ERR_CUDA, std::string("MLP setup: ") + cudaGetErrorString(e));
    }
    *out = M;
    return ES_OK;
}

int es_mlp_num_params(const es_mlp* M, uint64_t* n) {
    if (!M || !n) return mlp_fail(ES_ERR_ARG, "null argument");
    *n = (uint64_t)M->d.n();
    return ES_OK;
}

int es_mlp_get_params(es_mlp* M, float* out, uint64_t n) {
    if (!M || !out || n != (uint64_t)M->d.n()) return mlp_fail(ES_ERR_ARG, "bad parameter buffer");
    cudaError_t e = cudaMemcpy(out, M->P, 4ull * n, cudaMemcpyDeviceToHost);
    return e == cudaSuccess ? ES_OK : mlp_fail(ES_ERR_CUDA, cudaGetErrorString(e));
}

int es_mlp_set_params(es_mlp* M, const float* in, uint64_t n) {
    if (!M || !in || n != (uint64_t)M->d.n()) return mlp_fail(ES_ERR_ARG, "bad parameter buffer");
    cudaError_t e = cudaMemcpy(M->P, in, 4ull * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(M->m, 0, 8ull * n);   // both moments
    M->steps = 0;
    return e == cudaSuccess ? ES_OK : mlp_fail(ES_ERR_CUDA, cudaGetErrorString(e));
}

// Y[n][O] = MLP(X[n][D]); host buffers.
int es_mlp_forward(es_mlp* M, const float* X, uint64_t n, float* Y) {
    if (!M || (n && (!X || !Y))) return mlp_fail(ES_ERR_ARG, "null argument");
    if (n == 0) return ES_OK;
    const Dims d = M->d;
    cudaError_t e = M->X.need(4ull * n * d.D);
    if (e == cudaSuccess) e = M->Y.need(4ull * n * d.O);
    if (e == cudaSuccess) e = cudaMemcpy(M->X.p, X, 4ull * n * d.D, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        const unsigned tiles = (unsigned)((n + kTile - 1) / kTile);
        auto* f = d.H == 32 ? mlp_forward_kernel<32> : mlp_forward_kernel<64>;
        f<<<tiles, kThreads, fwd_smem(d)>>>(d, M->P, M->X.as<float>(), n, M->Y.as<float>());
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(Y, M->Y.p, 4ull * n * d.O, cudaMemcpyDeviceToHost);
    M->trim();
    return e == cudaSuccess ? ES_OK : mlp_fail(ES_ERR_CUDA, cudaGetErrorString(e));
}

// Loss and gradient of the rows in M->X, M->T (on the device already).
static cudaError_t device_loss_grad(es_mlp* M, uint64_t n, float* loss, float* grad) {
    const Dims d = M->d;
    const int np = d.n();
    const unsigned tiles = (unsigned)((n + kTile - 1) / kTile);
    cudaError_t e = M->G.need(4ull * tiles * np);
    if (e == cudaSuccess) e = M->L.need(4ull * tiles);
    if (e == cudaSuccess) {
        const float scale = 1.f / (float)(n * d.O);
        auto* f = d.H == 32 ? mlp_grad_kernel<32> : mlp_grad_kernel<64>;
        f<<<tiles, kThreads, grad_smem(d)>>>(d, M->P, M->X.as<float>(), M->T.as<float>(), n, scale, M->G.as<float>(),
                                             M->L.as<float>());
        mlp_reduce_kernel<<<(np + 255) / 256, 256>>>(M->G.as<float>(), (int)tiles, np, M->g, M->L.as<float>(), M->loss);
        e = cudaGetLastError();
    }
    float l = 0.f;
    if (e == cudaSuccess) e = cudaMemcpy(&l, M->loss, 4, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && grad) e = cudaMemcpy(grad, M->g, 4ull * np, cudaMemcpyDeviceToHost);
    *loss = l / (float)(n * d.O);
    return e;
}

// Full-batch loss (mean squared error) and its gradient with respect to every parameter.
int es_mlp_loss_grad(es_mlp* M, const float* X, const float* T, uint64_t n, float* loss, float* grad) {
    if (!M || !X || !T || n == 0 || !loss) return mlp_fail(ES_ERR_ARG, "null argument or empty set");
    const Dims d = M->d;
    cudaError_t e = M->X.need(4ull * n * d.D);
    if (e == cudaSuccess) e = M->T.need(4ull * n * d.O);
    if (e == cudaSuccess) e = cudaMemcpy(M->X.p, X, 4ull * n * d.D, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(M->T.p, T, 4ull * n * d.O, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = device_loss_grad(M, n, loss, grad);
    M->trim();
    return e == cudaSuccess ? ES_OK : mlp_fail(ES_ERR_CUDA, cudaGetErrorString(e));
}

// Minibatch Adam on (X, T): `epochs` passes over a seeded permutation, `batch` samples a step.  One
// launch per epoch: the host draws the next epoch's order, and a second stream uploads it, while the
// cluster works on the last one.
int es_mlp_train(es_mlp* M, const float* X, const float* T, uint64_t n, uint32_t epochs, uint32_t batch,
                 float lr, uint64_t seed, float* final_loss) {
    if (!M || !X || !T || n == 0 || batch == 0) return mlp_fail(ES_ERR_ARG, "null argument or empty set");
    if (n > 0xffffffffull) return mlp_fail(ES_ERR_RANGE, "more than 2^32 samples");
    const Dims d = M->d;
    const uint32_t step_batch = (uint32_t)std::min<uint64_t>(batch, n);
    const uint32_t spe = (uint32_t)((n + batch - 1) / batch);
    // epochs whose orders and step constants are on the device at a time
    const uint64_t per_epoch = 4ull * n + 8ull * spe;
    const uint32_t hold = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(epochs, (32ull << 20) / per_epoch));
    cudaError_t e = allow_smem();
    if (e == cudaSuccess && !M->copy) e = cudaStreamCreateWithFlags(&M->copy, cudaStreamNonBlocking);
    if (e == cudaSuccess && !M->up) e = cudaEventCreateWithFlags(&M->up, cudaEventDisableTiming);
    if (e == cudaSuccess) e = M->X.need(4ull * n * d.D);
    if (e == cudaSuccess) e = M->T.need(4ull * n * d.O);
    if (e == cudaSuccess) e = M->idx.need(4ull * n * hold);
    if (e == cudaSuccess) e = M->bias.need(8ull * spe * hold);
    if (e == cudaSuccess) e = cudaMemcpy(M->X.p, X, 4ull * n * d.D, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(M->T.p, T, 4ull * n * d.O, cudaMemcpyHostToDevice);
    std::vector<uint32_t> perm(n);
    std::vector<float2> bias(spe);
    for (uint64_t i = 0; i < n; ++i) perm[i] = (uint32_t)i;
    uint64_t s = seed;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    auto* kernel = d.H == 32 ? mlp_train_kernel<32> : mlp_train_kernel<64>;
    for (uint32_t ep = 0; ep < epochs && e == cudaSuccess; ++ep) {
        for (uint64_t i = n - 1; i > 0; --i) {   // Fisher-Yates with a seeded generator
            const uint64_t j = splitmix(s) % (i + 1);
            std::swap(perm[i], perm[j]);
        }
        for (uint32_t i = 0; i < spe; ++i) {
            M->steps += 1;
            bias[i] = make_float2(1.f - std::pow(b1, (float)M->steps), 1.f - std::pow(b2, (float)M->steps));
        }
        const uint32_t at = ep % hold;
        if (at == 0 && ep) e = cudaStreamSynchronize(nullptr);   // the held orders are used up
        uint32_t* idx = M->idx.as<uint32_t>() + n * at;
        float2* bs = M->bias.as<float2>() + (uint64_t)spe * at;
        if (e == cudaSuccess) e = cudaMemcpyAsync(idx, perm.data(), 4ull * n, cudaMemcpyHostToDevice, M->copy);
        if (e == cudaSuccess) e = cudaMemcpyAsync(bs, bias.data(), 8ull * spe, cudaMemcpyHostToDevice, M->copy);
        // the pageable copies have read the host arrays once the copy stream is idle
        if (e == cudaSuccess) e = cudaEventRecord(M->up, M->copy);
        if (e == cudaSuccess) e = cudaStreamWaitEvent(nullptr, M->up, 0);
        if (e == cudaSuccess) e = cudaEventSynchronize(M->up);
        if (e != cudaSuccess) break;
        TrainArgs a{d, M->P, M->m, M->v, M->X.as<float>(), M->T.as<float>(), idx, bs, (uint32_t)n, step_batch, spe, spe,
                    lr, b1, b2, eps};
        kernel<<<kCluster, kThreads, train_smem(d)>>>(a);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (final_loss && e == cudaSuccess) {
        float l = 0.f;
        e = device_loss_grad(M, n, &l, nullptr);
        *final_loss = l;
    }
    M->trim();
    return e == cudaSuccess ? ES_OK : mlp_fail(ES_ERR_CUDA, cudaGetErrorString(e));
}

}  // extern "C"
