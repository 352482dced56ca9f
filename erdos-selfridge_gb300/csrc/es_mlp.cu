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
// One CTA works on one tile with the parameters in shared memory.  A thread has two units x four samples
// of a layer, or four units x four inputs of a weight gradient, in pairs: two FMAs per instruction
// (fma.rn.f32x2: each rounds as it would alone).  Activations are kept unit by unit, and the inputs of a
// weight gradient sample by sample too, so that pairs come from 16-byte loads; row strides are odd
// multiples of 16 bytes, so that the rows of eight lanes fall on different banks.
//
// Training is one launch per epoch, a cluster of eight CTAs that keeps parameters, moments and gradients
// on chip: each CTA differentiates its tile, the owners sum the tiles (each CTA owns an eighth of the
// parameters and their Adam moments, in registers) and send the new parameters to the others, as bulk
// copies between the CTAs' shared memories counted by the receivers' barriers.  What bounds a step is
// the chain of its phases on two warps per scheduler.  34 inputs, 64 hidden, batches of 256, per step:
// 204 us with a launch per pass; 13.8 us on a cluster with gradients read and parameters written in
// place between two cluster barriers (9.2 thousand of 24.7 thousand cycles) and one unit x eight samples
// per thread; 10.6 us like this.  512 threads of one unit x four samples took 12.2 us.  Of the 17.9
// thousand cycles now 12 are the four products and gradients over 64 terms (0.7, 2.5, 2.4 and 4.2), 2.7
// the sums and Adam's divisions, 2.3 waits and copies.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <exception>
#include <memory>
#include <string>
#include <vector>

#include "../../include/es_gb300.h"

namespace {

constexpr int kTile = 32;        // samples per tile
constexpr int kMaxD = 64, kMaxH = 64, kMaxO = 8;
constexpr int kRow = 68;         // stride of rows over units or inputs, sample by sample
constexpr int kCol = 36;         // stride of rows over samples, unit by unit
constexpr int kCluster = 8;
__host__ __device__ constexpr int threads_of(int H) { return 4 * H; }   // a thread has 2 units x 4 samples of a layer

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
    // the same in shared memory, with padded rows: W1 rows of sD (zeros past D), W2 rows of H + 4
    __host__ __device__ int D4() const { return (D + 3) / 4 * 4; }
    __host__ __device__ int sD() const { return D4() / 4 % 2 ? D4() : D4() + 4; }
    __host__ __device__ int sH() const { return H + 4; }
    __host__ __device__ int pB1() const { return H * sD(); }
    __host__ __device__ int pW2() const { return pB1() + H; }
    __host__ __device__ int pB2() const { return pW2() + H * sH(); }
    __host__ __device__ int pW3() const { return pB2() + H; }
    __host__ __device__ int pB3() const { return pW3() + O * H; }
    __host__ __device__ int pn() const { return (pB3() + O + 3) / 4 * 4; }
    // padded place of flat parameter p
    __host__ __device__ int place(int p) const {
        if (p < nW1()) return p / D * sD() + p % D;
        if (p < oW2()) return pB1() + (p - oB1());
        if (p < oB2()) return pW2() + (p - oW2()) / H * sH() + (p - oW2()) % H;
        return pB2() + (p - oB2());   // b2, W3 and b3 keep their order
    }
};

// Two FP32 values in one 64-bit register pair.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpair(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ ulonglong2 ld_pairs(const float* p) { return *reinterpret_cast<const ulonglong2*>(p); }

// How the threads share a layer of H units: a warp has 16 units from u0 on and 16 samples, a thread the
// units u0 + g and u0 + g + 8 (or u0 + 2 g and u0 + 2 g + 1) and the samples t0 .. t0 + 3.  A 16-byte load
// takes a pass over the banks per half-warp and 128 bytes of different addresses: eight rows of weights
// and two of samples per half-warp is the least for a tile of 2 x 4 per thread.
template <int H>
struct Share {
    int u0, g, t0;
    __device__ Share() {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        u0 = 16 * (warp % (H / 16));
        g = lane & 7;
        t0 = 16 * (warp / (H / 16)) + 4 * (lane >> 3);
    }
};

// `rows` rows of n values to rows of `stride`, zeros past n: a warp per row.
__device__ __forceinline__ void load_rows(const float* __restrict__ src, int rows, int n, int stride, float* dst) {
    const int lane = threadIdx.x & 31;
#pragma unroll 8
    for (int j = threadIdx.x >> 5; j < rows; j += blockDim.x >> 5) {
        float v[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k] = lane + 32 * k < n ? __ldg(src + j * n + lane + 32 * k) : 0.f;
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (lane + 32 * k < stride) dst[j * stride + lane + 32 * k] = v[k];
    }
}
// Copies the flat parameters to their padded places, zeros between them.
__device__ __forceinline__ void load_params(const Dims& d, const float* __restrict__ P, float* sp) {
    load_rows(P, d.H, d.D, d.sD(), sp);
    load_rows(P + d.oW2(), d.H, d.H, d.sH(), sp + d.pW2());
    const int tail = d.pn() - d.pB2(), n = d.n() - d.oB2();
    for (int i = threadIdx.x; i < d.H; i += blockDim.x) sp[d.pB1() + i] = P[d.oB1() + i];
    for (int i = threadIdx.x; i < tail; i += blockDim.x) sp[d.pB2() + i] = i < n ? P[d.oB2() + i] : 0.f;
}

// four samples' values of one unit
__device__ __forceinline__ float4 four(const f32x2 (&a)[2]) {
    float4 y;
    unpair(a[0], y.x, y.y);
    unpair(a[1], y.z, y.w);
    return y;
}
__device__ __forceinline__ float4 where_positive(const float4 a, const float4 y) {
    return make_float4(a.x > 0.f ? y.x : 0.f, a.y > 0.f ? y.y : 0.f, a.z > 0.f ? y.z : 0.f, a.w > 0.f ? y.w : 0.f);
}
__device__ __forceinline__ void store4(float* p, const float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// acc[unit][t] += w[unit] in[t] for the thread's two units and four samples
__device__ __forceinline__ void fma_tile(float w0, float w1, const float* in, f32x2 (&a0)[2], f32x2 (&a1)[2]) {
    const ulonglong2 x = ld_pairs(in);
    const f32x2 p0 = pair(w0, w0), p1 = pair(w1, w1);
    a0[0] = fma2(p0, x.x, a0[0]);
    a0[1] = fma2(p0, x.y, a0[1]);
    a1[0] = fma2(p1, x.x, a1[0]);
    a1[1] = fma2(p1, x.y, a1[1]);
}

// out[j][t] = relu(b[j] + sum_i W[j][i] in[i][t]) for the tile (W rows of `stride`, K inputs, a multiple
// of 4, zero-padded), and the same sample by sample in `rows` (or null).
template <int H>
__device__ __forceinline__ void layer(const float* W, int stride, const float* b, const float* in, int K, float* out,
                                      float* rows) {
    const Share<H> me;
    f32x2 acc[2][2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const float bu = b[me.u0 + me.g + 8 * u];
        acc[u][0] = acc[u][1] = pair(bu, bu);
    }
    const float *w0 = W + (me.u0 + me.g) * stride, *w1 = w0 + 8 * stride, *x = in + me.t0;
#pragma unroll 4
    for (int i = 0; i < K; i += 4) {
        const float4 c0 = load4(w0 + i), c1 = load4(w1 + i);
        fma_tile(c0.x, c1.x, x + i * kCol, acc[0], acc[1]);
        fma_tile(c0.y, c1.y, x + (i + 1) * kCol, acc[0], acc[1]);
        fma_tile(c0.z, c1.z, x + (i + 2) * kCol, acc[0], acc[1]);
        fma_tile(c0.w, c1.w, x + (i + 3) * kCol, acc[0], acc[1]);
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int j = me.u0 + me.g + 8 * u;
        float4 y = four(acc[u]);
        y = make_float4(fmaxf(y.x, 0.f), fmaxf(y.y, 0.f), fmaxf(y.z, 0.f), fmaxf(y.w, 0.f));
        store4(out + j * kCol + me.t0, y);
        if (rows) {
            float* r = rows + me.t0 * kRow + j;
            r[0] = y.x;
            r[kRow] = y.y;
            r[2 * kRow] = y.z;
            r[3 * kRow] = y.w;
        }
    }
}

// y of sample t, output o: b3[o] + sum_i W3[o][i] a2[i][t]
template <int H>
__device__ __forceinline__ float output(const Dims& d, const float* sp, const float* a2, int t, int o) {
    const float* w = sp + d.pW3() + o * H;
    float acc = sp[d.pB3() + o];
#pragma unroll
    for (int i = 0; i < H; ++i) acc = fmaf(w[i], a2[i * kCol + t], acc);
    return acc;
}

// dW[j][i] = sum_t g[j][t] x[t][i] for i < D4 (a multiple of 4; x is zero past the inputs), into rows of
// `stride`; db[j] = sum_t g[j][t].  A thread has four units, eight apart, and four inputs.
template <int H>
__device__ __forceinline__ void weight_grad(const float* g, const float* x, int D4, float* dW, int stride, float* db) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int u0 = 32 * (warp % (H / 32)), j = u0 + (lane & 7), quarter = warp / (H / 32), i = 16 * quarter + 4 * (lane >> 3);
    if (16 * quarter < D4) {
        f32x2 acc[4][2];
#pragma unroll
        for (int u = 0; u < 4; ++u) acc[u][0] = acc[u][1] = pair(0.f, 0.f);
#pragma unroll 2
        for (int t = 0; t < kTile; t += 4) {
            float gs[4][4];
            ulonglong2 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float4 gv = load4(g + (j + 8 * u) * kCol + t);
                gs[u][0] = gv.x;
                gs[u][1] = gv.y;
                gs[u][2] = gv.z;
                gs[u][3] = gv.w;
                v[u] = ld_pairs(x + (t + u) * kRow + i);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const f32x2 gg = pair(gs[u][q], gs[u][q]);
                    acc[u][0] = fma2(gg, v[q].x, acc[u][0]);
                    acc[u][1] = fma2(gg, v[q].y, acc[u][1]);
                }
        }
        if (i < D4)
#pragma unroll
            for (int u = 0; u < 4; ++u) store4(dW + (j + 8 * u) * stride + i, four(acc[u]));
    }
    if (quarter == 3) {
        float a = 0.f;
#pragma unroll
        for (int t = 0; t < kTile; t += 4) {
            const float4 gv = load4(g + (u0 + lane) * kCol + t);
            a += gv.x;
            a += gv.y;
            a += gv.z;
            a += gv.w;
        }
        db[u0 + lane] = a;
    }
}

// Shared memory of one tile's forward and backward pass, after the parameters: x and a1 sample by
// sample (r) and unit by unit, the others unit by unit; targets and output gradients output by output.
struct TileMem {
    float *xr, *a1r, *xs, *a1, *a2, *g2, *g1, *ts, *go, *G;
};
constexpr int kRows = kTile * kRow, kCols = kMaxH * kCol;

// Gradient of one tile of nt samples (rows past nt are zero) into G, in the parameters' padded
// places, of the loss sum (y - t)^2 * scale over all tiles.  err (or null): y - t of sample t, output o
// at [32 o + t].
template <int H>
__device__ __forceinline__ void tile_grad(const Dims& d, const float* sp, const TileMem& m, int nt, float scale, float* err) {
    const Share<H> me;
    layer<H>(sp, d.sD(), sp + d.pB1(), m.xs, d.D4(), m.a1, m.a1r);
    __syncthreads();
    layer<H>(sp + d.pW2(), d.sH(), sp + d.pB2(), m.a1, H, m.a2, nullptr);
    __syncthreads();
    // d loss / d out of sample t (a lane) and output o (a warp)
    for (int o = threadIdx.x >> 5; o < d.O; o += H / 8) {
        const int t = threadIdx.x & 31;
        float e = 0.f;
        if (t < nt) e = output<H>(d, sp, m.a2, t, o) - m.ts[o * kTile + t];
        if (err) err[32 * o + t] = e;
        m.go[o * kTile + t] = 2.f * e * scale;
    }
    __syncthreads();
    // back through layer 3: g2 = (W3^T go) * [a2 > 0]
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int j = me.u0 + me.g + 8 * u, at = j * kCol + me.t0;
        float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int o = 0; o < d.O; ++o) {
            const float w = sp[d.pW3() + o * H + j];
            const float4 v = load4(m.go + o * kTile + me.t0);
            y.x = fmaf(w, v.x, y.x);
            y.y = fmaf(w, v.y, y.y);
            y.z = fmaf(w, v.z, y.z);
            y.w = fmaf(w, v.w, y.w);
        }
        store4(m.g2 + at, where_positive(load4(m.a2 + at), y));
    }
    __syncthreads();
    // g1 = (W2^T g2) * [a1 > 0]
    {
        f32x2 acc[2][2];
#pragma unroll
        for (int u = 0; u < 2; ++u) acc[u][0] = acc[u][1] = pair(0.f, 0.f);
        const float *w = sp + d.pW2() + me.u0 + 2 * me.g, *x = m.g2 + me.t0;
        const int sH = d.sH();
#pragma unroll 16
        for (int i = 0; i < H; ++i) {
            const float2 c = *reinterpret_cast<const float2*>(w + i * sH);
            fma_tile(c.x, c.y, x + i * kCol, acc[0], acc[1]);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int at = (me.u0 + 2 * me.g + u) * kCol + me.t0;
            store4(m.g1 + at, where_positive(load4(m.a1 + at), four(acc[u])));
        }
    }
    weight_grad<H>(m.g2, m.a1r, H, m.G + d.pW2(), d.sH(), m.G + d.pB2());
    // dW3[o][j], db3[o]
    for (int x = threadIdx.x; x < d.O * H; x += threads_of(H)) {
        const int o = x / H, j = x % H;
        float acc = 0.f;
#pragma unroll
        for (int t = 0; t < kTile; t += 4) {
            const float4 gv = *reinterpret_cast<const float4*>(m.go + o * kTile + t);
            const float4 av = *reinterpret_cast<const float4*>(m.a2 + j * kCol + t);
            acc = fmaf(gv.x, av.x, acc);
            acc = fmaf(gv.y, av.y, acc);
            acc = fmaf(gv.z, av.z, acc);
            acc = fmaf(gv.w, av.w, acc);
        }
        m.G[d.pW3() + x] = acc;
    }
    if (threadIdx.x < d.O) {
        float acc = 0.f;
        for (int t = 0; t < kTile; ++t) acc += m.go[threadIdx.x * kTile + t];
        m.G[d.pB3() + threadIdx.x] = acc;
    }
    __syncthreads();
    weight_grad<H>(m.g1, m.xr, d.D4(), m.G, d.sD(), m.G + d.pB1());
}

// The tile memory carved out of `at` (16-byte aligned).
__device__ __forceinline__ TileMem carve(float* at, float* G) {
    TileMem m;
    m.xr = at;
    m.a1r = m.xr + kRows;
    m.xs = m.a1r + kRows;
    m.a1 = m.xs + kCols;
    m.a2 = m.a1 + kCols;
    m.g2 = m.a2 + kCols;
    m.g1 = m.g2 + kCols;
    m.ts = m.g1 + kCols;
    m.go = m.ts + kTile * kMaxO;
    m.G = G;
    return m;
}
constexpr int kTileFloats = 2 * kRows + 5 * kCols + 2 * kTile * kMaxO;

// Forward of one tile per CTA.  Shared memory: parameters, x and two activations.
template <int H>
__global__ void __launch_bounds__(threads_of(H)) mlp_forward_kernel(Dims d, const float* __restrict__ P,
                                                               const float* __restrict__ X, uint64_t n,
                                                               float* __restrict__ Y) {
    extern __shared__ __align__(16) float sm[];
    float* sp = sm;
    float* xs = sm + d.pn();
    float *a1 = xs + kCols, *a2 = xs;   // layer 2 writes over x, which nothing reads any more
    const uint64_t n0 = (uint64_t)blockIdx.x * kTile;
    load_params(d, P, sp);
    for (int i = threadIdx.x; i < kTile * d.D4(); i += threads_of(H)) {
        const int t = i / d.D4(), c = i % d.D4();
        xs[c * kCol + t] = (n0 + t < n && c < d.D) ? X[(n0 + t) * d.D + c] : 0.f;
    }
    __syncthreads();
    layer<H>(sp, d.sD(), sp + d.pB1(), xs, d.D4(), a1, nullptr);
    __syncthreads();
    layer<H>(sp + d.pW2(), d.sH(), sp + d.pB2(), a1, H, a2, nullptr);
    __syncthreads();
    const int t = threadIdx.x & 31;
    for (int o = threadIdx.x >> 5; o < d.O; o += H / 8)
        if (n0 + t < n) Y[(n0 + t) * d.O + o] = output<H>(d, sp, a2, t, o);
}

// Gradient of one tile per CTA to Gout[blockIdx.x][n_params] and its squared error to L[blockIdx.x].
template <int H>
__global__ void __launch_bounds__(threads_of(H)) mlp_grad_kernel(Dims d, const float* __restrict__ P,
                                                            const float* __restrict__ X, const float* __restrict__ T,
                                                            uint64_t n, float scale, float* __restrict__ Gout,
                                                            float* __restrict__ L) {
    extern __shared__ __align__(16) float sm[];
    float* sp = sm;
    const TileMem m = carve(sm + d.pn(), sm + d.pn() + kTileFloats);
    __shared__ float red[kTile * kMaxO];
    const uint64_t n0 = (uint64_t)blockIdx.x * kTile;
    const int nt = (int)((n - n0) < (uint64_t)kTile ? (n - n0) : (uint64_t)kTile);
    load_params(d, P, sp);
    for (int i = threadIdx.x; i < kTile * d.D4(); i += threads_of(H)) {
        const int t = i / d.D4(), c = i % d.D4();
        const float v = (t < nt && c < d.D) ? X[(n0 + t) * d.D + c] : 0.f;
        m.xr[t * kRow + c] = v;
        m.xs[c * kCol + t] = v;
    }
    for (int i = threadIdx.x; i < kTile * d.O; i += threads_of(H))
        m.ts[i % d.O * kTile + i / d.O] = i / d.O < nt ? T[(n0 + i / d.O) * d.O + i % d.O] : 0.f;
    __syncthreads();
    tile_grad<H>(d, sp, m, nt, scale, red);
    __syncthreads();
    float* g = Gout + (uint64_t)blockIdx.x * d.n();
    for (int p = threadIdx.x; p < d.n(); p += threads_of(H)) g[p] = m.G[d.place(p)];
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
__device__ __forceinline__ void bar_init(uint32_t bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
// the barrier's current phase ends with this arrival and `bytes` of incoming copies
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Waits for the phase of `parity`; false after far more tries than a step can take.
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity) {
    for (int i = 0; i < (1 << 20); ++i) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
// Copies `bytes` of this CTA's shared memory at `src` to `dst`, counted by `bar` (both in one CTA of the cluster).
__device__ __forceinline__ void peer_copy(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "r"(src), "r"(bytes), "r"(bar) : "memory");
}
// orders this thread's writes to shared memory before copies of it
__device__ __forceinline__ void fence_copies() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

struct TrainArgs {
    Dims d;
    float *P, *m, *v;
    const float *X, *T;
    const uint32_t* idx;      // [epochs][n] sample order
    const float2* bias;       // per step: 1 - b1^s, 1 - b2^s
    int* err;                 // set to 1 when a wait ran out
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
//
// A CTA sends each eighth of its gradient to that eighth's owner, and an owner its new parameters to
// the seven others, as bulk copies counted by the receiver's barriers, and nothing else synchronises a
// step: an owner has all eight gradients only when no CTA reads the old parameters any more, and a CTA
// has all parameters only when its gradient has been read.  Every CTA sends in every iteration, also
// without a tile, so that no sender is ever a phase ahead.
template <int H>
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(threads_of(H)) mlp_train_kernel(const TrainArgs A) {
    extern __shared__ __align__(16) float sm[];
    constexpr int kThreads = threads_of(H);
    const Dims d = A.d;
    const int n4 = d.pn() / 4, slice = (n4 + kCluster - 1) / kCluster;   // float4s: all, of an owner
    float* sp = sm;
    float* G = sm + d.pn();
    float* part = G + d.pn();   // [8][4 slice]: the CTAs' gradients of this CTA's parameters
    float* tile = part + 4 * kCluster * slice;
    TileMem m = carve(tile, G);
    uint32_t* rows = reinterpret_cast<uint32_t*>(tile + kTileFloats);   // [2][32] sample indices
    __shared__ uint64_t bars[2];
    const uint32_t bar_g = (uint32_t)__cvta_generic_to_shared(&bars[0]), bar_p = bar_g + 8;
    const uint32_t rank = cluster_rank();
    const int tid = threadIdx.x;
    // CTA `rank` owns a contiguous eighth of the padded parameters; the padding has zero gradients and
    // stays zero
    constexpr int kMaxPadded = H * (kMaxD + 4) + H + H * (H + 4) + H + kMaxO * H + kMaxO + 4;
    constexpr int kOwn = (kMaxPadded / kCluster + 4 + kThreads - 1) / kThreads;
    constexpr int kFetch = kTile * kMaxD / kThreads;
    const int np = d.n(), lo = 4 * slice * (int)rank, mine = 4 * min(slice, n4 - slice * (int)rank);
    load_params(d, A.P, sp);
    for (int i = tid; i < kRows; i += kThreads) m.xr[i] = 0.f;
    for (int i = tid; i < kCols; i += kThreads) m.xs[i] = 0.f;
    float mo[kOwn], ve[kOwn], acc[kOwn];   // of own parameters lo + tid + kThreads k
    auto moments = [&](const float* src, float (&dst)[kOwn]) {   // flat global -> padded, own part
        for (int i = tid; i < d.pn(); i += kThreads) G[i] = 0.f;
        __syncthreads();
        for (int p = tid; p < np; p += kThreads) G[d.place(p)] = src[p];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kOwn; ++k) dst[k] = tid + kThreads * k < mine ? G[lo + tid + kThreads * k] : 0.f;
        __syncthreads();
    };
    // which of those are parameters: the division and the root of a padding's zeros would take their slow paths
    for (int i = tid; i < d.pn(); i += kThreads) G[i] = 0.f;
    __syncthreads();
    for (int p = tid; p < np; p += kThreads) G[d.place(p)] = 1.f;
    __syncthreads();
    uint32_t real = 0;
#pragma unroll
    for (int k = 0; k < kOwn; ++k)
        if (tid + kThreads * k < mine && G[lo + tid + kThreads * k] != 0.f) real |= 1u << k;
    __syncthreads();
    moments(A.m, mo);
    moments(A.v, ve);
    for (int i = tid; i < d.pn(); i += kThreads) G[i] = 0.f;
    const uint32_t rounds = ((A.batch + kTile - 1) / kTile + kCluster - 1) / kCluster;
    // an iteration: its round within the step, the step's first sample within the epoch
    struct Iter {
        uint32_t left, round, b0, epoch;   // iterations left with this one; epoch: where its order starts
    };
    auto next = [&](Iter c) {
        if (c.left) --c.left;
        if (++c.round == rounds) {
            c.round = 0;
            c.b0 += A.batch;
            if (c.b0 >= A.n) {
                c.b0 = 0;
                c.epoch += A.n;
            }
        }
        return c;
    };
    // samples of an iteration for this CTA: first position in the epochs' orders, and how many
    auto tile_of = [&](const Iter& c, uint32_t& base, int& nt) {
        const uint32_t at = (c.round * kCluster + rank) * kTile, nb = min(A.batch, A.n - c.b0);
        nt = c.left && at < nb ? (int)min(nb - at, (uint32_t)kTile) : 0;
        base = c.epoch + c.b0 + at;
    };
    // value e = tid + kThreads k of a tile's x is input xc[k] of sample xt[k] (32 and above: none)
    int xt[kFetch], xc[kFetch];
#pragma unroll
    for (int k = 0; k < kFetch; ++k) {
        xt[k] = (tid + kThreads * k) / d.D;
        xc[k] = (tid + kThreads * k) % d.D;
    }
    // the same for the targets
    constexpr int kFetchT = kTile * kMaxO / kThreads;
    int tt[kFetchT], to[kFetchT];
#pragma unroll
    for (int k = 0; k < kFetchT; ++k) {
        tt[k] = (tid + kThreads * k) / d.O;
        to[k] = (tid + kThreads * k) % d.O;
    }
    float fx[kFetch], ft[kFetchT];
    auto fetch_rows = [&](const Iter& c) -> uint32_t {   // lanes of warp 0: one sample index each
        uint32_t base, v = 0;
        int nt;
        tile_of(c, base, nt);
        if (tid < nt) v = __ldg(A.idx + base + tid);
        return v;
    };
    auto fetch = [&](const Iter& c, uint32_t half) {
        uint32_t base;
        int nt;
        tile_of(c, base, nt);
        const uint32_t* r = rows + half * kTile;
#pragma unroll
        for (int k = 0; k < kFetch; ++k) fx[k] = xt[k] < nt ? __ldg(A.X + (uint64_t)r[xt[k]] * d.D + xc[k]) : 0.f;
#pragma unroll
        for (int k = 0; k < kFetchT; ++k) ft[k] = tt[k] < nt ? __ldg(A.T + (uint64_t)r[tt[k]] * d.O + to[k]) : 0.f;
    };
    auto put = [&]() {
#pragma unroll
        for (int k = 0; k < kFetch; ++k)
            if (xt[k] < kTile) {
                m.xr[xt[k] * kRow + xc[k]] = fx[k];
                m.xs[xc[k] * kCol + xt[k]] = fx[k];
            }
#pragma unroll
        for (int k = 0; k < kFetchT; ++k)
            if (tt[k] < kTile) m.ts[to[k] * kTile + tt[k]] = ft[k];
    };
    Iter cur{A.steps * rounds, 0, 0, 0}, after = next(cur);
    if (tid < kTile) {
        rows[tid] = fetch_rows(cur);
        rows[kTile + tid] = fetch_rows(after);
    }
    if (tid == 0) {
        bar_init(bar_g);
        bar_init(bar_p);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    fetch(cur, 0);
    put();
    cluster_sync();   // every CTA of the cluster runs, and its barriers are set up
    const uint32_t g_addr = (uint32_t)__cvta_generic_to_shared(G), p_addr = (uint32_t)__cvta_generic_to_shared(sp);
    const uint32_t part_addr = (uint32_t)__cvta_generic_to_shared(part);
#pragma unroll
    for (int k = 0; k < kOwn; ++k) acc[k] = 0.f;
    bool ok = true;
    uint32_t step = 0;
    for (uint32_t it = 0; cur.left; ++it) {
        uint32_t base;
        int nt;
        tile_of(cur, base, nt);
        const bool last = cur.round + 1 == rounds;
        const uint32_t nb = min(A.batch, A.n - cur.b0);
        if (tid == 0) {
            bar_expect(bar_g, 4u * kCluster * mine);
            if (last) bar_expect(bar_p, 4u * (4 * n4 - mine));
        }
        const float2 c = __ldg(A.bias + step);
        fetch(after, ~it & 1u);
        const Iter after2 = next(after);
        const uint32_t next_row = tid < kTile ? fetch_rows(after2) : 0u;
        if (nt > 0) tile_grad<H>(d, sp, m, nt, 1.f / (float)((uint64_t)nb * d.O), nullptr);
        fence_copies();
        if (!__syncthreads_and(ok)) break;
        if ((tid & 31) == 0)   // a warp issues its lanes' copies one after another: a lane of each warp
            for (uint32_t r = tid >> 5; r < kCluster; r += kThreads / 32) {
                const uint32_t at = slice * r, n = min((uint32_t)slice, n4 - at);
                peer_copy(peer_addr(part_addr + 16u * slice * rank, r), g_addr + 16u * at, 16u * n, peer_addr(bar_g, r));
            }
        put();
        if (tid < kTile) rows[(it & 1u) * kTile + tid] = next_row;
        ok = bar_wait(bar_g, it & 1u);
        const uint32_t tiles = (nb + kTile - 1) / kTile;
        const uint32_t first = cur.round * kCluster;
        const uint32_t here = tiles > first ? min(tiles - first, (uint32_t)kCluster) : 0u;
#pragma unroll
        for (int k = 0; k < kOwn; ++k) {
            const int i = tid + kThreads * k;
            if (!(real >> k & 1u)) continue;
#pragma unroll
            for (uint32_t r = 0; r < kCluster; ++r)
                if (r < here) acc[k] += part[4 * slice * r + i];
            if (last) {
                sp[lo + i] = adam(sp[lo + i], acc[k], mo[k], ve[k], A, c);
                acc[k] = 0.f;
            }
        }
        fence_copies();
        if (!__syncthreads_and(ok)) break;
        if (last) {
            if ((tid & 31) == 0)
                for (uint32_t r = tid >> 5; r < kCluster; r += kThreads / 32)
                    if (r != rank) peer_copy(peer_addr(p_addr + 4u * lo, r), p_addr + 4u * lo, 4u * mine, peer_addr(bar_p, r));
            ok = bar_wait(bar_p, step & 1u);
            ++step;
        } else {
            cluster_sync();   // every owner has read this round's gradients
        }
        cur = after;
        after = after2;
    }
    if (!ok) *A.err = 1;
    cluster_sync();   // no copy of or into this CTA's memory is under way
    // this CTA's part of the parameters and moments back to the flat arrays
    auto store = [&](const float* padded, float* dst) {
        for (int p = tid; p < np; p += kThreads) {
            const int at = d.place(p);
            if (at >= lo && at < lo + mine) dst[p] = padded[at];
        }
    };
    store(sp, A.P);
    auto flat = [&](const float (&src)[kOwn], float* dst) {
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kOwn; ++k)
            if (tid + kThreads * k < mine) G[lo + tid + kThreads * k] = src[k];
        __syncthreads();
        store(G, dst);
    };
    flat(mo, A.m);
    flat(ve, A.v);
}

size_t fwd_smem(const Dims& d) { return sizeof(float) * (size_t)(d.pn() + 2 * kCols); }
size_t grad_smem(const Dims& d) { return sizeof(float) * (size_t)(2 * d.pn() + kTileFloats); }
size_t train_smem(const Dims& d) {
    return grad_smem(d) + sizeof(float) * (size_t)(d.pn() + 4 * kCluster) + 2 * kTile * sizeof(uint32_t);
}

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
    int* err = nullptr;      // set by a training kernel whose waits ran out
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

int es_mlp_create(uint32_t in_dim, uint32_t hidden, uint32_t out_dim, uint64_t seed, es_mlp** out) try {
    if (!out) return mlp_fail(ES_ERR_ARG, "null output");
    *out = nullptr;
    if (in_dim < 1 || in_dim > kMaxD || hidden < 8 || hidden > kMaxH || hidden % 32 || out_dim < 1 ||
        out_dim > kMaxO || out_dim > hidden)
        return mlp_fail(ES_ERR_RANGE, "MLP dims must be in <= 64, hidden 32 or 64, out <= 8");
    std::unique_ptr<es_mlp, int (*)(es_mlp*)> own(new es_mlp(), es_mlp_destroy);
    es_mlp* M = own.get();
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
    if (e == cudaSuccess) e = cudaMalloc(&M->P, 4ull * (4 * np + 2));
    if (e == cudaSuccess) e = cudaMemcpy(M->P, h.data(), 12ull * np, cudaMemcpyHostToDevice);
    M->m = M->P + np;
    M->v = M->m + np;
    M->g = M->v + np;
    M->loss = M->g + np;
    M->err = reinterpret_cast<int*>(M->loss + 1);
    if (e == cudaSuccess) e = cudaMemset(M->err, 0, 4);
    if (e != cudaSuccess) return mlp_fail(ES_ERR_CUDA, std::string("MLP setup: ") + cudaGetErrorString(e));
    *out = own.release();
    return ES_OK;
} catch (const std::exception&) {   // nothing throws across the ABI
    return mlp_fail(ES_ERR_NOMEM, "host allocation");
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
        f<<<tiles, threads_of(d.H), fwd_smem(d)>>>(d, M->P, M->X.as<float>(), n, M->Y.as<float>());
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
        f<<<tiles, threads_of(d.H), grad_smem(d)>>>(d, M->P, M->X.as<float>(), M->T.as<float>(), n, scale, M->G.as<float>(),
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
                 float lr, uint64_t seed, float* final_loss) try {
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
        TrainArgs a{d, M->P, M->m, M->v, M->X.as<float>(), M->T.as<float>(), idx, bs, M->err, (uint32_t)n, step_batch, spe, spe,
                    lr, b1, b2, eps};
        kernel<<<kCluster, threads_of(d.H), train_smem(d)>>>(a);
        e = cudaGetLastError();
    }
    int late = 0;
    if (e == cudaSuccess) e = cudaMemcpy(&late, M->err, 4, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess && late) {
        cudaMemset(M->err, 0, 4);
        M->trim();
        return mlp_fail(ES_ERR_CUDA, "a training step did not finish");
    }
    if (final_loss && e == cudaSuccess) {
        float l = 0.f;
        e = device_loss_grad(M, n, &l, nullptr);
        *final_loss = l;
    }
    M->trim();
    return e == cudaSuccess ? ES_OK : mlp_fail(ES_ERR_CUDA, cudaGetErrorString(e));
} catch (const std::exception&) {
    return mlp_fail(ES_ERR_NOMEM, "host allocation");
}

}  // extern "C"
