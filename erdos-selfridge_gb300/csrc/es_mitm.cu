// Meet-in-the-middle search kernel of the GB300 Erdős–Selfridge engine (sm_103a) and its C ABI
// (es_mitm_* in include/es_gb300.h).
//
// What one scan computes (the semantics of sieve/gpu_mitm.py:33-125): the wheel residues are
// n = (s1 + s2) mod M with s1 a sum of one term per prime of the large half W1 and s2 one per
// prime of the small half W2 (terms a * c_p mod M, c_p the CRT basis).  For a bound B <= M and
// every s1 index in [s1_begin, s1_end), the n < B are exactly s1 + S2[u] for the u of one
// circular run of the sorted S2: [lower_bound(M - s1), lower_bound(M - s1 + B)) mod M, the run
// wrapping to the front of S2 when M - s1 + B >= M.  Each such n runs through the residual-prime
// cascade (n mod q for every filter in order, early exit) and the survivors are emitted; the
// number of n tested is counted.
//
// GB300-first organisation (not the reference's one-thread-per-s1 kernel with two full binary
// searches):
//  * S2 is sorted once on the host and uploaded with a directory over the top bits of its values
//    (bucket b -> first index whose value >= b << shift), about one entry per bucket.  A run is
//    walked from its bucket's first entry: the few entries below M - s1 are passed over, and it
//    ends at the first n >= B, so no search is needed for either end.
//  * S1 is swept in value order, tile by tile: with A the sums over the first rings of the large
//    half (sorted on the host) and b those over the rest, the s1 = a + b of one slice [X, X') of
//    [0, M) are, for every b, one circular range of A.  Warps claim up to 16 values of b of one slice
//    from an atomic counter (persistent grid, no waits), search their ranges, a lane per end,
//    and sweep them, so that the warps at work read one slice of S2 and its directory, which stay
//    in L2, and a slice comes from memory once.  (In index order every s1 falls anywhere in S2.)
//  * Runs have a handful of entries and differ from lane to lane, and four of five candidates
//    fail the first filter: the walk only queues its candidates (per warp, in shared memory), and
//    a full warp of them at a time goes through the cascade.  Two bit tables in shared memory come
//    first, each over a product of projections of filters (es_cascade.h), so that one limb-weight
//    and Barrett reduction tests several filters; the full cascade runs for what is left.
//
// What bounds it: instruction issue and the latency of the S2 reads.  With per-lane searches and
// per-lane cascades the warps ran at 8.6 of 32 lanes: k = 150, bound 3E (1.2e7 s1, 1.7e7
// candidates) took 930 us of kernel time (7.7e8 warp instructions) and takes 290 (2.1e8); k = 160, whose
// S2 is twice the L2, 4.2 ms and 1.2 ms.  (More CTAs per SM are slower: 5 of 256 threads 507 against
// 474 us a scan, 8 895 us.  Their shared memory is taken from the L1 that S2 and the directory use.)
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <functional>
#include <memory>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "../../include/es_gb300.h"
#include "es_cascade.h"
#include "es_internal.h"
#include "es_scan_kernel.cuh"

typedef unsigned __int128 u128m;

namespace {

int mfail(int code, const std::string& msg) {
    es_set_last_error(msg.c_str());
    return code;
}

int mcuda(cudaError_t e, const char* what) {
    es_set_last_error((std::string(what) + ": " + cudaGetErrorString(e)).c_str());
    return ES_ERR_CUDA;
}

#define ES_MCUDA(call, what)                               \
    do {                                                   \
        cudaError_t _e = (call);                           \
        if (_e != cudaSuccess) return mcuda(_e, what);     \
    } while (0)

constexpr uint32_t kMitmMaxRings = 32;
constexpr uint32_t kMitmThreads = 512;
constexpr uint32_t kMitmChunk = 16;  // values of b per claimed unit, at most (two lanes each for its range)
constexpr uint32_t kMitmQueue = 64;  // candidates queued per warp
constexpr uint32_t kMitmTables = 2;  // merged bit tables ahead of the cascade
// Bits of both: 32 KB less a word that each may round up to, so that with 16 KB of queues the kernel stays
// within the 48 KB of shared memory that need no opt-in.
constexpr uint32_t kMitmTableBits = (1u << 18) - 64u;
// Rings are grouped while their sums stay within this, and A's within a quarter of S1 as well: sorting a
// large A costs more than a short scan gains from it.  Creation and one scan, A within 2^17 alone and
// within a quarter of S1: k = 90 (S1 90,720) 4.19 + 0.080 and 2.53 + 0.080 ms, k = 100 (119,808) 4.89 +
// 0.092 and 2.86 + 0.083, k = 130 (7.4 million, the same A) 9.50 + 0.263 and 9.45 + 0.270.
constexpr uint64_t kMitmGroup = 1u << 17;
constexpr uint64_t kMitmShare = 4;
constexpr uint64_t kMitmRange = 64;             // values of A per b and slice, at least
constexpr uint32_t kMitmSlicesLog2 = 12;        // slices at most

static_assert(kMitmThreads / 32u * kMitmQueue * sizeof(uint4) + (kMitmTableBits / 32u + kMitmTables) * 4u <= 48u << 10,
              "queues and merged tables exceed what a launch has without an opt-in");

struct MitmParams {
    const uint4* S2;              // sorted small half: {lo.x, lo.y, hi.x, hi.y} per entry
    const uint32_t* dir;          // [2^D + 1] first S2 index with value >= b << shift
    const uint4* A;               // large half: sorted sums over its first rings
    const uint32_t* a_index;      // their indices (mixed radix, first ring fastest)
    const uint4* sums1;           // sums over the groups of the other rings
    const uint4* slices;          // [n_slices + 1] slice boundaries, 0 .. M
    const EsFilterC* filt;        // residual filters (q, limb weights, Barrett reciprocal, offset)
    const uint32_t* allowed;      // packed admissible-residue bits of every filter
    const uint32_t* merged;       // the merged tables' bits
    uint4* out;                   // survivors {n_lo, n_hi} as uint4
    unsigned long long* counters; // [0] survivors, [1] candidates tested, [2] work counter
    uint64_t out_cap;
    uint64_t n2;
    uint64_t s1_begin, s1_end;
    uint64_t M_lo, M_hi, B_lo, B_hi;
    uint32_t shift;               // directory bucket = value >> shift
    uint32_t n_a, n_slices;
    uint32_t chunk;               // values of b per claimed unit
    uint32_t n_groups;
    uint32_t n_filters;
    uint32_t merged_words;
    EsFilterC table[kMitmTables];   // merged moduli; off: word offset in the merged bits
    EsGroup group[kMitmMaxRings];
};

__device__ __forceinline__ U4 ld_s2(const uint4* S2, uint64_t i) { return u4(__ldg(S2 + i)); }

// 128-bit value >> shift (shift < 128), low 32 bits (the directory bucket of a value < M)
__device__ __forceinline__ uint32_t bucket_of(const U4 v, uint32_t shift) {
    const uint64_t lo = lo64(v), hi = hi64(v);
    uint64_t r;
    if (shift >= 64) r = hi >> (shift - 64);
    else if (shift == 0) r = lo;
    else r = (lo >> shift) | (hi << (64 - shift));
    return (uint32_t)r;
}

// b of index idx: mixed radix over the groups of rings after A's, the first fastest
__device__ __forceinline__ U4 decode_b(const MitmParams& P, uint64_t idx, const U4 M) {
    U4 acc{0u, 0u, 0u, 0u};
    uint64_t rem = idx;
    for (uint32_t g = 0; g < P.n_groups; ++g) {
        const EsGroup G = P.group[g];
        // floor(rem / size) or one less (magic = floor((2^64 - 1) / size)), then corrected
        uint64_t q = __umul64hi(rem, G.magic);
        uint64_t d = rem - q * G.size;
        if (d >= G.size) {
            d -= G.size;
            ++q;
        }
        rem = q;
        uint32_t wm;
        acc = addmod(acc, u4(__ldg(P.sums1 + (G.off + d))), M, wm);
    }
    return acc;
}

// first index of the sorted A with A[i] >= v (n_a when none)
__device__ __forceinline__ uint32_t lower_bound_a(const MitmParams& P, const U4 v) {
    uint32_t a = 0, e = P.n_a;
    while (a < e) {
        const uint32_t m = (a + e) >> 1;
        if (lt128(u4(__ldg(P.A + m)), v)) a = m + 1; else e = m;
    }
    return a;
}

// warp-uniform: the first min(32, size) queued candidates through the cascade; survivors are emitted
__device__ __forceinline__ void mitm_flush(const MitmParams& P, const uint4* queue, const uint32_t* bits, uint32_t lane,
                                           uint32_t head, uint32_t size) {
    __syncwarp();
    bool ok = lane < size;
    const U4 n = u4(queue[(head + lane) & (kMitmQueue - 1u)]);   // (stale beyond size: not used)
    for (uint32_t i = 0; i < kMitmTables; ++i) {
        const EsFilterC& fc = P.table[i];
        const uint32_t r = mod128(n, fc);
        ok = ok && ((bits[fc.off + (r >> 5)] >> (r & 31u)) & 1u);
        if (!__any_sync(0xffffffffu, ok)) break;
    }
    if (ok) {
        for (uint32_t f = 0; f < P.n_filters && ok; ++f) {
            const EsFilterC fc = P.filt[f];
            const uint32_t r = mod128(n, fc);
            ok = (__ldg(P.allowed + fc.off + (r >> 5)) >> (r & 31u)) & 1u;
        }
        if (ok) {
            const unsigned long long slot = atomicAdd(P.counters + 0, 1ull);
            if (slot < P.out_cap) P.out[slot] = make_uint4(n.x, n.y, n.z, n.w);
        }
    }
    __syncwarp();
}

__global__ void __launch_bounds__(kMitmThreads) es_mitm_kernel(const __grid_constant__ MitmParams P) {
    extern __shared__ __align__(16) uint32_t bits[];   // the merged tables
    __shared__ uint4 queues[kMitmThreads / 32][kMitmQueue];
    const uint32_t lane = threadIdx.x & 31u;
    uint4* queue = queues[threadIdx.x >> 5];
    for (uint32_t i = threadIdx.x; i < P.merged_words; i += kMitmThreads) bits[i] = __ldg(P.merged + i);
    for (uint32_t i = lane; i < kMitmQueue; i += 32u) queue[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const U4 M{(uint32_t)P.M_lo, (uint32_t)(P.M_lo >> 32), (uint32_t)P.M_hi, (uint32_t)(P.M_hi >> 32)};
    const U4 B{(uint32_t)P.B_lo, (uint32_t)(P.B_lo >> 32), (uint32_t)P.B_hi, (uint32_t)(P.B_hi >> 32)};
    // the values of b that the s1 indices touch; the first and the last may take part of A only
    const uint64_t b_lo = P.s1_begin / P.n_a, b_hi = (P.s1_end + P.n_a - 1) / P.n_a;
    const uint64_t chunks = (b_hi - b_lo + P.chunk - 1) / P.chunk;
    const uint32_t n2 = (uint32_t)P.n2;   // below 2^31
    unsigned long long tested = 0;
    uint32_t head = 0, size = 0;
    for (;;) {
        unsigned long long c = 0;
        if (lane == 0) c = atomicAdd(P.counters + 2, 1ull);
        c = __shfl_sync(0xffffffffu, c, 0);
        if (c >= chunks * P.n_slices) break;
        const uint64_t slice = c / chunks, b0 = b_lo + (c - slice * chunks) * P.chunk;
        // lanes 2 i and 2 i + 1: b0 + i, and where its range of A starts and ends.  The slice's upper
        // boundary less b is taken mod M too: an end that is not above the start goes round.
        const U4 bv = decode_b(P, min(b0 + (lane >> 1), b_hi - 1), M);
        uint32_t br;
        U4 v = sub128(u4(__ldg(P.slices + slice + (lane & 1u))), bv, br);
        if (br) v = add128(v, M);
        if (((v.x ^ M.x) | (v.y ^ M.y) | (v.z ^ M.z) | (v.w ^ M.w)) == 0u) v = U4{0u, 0u, 0u, 0u};
        const uint32_t at = lower_bound_a(P, v);
        const U4 other{__shfl_xor_sync(0xffffffffu, v.x, 1), __shfl_xor_sync(0xffffffffu, v.y, 1),
                       __shfl_xor_sync(0xffffffffu, v.z, 1), __shfl_xor_sync(0xffffffffu, v.w, 1)};
        const bool round = (lane & 1u) ? !lt128(other, v) : !lt128(v, other);
        for (uint32_t i = 0; i < P.chunk && b0 + i < b_hi; ++i) {
            const uint64_t b = b0 + i;
            const U4 bs{__shfl_sync(0xffffffffu, bv.x, 2 * i), __shfl_sync(0xffffffffu, bv.y, 2 * i),
                        __shfl_sync(0xffffffffu, bv.z, 2 * i), __shfl_sync(0xffffffffu, bv.w, 2 * i)};
            const uint32_t start = __shfl_sync(0xffffffffu, at, 2 * i), stop = __shfl_sync(0xffffffffu, at, 2 * i + 1);
            const uint32_t count = __shfl_sync(0xffffffffu, round, 2 * i) ? P.n_a - start + stop : stop - start;
            const bool partial = b * P.n_a < P.s1_begin || (b + 1) * P.n_a > P.s1_end;
            for (uint32_t from = 0; from < count; from += 32u) {
                bool active = from + lane < count;
                uint32_t ia = start + (active ? from + lane : from);
                if (ia >= P.n_a) ia -= P.n_a;
                if (partial) {
                    const uint64_t index = b * P.n_a + __ldg(P.a_index + ia);
                    active = active && index >= P.s1_begin && index < P.s1_end;
                }
                uint32_t wa;
                const U4 s1 = addmod(u4(__ldg(P.A + ia)), bs, M, wa);
                // The run starts at the first entry >= lo = (M - s1) mod M.  Up to the end of S2,
                // n = s2 - lo (below 0 for the entries passed over); past it, n = s2 + s1.
                const bool zero = (s1.x | s1.y | s1.z | s1.w) == 0u;
                U4 off = sub128(s1, M, br);   // -lo
                if (zero) off = U4{0u, 0u, 0u, 0u};
                const U4 lo = sub128(U4{0u, 0u, 0u, 0u}, off, br);
                uint32_t u = __ldg(P.dir + bucket_of(lo, P.shift));
                if (u == n2) {
                    u = 0;
                    off = s1;
                }
                uint32_t left = n2;        // entries the run may still take (B = M: all of S2)
                U4 s2 = ld_s2(P.S2, u);
                while (__any_sync(0xffffffffu, active)) {
                    // the next entry, circularly, is on its way while this one is looked at
                    const U4 n = add128(s2, off);
                    ++u;
                    if (u == n2) {
                        u = 0;
                        off = s1;
                    }
                    if (active) s2 = ld_s2(P.S2, u);
                    const bool cand = active && lt128(n, B) && left != 0u;   // (a negative n is above B)
                    left -= cand ? 1u : 0u;
                    active = cand || (active && (int32_t)n.w < 0);
                    const uint32_t has = __ballot_sync(0xffffffffu, cand);
                    if (has) {
                        if (cand) {
                            queue[(head + size + __popc(has & ((1u << lane) - 1u))) & (kMitmQueue - 1u)] =
                                make_uint4(n.x, n.y, n.z, n.w);
                            ++tested;
                        }
                        size += __popc(has);   // at most 31 + 32
                        if (size >= 32u) {
                            mitm_flush(P, queue, bits, lane, head, 32u);
                            head = (head + 32u) & (kMitmQueue - 1u);
                            size -= 32u;
                        }
                    }
                }
            }
        }
    }
    if (size) mitm_flush(P, queue, bits, lane, head, size);
    for (uint32_t o = 16; o > 0; o >>= 1) tested += __shfl_down_sync(0xffffffffu, tested, o);
    if (lane == 0 && tested) atomicAdd(P.counters + 1, tested);
}

}  // namespace

struct es_mitm {
    cudaStream_t stream = nullptr;
    MitmParams P{};
    unsigned char* tables = nullptr;   // every array that scans read, in one allocation
    uint4* d_out = nullptr;
    unsigned long long* d_cnt = nullptr;
    unsigned long long* h_cnt = nullptr;
    uint64_t n1 = 0, n2 = 0, cap = 0;
    int grid = 0;
};

namespace {

// Sorts items by their keys (below 2^bits): scattered to about one bucket per item (at most
// 2^16) by the keys' top bits, then the buckets one by one.
template <class T, class Key>
void bucket_sort(std::vector<T>& v, uint32_t bits, const Key& key) {
    const size_t n = v.size();
    uint32_t P = 0;
    while (P < std::min(bits, 16u) && ((size_t)1 << P) < n) ++P;
    const uint32_t sh = bits - P;
    std::vector<uint32_t> at(((size_t)1 << P) + 1, 0);   // bucket p's items end at at[p], start at at[p - 1]
    for (const T& x : v) ++at[(size_t)(key(x) >> sh) + 1];
    for (size_t p = 1; p < at.size(); ++p) at[p] += at[p - 1];
    std::vector<T> out(n);
    for (const T& x : v) out[at[(size_t)(key(x) >> sh)]++] = x;
    for (size_t p = 0, from = 0; p + 1 < at.size(); from = at[p++])
        if (at[p] - from > 1)
            std::sort(out.begin() + from, out.begin() + at[p], [&](const T& a, const T& b) { return key(a) < key(b); });
    v.swap(out);
}

// body(0) .. body(T - 1), each on a thread of its own where the system gives one (body must not throw).
template <class Body>
void on_threads(unsigned T, const Body& body) {
    std::vector<std::thread> th;
    th.reserve(T);
    unsigned t = 1;
    try {
        for (; t < T; ++t) th.emplace_back(std::cref(body), t);
    } catch (const std::exception&) {   // no more threads: the rest runs here
    }
    body(0);
    for (; t < T; ++t) body(t);
    for (auto& x : th) x.join();
}

}  // namespace

extern "C" {

int es_mitm_destroy(es_mitm* m) {
    if (!m) return ES_OK;
    if (m->stream) cudaStreamSynchronize(m->stream);
    cudaFree(m->tables);
    cudaFree(m->d_out);
    cudaFree(m->d_cnt);
    if (m->h_cnt) cudaFreeHost(m->h_cnt);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return ES_OK;
}

namespace {

// Sorts v (values below 2^bits) on the host cores: each thread counts its share of the values
// per partition of their top P bits, the values are scattered to their partitions, and the
// partitions are sorted, shared out among the threads.  The result equals std::sort's.
void parallel_sort(std::vector<u128m>& v, uint32_t bits) {
    const size_t n = v.size();
    const unsigned T = std::max(1u, std::min(64u, std::thread::hardware_concurrency()));
    if (n < (1u << 16) || T == 1 || bits == 0) {
        bucket_sort(v, bits, [](u128m x) { return x; });
        return;
    }
    const uint32_t P = std::min<uint32_t>(12, bits);
    const uint32_t sh = bits - P;
    const size_t np = (size_t)1 << P;
    std::vector<std::vector<size_t>> at(T, std::vector<size_t>(np, 0));
    on_threads(T, [&](unsigned t) {
        for (size_t i = n * t / T, e = n * (t + 1) / T; i < e; ++i) ++at[t][(size_t)(v[i] >> sh)];
    });
    std::vector<size_t> start(np + 1);
    size_t acc = 0;
    for (size_t p = 0; p < np; ++p) {   // partition-major, thread-minor write positions
        start[p] = acc;
        for (unsigned t = 0; t < T; ++t) {
            const size_t c = at[t][p];
            at[t][p] = acc;
            acc += c;
        }
    }
    start[np] = acc;
    std::vector<u128m> out(n);
    on_threads(T, [&](unsigned t) {
        for (size_t i = n * t / T, e = n * (t + 1) / T; i < e; ++i) out[at[t][(size_t)(v[i] >> sh)]++] = v[i];
    });
    std::atomic<size_t> next(0);
    on_threads(T, [&](unsigned) {
        for (size_t p = next++; p < np; p = next++) std::sort(out.begin() + start[p], out.begin() + start[p + 1]);
    });
    v.swap(out);
}

}  // namespace

int es_mitm_create(const es_mitm_desc* d, es_mitm** out) try {
    if (!d || !out) return mfail(ES_ERR_ARG, "null descriptor or output pointer");
    *out = nullptr;
    const u128m M = ((u128m)d->M_hi << 64) | d->M_lo;
    if (M < 2 || (M >> 126) != 0) return mfail(ES_ERR_RANGE, "wheel modulus must be in [2, 2^126)");
    if (d->n_rings1 > kMitmMaxRings || d->n_rings2 > kMitmMaxRings)
        return mfail(ES_ERR_RANGE, "too many wheel primes in one half (max 32)");
    if (d->n_filters > ES_MAX_FILTERS) return mfail(ES_ERR_RANGE, "too many residual filters");
    if ((d->n_rings1 && (!d->radix1 || !d->term1_lo || !d->term1_hi)) ||
        (d->n_rings2 && (!d->radix2 || !d->term2_lo || !d->term2_hi)) ||
        (d->n_filters && (!d->filter_q || !d->allowed)))
        return mfail(ES_ERR_ARG, "null array in descriptor");
    int dev = 0, major = 0, minor = 0, sms = 0;
    ES_MCUDA(cudaGetDevice(&dev), "cudaGetDevice");
    ES_MCUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev), "attr");
    ES_MCUDA(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev), "attr");
    ES_MCUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "attr");
    if (major != 10 || minor != 3) return mfail(ES_ERR_NODEV, "this library is built for sm_103a only");

    // ---- the two halves --------------------------------------------------------------------
    uint64_t n1 = 1, n2 = 1;
    std::vector<u128m> t1, t2;
    std::vector<uint32_t> r1(d->radix1, d->radix1 + d->n_rings1), r2(d->radix2, d->radix2 + d->n_rings2);
    for (uint32_t j = 0; j < d->n_rings1; ++j) {
        const uint32_t r = r1[j];
        if (r == 0 || r > 65535) return mfail(ES_ERR_RANGE, "radix must be in [1, 65535]");
        if (n1 > (1ull << 62) / r) return mfail(ES_ERR_RANGE, "|S1| exceeds 2^62");
        n1 *= r;
    }
    for (uint32_t j = 0; j < d->n_rings2; ++j) {
        const uint32_t r = r2[j];
        if (r == 0 || r > 65535) return mfail(ES_ERR_RANGE, "radix must be in [1, 65535]");
        if (n2 > (1ull << 31) / r) return mfail(ES_ERR_RANGE, "|S2| must stay below 2^31 entries");
        n2 *= r;
    }
    size_t pos = 0;
    for (uint32_t j = 0; j < d->n_rings1; ++j)
        for (uint32_t i = 0; i < r1[j]; ++i, ++pos) {
            const u128m v = ((u128m)d->term1_hi[pos] << 64) | d->term1_lo[pos];
            if (v >= M) return mfail(ES_ERR_ARG, "term not reduced mod M");
            t1.push_back(v);
        }
    pos = 0;
    for (uint32_t j = 0; j < d->n_rings2; ++j)
        for (uint32_t i = 0; i < r2[j]; ++i, ++pos) {
            const u128m v = ((u128m)d->term2_hi[pos] << 64) | d->term2_lo[pos];
            if (v >= M) return mfail(ES_ERR_ARG, "term not reduced mod M");
            t2.push_back(v);
        }
    // S2: every sum of one term per ring of the small half, mod M, sorted
    std::vector<u128m> S2(1, 0);
    pos = 0;
    for (uint32_t j = 0; j < d->n_rings2; ++j) {
        const size_t have = S2.size();
        std::vector<u128m> next;
        next.reserve(have * r2[j]);
        for (size_t a = 0; a < have; ++a)
            for (uint32_t i = 0; i < r2[j]; ++i) {
                u128m v = S2[a] + t2[pos + i];
                if (v >= M) v -= M;
                next.push_back(v);
            }
        S2.swap(next);
        pos += r2[j];
    }
    uint32_t bits = 0;   // values < M < 2^bits
    for (u128m x = M - 1; x; x >>= 1) ++bits;
    parallel_sort(S2, bits);
    // directory over the top bits of values < M: about one entry per bucket
    uint32_t D = 8;
    while (D < 28 && (1ull << D) < n2) ++D;
    if (D > bits) D = bits;
    const uint32_t shift = bits - D;
    std::vector<uint32_t> dir((1ull << D) + 1);
    {
        // every core fills the buckets of its share of the entries: bucket b holds the first entry i
        // with value >= b << shift, so entry i fills the buckets above entry i - 1's, up to its own
        const unsigned T = n2 < (1u << 16) ? 1u : std::max(1u, std::min(64u, std::thread::hardware_concurrency()));
        auto fill = [&](unsigned t) {
            const size_t from = n2 * t / T, to = n2 * (t + 1) / T;
            uint64_t b = from == 0 ? 0 : (uint64_t)(S2[from - 1] >> shift) + 1;
            for (size_t i = from; i < to; ++i)
                for (const uint64_t own = (uint64_t)(S2[i] >> shift); b <= own; ++b) dir[b] = (uint32_t)i;
            if (t + 1 == T)
                for (; b <= (1ull << D); ++b) dir[b] = (uint32_t)n2;
        };
        on_threads(T, fill);
    }
    // ---- filters ---------------------------------------------------------------------------
    std::vector<EsFilterC> fc(d->n_filters);
    uint32_t words = 0;
    for (uint32_t f = 0; f < d->n_filters; ++f) {
        const uint32_t q = d->filter_q[f];
        if (q < 2 || q >= ES_MAX_Q) return mfail(ES_ERR_RANGE, "filter modulus must be in [2, 2^20)");
        fc[f].q = q;
        fc[f].corr = 0;
        fc[f].w1 = (uint32_t)(((u128m)1 << 32) % q);
        fc[f].w2 = (uint32_t)(((u128m)1 << 64) % q);
        fc[f].w3 = (uint32_t)(((u128m)1 << 96) % q);
        fc[f].off = words;
        fc[f].rcp = (uint64_t)(((u128m)1 << 64) / q);
        words += (q + 31) / 32;
    }

    std::unique_ptr<es_mitm, int (*)(es_mitm*)> own(new es_mitm(), es_mitm_destroy);
    es_mitm* m = own.get();
    m->n1 = n1;
    m->n2 = n2;
    // ---- merged tables: products of projections of filters, tested ahead of the cascade ---------
    EsHostPlan hp;
    hp.k = d->k;
    hp.M = M;
    hp.q.assign(d->filter_q, d->filter_q + d->n_filters);
    hp.bit_off.assign(1, 0);
    for (uint32_t f = 0; f < d->n_filters; ++f) hp.bit_off.push_back(hp.bit_off.back() + (hp.q[f] + 31) / 32);
    if (d->n_filters) hp.allowed.assign(d->allowed, d->allowed + words);
    // (rows of one byte, two per residue: kMitmTableBits residues in all, padded to 16 rows a table)
    const EsCascade cascade = es_choose_cascade(hp, kMitmTables, 1, true, 2u * kMitmTableBits);
    std::vector<uint32_t> merged;
    for (uint32_t i = 0; i < kMitmTables; ++i) {
        uint32_t q = 1;
        for (const EsPart& p : cascade.inner[i]) q *= p.d;
        if (q == 1) q = 2;   // a fill-in that passes everything
        const uint32_t off = (uint32_t)merged.size();
        merged.resize(off + (q + 31) / 32, 0xffffffffu);
        for (const EsPart& p : cascade.inner[i])
            es_and_periodic(hp.allowed.data() + hp.bit_off[p.f], hp.q[p.f], p.d, q, &merged[off]);
        m->P.table[i] = es_filter_consts(M, q, off);
    }
    // ---- large half: sums over groups of consecutive rings; the first group is A, sorted -----------
    std::vector<u128m> A(1, 0), sums;
    const uint64_t a_most = std::min(kMitmGroup, std::max<uint64_t>(n1 / kMitmShare, 1024));
    for (uint32_t j = 0, o = 0; j < d->n_rings1;) {
        uint64_t size = 1;
        const bool first = j == 0;
        std::vector<u128m> sum(1, 0);
        do {
            std::vector<u128m> next;
            next.reserve(sum.size() * r1[j]);
            for (uint32_t i = 0; i < r1[j]; ++i)
                for (const u128m v : sum) {
                    const u128m x = v + t1[o + i];
                    next.push_back(x >= M ? x - M : x);
                }
            sum.swap(next);
            size *= r1[j];
            o += r1[j++];
        } while (j < d->n_rings1 && size * r1[j] <= (first ? a_most : kMitmGroup));
        if (first) {
            A.swap(sum);
            continue;
        }
        EsGroup& G = m->P.group[m->P.n_groups++];
        G.size = (uint32_t)size;
        G.magic = ~0ull / size;
        G.off = (uint32_t)sums.size();
        sums.insert(sums.end(), sum.begin(), sum.end());
    }
    if (sums.empty()) sums.push_back(0);
    struct Sum {
        u128m v;
        uint32_t index;
    };
    std::vector<Sum> by_value(A.size());
    for (size_t i = 0; i < A.size(); ++i) by_value[i] = Sum{A[i], (uint32_t)i};
    // (the indices sorted by the values they stand for took 11 ms where this takes 3: 90,720 values)
    bucket_sort(by_value, bits, [](const Sum& x) { return x.v; });
    std::vector<u128m> a_sorted(A.size());
    std::vector<uint32_t> a_index(A.size());
    for (size_t i = 0; i < A.size(); ++i) {
        a_sorted[i] = by_value[i].v;
        a_index[i] = by_value[i].index;
    }
    // slices of [0, M): a power of two of them, none so thin that a b's range of A is a few values, and
    // none empty (an end that is not above the start goes round, so an empty one would hold all of A)
    uint32_t sl = 0;
    while (sl < kMitmSlicesLog2 && (A.size() >> (sl + 1)) >= kMitmRange && (M >> (sl + 1)) != 0) ++sl;
    std::vector<u128m> slices;
    for (uint64_t i = 0; i < (1ull << sl); ++i) slices.push_back((M >> sl) * i);
    slices.push_back(M);
    static_assert(sizeof(u128m) == sizeof(uint4), "values are uploaded as they are (little endian)");
    cudaError_t ce = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
    // one allocation and three copies: S2, its directory, and the small arrays in one image
    size_t total = 0;
    auto take = [&](size_t bytes) {
        const size_t at = total;
        total = es_align_up(total + std::max<size_t>(bytes, 16), 256);
        return at;
    };
    std::vector<unsigned char> small;
    size_t small_at = 0;
    auto put = [&](const void* src, size_t bytes) {
        const size_t at = take(bytes);
        small.resize(total - small_at, 0);
        if (bytes) memcpy(&small[at - small_at], src, bytes);
        return at;
    };
    const size_t o_S2 = take(sizeof(uint4) * S2.size()), o_dir = take(4 * dir.size());
    small_at = total;
    const size_t o_sums = put(sums.data(), sizeof(uint4) * sums.size());
    const size_t o_filt = put(fc.data(), sizeof(EsFilterC) * fc.size());
    const size_t o_allowed = put(d->allowed, 4ull * words);
    const size_t o_A = put(a_sorted.data(), sizeof(uint4) * a_sorted.size());
    const size_t o_index = put(a_index.data(), 4 * a_index.size());
    const size_t o_slices = put(slices.data(), sizeof(uint4) * slices.size());
    const size_t o_merged = put(merged.data(), 4 * merged.size());
    if (ce == cudaSuccess) ce = cudaMalloc(&m->tables, total);
    if (ce == cudaSuccess) ce = cudaMalloc(&m->d_cnt, 8ull * 4);
    if (ce == cudaSuccess) ce = cudaHostAlloc(&m->h_cnt, 8ull * 4, cudaHostAllocDefault);
    if (ce == cudaSuccess) ce = cudaMemcpy(m->tables + o_S2, S2.data(), sizeof(uint4) * S2.size(), cudaMemcpyHostToDevice);
    if (ce == cudaSuccess) ce = cudaMemcpy(m->tables + o_dir, dir.data(), 4 * dir.size(), cudaMemcpyHostToDevice);
    if (ce == cudaSuccess) ce = cudaMemcpy(m->tables + small_at, small.data(), small.size(), cudaMemcpyHostToDevice);
    // the scans' stream is not ordered after the default stream: wait for the copies, and zero the
    // counters on the former
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(nullptr);
    if (ce == cudaSuccess) ce = cudaMemsetAsync(m->d_cnt, 0, 8ull * 4, m->stream);
    if (ce != cudaSuccess) return mcuda(ce, "MITM setup");
    MitmParams& P = m->P;
    P.S2 = reinterpret_cast<const uint4*>(m->tables + o_S2);
    P.dir = reinterpret_cast<const uint32_t*>(m->tables + o_dir);
    P.sums1 = reinterpret_cast<const uint4*>(m->tables + o_sums);
    P.filt = reinterpret_cast<const EsFilterC*>(m->tables + o_filt);
    P.allowed = reinterpret_cast<const uint32_t*>(m->tables + o_allowed);
    P.counters = m->d_cnt;
    P.n2 = n2;
    P.M_lo = d->M_lo;
    P.M_hi = d->M_hi;
    P.shift = shift;
    P.n_filters = d->n_filters;
    P.merged = reinterpret_cast<const uint32_t*>(m->tables + o_merged);
    P.A = reinterpret_cast<const uint4*>(m->tables + o_A);
    P.a_index = reinterpret_cast<const uint32_t*>(m->tables + o_index);
    P.n_a = (uint32_t)A.size();
    P.slices = reinterpret_cast<const uint4*>(m->tables + o_slices);
    P.n_slices = 1u << sl;
    P.merged_words = (uint32_t)merged.size();
    int occ = 0;
    ce = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, es_mitm_kernel, kMitmThreads, 4ull * merged.size());
    if (ce != cudaSuccess || occ < 1) return mcuda(ce == cudaSuccess ? cudaErrorInvalidConfiguration : ce, "MITM occupancy");
    m->grid = sms * occ;
    if (int e = es_mitm_set_capacity(m, 1u << 20)) return e;
    *out = own.release();
    return ES_OK;
} catch (const std::exception&) {   // nothing throws across the ABI
    return mfail(ES_ERR_NOMEM, "host allocation");
}

int es_mitm_info(const es_mitm* m, uint64_t* n1, uint64_t* n2) {
    if (!m) return mfail(ES_ERR_ARG, "null MITM engine");
    if (n1) *n1 = m->n1;
    if (n2) *n2 = m->n2;
    return ES_OK;
}

int es_mitm_set_capacity(es_mitm* m, uint64_t cap) {
    if (!m || cap == 0 || cap > (1ull << 32)) return mfail(ES_ERR_ARG, "capacity must be in [1, 2^32]");
    ES_MCUDA(cudaStreamSynchronize(m->stream), "sync");
    cudaFree(m->d_out);
    m->d_out = m->P.out = nullptr;
    m->cap = m->P.out_cap = 0;   // until there is a new one, scans count and store nothing
    ES_MCUDA(cudaMalloc(&m->d_out, sizeof(uint4) * cap), "cudaMalloc(survivors)");
    m->cap = cap;
    m->P.out = m->d_out;
    m->P.out_cap = cap;
    return ES_OK;
}

int es_mitm_reset(es_mitm* m) {
    if (!m) return mfail(ES_ERR_ARG, "null MITM engine");
    ES_MCUDA(cudaMemsetAsync(m->d_cnt, 0, 8ull * 2, m->stream), "memset");
    return ES_OK;
}

int es_mitm_scan(es_mitm* m, uint64_t B_lo, uint64_t B_hi, uint64_t s1_begin, uint64_t s1_end) {
    if (!m) return mfail(ES_ERR_ARG, "null MITM engine");
    const u128m B = ((u128m)B_hi << 64) | B_lo;
    const u128m M = ((u128m)m->P.M_hi << 64) | m->P.M_lo;
    if (B == 0 || B > M) return mfail(ES_ERR_RANGE, "bound B must be in [1, M]");
    if (s1_begin > s1_end || s1_end > m->n1) return mfail(ES_ERR_RANGE, "s1 range outside [0, |S1|)");
    if (s1_begin == s1_end) return ES_OK;
    MitmParams P = m->P;
    P.B_lo = B_lo;
    P.B_hi = B_hi;
    P.s1_begin = s1_begin;
    P.s1_end = s1_end;
    ES_MCUDA(cudaMemsetAsync(m->d_cnt + 2, 0, 8, m->stream), "memset");
    // persistent grid, no more CTAs than there are units for their warps
    const uint64_t nb = (s1_end + P.n_a - 1) / P.n_a - s1_begin / P.n_a;
    // (several units per warp where there is work for that)
    const uint64_t warps = (uint64_t)m->grid * (kMitmThreads / 32);
    P.chunk = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(kMitmChunk, nb * P.n_slices / (4 * warps)));
    const uint64_t claims = (nb + P.chunk - 1) / P.chunk * P.n_slices;
    const int grid = (int)std::max<uint64_t>(1, std::min<uint64_t>(m->grid, (claims + kMitmThreads / 32 - 1) /
                                                                              (kMitmThreads / 32)));
    es_mitm_kernel<<<grid, kMitmThreads, 4u * P.merged_words, m->stream>>>(P);
    ES_MCUDA(cudaGetLastError(), "MITM launch");
    return ES_OK;
}

int es_mitm_results(es_mitm* m, uint64_t* n_lo, uint64_t* n_hi, uint64_t cap, uint64_t* n_surv,
                    uint64_t* n_cand) try {
    if (!m || !n_surv) return mfail(ES_ERR_ARG, "null argument");
    ES_MCUDA(cudaMemcpyAsync(m->h_cnt, m->d_cnt, 16, cudaMemcpyDeviceToHost, m->stream), "copy");
    ES_MCUDA(cudaStreamSynchronize(m->stream), "MITM kernel execution");
    const uint64_t cnt = m->h_cnt[0];
    *n_surv = cnt;
    if (n_cand) *n_cand = m->h_cnt[1];
    if (cnt > m->cap)
        return mfail(ES_ERR_OVERFLOW, "MITM survivor buffer overflow (" + std::to_string(cnt) + " > " +
                                          std::to_string(m->cap) + ")");
    if (cnt > cap) return mfail(ES_ERR_OVERFLOW, "output buffer smaller than the survivor count");
    if (!cnt) return ES_OK;
    std::vector<uint4> tmp(cnt);
    ES_MCUDA(cudaMemcpy(tmp.data(), m->d_out, sizeof(uint4) * cnt, cudaMemcpyDeviceToHost), "copy");
    for (uint64_t i = 0; i < cnt; ++i) {
        if (n_lo) n_lo[i] = ((uint64_t)tmp[i].y << 32) | tmp[i].x;
        if (n_hi) n_hi[i] = ((uint64_t)tmp[i].w << 32) | tmp[i].z;
    }
    return ES_OK;
} catch (const std::exception&) {
    return mfail(ES_ERR_NOMEM, "host allocation");
}

}  // extern "C"
