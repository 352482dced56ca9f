// The production scan kernel of the GB300 Erdős–Selfridge CRT-wheel sieve (sm_103a): launches that
// report survivors and count no filter stages.  It computes what es_scan_kernel.cuh computes (see
// there for the semantics and the reference's files) with the library's own cascade (es_cascade.h)
// in place of the caller's filter order; the survivors are the same.
//
// Work distribution, lanes and strips are those of es_scan_kernel.cuh: warps claim warp-units, the
// 32 lanes of a warp take 32 consecutive ring-2 rows over one window of ring-2 digits, ring 1 is
// swept in a warp-uniform loop and the inner ring is tested 32 candidates at a time.  What differs:
//
//  * Every inner table lies in shared memory, whatever the filters' moduli (the cascade's tables
//    are products of small projections), so one kernel serves every plan and no filter reads its
//    phases through L2.
//  * No residue is reduced in the sweep: a table has a row for every unreduced phase
//    BQ2 + TQ1 < 2 d.  In one-word rings a row holds the masks of both sides of the carry split
//    (phase x and x + corr), so a lookup is: select BQ2 with or without the ring-1 wrap, add the
//    digit's residue, load.  Wider rings have the wrapped row a fixed distance away.  Residues
//    are kept as byte offsets and BQ2 as the shared address itself.
//  * The tables after the first two are read only by lanes that still hold a candidate: a random
//    gather costs shared-memory wavefronts by its active lanes.
//  * The carry split is one 4-byte load: a bucket entry holds the first slot and the low bits of
//    the one key that may lie in the bucket.  Buckets with more keys, key ties and keys within the
//    rounding band take the exact 128-bit path out of line.
//  * A lane's record is b3, the sum of its terms of rings >= 3, and its residues.  They hold for
//    the whole window, ring 2 is added where it is needed, and so the queue of candidates outlives
//    a strip step: it is flushed 32 entries at a time and drained once per warp-unit.
//  * b3 is decoded from tables of sums over groups of rings (es_cascade.cu), a few 64-bit
//    divisions by reciprocal instead of one division per ring.
//  * Lanes outside the scanned range sweep along and are dropped at the end of the cascade (only
//    candidates that pass the residue stage get that far), so the sweep has no per-digit test for
//    partial cycles.  An explicit list of outer indices gives each lane its own ring-1 digit and
//    no sweep.
//
// CTA: one per SM, 20 warps at 96 registers.  16 warps at 128 registers leave the scheduler short of
// ready warps (k = 300, 2^34 positions: 1469 against 1369 us), 24 at 80 spill in wide rings (k = 379:
// 2209 against 1842 us).
//
// What bounds it: shared-memory wavefronts (l1tex 87 to 90 % busy, a third of them bank conflicts), then
// the ALU pipe (57 to 66 %) and instruction issue (62 to 72 %).  Through the drop-in calls, against the caller's cascade by word-mask
// or pair tables (es_scan_kernel.cuh): k = 300, 2^34 positions 3069 -> 1359 us (1290 of
// them the kernel), 2^30 positions 319 -> 155 (102); the three-word k = 379 wheel, 2^34 positions, 5506 ->
// 1730 (1661); both k = 390 wheels, 2^35 positions each, 17,024 -> 5580 us (5497; their caller-order
// tables, 1.75 MB per wheel, came through L2).  Figures beside single choices, here and in the host
// code, compare their two sides with the kernel of the day and are not its time now.
#pragma once
#include "es_scan_kernel.cuh"

namespace {

// Everything the flush, the exact tail and the emit need for one warp-unit (in the warp's slot in
// shared memory, written once per unit).
struct ProdCtx {
    U4 M;
    uint64_t M_lo;
    uint64_t t_blk;
    uint64_t e_base;                   // strip entry of lane 0 (ring-1 cycle or list position)
    uint64_t e_min, e_max;             // entries in range: ring-1 cycles or list positions
    uint64_t o_begin, o_end;           // outer indices in range
    const unsigned long long* list;    // outer-index list of the item, or null (a range)
    const uint32_t* tc;
    const uint32_t* allowed_g;
    es_survivor* surv;
    unsigned long long* surv_n;
    unsigned long long* group_found;
    uint64_t surv_cap;
    uint32_t kp1, nf, item_id, group, r0, r1;
    uint32_t lstride;                  // entries between the strips of consecutive lanes
    uint64_t row0;                     // ring-2 row of lane 0 (where lanes stay on their rows)
    uint32_t d2;                       // ring-2 digit of step 0
    uint32_t M_big;
};

struct ProdQueue {
    uint4 ent[ES_QCAP];
    uint4 rec0[32];                    // per lane: b3 = sum of the terms of rings >= 3, mod M (limbs)
    uint4 rec1[32];                    // per lane: b3 + block term mod the residue-stage filters
    uint16_t own_d2[32];               // per lane: ring-2 digit, where lanes do not share it
    ProdCtx ctx;
};
#define ES_OWN_DIGIT 0xffffffffu       // ProdCtx::d2 where lanes do not share the ring-2 digit
static_assert(sizeof(ProdQueue) <= ES_QUEUE_BYTES, "per-warp slot overflows its shared-memory share");

__device__ __forceinline__ uint32_t shl_c(uint32_t v, uint32_t n) {   // shifts of 32 and more give 0
    uint32_t r;
    asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(n));
    return r;
}

// The sweep is bound by the ALU pipe next to shared memory, and selects and three-input adds are ALU
// work: a select between x and x + d is a multiply-add on the FMA pipe instead (k = 390, 2^34
// positions 1480 -> 1401 us, k = 378 1310 -> 1217).  Inline assembly, so that they stay so.
__device__ __forceinline__ uint32_t mad_lo(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}
__device__ __forceinline__ uint32_t zero_or_one(bool p) {
    uint32_t r;
    asm("mov.u32 %0, %1;" : "=r"(r) : "r"((uint32_t)p));
    return r;
}

// Predicated loads: lanes whose `alive` is 0 load nothing and get an arbitrary value.
__device__ __forceinline__ uint2 lds64_if(uint32_t a, uint32_t alive) {
    uint2 v;
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p ld.shared.v2.u32 {%0, %1}, [%2];\n\t}"
        : "=r"(v.x), "=r"(v.y) : "r"(a), "r"(alive));
    return v;
}
__device__ __forceinline__ uint4 lds128_if(uint32_t a, uint32_t alive) {
    uint4 v;
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\t@p ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
        : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a), "r"(alive));
    return v;
}

// x mod q times the multiplier of an inner table (limb weights from `off` on carry it)
__device__ __forceinline__ uint32_t mod128_times(const U4 x, const EsFilterC& f) {
    const uint64_t y = (uint64_t)x.x * f.off + (uint64_t)x.y * f.w1 + (uint64_t)x.z * f.w2 + (uint64_t)x.w * f.w3;
    const uint64_t qt = __umul64hi(y, f.rcp);
    uint64_t r = y - qt * f.q;
    if (r >= f.q) r -= f.q;
    return (uint32_t)r;
}

// b3 = sum_{j>=3} term_j[d_j] mod M for ring-2 row `row`, from the sums over groups of rings.
__device__ __noinline__ U4 decode_row(const EsInst& si, uint64_t row, const U4 M) {
    U4 acc{0u, 0u, 0u, 0u};
    uint64_t rem = row;
    for (uint32_t g = 0; g < si.n_groups; ++g) {
        const EsGroup G = si.group[g];
        // floor(rem / size) or one less (magic = floor((2^64 - 1) / size)), then corrected
        uint64_t q = __umul64hi(rem, G.magic);
        uint64_t d = rem - q * G.size;
        if (d >= G.size) {
            d -= G.size;
            ++q;
        }
        rem = q;
        uint32_t wm;
        acc = addmod(acc, u4(__ldg(reinterpret_cast<const uint4*>(si.ring_terms) + (G.off + d))), M, wm);
    }
    return acc;
}

// The candidates that passed the residue stage: range test, n mod M in 128 bits, the rest of the
// cascade by limb weights and Barrett, then the emit.
__device__ __forceinline__ void prod_tail(const ProdQueue* Q, const unsigned char* smem, const EsInst& si, uint32_t f0,
                                          const U4 b2, uint32_t own, uint32_t d1, uint32_t slot, uint32_t step) {
    const ProdCtx& C = Q->ctx;
    const uint64_t e = C.e_base + (uint64_t)own * C.lstride + step;
    if (e < C.e_min || e >= C.e_max) return;
    const uint64_t oidx = C.list ? __ldg(C.list + e) : e * C.r1 + d1;
    if (oidx < C.o_begin || oidx >= C.o_end) return;
    const EsFilterC* sFC = reinterpret_cast<const EsFilterC*>(smem + si.o_FC);
    uint32_t wm;
    const U4 b = addmod(b2, u4(reinterpret_cast<const uint4*>(smem + si.o_T1)[d1]), C.M, wm);
    const U4 s = addmod(b, u4(reinterpret_cast<const uint4*>(smem + si.o_S0)[slot]), C.M, wm);
    for (uint32_t f = f0; f < C.nf; ++f) {
        const EsFilterC fc = sFC[f];
        uint32_t r = mod128(s, fc) + C.tc[f];
        if (r >= fc.q) r -= fc.q;
        const uint32_t wv = __ldg(C.allowed_g + fc.off + (r >> 5));
        if (!((wv >> (r & 31u)) & 1u)) return;
    }
    bool good;
    if (C.M_big) {
        good = (C.t_blk > 0) || s.w || s.z || s.y || (s.x > C.kp1);
    } else {
        const uint64_t n = C.t_blk * C.M_lo + s.x;   // M <= k+1 <= 1025: n fits easily
        good = n > C.kp1;
    }
    const unsigned long long at = atomicAdd(C.surv_n, 1ull);
    if (at < C.surv_cap) {
        es_survivor* rec = C.surv + at;
        rec->idx = oidx * (uint64_t)C.r0 + reinterpret_cast<const uint32_t*>(smem + si.o_I0)[slot];
        rec->s_lo = lo64(s);
        rec->s_hi = hi64(s);
        rec->t = C.t_blk;
        rec->item = C.item_id;
        rec->good = good ? 1u : 0u;
    }
    if (good && C.group_found) atomicMin(C.group_found + C.group, (unsigned long long)C.t_blk);
}

// warp-uniform: one pass over up to 32 queued entries.  Each lane takes the lowest candidate of its
// entry and puts the rest of the entry back.  Entry formats: words (w, w + 1) of one ring-1 digit:
// {bits of w, bits of w + 1, d1 | split << 16, lane | wrap << 5 | w << 6 | step << 17}; or, with PD
// (one-word inner rings), the words of two consecutive digits d1, d1 + 1: {bits of d1, bits of
// d1 + 1, d1 | split(d1) << 16 | split(d1 + 1) << 24, lane | wrap(d1) << 5 | wrap(d1 + 1) << 6 |
// step << 17}.  Where lanes do not share the ring-2 digit it is in the lane's record (own_d2), and
// the queue is drained before the next step.
template <int F, bool PD>
__device__ __forceinline__ void prod_flush(ProdQueue* Q, const unsigned char* smem, const EsInst& si, uint32_t lane,
                                           uint32_t& qhead, uint32_t& qsize) {
    __syncwarp();
    const uint32_t n = qsize < 32u ? qsize : 32u;
    const uint4 en = Q->ent[(qhead + lane) & (ES_QCAP - 1)];
    const uint64_t bits = lane < n ? ((uint64_t)en.y << 32) | en.x : 0ull;
    const uint64_t rest = bits & (bits - 1ull);
    const uint32_t back = __ballot_sync(0xffffffffu, rest != 0u);
    __syncwarp();   // every lane holds its entry before any slot is reused
    qhead = (qhead + n) & (ES_QCAP - 1);
    qsize -= n;
    if (rest) {
        // lands on a free or just-consumed slot: qsize - n + popc(back) <= old qsize < ES_QCAP
        const uint32_t pos = (qhead + qsize + __popc(back & ((1u << lane) - 1u))) & (ES_QCAP - 1);
        Q->ent[pos] = make_uint4((uint32_t)rest, (uint32_t)(rest >> 32), en.z, en.w);
    }
    qsize += __popc(back);
    const bool has = bits != 0ull;
    const uint32_t i = has ? __ffsll((long long)bits) - 1u : 0u;
    const uint32_t hw = PD ? (i >> 5) : 0u;        // PD: the candidate is in the second digit's word
    const uint32_t d1 = has ? (en.z & 0xffffu) + hw : 0u;
    const uint32_t slot = has ? (PD ? (i & 31u) : (((en.w >> 6) & 0x7ffu) << 5) + i) : 0u;
    const uint32_t own = has ? (en.w & 31u) : 0u;
    const uint32_t step = has ? en.w >> 17 : 0u;
    const bool wrap1 = has && ((en.w >> (5u + hw)) & 1u);
    const uint32_t split = PD ? (hw ? (en.z >> 24) : ((en.z >> 16) & 0xffu)) : (en.z >> 16);
    const bool cw = has && slot >= split;          // sorted slots from the split on wrap past M
    const EsFilterC* sFC = reinterpret_cast<const EsFilterC*>(smem + si.o_FC);
    const uint32_t* allowed = si.allowed;
    const uint32_t d2 = Q->ctx.d2 == ES_OWN_DIGIT ? Q->own_d2[own] : Q->ctx.d2 + step;
    uint32_t wm2;
    const U4 b2 = addmod(u4(Q->rec0[own]), u4(reinterpret_cast<const uint4*>(smem + si.o_T2)[d2]), ldv_M(si), wm2);
    const uint4 bq = Q->rec1[own];
    const uint4 t2 = reinterpret_cast<const uint4*>(smem + si.o_TQ2r)[d2];
    const uint4 tq = reinterpret_cast<const uint4*>(smem + si.o_TQr)[d1];
    const uint4 sq = reinterpret_cast<const uint4*>(smem + si.o_Qr)[slot];
    const uint32_t bqv[ES_PRES] = {bq.x + t2.x, bq.y + t2.y, bq.z + t2.z, bq.w + t2.w};
    const uint32_t sqv[ES_PRES] = {sq.x + tq.x, sq.y + tq.y, sq.z + tq.z, sq.w + tq.w};
    // n mod q = b3 + T2[d2] + T1[d1] + S0[slot] mod q, with -M mod q per wrap
    const uint32_t wraps = (wm2 & 1u) + (wrap1 ? 1u : 0u) + (cw ? 1u : 0u);
    bool ok = has;
#pragma unroll
    for (uint32_t j = 0; j < ES_PRES; ++j) {
        if (j == 0 || __any_sync(0xffffffffu, ok)) {
            const EsFilterC& fc = sFC[F + j];
            const uint32_t q = fc.q;
            uint32_t x = bqv[j] + sqv[j] + wraps * fc.corr;   // < 7 q
            x = min(x, x - 4u * q);
            x = min(x, x - 2u * q);
            x = min(x, x - q);
            const uint32_t wv = __ldg(allowed + fc.off + (x >> 5));
            ok = ok && ((wv >> (x & 31u)) & 1u);
        }
    }
    if (ok) prod_tail(Q, smem, si, F + ES_PRES, b2, own, d1, slot, step);
    __syncwarp();
}

// warp-uniform (has = ballot of (lo | hi) != 0, nonzero; qsize < 32 on entry): queue the entry of
// every lane that has candidates, then flush while 32 entries wait
template <int F, bool PD>
__device__ __forceinline__ void prod_push(ProdQueue* Q, const unsigned char* smem, const EsInst& si, uint32_t lane,
                                          uint32_t& qhead, uint32_t& qsize, uint32_t has, uint32_t lo, uint32_t hi,
                                          uint32_t ez, uint32_t ew) {
    if (lo | hi) {
        const uint32_t pos = (qhead + qsize + __popc(has & ((1u << lane) - 1u))) & (ES_QCAP - 1);
        Q->ent[pos] = make_uint4(lo, hi, ez, ew);
    }
    qsize += __popc(has);
    // each pass retires one candidate per lane, so this ends
    while (qsize >= 32u) prod_flush<F, PD>(Q, smem, si, lane, qhead, qsize);
}

// The exact ring-1 wrap and carry split of digit d1 for one lane, in 128 bits: b = b2 + T1[d1] mod
// M, then the first sorted slot whose term is >= M - b.  Returns the slot, with the top bit set on a
// wrap.  Out of line: it runs for a tiny share of (lane, digit) pairs.
__device__ __noinline__ uint32_t prod_split(const ProdQueue* Q, const unsigned char* smem, const EsInst& si,
                                            uint32_t lane, uint32_t d2, uint32_t d1) {
    const U4 M = ldv_M(si);
    uint32_t wm, br;
    const U4 b2 = addmod(ldv128(&Q->rec0[lane]), ldv128(smem + si.o_T2 + 16u * d2), M, wm);
    const U4 b = addmod(b2, ldv128(smem + si.o_T1 + 16u * d1), M, wm);
    const U4 thr = sub128(M, b, br);
    const uint4* S0 = reinterpret_cast<const uint4*>(smem + si.o_S0);
    uint32_t lo = 0, hi = si.r0;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (lt128(u4(S0[mid]), thr)) lo = mid + 1; else hi = mid;
    }
    return lo | (wm & 0x80000000u);
}

// Words of a ring-1 row: the key and F scaled residues.
template <int F>
struct ProdRow {
    static constexpr uint32_t kWords = F <= 3 ? 4u : 8u;
    static constexpr uint32_t kBytes = 4u * kWords;
};

template <int F>
__device__ __forceinline__ void load_row(uint32_t a, uint32_t& key, uint32_t (&tq)[F]) {
    const uint4 r = lds128(a);
    key = r.x;
    tq[0] = r.y;
    if (F > 1) tq[1] = r.z;
    if (F > 2) tq[2] = r.w;
    if (F == 4) tq[3] = lds32(a + 16u);
    if (F > 4) {
        const uint4 s = lds128(a + 16u);
        tq[3] = s.x;
        tq[4] = s.y;
        if (F > 5) tq[5] = s.z;
    }
}

// Warp-uniform: scan one warp-unit w of `item`, whose plan is staged in smem / si.
template <int F, int WT>
__device__ __forceinline__ void prod_unit(const EsLaunch& L, const EsInst& si, unsigned char* smem, ProdQueue* Q,
                                          uint32_t lane, unsigned long long w, const EsItem& item) {
    constexpr uint32_t NW = WT == 0 ? 1u : (uint32_t)WT;   // inner words held at a time
    constexpr uint32_t NU = WT == 1 ? 2u : 1u;             // ring-1 digits per loop iteration
    constexpr bool PD = WT == 1;
    const uint32_t r1 = si.r1, r2 = si.r2;
    const EsFilterC* sFC = reinterpret_cast<const EsFilterC*>(smem + si.o_FC);
    const bool list = item.list != nullptr;
    // This unit's entries, decoded as in es_scan_kernel.cuh's scan_unit (units_of in es_abi.cu).
    const uint64_t u = w - item.unit_begin;
    const uint64_t c_lo = list ? item.o_begin : item.c_begin, c_hi = list ? item.o_end : item.c_end;
    uint64_t e_base, e_lo, row0 = 0;
    uint32_t lstride, nsteps, wlo = 0;
    if (!list && r2 > 1u) {
        const uint32_t J = (r2 + L.strip - 1u) / L.strip;
        const uint64_t rb = u / J;
        const uint32_t j = (uint32_t)(u - rb * J);
        wlo = j * r2 / J;
        nsteps = (j + 1u) * r2 / J - wlo;
        lstride = r2;
        row0 = item.c_begin / r2 + rb * 32ull;
        e_base = row0 * r2 + wlo;
    } else {
        nsteps = lstride = L.strip;
        e_base = c_lo + u * 32ull * L.strip;
    }
    e_lo = e_base + (uint64_t)lane * lstride;
    const bool rows = !list && r2 > 1u;   // each lane stays on its ring-2 row for the whole unit
    // this lane's steps in range: [first, last); the unit takes as many steps as its longest lane
    const uint64_t e_end = min(e_lo + nsteps, c_hi);
    const uint32_t last = e_end > e_lo ? (uint32_t)(e_end - e_lo) : 0u;
    const uint32_t first = e_lo >= c_lo ? 0u : (uint32_t)min(c_lo - e_lo, (uint64_t)nsteps);
    nsteps = __reduce_max_sync(0xffffffffu, last);
    ProdCtx& C = Q->ctx;
    if (lane == 0) {
        C.M = U4{(uint32_t)si.M_lo, (uint32_t)(si.M_lo >> 32), (uint32_t)si.M_hi, (uint32_t)(si.M_hi >> 32)};
        C.M_lo = si.M_lo;
        C.kp1 = si.k + 1u;
        C.M_big = (si.M_hi != 0) || (si.M_lo > C.kp1);
        C.nf = si.n_filters;
        C.r0 = si.r0;
        C.r1 = r1;
        C.tc = L.items ? item.tconst : L.tconst0;
        C.allowed_g = si.allowed;
        C.surv = L.surv;
        C.surv_n = L.surv_n;
        C.group_found = L.group_found;
        C.surv_cap = L.surv_cap;
        C.item_id = item.caller;
        C.group = item.group;
        C.t_blk = item.t;
        C.lstride = lstride;
        C.d2 = rows ? wlo : ES_OWN_DIGIT;
        C.row0 = row0;
        C.list = reinterpret_cast<const unsigned long long*>(item.list);
        C.e_base = e_base;
        C.e_min = c_lo;
        C.e_max = c_hi;
        C.o_begin = list ? 0ull : item.o_begin;
        C.o_end = list ? ~0ull : item.o_end;
    }
    // lanes that never reach a cycle of the range sweep with b3 = 0 (their candidates are dropped)
    Q->rec0[lane] = make_uint4(0u, 0u, 0u, 0u);
    Q->rec1[lane] = make_uint4(0u, 0u, 0u, 0u);
    Q->own_d2[lane] = 0;
    __syncwarp();

    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
    const uint32_t rb = si.row_bytes, KM = si.km;
    constexpr uint32_t bsh = 32u - ES_PBUCKET_LOG2, ssh = ES_PBUCKET_LOG2, smask = (1u << ssh) - 1u, band = 3u << ssh;
    const uint32_t bk = sbase + si.o_BK;
    int32_t wrap[F];   // (one- and two-word rings have the wrapped row in the row itself)
#pragma unroll
    for (int f = 0; f < F; ++f) wrap[f] = si.tab_wrap[f];
    uint32_t BQ3[F];   // b3 + block term mod the inner tables' moduli
#pragma unroll
    for (int f = 0; f < F; ++f) BQ3[f] = 0u;
    uint32_t qhead = 0, qsize = 0;
    for (uint32_t step = 0; step < nsteps; ++step) {
        uint32_t lo1 = 0u, d2 = rows ? wlo + step : 0u;
        const U4 Mv = ldv_M(si);
        if (rows ? (step == 0u && first < last) : (step >= first && step < last)) {
            const uint64_t e = Q->ctx.e_base + (uint64_t)lane * Q->ctx.lstride + step;
            const uint32_t* tcv = Q->ctx.tc;
            uint64_t row;
            if (rows) {
                row = Q->ctx.row0 + lane;
            } else {
                uint64_t c = e;
                if (list) {
                    const uint64_t o = __ldg(Q->ctx.list + e);
                    c = o / r1;
                    lo1 = (uint32_t)(o - c * r1);
                }
                row = c / r2;
                d2 = (uint32_t)(c - row * r2);
                Q->own_d2[lane] = (uint16_t)d2;
            }
            const U4 b3 = decode_row(si, row, Mv);
#pragma unroll
            for (int f = 0; f < F; ++f) BQ3[f] = red1(mod128_times(b3, sFC[f]) + tcv[f], sFC[f].q);
            uint32_t rv[ES_PRES];
#pragma unroll
            for (uint32_t j = 0; j < ES_PRES; ++j) rv[j] = red1(mod128(b3, sFC[F + j]) + tcv[F + j], sFC[F + j].q);
            Q->rec0[lane] = make_uint4(b3.x, b3.y, b3.z, b3.w);
            Q->rec1[lane] = make_uint4(rv[0], rv[1], rv[2], rv[3]);
        }
        uint32_t wm2;
        const U4 b2 = addmod(ldv128(&Q->rec0[lane]), u4(reinterpret_cast<const uint4*>(smem + si.o_T2)[d2]), Mv, wm2);
        // shared addresses of the tables' rows at BQ2, and what the ring-1 wrap adds to them
        uint32_t B[F], Bw[F];
        constexpr uint32_t DS = F <= 4 ? 4u : 8u;
        const uint32_t* tq2 = reinterpret_cast<const uint32_t*>(smem + si.o_TQ2) + d2 * DS;
#pragma unroll
        for (int f = 0; f < F; ++f) {
            // (volatile loads: constants of the step are not worth registers in the sweep)
            const uint32_t q = ldv32(&sFC[f].q), corr = ldv32(&sFC[f].corr);
            const uint32_t base = sbase + L.stage_off + ldv32(&si.tab_base[f]);
            const uint32_t BQ2 = red2(BQ3[f] + tq2[f] + (corr & wm2), q);
            B[f] = base + rb * BQ2;
            Bw[f] = base + rb * red1(BQ2 + corr, q) - B[f];
        }
        const uint32_t ews = lane | (step << 17);   // entry fields that belong to the step
        // A = M - b2 and its 32-bit key, once per ring-1 cycle
        uint32_t brA;
        const uint32_t KA = key32(sub128(Mv, b2, brA), si.sh) << si.lsh;

        // ---- ring 1 (a list has one digit per lane) -----------------------------------------
        const uint32_t nd = list ? 1u : r1;
        uint32_t row = sbase + si.o_R1 + lo1 * ProdRow<F>::kBytes;
        for (uint32_t i = 0; i < nd; i += NU, row += NU * ProdRow<F>::kBytes) {
            const uint32_t d1 = lo1 + i;
            uint32_t split[NU], wm1[NU], bits[NU][NW];
            uint32_t a[NU][F];
            bool rare[NU], any_rare = false;
#pragma unroll
            for (uint32_t v = 0; v < NU; ++v) {
                uint32_t k1, tq[F];
                load_row<F>(row + v * ProdRow<F>::kBytes, k1, tq);
                // ring-1 wrap (b2 + T1 >= M, i.e. T1 >= A) from the 32-bit keys, and t, the key of
                // thr = M - b to within +-1 (0 <= t <= KM away from a key tie)
                const uint32_t p = zero_or_one(k1 > KA);
                const uint32_t t = mad_lo(p, KM, KA - k1);
                const uint32_t e4 = lds32(bk + ((t >> bsh) << 2));
                const uint32_t ts = t << ssh;
                const uint32_t sp = e4 & smask;
                split[v] = sp + (e4 < ts ? 1u : 0u);
                rare[v] = (e4 - ts < band) || (sp == smask) || (k1 == KA);
                any_rare = any_rare || rare[v];
                wm1[v] = 0u - p;
#pragma unroll
                for (int f = 0; f < F; ++f) a[v][f] = mad_lo(p, Bw[f], B[f] + tq[f]);
            }
            // The first table's row is on its way before the vote on the exact path (whose lanes load
            // theirs again if the wrap was other than the keys said): k = 390, 2^34 positions 1659 ->
            // 1599 us, k = 384 2312 -> 2202, k = 379 1866 -> 1808, k = 300 1371 -> 1364.  Two rows cost
            // registers in wide rings (k = 378 1343 -> 1524).
            constexpr int PRE = WT == 0 ? 0 : 1;
            uint32_t pre0[NU][PRE + 1][4], pre1[NU][PRE + 1][4];
            auto load_pair = [&](uint32_t at, int f, uint32_t (&x0)[4], uint32_t (&x1)[4]) {
                if (WT == 1) {
                    const uint2 y = lds64(at);
                    x0[0] = y.x;
                    x1[0] = y.y;
                } else if (WT == 2) {
                    const uint2 y0 = lds64(at), y1 = lds64(at + wrap[f]);
                    x0[0] = y0.x; x0[1] = y0.y;
                    x1[0] = y1.x; x1[1] = y1.y;
                } else {
                    const uint4 y0 = lds128(at), y1 = lds128(at + wrap[f]);
                    x0[0] = y0.x; x0[1] = y0.y; x0[2] = y0.z; x0[3] = y0.w;
                    x1[0] = y1.x; x1[1] = y1.y; x1[2] = y1.z; x1[3] = y1.w;
                }
            };
#pragma unroll
            for (uint32_t v = 0; v < NU; ++v)
#pragma unroll
                for (int f = 0; f < PRE; ++f) load_pair(a[v][f], f, pre0[v][f], pre1[v][f]);
            if (__any_sync(0xffffffffu, any_rare)) {
#pragma unroll
                for (uint32_t v = 0; v < NU; ++v) {
                    // the padding row after the last digit has no term of its own
                    if (rare[v] && d1 + v < r1) {
                        const uint32_t was = wm1[v], x = prod_split(Q, smem, si, lane, d2, d1 + v);
                        split[v] = x & 0x7fffffffu;
                        wm1[v] = (x >> 31) ? 0xffffffffu : 0u;
                        if (was != wm1[v]) {
#pragma unroll
                            for (int f = 0; f < F; ++f) a[v][f] += wm1[v] ? Bw[f] : 0u - Bw[f];
#pragma unroll
                            for (int f = 0; f < PRE; ++f) load_pair(a[v][f], f, pre0[v][f], pre1[v][f]);
                        }
                    }
                }
            }
            if constexpr (WT == 0) {
                // any inner width: word by word, two words per entry
                const uint32_t Wn = si.W, tail = si.tail_mask;
                uint32_t lo = 0u;
                for (uint32_t wd = 0; wd < Wn; ++wd) {
                    const uint32_t from = wd << 5;
                    const uint32_t cm = shl_c(0xffffffffu, max(split[0], from) - from);
                    uint32_t m0 = wd + 1u == Wn ? tail : 0xffffffffu, m1 = m0;
#pragma unroll
                    for (int f = 0; f < F; ++f) {
                        m0 &= lds32(a[0][f] + 4u * wd);
                        m1 &= lds32(a[0][f] + wrap[f] + 4u * wd);
                    }
                    const uint32_t x = (m0 & ~cm) | (m1 & cm);
                    if ((wd & 1u) == 0u && wd + 1u < Wn) {
                        lo = x;
                        continue;
                    }
                    const bool odd = (wd & 1u) != 0u;
                    const uint32_t p0 = odd ? lo : x, p1 = odd ? x : 0u;
                    const uint32_t has = __ballot_sync(0xffffffffu, (p0 | p1) != 0u);
                    if (has)
                        prod_push<F, PD>(Q, smem, si, lane, qhead, qsize, has, p0, p1, ent_z(d1, split[0]),
                                         ent_w(ews, wm1[0], wd & ~1u));
                }
            } else {
#pragma unroll
                for (uint32_t v = 0; v < NU; ++v) {
                    // candidates on either side of the split that every table so far admits
                    uint32_t m0[NW], m1[NW];
#pragma unroll
                    for (uint32_t j = 0; j < NW; ++j) {
                        m1[j] = shl_c(0xffffffffu, j == 0 ? split[v] : max(split[v], 32u * j) - 32u * j);
                        m0[j] = ~m1[j];
                    }
#pragma unroll
                    for (int f = 0; f < F; ++f) {
                        uint32_t x0[4], x1[4];
                        if (f < PRE) {
#pragma unroll
                            for (uint32_t j = 0; j < NW; ++j) {
                                x0[j] = pre0[v][f < PRE ? f : 0][j];
                                x1[j] = pre1[v][f < PRE ? f : 0][j];
                            }
                        } else if (f < 2) {
                            load_pair(a[v][f], f, x0, x1);
                        } else if (WT == 1) {
                            const uint2 y = lds64_if(a[v][f], m0[0] | m1[0]);
                            x0[0] = y.x;
                            x1[0] = y.y;
                        } else if (WT == 2) {
                            const uint2 y0 = lds64_if(a[v][f], m0[0] | m0[NW - 1]);
                            const uint2 y1 = lds64_if(a[v][f] + wrap[f], m1[0] | m1[NW - 1]);
                            x0[0] = y0.x; x0[1] = y0.y;
                            x1[0] = y1.x; x1[1] = y1.y;
                        } else {
                            uint32_t l0 = 0u, l1 = 0u;
#pragma unroll
                            for (uint32_t j = 0; j < NW; ++j) {
                                l0 |= m0[j];
                                l1 |= m1[j];
                            }
                            const uint4 y0 = lds128_if(a[v][f], l0), y1 = lds128_if(a[v][f] + wrap[f], l1);
                            x0[0] = y0.x; x0[1] = y0.y; x0[2] = y0.z; x0[3] = y0.w;
                            x1[0] = y1.x; x1[1] = y1.y; x1[2] = y1.z; x1[3] = y1.w;
                        }
#pragma unroll
                        for (uint32_t j = 0; j < NW; ++j) {
                            m0[j] &= x0[j];
                            m1[j] &= x1[j];
                        }
                    }
#pragma unroll
                    for (uint32_t j = 0; j < NW; ++j) bits[v][j] = m0[j] | m1[j];
                }
                if (WT == 1) {
                    if (i + 1u >= nd) bits[NU - 1][0] = 0u;   // the padding row
                    const uint32_t has = __ballot_sync(0xffffffffu, (bits[0][0] | bits[NU - 1][0]) != 0u);
                    if (has)
                        prod_push<F, PD>(Q, smem, si, lane, qhead, qsize, has, bits[0][0], bits[NU - 1][0],
                                         d1 | (split[0] << 16) | (split[NU - 1] << 24),
                                         ews | (wm1[0] & 32u) | (wm1[NU - 1] & 64u));
                } else {
#pragma unroll 1
                    for (uint32_t j = 0; j < NW; j += 2) {   // (one copy of the push and flush)
                        const uint32_t p0 = j ? bits[0][NW - 2] : bits[0][0], p1 = j ? bits[0][NW - 1] : bits[0][1];
                        const uint32_t has = __ballot_sync(0xffffffffu, (p0 | p1) != 0u);
                        if (has)
                            prod_push<F, PD>(Q, smem, si, lane, qhead, qsize, has, p0, p1, ent_z(d1, split[0]),
                                             ent_w(ews, wm1[0], j));
                    }
                }
            }
        }
        // drain the queue after the last step, and where the lanes' records change with the next one
        if (!rows || step + 1u == nsteps)
            while (qsize) prod_flush<F, PD>(Q, smem, si, lane, qhead, qsize);
    }
    __syncwarp();
}

// Copies nwords words (both ends 16-byte aligned) with several loads in flight per thread.
__device__ __forceinline__ void stage_words(unsigned char* dst, const void* src, uint32_t nwords) {
    const uint4* s4 = reinterpret_cast<const uint4*>(src);
    uint4* d4 = reinterpret_cast<uint4*>(dst);
    const uint32_t n4 = nwords >> 2;
    uint32_t i = threadIdx.x;
    for (; i + 3u * blockDim.x < n4; i += 4u * blockDim.x) {
        uint4 v[4];
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) v[j] = __ldg(s4 + i + j * blockDim.x);
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) d4[i + j * blockDim.x] = v[j];
    }
    for (; i < n4; i += blockDim.x) d4[i] = __ldg(s4 + i);
}

__device__ __forceinline__ void stage_plan(const EsLaunch& L, EsInst& si, const EsInst* inst, unsigned char* smem) {
    load_inst(si, inst);
    if (L.small) {   // the launch has one plan and brings its table addresses
        stage_words(smem, L.small, L.small_bytes >> 2);
        stage_words(smem + L.stage_off, L.tabs, L.tab_words);
    } else {
        __syncthreads();
        stage_words(smem, si.small, si.small_bytes >> 2);
        stage_words(smem + L.stage_off, si.masks, si.tab_words);
    }
    __syncthreads();
}

// Template: F = inner tables, WT = inner-ring words (1, 2; 4 for three and four, rows of 16 bytes;
// 0 for wider rings).  Work distribution as in es_scan_kernel.
template <int F, int WT>
__global__ void __launch_bounds__(ES_PROD_THREADS, 1) es_prod_kernel(const __grid_constant__ EsLaunch L) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ EsInst si;
    __shared__ uint32_t s_item;

    const uint32_t tid = threadIdx.x;
    const uint32_t lane = tid & 31u;
    ProdQueue* Q = reinterpret_cast<ProdQueue*>(smem + L.queue_off + (tid >> 5) * ES_QUEUE_BYTES);
    const EsItem* items = L.items ? L.items : &L.item0;
    const unsigned long long total = L.total_units;

    if (L.direct) {
        // one plan: stage it, then warps claim warp-units on their own (the first claim is on its way
        // meanwhile).  With no more units than warps each warp has one at most and claims once.
        unsigned long long w = 0;
        if (lane == 0) w = atomicAdd(L.unit_counter, 1ull);
        const bool single = total <= (unsigned long long)gridDim.x * (blockDim.x >> 5);
        stage_plan(L, si, items[0].inst, smem);
        for (bool first = true;; first = false) {
            if (!first && single) break;
            uint32_t it_id = 0;
            int skip = 0;
            if (lane == 0) {
                if (!first) w = atomicAdd(L.unit_counter, 1ull);
                if (w < total) {
                    uint32_t lo = 0, hi = L.n_items;
                    while (hi - lo > 1) {
                        const uint32_t mid = (lo + hi) >> 1;
                        if (items[mid].unit_begin <= w) lo = mid; else hi = mid;
                    }
                    it_id = lo;
                    if (L.group_found) {
                        const unsigned long long fnd =
                            *reinterpret_cast<volatile unsigned long long*>(L.group_found + items[lo].group);
                        if (items[lo].t > fnd) skip = 1;
                    }
                }
            }
            w = __shfl_sync(0xffffffffu, w, 0);
            if (w >= total) break;
            it_id = __shfl_sync(0xffffffffu, it_id, 0);
            skip = __shfl_sync(0xffffffffu, skip, 0);
            if (skip) continue;
            prod_unit<F, WT>(L, si, smem, Q, lane, w, items[it_id]);
        }
        leave(L);
        return;
    }

    // several plans: a CTA works on one item at a time and synchronises only to move to another
    uint32_t cur_inst = 0xffffffffu;
    if (tid == 0) {
        const unsigned long long u0 = (unsigned long long)blockIdx.x * total / gridDim.x;
        uint32_t lo = 0, hi = L.n_items;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (items[mid].unit_begin <= u0) lo = mid; else hi = mid;
        }
        s_item = lo;
    }
    __syncthreads();
    for (;;) {
        const uint32_t item_id = s_item;
        if (item_id >= L.n_items) break;
        const EsItem& item = items[item_id];
        if (item.inst_id != cur_inst) {
            stage_plan(L, si, item.inst, smem);
            cur_inst = item.inst_id;
        }
        for (;;) {
            unsigned long long w = 0;
            int stop = 0;
            if (lane == 0) {
                const unsigned long long c = atomicAdd(L.item_next + item_id, 1ull);
                if (c >= item.n_units) {
                    stop = 1;
                } else if (L.group_found) {
                    const unsigned long long fnd =
                        *reinterpret_cast<volatile unsigned long long*>(L.group_found + item.group);
                    if (item.t > fnd) stop = 1;
                }
                w = item.unit_begin + c;
            }
            stop = __shfl_sync(0xffffffffu, stop, 0);
            w = __shfl_sync(0xffffffffu, w, 0);
            if (stop) break;
            prod_unit<F, WT>(L, si, smem, Q, lane, w, item);
        }
        __syncthreads();   // every warp is done with this item before its tables may be replaced
        if (tid == 0) {
            // the next item with unclaimed warp-units, after this one cyclically; each pass of
            // the loop above claims at least one unit, so the counters only grow and this ends
            uint32_t nxt = L.n_items;
            for (uint32_t j = 1; j <= L.n_items; ++j) {
                const uint32_t i = (item_id + j) % L.n_items;
                const EsItem& it = items[i];
                const unsigned long long c = *reinterpret_cast<volatile unsigned long long*>(L.item_next + i);
                if (c >= it.n_units) continue;
                if (L.group_found) {
                    const unsigned long long fnd =
                        *reinterpret_cast<volatile unsigned long long*>(L.group_found + it.group);
                    if (it.t > fnd) continue;
                }
                nxt = i;
                break;
            }
            s_item = nxt;
        }
        __syncthreads();
    }
}

template <int WT>
ScanFn pick_prod(uint32_t f) {
    switch (f) {
        case 1: return es_prod_kernel<1, WT>;
        case 2: return es_prod_kernel<2, WT>;
        case 3: return es_prod_kernel<3, WT>;
        case 4: return es_prod_kernel<4, WT>;
        case 5: return es_prod_kernel<5, WT>;
        case 6: return es_prod_kernel<6, WT>;
        default: return nullptr;
    }
}

}  // namespace
