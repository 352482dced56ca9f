// Host side of the production cascade (es_cascade.h): the plan, which projections the inner tables
// hold, and the tables themselves.
#include "es_cascade.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "../../include/es_gb300.h"

typedef es_u128 u128;

namespace {

int refuse(std::string& why, int code, const std::string& msg) {
    why = msg;
    return code;
}

}  // namespace

int es_check_desc(const es_plan_desc& d, std::string& why) {
    if (d.flags != 0) return refuse(why, ES_ERR_ARG, "descriptor flags must be 0");
    const u128 M = ((u128)d.M_hi << 64) | d.M_lo;
    if (M == 0 || es_bitlen(M) > 126) return refuse(why, ES_ERR_RANGE, "wheel modulus must be in [1, 2^126)");
    if (d.n_filters > ES_MAX_FILTERS)
        return refuse(why, ES_ERR_RANGE, "too many residual filters (max " + std::to_string(ES_MAX_FILTERS) + ")");
    if (d.n_rings > ES_MAX_RINGS - 3) return refuse(why, ES_ERR_RANGE, "too many wheel rings");
    if (d.n_rings && (!d.radix || !d.term_lo || !d.term_hi))
        return refuse(why, ES_ERR_ARG, "null ring arrays");
    if (d.n_filters && (!d.filter_q || !d.allowed)) return refuse(why, ES_ERR_ARG, "null filter arrays");
    return ES_OK;
}

int es_parse_plan(const es_plan_desc& d, EsHostPlan& P, EsInst& I, std::string& why) {
    const u128 M = ((u128)d.M_hi << 64) | d.M_lo;
    P.k = d.k;
    P.M = M;
    uint64_t R = 1;
    size_t pos = 0;
    for (uint32_t j = 0; j < d.n_rings; ++j) {
        const uint32_t r = d.radix[j];
        if (r == 0 || r > 65535) return refuse(why, ES_ERR_RANGE, "ring radix must be in [1, 65535]");
        P.roff.push_back((uint32_t)P.terms.size());
        P.radix.push_back(r);
        for (uint32_t i = 0; i < r; ++i, ++pos) {
            const u128 v = ((u128)d.term_hi[pos] << 64) | d.term_lo[pos];
            if (v >= M) return refuse(why, ES_ERR_ARG, "ring term not reduced mod M");
            P.terms.push_back(v);
        }
        if (R > (1ull << 62) / r) return refuse(why, ES_ERR_RANGE, "residues per block exceed 2^62");
        R *= r;
    }
    // rings are padded to three with radix-1 rings whose only term is 0
    while (P.radix.size() < 3) {
        P.roff.push_back((uint32_t)P.terms.size());
        P.radix.push_back(1);
        P.terms.push_back(0);
    }
    const uint32_t nf = d.n_filters;
    P.bit_off.assign(1, 0);
    for (uint32_t f = 0; f < nf; ++f) {
        const uint32_t q = d.filter_q[f];
        if (q < 2 || q >= ES_MAX_Q) return refuse(why, ES_ERR_RANGE, "filter modulus must be in [2, 2^20)");
        P.q.push_back(q);
        P.bit_off.push_back(P.bit_off.back() + (q + 31) / 32);
    }
    if (nf) P.allowed.assign(d.allowed, d.allowed + P.bit_off[nf]);
    I.M_lo = (uint64_t)M;
    I.M_hi = (uint64_t)(M >> 64);
    I.n_outer = R / P.radix[0];
    I.n_cycles = I.n_outer / P.radix[1];
    I.k = d.k;
    I.n_rings = (uint32_t)P.radix.size();
    I.r0 = P.radix[0];
    I.W = (I.r0 + 31) / 32;
    I.r1 = P.radix[1];
    I.r2 = P.radix[2];
    I.n_filters = nf;
    const uint32_t bl = es_bitlen(M);
    I.sh = bl > 32 ? bl - 32 : 0;
    I.km = (uint32_t)(M >> I.sh);
    I.tail_mask = (I.r0 % 32) ? ((1u << (I.r0 % 32)) - 1u) : 0xffffffffu;
    return ES_OK;
}

EsSortedRing es_sort_inner(const EsHostPlan& P) {
    EsSortedRing R;
    const uint32_t r0 = P.radix[0];
    const u128* t = P.terms.data() + P.roff[0];
    R.digit.resize(r0);
    for (uint32_t i = 0; i < r0; ++i) R.digit[i] = i;
    std::stable_sort(R.digit.begin(), R.digit.end(), [&](uint32_t a, uint32_t b) { return t[a] < t[b]; });
    R.S0.resize(r0);
    for (uint32_t i = 0; i < r0; ++i) R.S0[i] = t[R.digit[i]];
    return R;
}

u128 es_ring2_delta(const EsHostPlan& P, uint32_t i) {
    const uint32_t r2 = P.radix[2];
    const u128 a = P.terms[P.roff[2] + i], b = P.terms[P.roff[2] + (i + 1) % r2];
    return b >= a ? b - a : b + (P.M - a);
}

EsFilterC es_filter_consts(u128 M, uint32_t q, uint32_t off) {
    EsFilterC f;
    f.q = q;
    f.corr = (uint32_t)((q - es_mod(M, q)) % q);
    f.w1 = es_mod((u128)1 << 32, q);
    f.w2 = es_mod((u128)1 << 64, q);
    f.w3 = es_mod((u128)1 << 96, q);
    f.off = off;
    f.rcp = (uint64_t)(((u128)1 << 64) / q);
    return f;
}

uint32_t EsSmallBlock::take(size_t bytes) {
    const size_t o = b.size();
    b.resize(es_align_up(o + bytes, 16), 0);
    return (uint32_t)o;
}
void EsSmallBlock::put128(uint32_t o, size_t i, u128 v) {
    const uint64_t lo = (uint64_t)v, hi = (uint64_t)(v >> 64);
    memcpy(&b[o + 16 * i], &lo, 8);
    memcpy(&b[o + 16 * i + 8], &hi, 8);
}
void EsSmallBlock::put32(uint32_t o, size_t i, uint32_t v) { memcpy(&b[o + 4 * i], &v, 4); }

namespace {

uint32_t gcd32(uint32_t a, uint32_t b) {
    while (b) {
        const uint32_t t = a % b;
        a = b;
        b = t;
    }
    return a;
}

// The prime p when q is a power of p, else 0 (q < 2^20: at most 512 trial divisions by odd numbers).
uint32_t prime_of_power(uint32_t q) {
    uint32_t p = 0;
    if (q % 2u == 0u) p = 2u;
    for (uint32_t x = 3; !p && x * x <= q; x += 2)
        if (q % x == 0u) p = x;
    if (!p) return q;
    while (q % p == 0u) q /= p;
    return q == 1u ? p : 0u;
}

// 32 packed bits from bit `at` on, of `words` words (0 past them)
inline uint32_t bits_at(const uint32_t* bits, uint32_t words, uint32_t at) {
    const uint32_t w = at >> 5, s = at & 31u;
    const uint64_t lo = w < words ? bits[w] : 0u, hi = w + 1u < words ? bits[w + 1u] : 0u;
    return (uint32_t)(((hi << 32) | lo) >> s);
}

// The packed admissible set of a filter (q residues) projected to d | q, packed: word by word.
void project_bits(const uint32_t* bits, uint32_t q, uint32_t d, std::vector<uint32_t>& out) {
    const uint32_t words = (q + 31u) / 32u, n = (d + 31u) / 32u;
    out.assign(n, 0u);
    for (uint32_t from = 0; from < q; from += d)
        for (uint32_t w = 0; w < n; ++w) out[w] |= bits_at(bits, words, from + 32u * w);
    if (d % 32u) out[n - 1u] &= (1u << (d % 32u)) - 1u;
}

uint32_t count_bits(const std::vector<uint32_t>& v) {
    uint32_t n = 0;
    for (uint32_t w : v) n += (uint32_t)__builtin_popcount(w);
    return n;
}

// -log of the share of candidates that pass "n mod d lies in the packed set `proj`", given the wheel:
// among the residues mod d whose projection to g = gcd(d, M) the set holds at all.
double value_of(const std::vector<uint32_t>& proj, uint32_t d, uint32_t g, std::vector<uint32_t>& tmp) {
    const uint32_t n = count_bits(proj);
    if (n == 0) return 64.0;   // nothing is admissible
    uint32_t ng = 1;
    if (g > 1u) {
        project_bits(proj.data(), d, g, tmp);
        ng = count_bits(tmp);
    }
    return -std::log(((double)n / d) * ((double)g / ng));
}

// A possible inner table: up to three parts.
struct Slot {
    uint32_t n, part[3];
    double rows, value;
    uint64_t bytes;   // of its rows, padded as es_prod_image lays them out
};

}  // namespace

void es_project(const uint32_t* bits, uint32_t q, uint32_t d, std::vector<uint8_t>& out) {
    out.assign(d, 0);
    for (uint32_t from = 0; from < q; from += d)
        for (uint32_t j = 0; j < d; ++j) out[j] |= (bits[(from + j) >> 5] >> ((from + j) & 31u)) & 1u;
}

void es_and_periodic(const uint32_t* bits, uint32_t q, uint32_t d, uint32_t n, uint32_t* out) {
    std::vector<uint32_t> proj;
    project_bits(bits, q, d, proj);
    // one period and the 32 bits after it, so that a word can start anywhere in the period
    const uint32_t words = (d + 31u) / 32u + 1u;
    std::vector<uint32_t> two(words, 0u);
    for (uint32_t at = 0; at < 32u * words; at += d)
        for (uint32_t w = 0; w < proj.size(); ++w) {
            const uint32_t to = at + 32u * w;
            if (to >= 32u * words) break;
            two[to / 32u] |= proj[w] << (to % 32u);
            if (to % 32u && to / 32u + 1u < words) two[to / 32u + 1u] |= proj[w] >> (32u - to % 32u);
        }
    for (uint32_t w = 0, at = 0; w < (n + 31u) / 32u; ++w) {
        out[w] &= bits_at(two.data(), words, at);
        at = (at + 32u) % d;
    }
}

EsCascade es_choose_cascade(const EsHostPlan& P, uint32_t F, uint32_t row_bytes, bool pair, uint32_t table_bytes) {
    const uint32_t nf = (uint32_t)P.q.size();
    const double budget = (double)(table_bytes / row_bytes);
    std::vector<EsPart> parts;
    std::vector<double> full(nf, 0.0);   // value of the whole filter
    std::vector<uint32_t> proj, tmp;
    for (uint32_t f = 0; f < nf; ++f) {
        const uint32_t q = P.q[f], gM = gcd32(q, (uint32_t)(P.M % q));
        const uint32_t* bits = P.allowed.data() + P.bit_off[f];
        const uint32_t p = prime_of_power(q);
        for (uint32_t d = p ? p : q;; d *= p) {
            const bool whole = d == q;
            if (whole || 2.0 * d <= budget) {
                project_bits(bits, q, d, proj);
                const double v = value_of(proj, d, gcd32(d, gM), tmp);
                if (whole) full[f] = v;
                if (v > 1e-3 && 2.0 * d <= budget) parts.push_back(EsPart{f, d, v});
            }
            if (whole) break;
        }
    }
    // The parts that reject most, then tables of one, two or three of them.
    std::stable_sort(parts.begin(), parts.end(), [](const EsPart& a, const EsPart& b) { return a.value > b.value; });
    if (parts.size() > 48) parts.resize(48);
    auto rows = [&](uint32_t d) {
        const uint32_t m = (uint32_t)(P.M % d);
        return es_planned_rows(d, m ? d - m : 0u, pair);
    };
    auto bytes_of = [&](uint32_t n) { return (uint64_t)es_align_up((uint64_t)n * row_bytes, 16); };
    const uint64_t fill_bytes = bytes_of(es_table_rows(2, 1, pair));
    std::vector<Slot> slots;
    const uint32_t np = (uint32_t)parts.size();
    auto add = [&](uint32_t n, uint32_t a, uint32_t b, uint32_t c) {
        const uint32_t at[3] = {a, b, c};
        uint64_t d = 1;
        double v = 0.0;
        for (uint32_t i = 0; i < n; ++i) {
            const EsPart& x = parts[at[i]];
            for (uint32_t j = 0; j < i; ++j)
                if (parts[at[j]].f == x.f || gcd32(parts[at[j]].d, x.d) != 1u) return;
            d *= x.d;
            v += x.value;
        }
        if (d >= ES_MAX_Q || 2.0 * (double)d > budget) return;
        const uint32_t r = rows((uint32_t)d);
        if (bytes_of(r) <= table_bytes) slots.push_back(Slot{n, {a, b, c}, (double)r, v, bytes_of(r)});
    };
    for (uint32_t a = 0; a < np; ++a) {
        add(1, a, 0, 0);
        for (uint32_t b = a + 1; b < np; ++b) {
            if (2.0 * parts[a].d * parts[b].d > budget) continue;
            add(2, a, b, 0);
            for (uint32_t c = b + 1; c < np; ++c)
                if (2.0 * parts[a].d * parts[b].d * parts[c].d <= budget) add(3, a, b, c);
        }
    }
    // F tables of disjoint filters with the largest summed value within the budget: greedy picks
    // by value minus a price per row, over a range of prices.
    std::vector<uint32_t> best;
    double best_value = -1.0;
    uint64_t spare = 0;
    std::vector<uint8_t> used(nf);
    for (int step = 0; step <= 28; ++step) {
        const double price = step == 0 ? 0.0 : std::exp2(-4.0 - 0.5 * step) * 4000.0 / std::max(budget, 1.0);
        std::fill(used.begin(), used.end(), (uint8_t)0);
        std::vector<uint32_t> pick;
        double sum = 0.0;
        uint64_t left = table_bytes;
        while (pick.size() < F) {
            const uint64_t later = fill_bytes * (F - 1 - pick.size());   // the other tables are fill-ins at least
            int at = -1;
            double score = 0.0;
            for (uint32_t i = 0; i < slots.size(); ++i) {
                const Slot& s = slots[i];
                if (s.bytes + later > left) continue;
                const double x = s.value - price * s.rows;
                if (x <= score) continue;
                bool free = true;
                for (uint32_t j = 0; j < s.n; ++j) free = free && !used[parts[s.part[j]].f];
                if (free) {
                    at = (int)i;
                    score = x;
                }
            }
            if (at < 0) break;
            const Slot& s = slots[at];
            for (uint32_t j = 0; j < s.n; ++j) used[parts[s.part[j]].f] = 1;
            left -= s.bytes;
            sum += s.value;
            pick.push_back((uint32_t)at);
        }
        if (sum > best_value) {
            best_value = sum;
            best = pick;
            const uint64_t fills = fill_bytes * (F - pick.size());
            spare = left > fills ? left - fills : 0;
        }
    }
    std::stable_sort(best.begin(), best.end(), [&](uint32_t a, uint32_t b) { return slots[a].value > slots[b].value; });

    EsCascade C;
    std::vector<double> open = full;     // value still to come from each filter
    std::vector<uint8_t> settled(nf, 0);
    for (uint32_t i : best) {
        std::vector<EsPart> t;
        for (uint32_t j = 0; j < slots[i].n; ++j) {
            const EsPart& x = parts[slots[i].part[j]];
            t.push_back(x);
            open[x.f] = full[x.f] - x.value;
            if (x.d == P.q[x.f]) settled[x.f] = 1;
        }
        C.inner.push_back(t);
    }
    C.inner.resize(F);
    C.rate = std::exp(-std::max(best_value, 0.0));
    C.spare = spare;
    std::vector<uint32_t> order;
    for (uint32_t f = 0; f < nf; ++f)
        if (!settled[f]) order.push_back(f);
    std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return open[a] > open[b]; });
    for (uint32_t i = 0; i < ES_PRES; ++i) C.residue.push_back(i < order.size() ? (int)order[i] : -1);
    for (uint32_t i = ES_PRES; i < order.size(); ++i) C.tail.push_back(order[i]);
    return C;
}

namespace {

uint64_t xorshift(uint64_t& s) {
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    return s;
}

// The multiplier of an inner table: its rows are indexed by u n mod d, u coprime to d.  The lanes of a
// warp take consecutive rows of ring 3's digits, so their phases are, wraps apart, an arithmetic
// progression whose difference is an accident of the wheel: a difference with many factors of two
// puts all lanes on the same few banks, an odd one spreads them better than chance.  So the library
// tries multipliers on sampled warps and takes the one with the fewest wavefronts.  2^34 positions,
// without and with them:
// k = 384 2200 -> 1636 us, k = 390 1585 -> 1482, k = 379 1775 -> 1727, k = 300 1356 -> 1323.
constexpr uint32_t kSampleWarps = 8;

// b3 of the 32 lanes of a few warps (no short scan gains from this: none for blocks below 2^26).
std::vector<u128> sample_rows(const EsHostPlan& P, uint64_t R, uint64_t& seed) {
    std::vector<u128> b3;
    if (R < (1ull << 26)) return b3;
    for (uint32_t w = 0; w < kSampleWarps; ++w) {
        const uint64_t row0 = xorshift(seed) >> 24;
        for (uint32_t l = 0; l < 32; ++l) {
            uint64_t rem = row0 + l;
            u128 v = 0;
            for (size_t j = 3; j < P.radix.size(); ++j) {
                v += P.terms[P.roff[j] + rem % P.radix[j]];
                if (v >= P.M) v -= P.M;
                rem /= P.radix[j];
            }
            b3.push_back(v);
        }
    }
    return b3;
}

// reach: how far away the wrapped row may lie, where it is a row of its own.
uint32_t spread_of(const std::vector<u128>& b3, uint64_t& seed, uint32_t d, uint32_t corr, bool pair, uint32_t row_bytes,
                   uint32_t reach) {
    if (row_bytes > 16u || d < 8u || b3.empty()) return 1u;
    const uint32_t lanes = 128u / row_bytes;   // per wavefront at best; rows across all banks
    std::vector<uint32_t> res(b3.size()), shift(2 * kSampleWarps);   // shifts: the other rings' terms
    for (size_t i = 0; i < b3.size(); ++i) res[i] = es_mod(b3[i], d);
    for (uint32_t& x : shift) x = (uint32_t)(xorshift(seed) % d);
    uint32_t best = 1, least = ~0u;
    for (uint32_t t = 0; t < 64; ++t) {
        const uint32_t u = t == 0 ? 1u : (uint32_t)(xorshift(seed) % (d - 1u)) + 1u;
        if (gcd32(u, d) != 1u) continue;
        const uint32_t c = (uint32_t)((uint64_t)u * corr % d);
        if (!pair && t && std::min(c, d - c) > reach) continue;
        uint32_t cost = 0;
        for (uint32_t w = 0; w < kSampleWarps; ++w)
            for (uint32_t from = 0; from < 32; from += lanes) {
                uint32_t at[16][16], n[16] = {0}, most = 0;   // distinct rows by bank
                for (uint32_t l = from; l < from + lanes; ++l) {
                    const uint32_t x = (uint32_t)(((uint64_t)u * res[32 * w + l] + shift[2 * w]) % d) + shift[2 * w + 1];
                    const uint32_t bank = x % lanes;
                    bool seen = false;
                    for (uint32_t i = 0; i < n[bank]; ++i) seen = seen || at[bank][i] == x;
                    if (!seen) at[bank][n[bank]++] = x;
                    most = std::max(most, n[bank]);
                }
                cost += most;
            }
        if (cost < least) {
            least = cost;
            best = u;
        }
    }
    return best;
}

// Bytes the inner tables may take: what the CTA has left, and no more than staging them is worth.
// Every CTA copies them at launch, so a plan whose whole block is a short scan keeps them small.  One
// block alone, and 64 in one launch, with 12, 48 and 144 KB, us: 2^15.1 positions (k = 92) 20.7, 18.7, 19.2
// and 46, 39, 42; 2^17.2 (k = 124) 21.7, 20.4, 21.1 and 43, 39, 47; 2^20.8 (k = 112) 21.2, 20.8, 21.0 and 64, 65,
// 64; 2^22.4 (k = 152) 24.5, 23.7, 24.6 and 152, 137, 124; one block of 2^26.2 (k = 168) 34.5, 33.3, 31.4, of
// 2^28.0 (k = 176) 53.5, 43.3, 44.1, of 2^29.8 (k = 212) 125, 117, 97.  (So the lower line could lie at 2^21
// and the middle step matters little; single blocks hardly tell 12 from 144 KB below 2^25.)
uint32_t table_bytes(uint64_t R, size_t smem_bytes, size_t small_bytes) {
    const size_t left = smem_bytes > small_bytes ? smem_bytes - small_bytes : 0;
    const size_t want = R < (1ull << 22) ? 12u << 10 : (R < (1ull << 28) ? 48u << 10 : 144u << 10);
    return (uint32_t)std::min(left, want);
}

}  // namespace

// Tables of the production cascade with F inner tables (es_cascade.h, es_prod_kernel.cuh).
void es_prod_image(const EsHostPlan& P, const EsInst& geo, uint32_t F, uint32_t smem_bytes, EsProdImage& out,
                   double max_rate) {
    EsInst& I = out.inst;
    I = geo;
    const u128 M = P.M;
    const uint32_t r0 = I.r0, r1 = I.r1, r2 = I.r2, W = I.W, nf = I.n_filters, sh = I.sh;
    const uint32_t RS = es_row_words(W);
    const bool pair = es_pair_rows(W);
    const uint32_t stride = pair ? 2u * RS : RS, row_bytes = 4u * stride;   // words, bytes from phase to phase
    const uint32_t n_max = nf + F + ES_PRES;
    const uint32_t row1 = F <= 3 ? 16u : 32u, ds = F <= 4 ? 4u : 8u;   // ring-1 row bytes, step row words
    EsSmallBlock S;
    I.o_T1 = S.take(16ull * r1);
    I.o_R1 = S.take((size_t)row1 * (r1 + 1));   // + a padding row: digits are swept in pairs
    I.o_TQr = S.take(16ull * r1);
    I.o_T2 = S.take(16ull * r2);
    I.o_TQ2 = S.take(4ull * ds * r2);
    I.o_TQ2r = S.take(16ull * r2);
    I.o_S0 = S.take(16ull * r0);
    I.o_I0 = S.take(4ull * r0);
    I.o_Qr = S.take(16ull * r0);
    I.o_BK = S.take(4ull << ES_PBUCKET_LOG2);
    I.o_FC = S.take(sizeof(EsFilterC) * n_max);
    const EsCascade C = es_choose_cascade(P, F, row_bytes, pair, table_bytes(geo.n_outer * r0, smem_bytes, S.b.size()));

    out.rate = C.rate;
    if (C.rate > max_rate) return;

    // ---- entries: inner tables, residue stage, tail ----------------------------------------
    std::vector<EsCascadeEntry>& entries = out.entries;
    entries.clear();
    std::vector<uint32_t>& bits = out.bits;
    bits = P.allowed;
    const uint32_t ones = (uint32_t)bits.size();   // a bit table that passes both residues mod 2
    bits.push_back(0xffffffffu);
    std::vector<EsFilterC> fc;
    auto whole = [&](uint32_t f) {
        entries.push_back(EsCascadeEntry{P.q[f], {EsCascadeEntry::Part{f, P.q[f], 1u}}});
        fc.push_back(es_filter_consts(M, P.q[f], P.bit_off[f]));
    };
    auto fill = [&]() {
        entries.push_back(EsCascadeEntry{2u, {}});
        fc.push_back(es_filter_consts(M, 2u, ones));
    };
    uint64_t seed = 0x9e3779b97f4a7c15ull;
    const std::vector<u128> sample = sample_rows(P, geo.n_outer * r0, seed);
    // The tables' multipliers: a wrapped row no further than its distance with u = 1 or d / 4; where the
    // tables then exceed their room, also within the bytes that those before it leave.
    std::vector<uint32_t> mul(F, 1u);
    for (const bool within : {false, true}) {
        uint64_t s = seed;
        int64_t spare = (int64_t)C.spare;
        for (uint32_t i = 0; i < F; ++i) {
            if (C.inner[i].empty()) continue;
            uint32_t d = 1;
            for (const EsPart& p : C.inner[i]) d *= p.d;
            const uint32_t corr = (d - es_mod(M, d)) % d;
            auto bytes_of = [&](uint32_t c) { return (int64_t)es_align_up((uint64_t)c * row_bytes, 16); };
            const int64_t room = bytes_of(es_planned_rows(d, corr, pair)) + spare;
            uint32_t reach = std::max(std::min(corr, d - corr), d / 4u);
            if (within) reach = (uint32_t)std::min<uint64_t>(reach, (uint64_t)room / row_bytes - (2u * d - 1u));
            mul[i] = spread_of(sample, s, d, corr, pair, row_bytes, reach);
            spare = room - bytes_of(es_table_rows(d, (uint32_t)((uint64_t)corr * mul[i] % d), pair));
        }
        if (spare >= 0) break;
    }
    for (const std::vector<EsPart>& table : C.inner) {
        if (table.empty()) {
            I.tab_mul[entries.size()] = 1;
            fill();
            fc.back().off = 1;
            continue;
        }
        EsCascadeEntry e{1u, {}};
        for (const EsPart& p : table) e.q *= p.d;
        for (const EsPart& p : table) {
            // unit: the multiple of the other parts' moduli that is 1 mod d
            const uint32_t co = e.q / p.d;
            uint32_t u = co % p.d, k = 1;
            while (p.d > 1u && (uint64_t)u * k % p.d != 1u) ++k;
            e.parts.push_back(EsCascadeEntry::Part{p.f, p.d, p.d > 1u ? (uint32_t)((uint64_t)co * k % e.q) : 0u});
        }
        // residues are kept times the table's multiplier: limb weights (`off`, which has no use here, is
        // the lowest limb's), wrap correction and block constant
        EsFilterC c = es_filter_consts(M, e.q, 0);
        const uint32_t u = mul[entries.size()];
        I.tab_mul[entries.size()] = u;
        for (uint32_t* w : {&c.corr, &c.w1, &c.w2, &c.w3}) *w = (uint32_t)((uint64_t)*w * u % e.q);
        c.off = u;
        for (EsCascadeEntry::Part& p : e.parts) p.unit = (uint32_t)((uint64_t)p.unit * u % e.q);
        entries.push_back(e);
        fc.push_back(c);
    }
    for (int f : C.residue) {
        if (f < 0)
            fill();
        else
            whole((uint32_t)f);
    }
    for (uint32_t f : C.tail) whole(f);

    // ---- inner tables: rows of every unreduced phase and of the wrapped ones beside them ----
    const EsSortedRing R = es_sort_inner(P);
    std::vector<uint32_t>& tabs = out.tabs;
    tabs.clear();
    std::vector<uint32_t> phase;   // one row per phase mod d
    std::vector<uint8_t> adm, one;
    for (uint32_t i = 0; i < F; ++i) {
        const EsCascadeEntry& e = entries[i];
        const uint32_t d = e.q, corr = fc[i].corr, u = I.tab_mul[i];
        adm.assign(d, 1);
        for (const EsCascadeEntry::Part& p : e.parts) {
            const uint32_t q = P.q[p.f];
            es_project(P.allowed.data() + P.bit_off[p.f], q, p.d, one);
            for (uint32_t r = 0, m = 0; r < d; ++r) {
                adm[r] &= one[m];
                if (++m == p.d) m = 0;
            }
        }
        phase.assign((size_t)d * RS, 0u);
        for (uint32_t s = 0; s < r0; ++s) {
            const uint32_t a = es_mod(R.S0[s], d), wd = s >> 5, at = s & 31u;
            // phase ph is row u ph mod d
            for (uint32_t ph = 0, r = 0, m = a; ph < d; ++ph) {
                phase[(size_t)r * RS + wd] |= (uint32_t)adm[m] << at;
                if (++m == d) m = 0;
                r += u;
                if (r >= d) r -= d;
            }
        }
        const bool up = pair || corr <= d - corr;
        const uint32_t lead = up ? 0u : d - corr, rows = es_table_rows(d, corr, pair);
        const size_t at = tabs.size();
        I.tab_base[i] = 4u * (uint32_t)at + lead * row_bytes;
        I.tab_wrap[i] = pair ? (int32_t)(4u * RS) : up ? (int32_t)(corr * row_bytes) : -(int32_t)((d - corr) * row_bytes);
        tabs.resize(at + (size_t)rows * stride);
        uint32_t ph = lead ? d - lead : 0u, ph1 = corr;   // the first row's phase (lead <= d), its wrapped one
        if (ph == d) ph = 0;
        for (uint32_t r = 0; r < rows; ++r) {
            memcpy(&tabs[at + (size_t)r * stride], &phase[(size_t)ph * RS], 4u * RS);
            if (pair) memcpy(&tabs[at + (size_t)r * stride + RS], &phase[(size_t)ph1 * RS], 4u * RS);
            if (++ph == d) ph = 0;
            if (++ph1 == d) ph1 = 0;
        }
        while (tabs.size() % 4) tabs.push_back(0u);
    }

    // ---- carry-split buckets -----------------------------------------------------------------
    // Keys are the top 32 bits of values scaled to M's width (shifted up where M is below 2^32), and
    // t, the key of thr = M - b, is a difference of such keys: exact to within +-1.  Slot keys are
    // stored plus one, so that a slot is certainly below thr when its key is < t and certainly not
    // when it is > t + 2.  Entry of bucket [lo, hi] of t: the slots certainly below thr for every t
    // of the bucket, and above them the low bits of the one key that lies in it.
    constexpr uint32_t nb = 1u << ES_PBUCKET_LOG2, bsh = 32u - ES_PBUCKET_LOG2, ssh = ES_PBUCKET_LOG2;
    constexpr uint32_t flag = (1u << ssh) - 1u;
    const uint32_t lsh = sh ? 0u : 32u - es_bitlen(M);
    auto key_of = [&](u128 v) { return (uint32_t)(v >> sh) << lsh; };
    std::vector<uint64_t> key(r0);
    for (uint32_t i = 0; i < r0; ++i) key[i] = std::min<uint64_t>((uint64_t)key_of(R.S0[i]) + 1u, 0xffffffffull);
    for (uint32_t b = 0, n = 0; b < nb; ++b) {
        const uint64_t lo = (uint64_t)b << bsh, hi = lo + (1ull << bsh) - 1;
        while (n < r0 && key[n] < lo) ++n;
        uint32_t m = n;
        while (m < r0 && key[m] <= hi + 2) ++m;
        uint32_t v = flag;   // several keys, or too many slots to hold: found exactly
        if (n < flag && m == n)
            v = (uint32_t)((((1ull << bsh) - 1) << ssh) | n);
        else if (n < flag && m == n + 1 && key[n] <= hi)
            v = (uint32_t)(((key[n] - lo) << ssh) | n);
        S.put32(I.o_BK, b, v);
    }

    // ---- the rest of the small block ---------------------------------------------------------
    auto scaled = [&](u128 v, uint32_t f) {   // residue of an inner table, times its multiplier
        return (uint32_t)((uint64_t)es_mod(v, entries[f].q) * I.tab_mul[f] % entries[f].q);
    };
    for (uint32_t i = 0; i < r1; ++i) {
        const u128 v = P.terms[P.roff[1] + i];
        S.put128(I.o_T1, i, v);
        S.put32(I.o_R1 + row1 * i, 0, key_of(v));
        for (uint32_t f = 0; f < F; ++f) S.put32(I.o_R1 + row1 * i, 1 + f, row_bytes * scaled(v, f));
        for (uint32_t f = 0; f < ES_PRES; ++f) S.put32(I.o_TQr, 4 * i + f, es_mod(v, entries[F + f].q));
    }
    for (uint32_t i = 0; i < r2; ++i) {
        const u128 v = P.terms[P.roff[2] + i];
        S.put128(I.o_T2, i, v);
        for (uint32_t f = 0; f < F; ++f) S.put32(I.o_TQ2, i * ds + f, scaled(v, f));
        for (uint32_t f = 0; f < ES_PRES; ++f) S.put32(I.o_TQ2r, 4 * i + f, es_mod(v, entries[F + f].q));
    }
    for (uint32_t i = 0; i < r0; ++i) {
        S.put128(I.o_S0, i, R.S0[i]);
        S.put32(I.o_I0, i, R.digit[i]);
        for (uint32_t f = 0; f < ES_PRES; ++f) S.put32(I.o_Qr, 4 * i + f, es_mod(R.S0[i], entries[F + f].q));
    }
    memcpy(&S.b[I.o_FC], fc.data(), sizeof(EsFilterC) * fc.size());
    // ---- sums over groups of rings >= 3 --------------------------------------------------------
    // (two neighbouring groups hold more than ES_GROUP_SIZE sums between them and R < 2^62, so there
    // are far fewer than ES_MAX_GROUPS)
    out.sums.clear();
    I.n_groups = 0;
    for (uint32_t j = 3; j < I.n_rings;) {
        uint64_t size = 1;
        std::vector<u128> sum(1, 0);
        do {
            std::vector<u128> next;
            next.reserve(sum.size() * P.radix[j]);
            for (uint32_t d = 0; d < P.radix[j]; ++d)   // the group's first ring is the fastest digit
                for (const u128 v : sum) {
                    const u128 x = v + P.terms[P.roff[j] + d];
                    next.push_back(x >= M ? x - M : x);
                }
            sum.swap(next);
            size *= P.radix[j++];
        } while (j < I.n_rings && size * P.radix[j] <= ES_GROUP_SIZE);
        EsGroup& G = I.group[I.n_groups++];
        G.size = (uint32_t)size;
        G.magic = ~0ull / size;
        G.off = (uint32_t)out.sums.size();
        out.sums.insert(out.sums.end(), sum.begin(), sum.end());
    }
    I.n_filters = (uint32_t)entries.size();
    I.F = F;
    I.lsh = lsh;
    I.km = key_of(M);
    I.row_bytes = row_bytes;
    I.tab_words = (uint32_t)tabs.size();
    I.small_bytes = (uint32_t)S.b.size();
    out.small = std::move(S.b);
}
