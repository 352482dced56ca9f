// The production cascade: how a launch that does not count filter stages tests the residual
// filters.  Which candidates pass does not depend on the order or the grouping of the tests, so
// the library chooses both itself, from the filters' moduli and admissible sets:
//
//  * An inner-stage table need not hold a whole filter.  For q = p^t the projection of the
//    admissible set to p^s (s < t) is a necessary condition with p^s phases instead of p^t, and
//    for the large primes of a plan nearly all of the rejection is in the lowest digit: at
//    k = 390, q = 223^2 passes 0.250 of the candidates and its projection to 223 passes 0.251,
//    with 223 phases instead of 49,729.
//  * Two or three coprime projections share one table (modulus d1 * d2): one lookup tests them
//    all.
//  * What a projection leaves open is tested exactly later, by the full filter.
//
// So the tables of any plan fit shared memory, with room for rows that save the residue
// reductions (see es_prod_kernel.cuh).
#pragma once
#include <stdint.h>

#include <string>
#include <vector>

#include "../../include/es_gb300.h"
#include "es_internal.h"

typedef unsigned __int128 es_u128;

// A plan as the host keeps it (es_plan_desc copied; rings padded to at least three).
struct EsHostPlan {
    uint32_t k = 0;
    es_u128 M = 1;
    std::vector<uint32_t> radix, roff;   // per ring: residues, first term
    std::vector<es_u128> terms;
    std::vector<uint32_t> q, bit_off;    // per filter: modulus, word offset of its bits
    std::vector<uint32_t> allowed;       // packed admissible-residue bits
};

// One condition: n mod d lies in the projection of filter f's admissible set to d (d divides q_f).
struct EsPart {
    uint32_t f, d;
    double value;    // -log(pass rate), given the wheel
};

// The chosen cascade: F inner tables (each a product of parts with coprime moduli; none for a
// table that fills the count and passes everything), ES_PRES residue-stage filters (f = -1: none),
// then the tail, every filter not settled by then, most selective first.
struct EsCascade {
    std::vector<std::vector<EsPart>> inner;
    std::vector<int> residue;
    std::vector<uint32_t> tail;
    double rate = 1.0;    // share of the candidates that pass the inner tables
    uint64_t spare = 0;   // bytes of table_bytes that the planned rows leave
};

// Inner rings of one word have the masks of a phase and of the phase a wrap past M selects side by
// side in one row: one 8-byte load instead of two 4-byte ones, for rows twice as long (but none
// beyond the 2 d - 1 unreduced phases).  Wider rings keep them apart, where the shorter tables let
// more projections share one: k = 390 (two words), 2^34 positions, 2004 us with pair rows and 1686
// without.
inline bool es_pair_rows(uint32_t W) { return W <= 1; }

// Rows of an inner table of modulus d whose wrap correction is corr: unreduced phases up to
// 2 d - 2 and, where the wrapped masks are rows of their own, the nearer of +corr and corr - d.
inline uint32_t es_table_rows(uint32_t d, uint32_t corr, bool pair) {
    const uint32_t ext = corr <= d - corr ? corr : d - corr;
    return 2u * d - 1u + (pair ? 0u : ext);
}

// The admissible set of a filter (packed bits of q residues) as bytes, projected to d | q.
void es_project(const uint32_t* bits, uint32_t q, uint32_t d, std::vector<uint8_t>& out);

// Packed residues 0 .. n-1 (whole words): those whose residue mod d is not in the filter's admissible set
// projected to d | q are cleared.
void es_and_periodic(const uint32_t* bits, uint32_t q, uint32_t d, uint32_t n, uint32_t* out);

// Rows kept for the table of modulus d when it is chosen, before its multiplier u is: the wrapped row
// then lies u corr away, at the nearer side.
inline uint32_t es_planned_rows(uint32_t d, uint32_t corr, bool pair) {
    return es_table_rows(d, corr > d / 4u ? corr : d / 4u, pair);
}

// Chooses F inner tables whose planned rows of row_bytes bytes, each table padded to 16 bytes, fit
// table_bytes in all.  Fill-ins count too; nothing but they can exceed table_bytes.
EsCascade es_choose_cascade(const EsHostPlan& P, uint32_t F, uint32_t row_bytes, bool pair, uint32_t table_bytes);

// An entry of a production cascade: the residue of n mod q is needed.  Its block constant follows
// from the caller's by CRT over the entry's parts (unit = 1 mod d of its own part, 0 mod the
// others).
struct EsCascadeEntry {
    struct Part {
        uint32_t f, d, unit;
    };
    uint32_t q;
    std::vector<Part> parts;   // none: a fill-in that passes everything
};

// The tables of a plan's production cascade, as the device gets them.
struct EsProdImage {
    EsInst inst{};
    double rate = 1.0;    // share of the candidates that pass the inner tables
    std::vector<unsigned char> small;
    std::vector<uint32_t> tabs, bits;
    std::vector<es_u128> sums;   // over the groups of rings >= 3
    std::vector<EsCascadeEntry> entries;
};

// The inner ring sorted by term: term and original digit of each slot.
struct EsSortedRing {
    std::vector<es_u128> S0;
    std::vector<uint32_t> digit;
};

inline uint32_t es_bitlen(es_u128 x) {
    uint32_t n = 0;
    while (x) { ++n; x >>= 1; }
    return n;
}
inline uint32_t es_mod(es_u128 x, uint32_t q) { return (uint32_t)(x % q); }
inline size_t es_align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }
// Words of a table row: the inner ring's words, padded to four for three-word rings so that one
// 16-byte load reads a row.
inline uint32_t es_row_words(uint32_t W) { return W == 3 ? 4u : W; }

// A byte image whose parts start on 16-byte boundaries.
struct EsSmallBlock {
    std::vector<unsigned char> b;
    uint32_t take(size_t bytes);
    void put128(uint32_t o, size_t i, es_u128 v);
    void put32(uint32_t o, size_t i, uint32_t v);
};

EsSortedRing es_sort_inner(const EsHostPlan& P);
es_u128 es_ring2_delta(const EsHostPlan& P, uint32_t i);   // step from ring-2 digit i to the next
EsFilterC es_filter_consts(es_u128 M, uint32_t q, uint32_t off);

// Descriptor checks that need no array contents, then the plan and its geometry; ES_OK or an error
// code with the reason.
int es_check_desc(const es_plan_desc& d, std::string& why);
int es_parse_plan(const es_plan_desc& d, EsHostPlan& P, EsInst& geo, std::string& why);

// The image of the production cascade with F inner tables; smem_bytes: shared memory for the small
// block and the inner tables together.  Where more than max_rate of the candidates would pass those
// tables, only out.rate is set.
void es_prod_image(const EsHostPlan& P, const EsInst& geo, uint32_t F, uint32_t smem_bytes, EsProdImage& out,
                   double max_rate = 1.0);
