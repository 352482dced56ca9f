// Pair-table instances of the scan kernel (inner rings of one or two words), counting launches.
#include "es_scan_kernel.cuh"

namespace {

template <int WT>
ScanFn pick_pr(uint32_t f) {
    switch (f) {
        case 0: return es_scan_kernel<0, ES_LAYOUT_PAIR, true, WT>;
        case 1: return es_scan_kernel<1, ES_LAYOUT_PAIR, true, WT>;
        case 2: return es_scan_kernel<2, ES_LAYOUT_PAIR, true, WT>;
        case 3: return es_scan_kernel<3, ES_LAYOUT_PAIR, true, WT>;
        case 4: return es_scan_kernel<4, ES_LAYOUT_PAIR, true, WT>;
        case 5: return es_scan_kernel<5, ES_LAYOUT_PAIR, true, WT>;
        case 6: return es_scan_kernel<6, ES_LAYOUT_PAIR, true, WT>;
        default: return es_scan_kernel<8, ES_LAYOUT_PAIR, true, WT>;
    }
}

}  // namespace

// Only inner rings of exactly one or two words (every plan of the launch): anything else has no
// pair instance.
ScanFn es_pick_pair(uint32_t words, uint32_t f) {
    if (words == 1) return pick_pr<1>(f);
    if (words == 2) return pick_pr<2>(f);
    return nullptr;
}
