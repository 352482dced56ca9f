// Word-mask instances of the scan kernel for counting launches (per-stage pass counts): F in
// {0..6, 8}, inner rings of 1, 2, 3-4 or any words.
#include "es_scan_kernel.cuh"

namespace {

template <int WT>
ScanFn pick_wm(uint32_t f) {
    switch (f) {
        case 0: return es_scan_kernel<0, ES_LAYOUT_WORDMASK, true, WT>;
        case 1: return es_scan_kernel<1, ES_LAYOUT_WORDMASK, true, WT>;
        case 2: return es_scan_kernel<2, ES_LAYOUT_WORDMASK, true, WT>;
        case 3: return es_scan_kernel<3, ES_LAYOUT_WORDMASK, true, WT>;
        case 4: return es_scan_kernel<4, ES_LAYOUT_WORDMASK, true, WT>;
        case 5: return es_scan_kernel<5, ES_LAYOUT_WORDMASK, true, WT>;
        case 6: return es_scan_kernel<6, ES_LAYOUT_WORDMASK, true, WT>;
        default: return es_scan_kernel<8, ES_LAYOUT_WORDMASK, true, WT>;
    }
}

}  // namespace

ScanFn es_pick_wordmask(uint32_t words, uint32_t f) {
    if (words == 1) return pick_wm<1>(f);
    if (words == 2) return pick_wm<2>(f);
    if (words == 3 || words == 4) return pick_wm<4>(f);
    return pick_wm<0>(f);
}
