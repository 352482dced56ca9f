// Production scan kernel instances: inner rings of two words.
#include "es_prod_kernel.cuh"

ScanFn es_pick_prod2(uint32_t tables) { return pick_prod<2>(tables); }
