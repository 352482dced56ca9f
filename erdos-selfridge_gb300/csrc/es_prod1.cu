// Production scan kernel instances: inner rings of one word.
#include "es_prod_kernel.cuh"

ScanFn es_pick_prod1(uint32_t tables) { return pick_prod<1>(tables); }
