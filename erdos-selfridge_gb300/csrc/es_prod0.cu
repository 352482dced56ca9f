// Production scan kernel instances: inner rings of five or more words.
#include "es_prod_kernel.cuh"

ScanFn es_pick_prod0(uint32_t tables) { return pick_prod<0>(tables); }
