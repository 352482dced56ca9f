// Production scan kernel instances: inner rings of three or four words.
#include "es_prod_kernel.cuh"

ScanFn es_pick_prod4(uint32_t tables) { return pick_prod<4>(tables); }
