// Kernel instantiations: packed ViterbiFilter, 1793 to 2560 nodes (transitions in shared memory).
#include "msv_vit_fast.cuh"
MSVGB_INSTANTIATE_VITF(32) MSVGB_INSTANTIATE_VITF(36) MSVGB_INSTANTIATE_VITF(40)
