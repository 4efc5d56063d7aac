// Kernel instantiations: packed ViterbiFilter, wide models (transitions in
// registers up to 16 words per lane, in shared memory above: 20 and up).
#include "msv_vit_fast.cuh"
MSVGB_INSTANTIATE_VITF(13) MSVGB_INSTANTIATE_VITF(14) MSVGB_INSTANTIATE_VITF(16)
MSVGB_INSTANTIATE_VITF(20) MSVGB_INSTANTIATE_VITF(24) MSVGB_INSTANTIATE_VITF(28)
