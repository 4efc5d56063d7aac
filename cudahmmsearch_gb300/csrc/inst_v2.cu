// Kernel instantiations: packed ViterbiFilter, eight warps per sequence (up to 8192 nodes).
#include "msv_vit_fast.cuh"
MSVGB_INSTANTIATE_VITF(9, 8) MSVGB_INSTANTIATE_VITF(10, 8) MSVGB_INSTANTIATE_VITF(12, 8) MSVGB_INSTANTIATE_VITF(14, 8)
MSVGB_INSTANTIATE_VITF(16, 8)
