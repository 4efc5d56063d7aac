// Kernel instantiations: lane-group SSV pass with the mixed-width (16-bit and
// 8-bit) cost table; the four inst_hyb units split MSVGB_HYB_LIST's 8- and
// 16-lane entries (msv_hyb_list.h) between them so they compile in parallel.
#include <algorithm>
#include "msv_group.cuh"
MSVGB_INSTANTIATE_HYB(12, 8, 4) MSVGB_INSTANTIATE_HYB(16, 8, 4) MSVGB_INSTANTIATE_HYB(20, 8, 8)
MSVGB_INSTANTIATE_HYB(24, 8, 8) MSVGB_INSTANTIATE_HYB(28, 8, 8) MSVGB_INSTANTIATE_HYB(32, 8, 8)
MSVGB_INSTANTIATE_HYB(14, 16, 4) MSVGB_INSTANTIATE_HYB(18, 16, 4) MSVGB_INSTANTIATE_HYB(22, 16, 4)
MSVGB_INSTANTIATE_HYB(26, 16, 8) MSVGB_INSTANTIATE_HYB(30, 16, 8) MSVGB_INSTANTIATE_HYB(29, 8, 12)
MSVGB_INSTANTIATE_HYB(18, 16, 8) MSVGB_INSTANTIATE_HYB(22, 16, 8) MSVGB_INSTANTIATE_HYB(30, 16, 12)
