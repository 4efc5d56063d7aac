// Kernel instantiations: lane-group SSV pass with the mixed-width (16-bit and
// 8-bit) cost table; the four inst_hyb units split MSVGB_HYB_LIST's 8- and
// 16-lane entries (msv_hyb_list.h) between them so they compile in parallel.
#include <algorithm>
#include "msv_group.cuh"
MSVGB_INSTANTIATE_HYB(13, 8, 4) MSVGB_INSTANTIATE_HYB(17, 8, 4) MSVGB_INSTANTIATE_HYB(21, 8, 8)
MSVGB_INSTANTIATE_HYB(25, 8, 8) MSVGB_INSTANTIATE_HYB(29, 8, 8) MSVGB_INSTANTIATE_HYB(26, 8, 12)
MSVGB_INSTANTIATE_HYB(15, 16, 4) MSVGB_INSTANTIATE_HYB(19, 16, 4) MSVGB_INSTANTIATE_HYB(23, 16, 4)
MSVGB_INSTANTIATE_HYB(27, 16, 8) MSVGB_INSTANTIATE_HYB(31, 16, 8) MSVGB_INSTANTIATE_HYB(30, 8, 12)
MSVGB_INSTANTIATE_HYB(19, 16, 8) MSVGB_INSTANTIATE_HYB(23, 16, 8) MSVGB_INSTANTIATE_HYB(31, 16, 12)
