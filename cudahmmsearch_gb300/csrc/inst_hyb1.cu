// Kernel instantiations: lane-group SSV pass with the mixed-width (16-bit and
// 8-bit) cost table; the four inst_hyb units split MSVGB_HYB_LIST's 8- and
// 16-lane entries (msv_hyb_list.h) between them so they compile in parallel.
#include <algorithm>
#include "msv_group.cuh"
MSVGB_INSTANTIATE_HYB(11, 8, 4) MSVGB_INSTANTIATE_HYB(15, 8, 4) MSVGB_INSTANTIATE_HYB(19, 8, 8)
MSVGB_INSTANTIATE_HYB(23, 8, 8) MSVGB_INSTANTIATE_HYB(27, 8, 8) MSVGB_INSTANTIATE_HYB(31, 8, 8)
MSVGB_INSTANTIATE_HYB(13, 16, 4) MSVGB_INSTANTIATE_HYB(17, 16, 4) MSVGB_INSTANTIATE_HYB(21, 16, 4)
MSVGB_INSTANTIATE_HYB(25, 16, 8) MSVGB_INSTANTIATE_HYB(29, 16, 8) MSVGB_INSTANTIATE_HYB(28, 8, 12)
MSVGB_INSTANTIATE_HYB(32, 8, 12) MSVGB_INSTANTIATE_HYB(21, 16, 8) MSVGB_INSTANTIATE_HYB(29, 16, 12)
