// Big-box window kernel instantiations for box sizes: 68 72
#include "window_big.cuh"
FLCT_INSTANTIATE_WINDOW_BIG(17)
FLCT_INSTANTIATE_WINDOW_BIG(18)
