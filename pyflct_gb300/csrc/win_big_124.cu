// Big-box window kernel instantiations for box sizes: 124 128
#include "window_big.cuh"
FLCT_INSTANTIATE_WINDOW_BIG(31)
FLCT_INSTANTIATE_WINDOW_BIG(32)
