// Big-box window kernel instantiations for box sizes: 108 112
#include "window_big.cuh"
FLCT_INSTANTIATE_WINDOW_BIG(27)
FLCT_INSTANTIATE_WINDOW_BIG(28)
