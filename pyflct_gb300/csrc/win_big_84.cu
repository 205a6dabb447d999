// Big-box window kernel instantiations for box sizes: 84 88
#include "window_big.cuh"
FLCT_INSTANTIATE_WINDOW_BIG(21)
FLCT_INSTANTIATE_WINDOW_BIG(22)
