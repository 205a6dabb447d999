// Big-box window kernel instantiations for box sizes: 92 96
#include "window_big.cuh"
FLCT_INSTANTIATE_WINDOW_BIG(23)
FLCT_INSTANTIATE_WINDOW_BIG(24)
