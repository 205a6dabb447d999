// Big-box window kernel instantiations for box sizes: 116 120
#include "window_big.cuh"
FLCT_INSTANTIATE_WINDOW_BIG(29)
FLCT_INSTANTIATE_WINDOW_BIG(30)
