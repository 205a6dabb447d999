// Big-box window kernel instantiations for box sizes: 76 80
#include "window_big.cuh"
FLCT_INSTANTIATE_WINDOW_BIG(19)
FLCT_INSTANTIATE_WINDOW_BIG(20)
