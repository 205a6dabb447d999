// Big-box window kernel instantiations for box sizes: 100 104
#include "window_big.cuh"
FLCT_INSTANTIATE_WINDOW_BIG(25)
FLCT_INSTANTIATE_WINDOW_BIG(26)
