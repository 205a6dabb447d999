// window_big.cu -- the big-box kernel's dispatch over the box sides 68..128
// (the kernels themselves are compiled in win_big_*.cu).
#include "window_big.cuh"

namespace flct {

namespace {

struct BigEntry {
    cudaError_t (*launch)(const BigArgs&, int, cudaStream_t, bool);
    int (*bps)();
};
#define FLCT_BIG(M) {&launch_big<M>, &big_blocks_per_sm<M>}
const BigEntry kBig[] = {FLCT_BIG(17), FLCT_BIG(18), FLCT_BIG(19), FLCT_BIG(20), FLCT_BIG(21), FLCT_BIG(22),
                         FLCT_BIG(23), FLCT_BIG(24), FLCT_BIG(25), FLCT_BIG(26), FLCT_BIG(27), FLCT_BIG(28),
                         FLCT_BIG(29), FLCT_BIG(30), FLCT_BIG(31), FLCT_BIG(32)};
#undef FLCT_BIG

const BigEntry* find_big(int n) { return n % 4 == 0 && n >= 68 && n <= kMaxBigBox ? kBig + (n / 4 - 17) : nullptr; }

}  // namespace

cudaError_t launch_window_big(const BigArgs& a, int grid, cudaStream_t st, bool pdl) {
    const BigEntry* b = find_big(a.n);
    return b ? b->launch(a, grid, st, pdl) : cudaErrorInvalidValue;
}

int window_big_blocks_per_sm(int n) {
    const BigEntry* b = find_big(n);
    return b ? b->bps() : 0;
}

}  // namespace flct
