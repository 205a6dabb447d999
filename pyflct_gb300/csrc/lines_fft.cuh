// lines_fft.cuh -- FP32 transforms of the lines of an array, any length up
// to kLineMax: the uniform shift (warp.c:757-881) and the spectrum of the
// non-uniform warp (warp.c:899-934).
//
// A line lives in shared memory and takes one pass per radix (2..16, chosen
// for the fewest passes), each thread's butterflies in registers between two
// barriers; lengths with a prime factor above 13 go through a chirp
// (X[k] = c[k] sum_j (x[j] c[j]) b[k - j], b = conj c, c[j] =
// e^{-i pi j^2 / L}), a convolution done by transforms of a smooth length
// M >= 2 L - 1.
//
// Kernels of a whole shift (shift_frac2d), against radix-2 passes at powers of
// two and O(L) circulant sums elsewhere: 256 x 256 40 us (was 52), 600 x 640
// 55 (429), 1024 x 1024 95 (131), 1009 x 1021 (chirps) 273 (1,019).  Bound by
// the latency of passes and launches at small sizes, by shared memory at large
// ones.  Errors against 64 bits fell from 1e-6 to 2e-7 of the image's norm.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace flct {

constexpr int kLineMax = 16384;  // longest transform (shared memory; 16 points per thread)

struct LinePlan {
    int L = 0;         // line length
    int M = 0;         // transform length: L, or the chirp convolution's
    int npass = 0;     // 0: no plan for this length
    unsigned long long radices = 0;  // a byte each, first pass lowest
    int T = 0;         // threads per line
    bool chirp = false;
};
// Lengths that need a chirp get a plan from chirp_min points on.
LinePlan line_plan(int L, int chirp_min);

// Tables of one axis on the device: tw[M] = e^{-2 pi i m / M}; chirp plans
// also c[L] and bhat[M] = transform of b, times 1 / M.  FP64, rounded once.
struct LineTab {
    float2* tw = nullptr;
    float2* c = nullptr;
    float2* bhat = nullptr;
};
size_t line_tab_bytes(const LinePlan& p);
LineTab line_tab(const LinePlan& p, void* mem);
// Fills both axes' tables in one launch (a second one where an axis has a
// chirp).  ph[k], where given, are the shift's phase factors for darg[k].
struct LineSetup {
    LinePlan p[2];
    LineTab t[2];
    double darg[2] = {};
    double2* ph[2] = {};
};
cudaError_t launch_line_setup(const LineSetup& a, cudaStream_t st);

// What a launch does to each line.
enum LineOp {
    kLineForward = 0,  // out = DFT (e^{-2 pi i j k / L})
    kLineShift = 1     // out = inverse DFT of (DFT times ph[k]), over L
};

// in: `lines` lines of L float2 (real_in: doubles, imaginary part 0), out the
// same as float2 (may not overlap in).
cudaError_t launch_lines(LineOp op, const LinePlan& p, const LineTab& t, const void* in, bool real_in, float2* out,
                         int lines, const double2* ph, int nsm, cudaStream_t st);

}  // namespace flct
