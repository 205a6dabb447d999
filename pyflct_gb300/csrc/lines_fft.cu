// lines_fft.cu -- transforms of an array's lines (see lines_fft.cuh).
#include "lines_fft.cuh"

#include <algorithm>

#include "common.cuh"
#include "fft_reg.cuh"
#include "warp_math.cuh"

namespace flct {

namespace {

constexpr double kRefPi = 3.1415926535898;  // warp.c:768

struct LineArgs {
    LinePlan p;
    LineTab t;
    const void* in;
    float2* out;
    const double2* ph;
    int lines, op, real_in, lpc;  // lpc: lines per CTA
};
struct LineArgs2 {
    LineArgs a[2];
};

// One unused place after 16: the first pass stores R apart.
__device__ __forceinline__ int lpad(int i) { return i + (i >> 4); }

// One radix-R pass of a length-n transform in place (p: product of the
// radices before): butterfly i takes the elements i + r n / R, times
// e^{-2 pi i r k / (p R)} (k = i mod p), and leaves its outputs where the
// next pass and finally natural order want them.
template <int R, int PTS>
__device__ __noinline__ void line_pass(float2* s, int n, int p, const float2* __restrict__ tw, int tid, int T) {
    constexpr int NB = (PTS + R - 1) / R;  // a thread's butterflies
    const int nb = n / R, ts = nb / p;
    const unsigned magic = p > 1 ? 0xffffffffu / (unsigned)p + 1u : 0u;  // i / p = umulhi(i, magic), i < 2^14
    float2 v[NB][R];
    sfor<0, NB>([&](auto bc) {
        constexpr int b = decltype(bc)::value;
        const int i = tid + b * T;
        if (i < nb) {
            const int k = p > 1 ? i - (int)__umulhi((unsigned)i, magic) * p : 0;
            sfor<0, R>([&](auto rc) {
                constexpr int r = decltype(rc)::value;
                float2 x = s[lpad(i + r * nb)];
                if constexpr (r > 0) {
                    if (p > 1) {
                        const float2 w = __ldg(tw + r * k * ts);
                        x = make_float2(x.x * w.x - x.y * w.y, x.x * w.y + x.y * w.x);
                    }
                }
                v[b][fft_in<R>(r)] = x;
            });
            fft<R, 0, -1>(v[b]);
        }
    });
    __syncthreads();
    sfor<0, NB>([&](auto bc) {
        constexpr int b = decltype(bc)::value;
        const int i = tid + b * T;
        if (i < nb) {
            const int q = p > 1 ? (int)__umulhi((unsigned)i, magic) * p : i;
            const int j = q * R + (i - q);
            sfor<0, R>([&](auto rc) {
                constexpr int r = decltype(rc)::value;
                s[lpad(j + r * p)] = v[b][fft_out<R>(r)];
            });
        }
    });
    __syncthreads();
}

template <int PTS>
__device__ __forceinline__ void line_fft(int M, int T, unsigned long long radices, float2* s, const float2* tw,
                                         int tid) {
    for (int p = 1; radices; radices >>= 8) {
        const int R = (int)(radices & 255u);
        switch (R) {
#define FLCT_PASS(R) \
    case R: line_pass<R, PTS>(s, M, p, tw, tid, T); break;
            FLCT_PASS(2) FLCT_PASS(3) FLCT_PASS(4) FLCT_PASS(5) FLCT_PASS(6) FLCT_PASS(7) FLCT_PASS(8)
            FLCT_PASS(9) FLCT_PASS(10) FLCT_PASS(11) FLCT_PASS(12) FLCT_PASS(13) FLCT_PASS(15) FLCT_PASS(16)
#undef FLCT_PASS
            default: break;
        }
        p *= R;
    }
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// Every line of the launch: load, transform, for the shift times the phase
// factors and back (the inverse as the forward transform on swapped re / im),
// store.  A CTA's lines share its barriers.
template <int PTS, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == 256 ? 3 : 1) k_lines(LineArgs2 two) {
    extern __shared__ float2 sm[];
    const LineArgs& a = two.a[blockIdx.y];
    const LinePlan P = a.p;
    grid_dep_wait();
    const int slot = threadIdx.x / P.T, tid = threadIdx.x - slot * P.T;
    const int L = P.L, M = P.M;
    // threads past the last whole team keep the barriers company
    const bool in_team = slot < a.lpc;
    float2* const s = sm + (size_t)(in_team ? slot : 0) * lpad(M);
    const int groups = (a.lines + a.lpc - 1) / a.lpc;
    const int me = in_team ? tid : M;  // idle threads have no points and no butterflies
    const int halves = P.chirp ? 2 : 1, ffts = halves * (a.op == kLineShift ? 2 : 1);
    for (int g = blockIdx.x; g < groups; g += gridDim.x) {
        const int line = g * a.lpc + slot;
        const bool act = in_team && line < a.lines;
        const size_t o = (size_t)line * L;
        for (int e = me; e < M; e += P.T) {
            float2 v = make_float2(0.f, 0.f);
            if (act && e < L) {
                if (a.real_in) v.x = (float)static_cast<const double*>(a.in)[o + e];
                else v = static_cast<const float2*>(a.in)[o + e];
                if (P.chirp) v = cmul(v, a.t.c[e]);
            }
            s[lpad(e)] = v;
        }
        __syncthreads();
        // one transform, or two around the chirp's product; twice for the shift
        for (int f = 0; f < ffts; ++f) {
            line_fft<PTS>(M, P.T, P.radices, s, a.t.tw, me);
            const bool inner = P.chirp && !(f & 1), last = f == ffts - 1;
            const float sc = 1.0f / (float)L;
            for (int e = me; e < (inner || (P.chirp && !last) ? M : L); e += P.T) {
                float2 v = s[lpad(e)];
                if (inner) {
                    v = cmul(v, a.t.bhat[e]);
                    s[lpad(e)] = make_float2(v.y, v.x);
                    continue;
                }
                if (P.chirp) v = e < L ? cmul(make_float2(v.y, v.x), a.t.c[e]) : make_float2(0.f, 0.f);
                if (last) {
                    if (act) a.out[o + e] = a.op == kLineForward ? v : make_float2(v.y * sc, v.x * sc);
                } else if (e < L) {
                    const double2 p = a.ph[e];
                    v = cmul(v, make_float2((float)p.x, (float)p.y));
                    v = make_float2(v.y, v.x);
                    s[lpad(e)] = P.chirp ? cmul(v, a.t.c[e]) : v;
                } else {
                    s[lpad(e)] = v;
                }
            }
            __syncthreads();
        }
    }
}

// Both axes' tables.  tw[m] = e^{-2 pi i m / M}; chirp plans: c[j] =
// e^{-i pi j^2 / L} and b = conj c around 0 modulo M, over M, in bhat + M
// (its transform goes to bhat); the shift's phase factors e^{2 pi i kf darg}
// with the reference's 2*pi*kf*darg (warp.c:818-829).
__global__ void __launch_bounds__(128) k_line_setup(LineSetup a) {
    grid_dep_wait();
    const LinePlan& p = blockIdx.y ? a.p[1] : a.p[0];
    const LineTab& t = blockIdx.y ? a.t[1] : a.t[0];
    double2* const ph = blockIdx.y ? a.ph[1] : a.ph[0];
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    double s, c;
    if (m < p.L && ph) {
        const double kf = (double)freq_of(m, p.L);
        sincos(2. * kRefPi * kf * (blockIdx.y ? a.darg[1] : a.darg[0]), &s, &c);
        ph[m] = make_double2(c, s);
    }
    if (m >= p.M) return;
    sincospi(2.0 * (double)m / (double)p.M, &s, &c);
    t.tw[m] = make_float2((float)c, (float)-s);
    if (!p.chirp) return;
    float2 b = make_float2(0.f, 0.f);
    const int j = m < p.L ? m : p.M - m;
    if (j < p.L) {
        const long long q = (long long)j * j % (2ll * p.L);
        sincospi((double)q / (double)p.L, &s, &c);
        if (m < p.L) t.c[m] = make_float2((float)c, (float)-s);
        b = make_float2((float)(c / p.M), (float)(s / p.M));
    }
    t.bhat[p.M + m] = b;
}

constexpr int kRadices[] = {16, 15, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2};

// The lengths up to kLineMax without a prime factor above 13 and the fewest
// passes of each, made once per process (20 us): a search at every call took
// 24 us for a length of many divisors and up to 1.1 ms for a chirp's length,
// more than its transforms.
struct Lengths {
    unsigned char passes[kLineMax + 1] = {};  // 0: a larger prime factor
    unsigned short smooth[1024];              // ascending
    int count = 0;
    Lengths() {
        for (int m = 1; m <= kLineMax; ++m) {
            if (m > 1 && !passes[m]) continue;
            if (count < 1024) smooth[count++] = (unsigned short)m;
            for (int r : kRadices)
                if (m * r <= kLineMax && (!passes[m * r] || passes[m * r] > passes[m] + 1))
                    passes[m * r] = (unsigned char)(passes[m] + 1);
        }
        passes[1] = 1;
    }
};
const Lengths& lengths() {
    static const Lengths t;
    return t;
}

// The radices of a length's fewest passes, a byte each, the largest first.
unsigned long long radices_of(int n) {
    const Lengths& t = lengths();
    unsigned long long out = 0;
    for (int shift = 0; n > 1; shift += 8)
        for (int r : kRadices)
            if (n % r == 0 && (n == r ? 0 : t.passes[n / r]) == t.passes[n] - 1) {
                out |= (unsigned long long)r << shift;
                n /= r;
                break;
            }
    return out;
}

// Points a thread carries through a pass: 8 while a line's threads fit a CTA.
int line_pts(const LinePlan& p) { return p.M <= 8192 ? 8 : 16; }

cudaError_t launch_lines2(const LineArgs2& a, int axes, int nsm, cudaStream_t st) {
    size_t smem = 0;
    int groups = 1, threads = 256, pts = 8;
    for (int k = 0; k < axes; ++k) {
        const LineArgs& x = a.a[k];
        smem = std::max(smem, (size_t)x.lpc * (x.p.M + x.p.M / 16) * sizeof(float2));
        groups = std::max(groups, (x.lines + x.lpc - 1) / x.lpc);
        threads = std::max(threads, (x.p.T * x.lpc + 31) / 32 * 32);
        pts = std::max(pts, line_pts(x.p));
    }
    void (*kern)(LineArgs2) = pts == 16 ? k_lines<16, 1024> : threads > 256 ? k_lines<8, 1024> : k_lines<8, 256>;
    // the limit is the kernel's, shared by every context and thread: always
    // what its longest line takes (256 threads carry 2048 points: 17 KB)
    if (pts == 16 || threads > 256) {
        const int most = pts == 16 ? kLineMax : 8192;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)((most + most / 16) * sizeof(float2)));
        if (e != cudaSuccess) return e;
    }
    return launch_kernel(kern, dim3(std::min(groups, nsm * 16), axes), dim3(threads), smem, st, true, a);
}

}  // namespace

LinePlan line_plan(int L, int chirp_min) {
    LinePlan p;
    p.L = L;
    if (L < 1) return p;
    const Lengths& t = lengths();
    if (L <= kLineMax && t.passes[L]) {
        p.M = L;
    } else if (L < chirp_min || 2 * (long)L - 1 > kLineMax) {
        return p;
    } else {
        // chirp length: the smooth one of least work, up to the next power of two
        long best = -1;
        for (const unsigned short* m = std::lower_bound(t.smooth, t.smooth + t.count, 2 * L - 1);
             m < t.smooth + t.count; ++m) {
            const long work = (long)*m * (t.passes[*m] + 1);
            if (best < 0 || work < best) {
                best = work;
                p.M = *m;
            }
            if ((*m & (*m - 1)) == 0) break;
        }
        p.chirp = true;
    }
    p.npass = t.passes[p.M];
    p.radices = radices_of(p.M);
    p.T = (p.M + line_pts(p) - 1) / line_pts(p);
    return p;
}

size_t line_tab_bytes(const LinePlan& p) {
    return ((size_t)p.M + (p.chirp ? p.L + 2 * (size_t)p.M : 0)) * sizeof(float2) + 256;
}

LineTab line_tab(const LinePlan& p, void* mem) {
    LineTab t;
    t.tw = static_cast<float2*>(mem);
    if (p.chirp) {
        t.c = t.tw + p.M;
        t.bhat = t.c + p.L;
    }
    return t;
}

cudaError_t launch_line_setup(const LineSetup& a, cudaStream_t st) {
    int n = 1;
    LineArgs2 two{};
    int chirps = 0;
    for (int k = 0; k < 2; ++k) {
        const LinePlan& p = a.p[k];
        n = std::max(n, std::max(p.L, p.M));
        if (!p.chirp) continue;
        LineArgs& x = two.a[chirps++];
        x.p = p;
        x.p.L = p.M;
        x.p.chirp = false;
        x.t.tw = a.t[k].tw;
        x.in = a.t[k].bhat + p.M;
        x.out = a.t[k].bhat;
        x.lines = x.lpc = 1;
        x.op = kLineForward;
    }
    cudaError_t e = launch_kernel(k_line_setup, dim3((n + 127) / 128, 2), dim3(128), 0, st, true, a);
    return e == cudaSuccess && chirps ? launch_lines2(two, chirps, 1, st) : e;
}

cudaError_t launch_lines(LineOp op, const LinePlan& p, const LineTab& t, const void* in, bool real_in, float2* out,
                         int lines, const double2* ph, int nsm, cudaStream_t st) {
    // lines share a CTA of 256 threads, but not so that SMs stay without one
    const int lpc = std::max(1, std::min(256 / p.T, lines / nsm));
    LineArgs2 a{};
    a.a[0] = LineArgs{p, t, in, out, ph, lines, (int)op, real_in ? 1 : 0, lpc};
    return launch_lines2(a, 1, nsm, st);
}

}  // namespace flct
