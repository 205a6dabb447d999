// window_big.cuh -- the window-correlation kernel for boxes above 64
// (sigma >= 16), FP32 form: box side n = 4 M, M = 17..32.
//
// Same contract as k_window_fp32 (source/flct.c:829-876, 1325-1532: window,
// transforms of both sub-images, conj(A) B times the optional squared
// filter, inverse, |c| in the half-shifted frame, first strict maximum,
// peak record).  One CTA owns one window, z = g1 + i g2 in shared memory.
//
// Four lanes share a line of length n: lane r holds the elements r + 4 j in
// registers, transforms them with a length-M register FFT (fft_reg.cuh),
// multiplies by e^{-2 pi i r k / n}, and the four combine by a radix-4
// butterfly over two lane exchanges: lane r ends with frequency k + M s,
// s = r bit-reversed, for every k, and stores it where element r + 4 k came
// from.  So spectra stay in that order ("position" 4 k + r) and the inverse
// runs the steps backwards; no pass moves data between lines.  The inverse
// takes half the lines: C is Hermitian, so the column pass runs for
// ky = 0..n/2 only (the real-imaged columns 0 and n/2 share one line), and
// the row pass makes two rows of the real correlation image at once.
//
// What bounds it: the shared-memory pipe (68% busy at side 84, lane exchanges
// and line loads and stores) and the barriers between passes (44% of issue
// slots used).  4,096 windows of side 84 take 245 us, 100 346 us, 128 508 us;
// summing n terms per output directly took 6.9, 13.6 and 20.5 ms, held to
// 92% of the shared-memory pipe by its table and line reads.  Its error
// against 64 bits is 4e-7 of the field where the direct sums had 2e-6.
#pragma once
#include "common.cuh"
#include "fft_reg.cuh"
#include "window_common.cuh"

namespace flct {

constexpr int kMaxBigBox = 128;  // largest box side of the big-box kernel

struct BigArgs {
    const float4* s12;    // both frames split per pixel (WinArgs::s12)
    const float4* means;  // per grid point at mean_slot(mg, i, j), or null: zero means
    MeanGrid mg;
    const int* work;
    const int* nwork;
    int nx, ny, nsize, n;
    int use_filter;
    int direct;           // windows given directly: box w starts at row w*n, unit weights
    PeakRec* peaks;
    PeakRecH* peaks_h;    // -h records instead (else null)
    const WinSeg* segs;   // batched launch (see WinArgs), else null
    const int* seg_start;
    int nseg;
    float2 tw[kMaxBigBox];             // e^{-2 pi i m / n}, m < n
    float gauss[2 * kMaxBigBox + 1];   // weight of offset d at d + n
    float filt2[kMaxBigBox];           // squared k-space filter by frequency index
};

template <int M>
struct BigShape {
    static constexpr int N = 4 * M, H = 2 * M;
    // row stride, 4 or 12 mod 16: four lines x four lanes of a half warp
    // touch 16 distinct 8-byte banks
    static constexpr int LD = N % 8 == 4 ? N : N + 4;
    static constexpr int THREADS = (4 * N + 31) / 32 * 32;  // a lane group of four per line
    static constexpr size_t smem =
        (size_t)N * LD * 8 + (size_t)N * 8 + (size_t)(3 * N + 1) * 4 + 8 * 4;
    // CTAs per SM the registers are held to: 4,096 windows of side 68 / 84 /
    // 96 took 194 / 243 / 291 us at 1, 161 / 243 / 303 at 2, 155 / 245 / 350
    // at 3 (above side 84 the line no longer fits the smaller share)
    static constexpr int MINB = M <= 18 ? 3 : M <= 21 ? 2 : 1;
};

// Frequency at spectrum position p = 4 k + r, and the position of -f.
template <int M>
__host__ __device__ constexpr int big_freq(int p) {
    const int r = p & 3;
    return (p >> 2) + M * ((r >> 1) | ((r & 1) << 1));
}
template <int M>
__host__ __device__ constexpr int big_mirror(int p) {
    const int k = p >> 2, r = p & 3;
    return k ? 4 * (M - k) + 3 - r : (r < 2 ? r : 5 - r);
}

// Lane r's share of a line: x[fft_in<M>(j)] = element r + 4 j in, frequency
// k + M s(r) in x[k] out.  The partners are X2 (r ^ 2) and X1 (r ^ 1) lanes
// away.
template <int M, int X2, int X1>
__device__ __forceinline__ void big_forward(float2 (&x)[M], int r, const float2* tw) {
    fft<M, 0, -1>(x);
    const float s2 = r & 2 ? -1.f : 1.f, s1 = r & 1 ? -1.f : 1.f;
    sfor<0, M>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        float2 y = x[k];
        if constexpr (k > 0) {
            const float2 w = tw[r * k];
            y = make_float2(y.x * w.x - y.y * w.y, y.x * w.y + y.y * w.x);
        }
        float2 p;
        p.x = __shfl_xor_sync(0xffffffffu, y.x, X2);
        p.y = __shfl_xor_sync(0xffffffffu, y.y, X2);
        y = cfma(y, s2, p);  // y_r + y_(r+2) | y_(r-2) - y_r
        if (r == 3) y = make_float2(y.y, -y.x);
        p.x = __shfl_xor_sync(0xffffffffu, y.x, X1);
        p.y = __shfl_xor_sync(0xffffffffu, y.y, X1);
        x[k] = cfma(y, s1, p);
    });
}

// The way back: x[k] = frequency k + M s(r) in, element r + 4 j in x[j] out
// (unnormalised).
template <int M, int X2, int X1>
__device__ __forceinline__ void big_inverse(float2 (&x)[M], int r, const float2* tw) {
    const float s2 = r & 2 ? -1.f : 1.f, s1 = r & 1 ? -1.f : 1.f;
    float2 u[M];
    sfor<0, M>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        float2 y = x[k], p;
        p.x = __shfl_xor_sync(0xffffffffu, y.x, X1);
        p.y = __shfl_xor_sync(0xffffffffu, y.y, X1);
        y = cfma(y, s1, p);
        if (r == 3) y = make_float2(-y.y, y.x);
        p.x = __shfl_xor_sync(0xffffffffu, y.x, X2);
        p.y = __shfl_xor_sync(0xffffffffu, y.y, X2);
        y = cfma(y, s2, p);
        if constexpr (k > 0) {
            const float2 w = tw[r * k];  // conjugate
            y = make_float2(y.x * w.x + y.y * w.y, y.y * w.x - y.x * w.y);
        }
        u[fft_in<M>(k)] = y;
    });
    fft<M, 0, +1>(u);
    sfor<0, M>([&](auto kc) { x[decltype(kc)::value] = u[decltype(kc)::value]; });
}

template <int M>
__global__ void __launch_bounds__(BigShape<M>::THREADS, BigShape<M>::MINB) k_window_big(BigArgs a) {
    using S = BigShape<M>;
    constexpr int N = S::N, H = S::H, LD = S::LD;
    extern __shared__ __align__(16) unsigned char sm[];
    float2* const z = reinterpret_cast<float2*>(sm);        // N x LD
    float2* const tw = z + N * LD;                          // N
    float* const s_g = reinterpret_cast<float*>(tw + N);    // weight of offset d at d + N
    float* const s_f = s_g + 2 * N + 1;                     // filter by position
    unsigned* const s_red = reinterpret_cast<unsigned*>(s_f + N);  // two windows' max f1, max f2, peak, index
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int k = t; k < N; k += S::THREADS) {
        tw[k] = a.tw[k];
        s_f[k] = a.use_filter ? a.filt2[big_freq<M>(k)] : 1.0f;
    }
    for (int k = t; k < 2 * N + 1; k += S::THREADS) s_g[k] = a.gauss[k];
    if (t < 8) s_red[t] = (t & 3) == 3 ? 0xffffffffu : 0u;
    grid_dep_wait();
    const int nwork = *a.nwork;
    __syncthreads();

    // lane groups of the column passes (eight neighbouring columns, so that
    // loads from the frames are whole 128-byte lines) and of the row passes.
    // Groups past the last line take part in the exchanges with the last
    // line's values (a line of their own warp, read before its owners store)
    // and store nothing.
    const int cr = ((lane >> 3) & 1) * 2 + (lane >> 4), cl = warp * 8 + (lane & 7);
    const int rr = lane & 3, rl = warp * 8 + (lane >> 2);

    for (int w = blockIdx.x, par = 0; w < nwork; w += gridDim.x, par ^= 1) {
        unsigned* const red = s_red + 4 * par;
        int gi = w;
        const float4* f12 = a.s12;
        int nx = a.nx, ny = a.ny;
        const float4* mp = a.means;
        MeanGrid mg = a.mg;
        if (a.nseg > 0) {
            const int k = seg_find(a.seg_start, a.nseg, gi);
            const WinSeg sg = a.segs[k];
            f12 = sg.s12;
            nx = sg.nx;
            ny = sg.ny.d;
            if (mp) mp += sg.base;
            mg = sg.mg;
            gi = sg.base + (gi - __ldg(a.seg_start + k));
        }
        const int pix = a.work[gi];
        int i, j, imin, jmin;
        if (a.direct) {
            imin = pix / ny;
            jmin = 0;
            i = imin;
            j = 0;
        } else {
            i = pix / ny;
            j = pix - i * ny;
            imin = box_start(i, nx, a.nsize);
            jmin = box_start(j, ny, a.nsize);
        }
        const float4 mm = (mp && !a.direct) ? __ldg(mp + mean_slot(mg, i, j)) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float2 mh = make_float2(mm.x, mm.y), ml = make_float2(mm.z, mm.w);  // (f1, f2) hi, lo

        float2 x[M];
        // forward, columns: windowed, mean-subtracted sub-images z = g1 + i g2
        float2 cs = make_float2(1.f, 1.f);
        for (bool scaled = false;; scaled = true) {
            const int col = min(cl, N - 1);
            const float wc = s_g[jmin - j + N + col];
            const float* gr = s_g + (imin - i + N + cr);
            const float4* src = f12 + (size_t)(imin + cr) * ny + jmin + col;
            float mx1 = 0.f, mx2 = 0.f;
            sfor<0, M>([&](auto jc) {
                constexpr int jj = decltype(jc)::value;
                const float4 v = __ldg(src + (size_t)(4 * jj) * ny);
                const float2 d = cadd(csub(make_float2(v.x, v.y), mh), csub(make_float2(v.z, v.w), ml));
                const float2 zz = cscale(d, wc * gr[4 * jj]);
                x[fft_in<M>(jj)] = emul(zz, cs);
                mx1 = fmaxf(mx1, fabsf(zz.x));
                mx2 = fmaxf(mx2, fabsf(zz.y));
            });
            if (!scaled) {
                const unsigned b1 = __reduce_max_sync(0xffffffffu, __float_as_uint(mx1));
                const unsigned b2 = __reduce_max_sync(0xffffffffu, __float_as_uint(mx2));
                if (lane == 0) {
                    atomicMax(red, b1);
                    atomicMax(red + 1, b2);
                }
            }
            big_forward<M, 8, 16>(x, cr, tw);
            if (cl < N) {
                sfor<0, M>([&](auto kc) {
                    constexpr int k = decltype(kc)::value;
                    z[(4 * k + cr) * LD + cl] = x[k];
                });
            }
            __syncthreads();
            // maxima within 2^+-40 of 1 need no scaling: every value of the
            // transforms then stays inside FP32's normal range; else the
            // columns are done again, each sub-image times an exact power of
            // two, or both times zero where one is zero (the correlation is)
            const unsigned b1 = red[0], b2 = red[1];
            auto near1 = [](unsigned b) { return (b >> 23) - 87u <= 80u; };
            if (scaled || (near1(b1) && near1(b2))) break;
            cs = b1 == 0u || b2 == 0u ? make_float2(0.f, 0.f) : make_float2(pow2_scale(b1), pow2_scale(b2));
            __syncthreads();  // every thread has read the maxima and its part of z
        }
        if (t < 4) s_red[4 * (par ^ 1) + t] = t == 3 ? 0xffffffffu : 0u;  // the next window's

        // forward, rows in place
        {
            float2* const row = z + min(rl, N - 1) * LD + rr;
            sfor<0, M>([&](auto jc) {
                constexpr int jj = decltype(jc)::value;
                x[fft_in<M>(jj)] = row[4 * jj];
            });
            big_forward<M, 2, 1>(x, rr, tw);
            if (rl < N) {
                sfor<0, M>([&](auto kc) {
                    constexpr int k = decltype(kc)::value;
                    row[4 * k] = x[k];
                });
            }
        }
        __syncthreads();

        // C = conj(A) B filt^2 with A, B separated from Z(k) and Z(-k), at
        // ky = 0..n/2: frequencies 0..n/2-1 sit at the even positions, n/2 at
        // position 1.  Columns 0 and n/2 merge into C[.][0] + i C[.][n/2] at
        // position 0 (their inverse images are real).
        {
            auto prod = [](float2 v, float2 vm, float f) {
                const float ax = v.x + vm.x, ay = v.y - vm.y;  // 2 s1 A
                const float bx = v.y + vm.y, by = vm.x - v.x;  // 2 s2 B
                return make_float2(f * (ax * bx + ay * by), f * (ax * by - ay * bx));
            };
            for (int e = t; e < N * (H - 1); e += S::THREADS) {
                const int pr = e / (H - 1), pc = 2 * (e - pr * (H - 1)) + 2;
                float2* const c = z + pr * LD + pc;
                *c = prod(*c, z[big_mirror<M>(pr) * LD + big_mirror<M>(pc)], s_f[pr] * s_f[pc]);
            }
            if (t < N) {
                const int mr = big_mirror<M>(t);
                if (t <= mr) {
                    float2 *const c = z + t * LD, *const cm = z + mr * LD;
                    const float2 c0 = prod(c[0], cm[0], s_f[t] * s_f[0]), ch = prod(c[1], cm[1], s_f[t] * s_f[1]);
                    c[0] = make_float2(c0.x - ch.y, c0.y + ch.x);
                    cm[0] = make_float2(c0.x + ch.y, ch.x - c0.y);
                }
            }
        }
        __syncthreads();

        // inverse, columns ky = 0..n/2-1 (even positions) in place: rows come
        // out in natural order
        if (warp * 8 < H) {
            float2* const col = z + 2 * min(cl, H - 1) + cr * LD;
            sfor<0, M>([&](auto kc) {
                constexpr int k = decltype(kc)::value;
                x[k] = col[4 * k * LD];
            });
            big_inverse<M, 8, 16>(x, cr, tw);
            if (cl < H) {
                sfor<0, M>([&](auto jc) {
                    constexpr int jj = decltype(jc)::value;
                    col[4 * jj * LD] = x[jj];
                });
            }
        }
        __syncthreads();

        // inverse, rows 2 a and 2 a + 1 as E = D[2a] + i D[2a+1], the upper
        // half from D's Hermitian rows; c[2a] + i c[2a+1] over row 2 a
        float mx = 0.f;
        if (warp * 8 < H) {
            float2* const r0 = z + 2 * min(rl, H - 1) * LD;
            const float sg = rr & 1 ? -1.f : 1.f;  // lanes 1 and 3 read conjugates from lanes 2 and 0
            const int off = rr & 1 ? 4 * M + (rr == 1 ? 2 : 0) : rr, step = rr & 1 ? -4 : 4;
            sfor<0, M>([&](auto kc) {
                constexpr int k = decltype(kc)::value;
                const int o = k ? off + step * k : (rr < 2 ? 0 : 2);
                const float2 v0 = r0[o], v1 = r0[LD + o];
                float2 e = make_float2(fmaf(-sg, v1.y, v0.x), fmaf(sg, v0.y, v1.x));
                if (k == 0 && rr < 2) e = rr ? make_float2(v0.y, v1.y) : make_float2(v0.x, v1.x);
                x[k] = e;
            });
            big_inverse<M, 2, 1>(x, rr, tw);
            if (rl < H) {
                sfor<0, M>([&](auto jc) {
                    constexpr int jj = decltype(jc)::value;
                    r0[rr + 4 * jj] = x[jj];
                    mx = fmaxf(mx, fmaxf(fabsf(x[jj].x), fabsf(x[jj].y)));
                });
            }
            const unsigned mw = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
            if (lane == 0) atomicMax(red + 2, mw);
        }
        __syncthreads();
        // first strict maximum of the sequential scan of |c| in the
        // half-shifted frame: the least row-major index that holds it
        const unsigned mb = red[2];
        if (mb != 0u && __float_as_uint(mx) == mb) {
            unsigned L = 0xffffffffu;
            const int I = (2 * rl + H) % N;  // n/2 is even: rows 2 a, 2 a + 1 stay neighbours
            sfor<0, M>([&](auto jc) {
                constexpr int jj = decltype(jc)::value;
                const int J = rr + 4 * jj < H ? rr + 4 * jj + H : rr + 4 * jj - H;
                if (__float_as_uint(fabsf(x[jj].x)) == mb) L = min(L, (unsigned)(I * N + J));
                if (__float_as_uint(fabsf(x[jj].y)) == mb) L = min(L, (unsigned)((I + 1) * N + J));
            });
            atomicMin(red + 3, L);
        }
        __syncthreads();
        auto shifted = [&](int r, int c) {
            const int i1 = r + H < N ? r + H : r - H, j1 = c + H < N ? c + H : c - H;
            const float2 v = z[(i1 & ~1) * LD + j1];
            return i1 & 1 ? v.y : v.x;
        };
        int I, J;
        bool have;
        const float v0 = shifted(0, 0);
        if (v0 != v0) {
            // a NaN first element stays the maximum of a sequential scan
            I = 0;
            J = 0;
            have = true;
        } else {
            const unsigned L = red[3];
            have = mb != 0u;
            I = have ? (int)(L / N) : H;
            J = have ? (int)(L % N) : H;
        }
        if (a.peaks_h) {
            if (t < kHiresPatch * kHiresPatch + 1) {
                float* rec = reinterpret_cast<float*>(a.peaks_h + gi);
                if (t < kHiresPatch * kHiresPatch) {
                    const int r = I - 2 + t / kHiresPatch, c = J - 2 + t % kHiresPatch;
                    rec[t] = (r >= 0 && r < N && c >= 0 && c < N) ? fabsf(shifted(r, c)) : 0.f;
                } else {
                    rec[t] = __uint_as_float(peak_meta(I, J, have));
                }
            }
        } else if (t < 10) {
            const bool dofit = have && I > 0 && I < N - 1 && J > 0 && J < N - 1;
            float* rec = reinterpret_cast<float*>(a.peaks + gi);
            if (t < 9)
                rec[t] = dofit ? fabsf(shifted(I - 1 + t / 3, J - 1 + t % 3)) : 0.f;
            else
                rec[9] = __uint_as_float(peak_meta(I, J, dofit));
        }
        __syncthreads();  // the record is read before the next window's columns are stored
    }
}

// Per box side n (a multiple of 4, 68..128): the kernel's launch and its CTAs
// per SM; null / 0 for other sides.  pdl: as a programmatic dependent.
template <int M>
cudaError_t launch_big(const BigArgs& a, int grid, cudaStream_t st, bool pdl);
template <int M>
int big_blocks_per_sm();

cudaError_t launch_window_big(const BigArgs& a, int grid, cudaStream_t st, bool pdl);
int window_big_blocks_per_sm(int n);

}  // namespace flct

#define FLCT_INSTANTIATE_WINDOW_BIG(M)                                                                       \
    namespace flct {                                                                                         \
    template <>                                                                                              \
    int big_blocks_per_sm<M>() {                                                                             \
        int nb = 0;                                                                                          \
        if (cudaFuncSetAttribute(k_window_big<M>, cudaFuncAttributeMaxDynamicSharedMemorySize,               \
                                 (int)BigShape<M>::smem) != cudaSuccess ||                                   \
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_window_big<M>, BigShape<M>::THREADS,        \
                                                          BigShape<M>::smem) != cudaSuccess)                 \
            return 0;                                                                                        \
        return nb;                                                                                           \
    }                                                                                                        \
    template <>                                                                                              \
    cudaError_t launch_big<M>(const BigArgs& a, int grid, cudaStream_t st, bool pdl) {                       \
        cudaError_t e = cudaFuncSetAttribute(k_window_big<M>, cudaFuncAttributeMaxDynamicSharedMemorySize,   \
                                             (int)BigShape<M>::smem);                                        \
        if (e != cudaSuccess) return e;                                                                      \
        return launch_kernel(k_window_big<M>, dim3(grid), dim3(BigShape<M>::THREADS), BigShape<M>::smem, st, \
                             pdl, a);                                                                        \
    }                                                                                                        \
    }
