// global.cu -- kernels of the sigma <= 0 mode (see global.cuh).
#include "global.cuh"

#include "fft_reg.cuh"
#include "warp_math.cuh"

namespace flct {

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block sums of (a, b) in a fixed order: lanes, then warps.
__device__ __forceinline__ void block_sum2(double& a, double& b) {
    __shared__ double s[2][32];
    a = warp_sum_d(a);
    b = warp_sum_d(b);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if (lane == 0) {
        s[0][warp] = a;
        s[1][warp] = b;
    }
    __syncthreads();
    if (warp == 0) {
        a = lane < nw ? s[0][lane] : 0.;
        b = lane < nw ? s[1][lane] : 0.;
        a = warp_sum_d(a);
        b = warp_sum_d(b);
    }
}

__global__ void k_gsum_part(const double* __restrict__ f1, const double* __restrict__ f2, long n,
                            double* __restrict__ part) {
    grid_dep_wait();
    const long chunk = (n + gridDim.x - 1) / gridDim.x;
    const long b0 = blockIdx.x * chunk, b1 = min(n, b0 + chunk);
    double a = 0., b = 0.;
    for (long k = b0 + threadIdx.x; k < b1; k += blockDim.x) {
        a = __dadd_rn(a, f1[k]);
        b = __dadd_rn(b, f2[k]);
    }
    block_sum2(a, b);
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = a;
        part[2 * blockIdx.x + 1] = b;
    }
}

__global__ void k_gsum_final(const double* __restrict__ part, int nparts, double dn, double* __restrict__ means) {
    grid_dep_wait();
    double a = 0., b = 0.;
    for (int k = threadIdx.x; k < nparts; k += blockDim.x) {
        a = __dadd_rn(a, part[2 * k]);
        b = __dadd_rn(b, part[2 * k + 1]);
    }
    block_sum2(a, b);
    if (threadIdx.x == 0) {
        means[0] = a / dn;  // flct.c:833-834
        means[1] = b / dn;
    }
}

__global__ void k_gz(const double* __restrict__ f1, const double* __restrict__ f2, long n,
                     const double* __restrict__ means, float2* __restrict__ z, unsigned* maxbits,
                     unsigned* status) {
    grid_dep_wait();
    const float2 m1 = split_double_fast(means[0]), m2 = split_double_fast(means[1]);
    float mx1 = 0.f, mx2 = 0.f;
    for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x) {
        const double fa = f1[k], fb = f2[k];
        const float2 a = split_double_fast(fa), b = split_double_fast(fb);
        if (((__float_as_uint(a.x) & 0x7fffffffu) == 0x7f800000u && finite_d(fa)) ||
            ((__float_as_uint(b.x) & 0x7fffffffu) == 0x7f800000u && finite_d(fb)))
            atomicOr(status, kStatusRange);
        const float d1 = (a.x - m1.x) + (a.y - m1.y), d2 = (b.x - m2.x) + (b.y - m2.y);
        z[k] = make_float2(d1, d2);
        mx1 = fmaxf(mx1, fabsf(d1));
        mx2 = fmaxf(mx2, fabsf(d2));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
        mx2 = fmaxf(mx2, __shfl_xor_sync(0xffffffffu, mx2, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(maxbits, __float_as_uint(mx1));
        atomicMax(maxbits + 1, __float_as_uint(mx2));
    }
}

// Tile of a direct DFT: 2 TL LP lines by 256 / TL KQ frequencies, LP pairs of
// lines by KQ frequencies per thread, on packed FMAs (two lines an instruction).
// Every output adds its L terms from j = 0 up, the real part x.x w.x after
// -x.y w.y, so results do not depend on the tile.  Chunks of kDftChunk points
// of the lines and their twiddles tw[(j k) mod L] go through shared memory;
// a thread steps the index of its twiddle column.  Bound by the FP32 pipe (65%
// busy; 4 FMAs per point and output, 2 where only the real part is wanted).
// The four passes of a 1000 x 1200 call: 5.1 -> 0.83 ms against one output a
// thread, which read the table once per 4 FMAs.  Tiles of 8 lines for as few:
// 8 x 10007 3.31 -> 1.29 ms, 8 x 4096 0.42 -> 0.37; no gain below (8 x 1000
// 0.113 -> 0.127).
constexpr int kDftChunk = 16;

// Both frames' exact scales from their maxima.  Where one frame is zero both
// are: the correlation is zero, not what the other frame's rounding leaves of
// the separation.
__device__ __forceinline__ float2 frame_scales(const unsigned* scale) {
    if (!scale) return make_float2(1.f, 1.f);
    if (scale[0] == 0u || scale[1] == 0u) return make_float2(0.f, 0.f);
    return make_float2(pow2_scale(scale[0]), pow2_scale(scale[1]));
}

template <int DIR, int TL, int LP, int KQ, bool REAL_OUT>
__global__ void __launch_bounds__(256) k_dft_rows(const float2* __restrict__ in, float2* __restrict__ out, int L,
                                                  int lines, const float2* __restrict__ tw,
                                                  const unsigned* __restrict__ scale) {
    constexpr int J = kDftChunk, TK = 256 / TL, WL = 2 * TL * LP, WK = TK * KQ;
    __shared__ __align__(16) float xr[J][WL + 2], xi[J][WL + 2];
    __shared__ float2 ws[J][WK];
    grid_dep_wait();
    // a thread's outputs lie TK frequencies (2 TL lines) apart, so that a warp
    // reads whole rows of ws
    const int t = threadIdx.x, tk = t % TK, tl = 2 * (t / TK);
    const int k0 = blockIdx.x * WK, l0 = blockIdx.y * WL;
    const float2 c = frame_scales(scale);
    // this thread's twiddle column, from its row on
    constexpr int WR = 256 / WK;  // twiddle rows a round
    const int wk = t % WK, wj = t / WK, k = min(k0 + wk, L - 1);
    int idx = (int)((long)wj * k % L);
    const int step = (int)((long)WR * k % L);
    float2 ax[LP][KQ] = {}, ay[LP][KQ] = {};
    // the next chunk travels while this one is summed; half a warp reads 16
    // points of a line
    constexpr int NX = (WL * J + 255) / 256, NW = J / WR;
    const int jx = t % J, lx = t / J;
    float2 nx[NX], nw[NW];
    auto fetch = [&](int j0) {
#pragma unroll
        for (int q = 0; q < NX; ++q) {
            const int l = l0 + lx + q * (256 / J);
            nx[q] = (l < lines && j0 + jx < L) ? __ldg(in + (size_t)l * L + j0 + jx) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            nw[q] = __ldg(tw + idx);
            idx += step;
            if (idx >= L) idx -= L;
        }
    };
    fetch(0);
    for (int j0 = 0; j0 < L; j0 += J) {
        __syncthreads();
#pragma unroll
        for (int q = 0; q < NX; ++q) {
            if (WL * J < 256 && lx >= WL) break;
            xr[jx][lx + q * (256 / J)] = nx[q].x * c.x;
            xi[jx][lx + q * (256 / J)] = nx[q].y * c.y;
        }
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            ws[wj + q * WR][wk] = make_float2(nw[q].x, DIR > 0 ? -nw[q].y : nw[q].y);
        }
        __syncthreads();
        if (j0 + J < L) fetch(j0 + J);
        const int jn = min(J, L - j0);
#pragma unroll 4
        for (int j = 0; j < jn; ++j) {
            float2 re[LP], im[LP], ni[LP];
            float2 w[KQ];
#pragma unroll
            for (int p = 0; p < LP; ++p) {
                re[p] = *reinterpret_cast<const float2*>(&xr[j][tl + 2 * TL * p]);
                im[p] = *reinterpret_cast<const float2*>(&xi[j][tl + 2 * TL * p]);
                ni[p] = make_float2(-im[p].x, -im[p].y);
            }
#pragma unroll
            for (int q = 0; q < KQ; ++q) w[q] = ws[j][tk + TK * q];
#pragma unroll
            for (int p = 0; p < LP; ++p)
#pragma unroll
                for (int q = 0; q < KQ; ++q) {
                    const float2 wx = make_float2(w[q].x, w[q].x), wy = make_float2(w[q].y, w[q].y);
                    ax[p][q] = efma(re[p], wx, efma(ni[p], wy, ax[p][q]));
                    if (!REAL_OUT) ay[p][q] = efma(re[p], wy, efma(im[p], wx, ay[p][q]));
                }
        }
    }
#pragma unroll
    for (int p = 0; p < LP; ++p)
#pragma unroll
        for (int q = 0; q < KQ; ++q) {
            const int l = l0 + tl + 2 * TL * p, kk = k0 + tk + TK * q;
            if (kk >= L) continue;
            if (l < lines) out[(size_t)l * L + kk] = make_float2(ax[p][q].x, ay[p][q].x);
            if (l + 1 < lines) out[(size_t)(l + 1) * L + kk] = make_float2(ax[p][q].y, ay[p][q].y);
        }
}

// The same sums, one output a thread, for one to three lines so long that tiles
// of 64 frequencies would share SMs: there the twiddle reads bound both, and
// these keep more of them in flight.  1 x 10007 (whole call) 1.26 -> 0.91 ms,
// 3 x 10007 1.27 -> 0.91, 1 x 30000 10.6 -> 6.7; 2 x 30000, two rounds of
// blocks, would take 14.0 for the tiles' 10.6.
template <int DIR, bool REAL_OUT>
__global__ void __launch_bounds__(256) k_dft_long(const float2* __restrict__ in, float2* __restrict__ out, int L,
                                                  const float2* __restrict__ tw, const unsigned* __restrict__ scale) {
    constexpr int J = 2048;
    __shared__ float2 x[J];
    grid_dep_wait();
    const int k = blockIdx.x * 256 + threadIdx.x;
    const float2* const src = in + (size_t)blockIdx.y * L;
    const float2 c = frame_scales(scale);
    float ax = 0.f, ay = 0.f;
    int idx = 0;  // (j k) mod L
    for (int j0 = 0; j0 < L; j0 += J) {
        const int jn = min(J, L - j0);
        __syncthreads();
        for (int j = threadIdx.x; j < jn; j += 256) {
            const float2 v = src[j0 + j];
            x[j] = make_float2(v.x * c.x, v.y * c.y);
        }
        __syncthreads();
        if (k >= L) continue;
        for (int j = 0; j < jn; ++j) {
            float2 w = __ldg(tw + idx);
            if (DIR > 0) w.y = -w.y;
            const float2 v = x[j];
            ax = fmaf(v.x, w.x, fmaf(-v.y, w.y, ax));
            if (!REAL_OUT) ay = fmaf(v.x, w.y, fmaf(v.y, w.x, ay));
            idx += k;
            if (idx >= L) idx -= L;
        }
    }
    if (k < L) out[(size_t)blockIdx.y * L + k] = make_float2(ax, ay);
}

cudaError_t launch_dft_rows(bool inverse, bool real_out, const float2* in, float2* out, int L, int lines,
                            const float2* tw, const unsigned* scale, int nsm, cudaStream_t st) {
    // the widest tile that still gives every SM one, but none that is mostly
    // lines that are not there: up to 32 lines 32 x 32, up to 8 lines 8 x 64
    // once tiles of 32 x 16 would share SMs
    auto grid = [&](int wl, int wk) { return dim3((L + wk - 1) / wk, (lines + wl - 1) / wl); };
    auto tiles = [&](int wl, int wk) { return (long)grid(wl, wk).x * grid(wl, wk).y; };
    const bool few = lines <= 8 && tiles(32, 16) > nsm;
    const dim3 one((L + 255) / 256, lines);  // one output a thread: in one round of the SMs
    if (few && tiles(8, 64) > nsm && (long)one.x * one.y <= nsm) {
        auto* kern = !inverse ? k_dft_long<-1, false> : real_out ? k_dft_long<1, true> : k_dft_long<1, false>;
        return launch_kernel(kern, one, dim3(256), 0, st, true, in, out, L, tw, scale);
    }
    const bool wide = lines > 32 && tiles(64, 64) >= nsm, mid = tiles(32, 32) >= nsm;
#define FLCT_DFT(D, TL, LP, KQ, R)                                                                             \
    launch_kernel(k_dft_rows<D, TL, LP, KQ, R>, grid(2 * TL * LP, 256 / TL * KQ), dim3(256), 0, st, true, in, \
                  out, L, lines, tw, scale)
#define FLCT_DFT_TILE(D, R)             \
    (few    ? FLCT_DFT(D, 4, 1, 1, R)   \
     : wide ? FLCT_DFT(D, 16, 2, 4, R)  \
     : mid  ? FLCT_DFT(D, 16, 1, 2, R)  \
            : FLCT_DFT(D, 16, 1, 1, R))
    return !inverse ? FLCT_DFT_TILE(-1, false) : real_out ? FLCT_DFT_TILE(1, true) : FLCT_DFT_TILE(1, false);
#undef FLCT_DFT_TILE
#undef FLCT_DFT
}

// Twiddles e^{-2 pi i m / L} of both axes and the squared -k filter factors
// exp(-2 (k / (kr n / 2))^2) by frequency index (flct.c:1694-1715, applied to
// both spectra; 1 without -k).
__global__ void k_gtables(int nx, int ny, int use, double kr, float2* __restrict__ twx, float2* __restrict__ twy,
                          float* __restrict__ fx2, float* __restrict__ fy2) {
    grid_dep_wait();
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nx + ny) return;
    const int n = e < nx ? nx : ny, k = e < nx ? e : e - nx;
    const double a = 2.0 * 3.14159265358979323846 * (double)k / (double)n;
    double s, c;
    sincos(a, &s, &c);
    (e < nx ? twx : twy)[k] = make_float2((float)c, (float)-s);
    float f = 1.0f;
    if (use) {
        const double x = (double)freq_of(k, n) / (kr * (double)(n / 2));
        f = (float)exp(-2.0 * x * x);
    }
    (e < nx ? fx2 : fy2)[k] = f;
}

__global__ void k_transpose(const float2* __restrict__ in, float2* __restrict__ out, int R, int C) {
    grid_dep_wait();
    __shared__ float2 t[32][33];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int dy = threadIdx.y; dy < 32; dy += blockDim.y) {
        const int r = r0 + dy, c = c0 + threadIdx.x;
        if (r < R && c < C) t[dy][threadIdx.x] = in[(size_t)r * C + c];
    }
    __syncthreads();
    for (int dy = threadIdx.y; dy < 32; dy += blockDim.y) {
        const int c = c0 + dy, r = r0 + threadIdx.x;
        if (r < R && c < C) out[(size_t)c * R + r] = t[threadIdx.x][dy];
    }
}

__global__ void k_gprod(const float2* __restrict__ zt, float2* __restrict__ ct, int nx, int ny,
                        const float* __restrict__ fx2, const float* __restrict__ fy2) {
    grid_dep_wait();
    const long n = (long)nx * ny;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x) {
        const int ky = (int)(e / nx), kx = (int)(e - (long)ky * nx);
        const int my = ky ? ny - ky : 0, mx = kx ? nx - kx : 0;
        const float2 z = zt[e], zm = zt[(size_t)my * nx + mx];
        const float ax = z.x + zm.x, ay = z.y - zm.y;  // 2 A
        const float bx = z.y + zm.y, by = zm.x - z.x;  // 2 B
        const float f = fx2[kx] * fy2[ky];
        ct[e] = make_float2(f * (ax * bx + ay * by), f * (ax * by - ay * bx));
    }
}

__global__ void k_gpeak(const float2* __restrict__ c, int nx, int ny, unsigned long long* key) {
    grid_dep_wait();
    const long n = (long)nx * ny;
    unsigned long long best = 0ull;
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x) {
        const int i = (int)(e / ny), j = (int)(e - (long)i * ny);
        const float v = fabsf(c[e].x);
        if (v != v) continue;
        const int I = (i + nx / 2) % nx, J = (j + ny / 2) % ny;  // shift2d (flct.c:1510, 2111-2140)
        const unsigned long long kk =
            ((unsigned long long)__float_as_uint(v) << 32) | (0xffffffffu - (unsigned)(I * ny + J));
        best = kk > best ? kk : best;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
        best = other > best ? other : best;
    }
    if ((threadIdx.x & 31) == 0 && best) atomicMax(key, best);
}

__global__ void k_gpatch(const float2* __restrict__ c, int nx, int ny, const unsigned long long* __restrict__ key,
                         PeakRec* rec, PeakRecH* rech, int* work, int* nwork) {
    grid_dep_wait();
    // |c| at shifted coordinates (I, J)
    auto sh = [&](int I, int J) -> float {
        const int i = (I - nx / 2 + nx) % nx, j = (J - ny / 2 + ny) % ny;
        return fabsf(c[(size_t)i * ny + j].x);
    };
    __shared__ int s_I, s_J, s_have;
    if (threadIdx.x == 0) {
        int I, J;
        bool have;
        if (sh(0, 0) != sh(0, 0)) {  // a NaN first element stays the maximum (maxloc, flct.c:2142-2161)
            I = 0;
            J = 0;
            have = true;
        } else {
            const unsigned long long k = *key;
            const unsigned L = 0xffffffffu - (unsigned)(k & 0xffffffffull);
            have = __uint_as_float((unsigned)(k >> 32)) != 0.0f;
            I = have ? (int)(L / ny) : nx / 2;
            J = have ? (int)(L % ny) : ny / 2;
        }
        s_I = I;
        s_J = J;
        s_have = have;
        work[0] = 0;
        *nwork = 1;
    }
    __syncthreads();
    const int I = s_I, J = s_J;
    const bool have = s_have;
    if (rech) {
        for (int k = threadIdx.x; k < kHiresPatch * kHiresPatch; k += blockDim.x) {
            const int r = I - 2 + k / kHiresPatch, q = J - 2 + k % kHiresPatch;
            rech->v[k] = (r >= 0 && r < nx && q >= 0 && q < ny) ? sh(r, q) : 0.f;
        }
        if (threadIdx.x == 0) rech->meta = peak_meta(I, J, have);
    } else {
        const bool dofit = have && I > 0 && I < nx - 1 && J > 0 && J < ny - 1;
        if (threadIdx.x < 9) rec->v[threadIdx.x] = dofit ? sh(I - 1 + threadIdx.x / 3, J - 1 + threadIdx.x % 3) : 0.f;
        if (threadIdx.x == 0) rec->meta = peak_meta(I, J, dofit);
    }
}

}  // namespace flct
