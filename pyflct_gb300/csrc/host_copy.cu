// host_copy.cu -- see host_copy.cuh.
#include "host_copy.cuh"

#include <stdint.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>

namespace flct {

namespace {

struct CopyArgs {
    const double* src[3];
    double* dst[3];
    size_t n;
};

// Bound by the host link: its latency below some 100 KB, 150-165 GB/s above.
__global__ void __launch_bounds__(256) k_copy_arrays(CopyArgs a) {
    const double* __restrict__ s = blockIdx.y == 0 ? a.src[0] : blockIdx.y == 1 ? a.src[1] : a.src[2];
    double* __restrict__ d = blockIdx.y == 0 ? a.dst[0] : blockIdx.y == 1 ? a.dst[1] : a.dst[2];
    const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x, nt = (size_t)gridDim.x * blockDim.x;
    if (((reinterpret_cast<uintptr_t>(s) | reinterpret_cast<uintptr_t>(d)) & 15) == 0) {
        for (size_t k = t; k < a.n / 2; k += nt)
            reinterpret_cast<double2*>(d)[k] = reinterpret_cast<const double2*>(s)[k];
        if (t == 0 && (a.n & 1)) d[a.n - 1] = s[a.n - 1];
    } else {
        for (size_t k = t; k < a.n; k += nt) d[k] = s[k];
    }
}

// The kernel moves doubles: every array has to start on their boundary (a view
// into a file's bytes may not), which the runtime's copies do not ask for.  It
// also moves all arrays at once: results that share memory, where a later one
// is to stay, are left to copies one after another.
bool kernel_copies(const double* const* src, double* const* dst, int count, size_t n) {
    if (count > 3 || n * sizeof(double) > kHostKernelBytes) return false;
    uintptr_t any = 0;
    for (int k = 0; k < count; ++k) any |= reinterpret_cast<uintptr_t>(src[k]) | reinterpret_cast<uintptr_t>(dst[k]);
    for (int k = 1; k < count; ++k)
        for (int q = 0; q < k; ++q) {
            const uintptr_t a = reinterpret_cast<uintptr_t>(dst[k]), b = reinterpret_cast<uintptr_t>(dst[q]);
            if ((a < b ? b - a : a - b) < n * sizeof(double)) return false;
        }
    return any % alignof(double) == 0;
}

}  // namespace

cudaError_t copy_arrays(const double* const* src, double* const* dst, int count, size_t n, cudaMemcpyKind kind,
                        bool direct, cudaStream_t st) {
    const bool staged = kind == cudaMemcpyHostToDevice && count * n * sizeof(double) <= kHostStagedBytes;
    if (direct && !staged && kernel_copies(src, dst, count, n)) {
        CopyArgs a{};
        for (int k = 0; k < count; ++k) {
            a.src[k] = src[k];
            a.dst[k] = dst[k];
        }
        a.n = n;
        k_copy_arrays<<<dim3((unsigned)std::max<size_t>(1, std::min<size_t>((n / 2 + 255) / 256, 152)), count), 256, 0,
                        st>>>(a);
        return cudaGetLastError();
    }
    for (int k = 0; k < count; ++k) {
        cudaError_t e = cudaMemcpyAsync(dst[k], src[k], n * sizeof(double), kind, st);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

bool populate_output(void* p, size_t bytes) {
#ifdef MADV_POPULATE_WRITE
    const int advice = MADV_POPULATE_WRITE;
#else
    const int advice = 23;
#endif
    static const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
    if (bytes < page) {  // on two pages at most: cheaper to touch (a call of 24 x 24 62 against 66 us)
        volatile char* const c = static_cast<volatile char*>(p);
        for (size_t k : {(size_t)0, bytes - 1}) c[k] = c[k];
        return true;
    }
    const uintptr_t a = reinterpret_cast<uintptr_t>(p) & ~(page - 1);
    return madvise(reinterpret_cast<void*>(a), reinterpret_cast<uintptr_t>(p) + bytes - a, advice) == 0;
}

}  // namespace flct
