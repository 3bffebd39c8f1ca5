// Exponent range of FP64 grids, for choosing the arithmetic of an FP64
// program: float pairs (df32) hold a value to 2^-48 of itself only between
// 2^-74 and 2^128, so a program runs df32 only when the largest magnitude,
// grown by (sum |c|)^T, stays well below 2^128 and the smallest nonzero
// magnitude well above 2^-74 (pair_range).  Both kernels fold the biased
// exponent fields with integer max and min.
//   k_run_scan        the cells a run reads (a's domain, both grids' shells); its
//                     verdict stays on the device, for the run's own kernels
//   k_exponent_range  a grid's whole span (padding included) as 64-bit words, for
//                     the host's choice: batches, temporal fusion, term-by-term 3D
//                     boxes of radius 2-3 from 8 sweeps on, and calls without
//                     scratch (one atomicMax and one atomicMin per warp)
// and k_shell_copy fills the shells of a run's copies.
#include "df32.cuh"
#include "resident.h"
#include "uhs_kernels.h"

namespace uhs {
namespace {

__global__ void __launch_bounds__(256) k_exponent_range(const unsigned long long *w, int64_t n, unsigned *max_out,
                                                        unsigned *min_out) {
    unsigned hi = 0u, lo = 0x7ffu;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const unsigned long long v = w[i];
        const unsigned e = static_cast<unsigned>(v >> 52) & 0x7ffu;
        hi = max(hi, e);
        if (v << 1) lo = min(lo, e);  // nonzero magnitude (the sign bit shifted out)
    }
    for (int o = 16; o > 0; o >>= 1) {
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(max_out, hi);
        atomicMin(min_out, lo);
    }
}

// Cells of a box that lie outside its inner domain (n0 x n1 x n2, reach r on
// each axis), counted along: planes before and after, then rows, then columns.
// Coordinates are relative to the domain.
struct Shell {
    int n0, n1, n2, r0, r1, r2;
    __host__ __device__ int64_t planes() const { return 2ll * r0 * (n1 + 2 * r1) * (n2 + 2 * r2); }
    __host__ __device__ int64_t rows() const { return 2ll * n0 * r1 * (n2 + 2 * r2); }
    __host__ __device__ int64_t cells() const { return planes() + rows() + 2ll * n0 * n1 * r2; }
    __device__ void at(int64_t i, int &z, int &y, int &x) const {
        const int w = n2 + 2 * r2, h = n1 + 2 * r1;
        if (i < planes()) {
            const int64_t row = i / w;
            const int p = static_cast<int>(row / h);
            x = static_cast<int>(i - row * w) - r2;
            y = static_cast<int>(row - static_cast<int64_t>(p) * h) - r1;
            z = p < r0 ? p - r0 : n0 + p - r0;
        } else if ((i -= planes()) < rows()) {
            const int64_t row = i / w;
            const int k = static_cast<int>(row % (2 * r1));
            x = static_cast<int>(i - row * w) - r2;
            y = k < r1 ? k - r1 : n1 + k - r1;
            z = static_cast<int>(row / (2 * r1));
        } else {
            i -= rows();
            const int64_t row = i / (2 * r2);
            const int k = static_cast<int>(i - row * 2 * r2);
            x = k < r2 ? k - r2 : n2 + k - r2;
            z = static_cast<int>(row / n1);
            y = static_cast<int>(row - static_cast<int64_t>(z) * n1);
        }
    }
};

struct RunScan {
    const double *a, *b;             // domain cell (0, 0, 0) of each grid; b NULL: not read
    int64_t as0, as1, bs0, bs1;
    Shell sh;
    double growth;
    unsigned *ctl;  // tickets, unused, largest exponent, largest 0x800 - exponent; zero between launches
    PairRun *run;
};

__device__ __forceinline__ void fold_exponent(double v, unsigned &hi, unsigned &lo) {
    const unsigned h = static_cast<unsigned>(__double2hiint(v)), e = (h >> 20) & 0x7ffu;
    hi = max(hi, e);
    if ((h << 1) | static_cast<unsigned>(__double2loint(v))) lo = max(lo, 0x800u - e);
}

// The cells an FP64 run reads -- a's domain and both grids' shells -- folded
// into the verdict that its kernels follow (pair_range): one read of a, no
// host round trip.  One warp per row; HBM-bound at large sizes.
__global__ void __launch_bounds__(256) k_run_scan(const RunScan s) {
    unsigned hi = 0u, lo = 0u;
    const int lane = threadIdx.x & 31;
    const int64_t rows = static_cast<int64_t>(s.sh.n0) * s.sh.n1;
    for (int64_t row = blockIdx.x * 8ll + (threadIdx.x >> 5); row < rows; row += gridDim.x * 8ll) {
        const int64_t z = row / s.sh.n1, y = row - z * s.sh.n1;
        const double *p = s.a + z * s.as0 + y * s.as1;
#pragma unroll 8
        for (int x = lane; x < s.sh.n2; x += 32) fold_exponent(p[x], hi, lo);
    }
    const int64_t n = s.sh.cells();
    for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < n; i += gridDim.x * 256ll) {
        int z, y, x;
        s.sh.at(i, z, y, x);
        fold_exponent(s.a[z * s.as0 + y * s.as1 + x], hi, lo);
        if (s.b) fold_exponent(s.b[z * s.bs0 + y * s.bs1 + x], hi, lo);
    }
    for (int o = 16; o > 0; o >>= 1) {
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        lo = max(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    }
    __shared__ unsigned sh_hi, sh_lo;
    if (threadIdx.x == 0) sh_hi = sh_lo = 0u;
    __syncthreads();
    if (lane == 0) {
        atomicMax(&sh_hi, hi);
        atomicMax(&sh_lo, lo);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicMax(s.ctl + 2, sh_hi);
        atomicMax(s.ctl + 3, sh_lo);
        __threadfence();
        if (atomicAdd(s.ctl, 1u) == gridDim.x - 1) {  // the last block
            __threadfence();
            const unsigned h = *reinterpret_cast<volatile unsigned *>(s.ctl + 2),
                           l = *reinterpret_cast<volatile unsigned *>(s.ctl + 3);
            const PairRange pr = pair_range(static_cast<int>(h), l ? static_cast<int>(0x800u - l) : -1, s.growth);
            s.run->state = pr.ok ? kRunPairs : kRunNative;
            s.run->bias = pair_bias(pr.shift);
            s.ctl[0] = s.ctl[2] = s.ctl[3] = 0u;
        }
    }
}

// Both grids' shells copied into a run's own copies: FP64 split into pairs
// (by the run's verdict), or 4-byte cells as they are.
struct ShellCopy {
    const void *src[2];
    void *dst[2];
    int64_t ss0[2], ss1[2], ds0, ds1;
    Shell sh;
    const PairRun *run;
};
template <bool F64>
__global__ void __launch_bounds__(256) k_shell_copy(const ShellCopy c) {
    const int g = blockIdx.y;
    int bias = 0;
    if constexpr (F64) {
        if (c.run->state != kRunPairs) return;
        bias = c.run->bias;
    }
    const int64_t n = c.sh.cells();
    unsigned range_err = 0u;  // (the scan has bounded every cell)
    for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < n; i += gridDim.x * 256ll) {
        int z, y, x;
        c.sh.at(i, z, y, x);
        const int64_t s = z * c.ss0[g] + y * c.ss1[g] + x, d = z * c.ds0 + y * c.ds1 + x;
        if constexpr (F64)
            static_cast<float2 *>(c.dst[g])[d] = split_f64(static_cast<const double *>(c.src[g])[s], range_err, bias);
        else
            static_cast<float *>(c.dst[g])[d] = static_cast<const float *>(c.src[g])[s];
    }
}

Shell shell_of(const int64_t lb[3], const int64_t ub[3], const int reach[3]) {
    return Shell{static_cast<int>(ub[0] - lb[0]), static_cast<int>(ub[1] - lb[1]), static_cast<int>(ub[2] - lb[2]),
                 reach[0], reach[1], reach[2]};
}
template <class T>
T *domain_origin(const GridView &g, const int64_t lb[3]) {
    return static_cast<T *>(g.data) + lb[0] * g.s[0] + lb[1] * g.s[1] + lb[2];
}

}  // namespace

cudaError_t launch_exponent_range(const void *data, int64_t n_words, unsigned *max_out, unsigned *min_out, int sms,
                                  cudaStream_t st) {
    if (n_words <= 0) return cudaSuccess;
    const int64_t blocks = std::min<int64_t>((n_words + 255) / 256, static_cast<int64_t>(sms) * 8);
    k_exponent_range<<<static_cast<unsigned>(blocks), 256, 0, st>>>(static_cast<const unsigned long long *>(data),
                                                                     n_words, max_out, min_out);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_run_scan(const GridView &a, const GridView *b, const int64_t lb[3], const int64_t ub[3],
                            const int reach[3], double growth, unsigned *ctl, PairRun *run, cudaStream_t st) {
    RunScan s{domain_origin<const double>(a, lb), b ? domain_origin<const double>(*b, lb) : nullptr, a.s[0], a.s[1],
              b ? b->s[0] : 0, b ? b->s[1] : 0, shell_of(lb, ub, reach), growth, ctl, run};
    const int64_t rows = static_cast<int64_t>(s.sh.n0) * s.sh.n1, want = (rows + 7) / 8;
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>(want, device_sm_count() * 8ll));
    k_run_scan<<<static_cast<unsigned>(blocks), 256, 0, st>>>(s);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_shell_copy(bool f64, const GridView &a, const GridView &b, const GridView &ca, const GridView &cb,
                              const int64_t lb[3], const int64_t ub[3], const int64_t clb[3], const int reach[3],
                              const PairRun *run, cudaStream_t st) {
    ShellCopy c{};
    const GridView *src[2] = {&a, &b}, *dst[2] = {&ca, &cb};
    for (int g = 0; g < 2; ++g) {
        if (f64) {
            c.src[g] = domain_origin<const double>(*src[g], lb);
            c.dst[g] = domain_origin<float2>(*dst[g], clb);
        } else {
            c.src[g] = domain_origin<const float>(*src[g], lb);
            c.dst[g] = domain_origin<float>(*dst[g], clb);
        }
        c.ss0[g] = src[g]->s[0];
        c.ss1[g] = src[g]->s[1];
    }
    c.ds0 = ca.s[0];
    c.ds1 = ca.s[1];
    c.sh = shell_of(lb, ub, reach);
    c.run = run;
    const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>((c.sh.cells() + 255) / 256, device_sm_count() * 8ll));
    const dim3 grid(static_cast<unsigned>(blocks), 2);
    if (f64) k_shell_copy<true><<<grid, 256, 0, st>>>(c);
    else k_shell_copy<false><<<grid, 256, 0, st>>>(c);
    count_launch();
    return cudaGetLastError();
}

}  // namespace uhs
