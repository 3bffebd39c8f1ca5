// Host-visible description of a resident run (resident.cuh holds the kernel,
// resident.cu the decomposition).
#pragma once
#include <cmath>

#include "stream_call.h"

namespace uhs {

// Threads of a CTA: float pairs 768 (at most 85 registers, one row pair per
// iteration), FP32 512 (the walk unrolled twice for radius 1).  us per sweep,
// 512 -> 768 threads: float pairs 2d1r star 1448^2 8.6 -> 7.6, 4000 x 400 7.4
// -> 6.0, others within 5 %; FP32 mostly 1-4 % slower.
constexpr int resident_threads(bool pairs) { return pairs ? 768 : 512; }
// dynamic shared memory a CTA may take (227 KB less the kernel's own words)
constexpr int kResidentSmem = 227 * 1024 - 256;

// Grids in the kernel's frame: rank-2 rows are z.
struct ResCall {
    void *a, *b;             // element (0, 0) of each grid
    int64_t as0, bs0;        // row strides, elements
    int lb0, lb2;            // domain origin (row, column)
    int nz, nx;              // domain extents
    int pz, px;              // boxes along each axis
    int G, L;                // rows between block barriers; rows a thread walks (both even, L at most 32)
    int halo_off;            // shared-memory byte offset of the halo list
    int T;
    int round64;             // FP64: round to FP64 between steps
    double growth;           // log2 of (sum |c|)^T where that exceeds 1
    void *pub;               // published cells, two buffers of the domain's cells
    unsigned *ctl;           // barrier counters and exponent words of the stream
    unsigned *err;
    int *verdict;            // FP64: 1 float pairs, 2 native
};

// The float pairs' scale from the exponent fields of a run's grids: emax the
// largest, emin the smallest of a nonzero value (negative: every cell zero).
// The largest magnitude grown over the run stays below 2^120; float pairs
// need every nonzero magnitude, scaled, at least 2^(-74 + kPairLowMargin).
// The scale is kept within +-800 so scaled exponents and their joins stay
// inside the FP64 range.
constexpr int kPairLowMargin = 24;
struct PairRange {
    bool ok;
    int shift;
};
__host__ __device__ inline PairRange pair_range(int emax, int emin, double growth) {
    if (emax >= 0x7ff) return PairRange{false, 0};  // Inf or NaN somewhere
    if (emin < 0) return PairRange{true, 0};
    const double top = static_cast<double>(emax - 1023) + 1.0 + growth;
    const double sd = floor(119.0 - top);
    if (!(sd >= -800.0)) return PairRange{false, 0};
    const int sh = static_cast<int>(sd < 800.0 ? sd : 800.0);
    if (emin - 1023 + sh < -74 + kPairLowMargin) return PairRange{false, 0};
    return PairRange{true, sh};
}

// The boxes of a resident run, or px = 0 when the domain does not fit.
struct ResPlan {
    int pz = 0, px = 0, G = 0, L = 0;
    int smem = 0, halo_off = 0;
    double cost = 0.0;  // estimated SM cycles per step
};
ResPlan plan_resident(bool corners, int R, int cell_bytes, int nterms, int64_t nz, int64_t nx, int sms, int max_smem);
cudaError_t launch_resident(int shape, int R, int st, const ResCall &c, int smem, const double *coef,
                            cudaStream_t stream);

}  // namespace uhs
