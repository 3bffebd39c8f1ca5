// Resident runs (resident.cuh): the split into one box per CTA, and the
// launch.
#include <atomic>
#include <cstring>

#include "resident.cuh"

namespace uhs {
namespace {

template <int SHAPE, int R, int ST>
cudaError_t launch_cfg(const ResCall &c, int smem, const double *coef, cudaStream_t st) {
    constexpr int NT = ResShape<SHAPE, R>::NT;
    ResArgs<NT> args;
    std::memset(&args, 0, sizeof args);
    args.c = c;
    double cd[NT];
    fill_coefs(cd, args.chl, args.cl_sum, coef, NT, SHAPE, R);
    if (ST == kStF64) fill_coef_anchor(args.cab, args.chl, NT, SHAPE, R, false);
    auto kern = k_resident<SHAPE, R, ST>;
    // the largest size once per device, so concurrent launches never see a smaller one
    static std::atomic<bool> ready[64];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const bool known = dev >= 0 && dev < 64;
    if (!known || !ready[dev].load(std::memory_order_acquire)) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kResidentSmem);
        if (e != cudaSuccess) return e;
        if (known) ready[dev].store(true, std::memory_order_release);
    }
    void *params[] = {&args};
    e = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(kern), dim3(c.px * c.pz), dim3(resident_threads(ST == kStF64)),
                                    params, static_cast<size_t>(smem), st);
    if (e == cudaSuccess) count_launch();
    return e;
}

template <int ST>
cudaError_t dispatch(int shape, int R, const ResCall &c, int smem, const double *coef, cudaStream_t st) {
    switch (shape * 4 + R) {
        case kStar2 * 4 + 1: return launch_cfg<kStar2, 1, ST>(c, smem, coef, st);
        case kStar2 * 4 + 2: return launch_cfg<kStar2, 2, ST>(c, smem, coef, st);
        case kStar2 * 4 + 3: return launch_cfg<kStar2, 3, ST>(c, smem, coef, st);
        case kBox2 * 4 + 1: return launch_cfg<kBox2, 1, ST>(c, smem, coef, st);
        case kBox2 * 4 + 2: return launch_cfg<kBox2, 2, ST>(c, smem, coef, st);
        case kBox2 * 4 + 3: return launch_cfg<kBox2, 3, ST>(c, smem, coef, st);
        case kSep2 * 4 + 1: return launch_cfg<kSep2, 1, ST>(c, smem, coef, st);
        case kSep2 * 4 + 2: return launch_cfg<kSep2, 2, ST>(c, smem, coef, st);
        case kSep2 * 4 + 3: return launch_cfg<kSep2, 3, ST>(c, smem, coef, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

cudaError_t launch_resident(int shape, int R, int st, const ResCall &c, int smem, const double *coef,
                            cudaStream_t stream) {
    return st == kStF64 ? dispatch<kStF64>(shape, R, c, smem, coef, stream)
                        : dispatch<kStF32>(shape, R, c, smem, coef, stream);
}

// The split that makes the slowest CTA's step shortest, by a rough count of SM
// cycles (fitted to GB300 timings): a walk's set-up, its iterations (two rows
// of a column each; the warps share the issue slots, a lone warp still takes
// its own latency), the halo cells and a fixed exchange latency.
ResPlan plan_resident(bool corners, int R, int cell_bytes, int nterms, int64_t nz, int64_t nx, int sms, int max_smem) {
    ResPlan best;
    // more than shared memory holds whatever the split
    if (nz <= 0 || nx <= 0 || nz * nx > static_cast<int64_t>(max_smem / cell_bytes) * sms) return best;
    const bool pairs = cell_bytes == 8;
    const double iter = pairs ? 48.0 * nterms + 140.0 : 8.0 * nterms + 100.0, lat = 0.4 * iter + 60.0;
    const double setup = 440.0;
    const int threads = resident_threads(pairs);
    for (int64_t px : {1, 2, 3, 4, 5, 6, 8, 10, 12, 15, 19, 25, 30, 38, 50, 76, 152}) {
        if (px > sms || px > nx) break;
        const int64_t bx = (nx + px - 1) / px;
        const int64_t pmax = std::min<int64_t>(sms / px, nz);
        const int64_t bz = (nz + pmax - 1) / pmax, pz = (nz + bz - 1) / bz;
        const int64_t w = bx + 2 * R, cells = 2 * R * (bz + (corners ? w : bx));
        const int64_t slots = (max_smem - 4 * cells) / (w * cell_bytes);
        if (slots < bz + 3 * R + 2 + 1) continue;
        const int64_t gmax = std::min<int64_t>(slots - (bz + 3 * R + 1), bz + 1) & ~int64_t(1);
        const int64_t groups = (bz + gmax - 1) / gmax;
        const int64_t g = ((bz + groups - 1) / groups + 1) & ~int64_t(1);  // even groups, at most gmax
        const double exchange = 2200.0 + (pairs ? 2.2 : 1.8) * static_cast<double>(cells);
        for (int64_t l = 2; l <= 32 && l <= g; l += 2) {
            const int64_t items = bx * ((std::min(g, bz) + l - 1) / l);
            const int64_t full = items / threads, rest = items % threads;
            const double part = std::max(lat, iter * static_cast<double>(rest) / threads);
            const double work = static_cast<double>(full) * (iter * (l / 2) + setup) +
                                (rest ? part * (l / 2) + setup : 0.0);
            const double cost = exchange + static_cast<double>(groups) * (work + 60.0);
            if (best.px && cost >= best.cost) continue;
            best.cost = cost;
            best.px = static_cast<int>(px);
            best.pz = static_cast<int>(pz);
            best.G = static_cast<int>(g);
            best.L = static_cast<int>(l);
            best.halo_off = static_cast<int>((bz + 3 * R + g + 1) * w * cell_bytes);
            best.smem = best.halo_off + static_cast<int>(4 * cells);
        }
    }
    return best;
}

}  // namespace uhs
