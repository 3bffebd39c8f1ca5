// Sweeps of runs on float-pair copies of FP64 grids: the first reads the FP64
// grid and writes pairs, the last ones read pairs and write the FP64 grid, so
// that a run needs no conversion passes; the ones between them sum without the
// anchored sums' factor.  One tile per shape, the planner's default.
#include "stream_launch.cuh"

namespace uhs {
namespace {

// stars: 256 columns by cp.async, two points per thread (radius 3: one), and
// 128 columns by TMA, two points; boxes: 128 columns, one point
template <int SHAPE, int R>
cudaError_t dispatch(const StreamCall &c) {
    if constexpr (SHAPE == kStar2) {
        if (c.io == kIoRun)
            return c.ld == kLdTma && c.tile == 3
                       ? launch_cfg<StreamCfg<SHAPE, R, kStF32x2, kArDf32, kLdTma, 64, 1, 1, 4, 0, 2, kIoRun>>(c)
                       : cudaErrorInvalidValue;
        if (c.io == kIoLast)
            return c.ld == kLdTma && c.tile == 3
                       ? launch_cfg<StreamCfg<SHAPE, R, kStF32x2, kArDf32, kLdTma, 64, 1, 1, 4, 0, 2, kIoLast>>(c)
                       : cudaErrorInvalidValue;
        if (c.ld != kLdCpAsync || c.tile != (R == 3 ? 2 : 4)) return cudaErrorInvalidValue;
        if constexpr (R == 3) return launch_cfg<StreamCfg<SHAPE, R, kStF64, kArDf32, kLdCpAsync, 256, 1, 1, 4, 0, 1, kIoFirst>>(c);
        else return launch_cfg<StreamCfg<SHAPE, R, kStF64, kArDf32, kLdCpAsync, 128, 1, 1, 4, 0, 2, kIoFirst>>(c);
    } else {
        constexpr int LAST = SHAPE == kBox2 ? kLdCpAsync : kLdTma;
        if (c.tile != 0) return cudaErrorInvalidValue;
        if (c.io == kIoRun) {
            if constexpr (SHAPE == kSep2)
                if (c.ld == kLdTma)
                    return launch_cfg<StreamCfg<SHAPE, R, kStF32x2, kArDf32, kLdTma, 128, 1, 1, 4, 0, 1, kIoRun>>(c);
            return cudaErrorInvalidValue;
        }
        if (c.io == kIoLast)
            return c.ld == LAST ? launch_cfg<StreamCfg<SHAPE, R, kStF32x2, kArDf32, LAST, 128, 1, 1, 4, 0, 1, kIoLast>>(c)
                                : cudaErrorInvalidValue;
        if (c.ld == kLdTma) {
            if constexpr (SHAPE == kSep2)
                return launch_cfg<StreamCfg<SHAPE, R, kStF64, kArDf32, kLdTma, 128, 1, 1, 4, 0, 1, kIoFirst>>(c);
            else
                return cudaErrorInvalidValue;
        }
        return launch_cfg<StreamCfg<SHAPE, R, kStF64, kArDf32, kLdCpAsync, 128, 1, 1, 4, 0, 1, kIoFirst>>(c);
    }
}

}  // namespace

cudaError_t launch_stream_ends_2d(const StreamCall &c) {
    switch (c.R * 3 + (c.shape == kStar2 ? 0 : c.shape == kSep2 ? 2 : 1)) {
        case 3: return dispatch<kStar2, 1>(c);
        case 4: return dispatch<kBox2, 1>(c);
        case 5: return dispatch<kSep2, 1>(c);
        case 6: return dispatch<kStar2, 2>(c);
        case 7: return dispatch<kBox2, 2>(c);
        case 8: return dispatch<kSep2, 2>(c);
        case 9: return dispatch<kStar2, 3>(c);
        case 10: return dispatch<kBox2, 3>(c);
        case 11: return dispatch<kSep2, 3>(c);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace uhs
