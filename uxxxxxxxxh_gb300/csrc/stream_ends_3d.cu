// Sweeps of runs on float-pair copies of FP64 grids: the first reads the FP64
// grid and writes pairs, the last ones read pairs and write the FP64 grid, so
// that a run needs no conversion passes; the ones between them sum without the
// anchored sums' factor.  One tile per shape, the planner's default.
// Term-by-term boxes of radius 2-3 have none: their sums dwarf the
// conversion passes.
#include "stream_launch.cuh"

namespace uhs {
namespace {

template <int SHAPE, int R>
cudaError_t dispatch(const StreamCall &c) {
    constexpr int TY = 4, VY = 4, PD = 3;
    if (c.io == kIoRun) {
        if constexpr (is_anchored(SHAPE, R))
            if (c.ld == kLdTma) return launch_cfg<StreamCfg<SHAPE, R, kStF32x2, kArDf32, kLdTma, 32, TY, VY, PD, 0, 1, kIoRun>>(c);
        return cudaErrorInvalidValue;
    }
    if (c.io == kIoLast)
        return c.ld == kLdTma ? launch_cfg<StreamCfg<SHAPE, R, kStF32x2, kArDf32, kLdTma, 32, TY, VY, PD, 0, 1, kIoLast>>(c)
                              : cudaErrorInvalidValue;
    return c.ld == kLdTma ? launch_cfg<StreamCfg<SHAPE, R, kStF64, kArDf32, kLdTma, 32, TY, VY, PD, 0, 1, kIoFirst>>(c)
                          : launch_cfg<StreamCfg<SHAPE, R, kStF64, kArDf32, kLdCpAsync, 32, TY, VY, PD, 0, 1, kIoFirst>>(c);
}

}  // namespace

cudaError_t launch_stream_ends_3d(const StreamCall &c) {
    if (c.tile != 1) return cudaErrorInvalidValue;
    switch (c.R * 3 + (c.shape == kStar3 ? 0 : c.shape == kSep3 ? 2 : 1)) {
        case 3: return dispatch<kStar3, 1>(c);
        case 4: return dispatch<kBox3, 1>(c);
        case 5: return dispatch<kSep3, 1>(c);
        case 6: return dispatch<kStar3, 2>(c);
        case 8: return dispatch<kSep3, 2>(c);
        case 9: return dispatch<kStar3, 3>(c);
        case 11: return dispatch<kSep3, 3>(c);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace uhs
