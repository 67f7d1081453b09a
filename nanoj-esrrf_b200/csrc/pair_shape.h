// pair_shape.h -- how the paired-tap kernels (rgc_pair.cuh, bic_pair.cuh) lay a launch's warps out.
#pragma once

namespace esrrf {

// How a launch's warps are laid out: warps of a CTA, and the row segments a strip is cut into (`segs`
// of `rows` rows each, the rest of the frame one more).
struct PairShape {
    int warps = 16, rows = 0, segs = 1;
    double cost = 0;  // modelled time, in rows of one warp
};

// The shape with the least modelled time for `units` (strip, frame) pairs of H rows, taps reaching R rows,
// `maxw` warps an SM.
PairShape pair_shape(int units, int H, int R, int maxw, int sms);

}  // namespace esrrf
