// rgc_pair_wide.cu -- the paired-tap RGC for tap boxes 20 .. 32 pixels wide, in a unit of its own so
// that the instantiations compile in parallel.  See rgc_pair.cuh.
#include "rgc_pair.cuh"

namespace esrrf {

cudaError_t fht_rgc_pair_wide(int R, const pair::PairArgs& a, int warps, cudaStream_t stream) {
    return pair::launch_pair_in<9, pair::kMaxR>(R, a, warps, stream);
}

}  // namespace esrrf
