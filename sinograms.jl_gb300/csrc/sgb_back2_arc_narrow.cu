// sgb_back2_arc_narrow.cu -- 2D back-projection, arc detector within +-31 degrees.
#include "sgb_back2_kernel.cuh"

namespace sgb {

int launch_back2_arc_narrow(const Back2Args &A, cudaStream_t st) { return back2::launch<back2::B2_ARC_NARROW>(A, st); }

}  // namespace sgb
