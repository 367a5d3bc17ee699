// sgb_back2_flat.cu -- 2D back-projection, flat detector.
#include "sgb_back2_kernel.cuh"

namespace sgb {

int launch_back2_flat(const Back2Args &A, cudaStream_t st) { return back2::launch<back2::B2_FLAT>(A, st); }

}  // namespace sgb
