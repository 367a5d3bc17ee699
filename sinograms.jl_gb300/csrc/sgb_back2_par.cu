// sgb_back2_par.cu -- 2D back-projection, parallel beam.
#include "sgb_back2_kernel.cuh"

namespace sgb {

int launch_back2_par(const Back2Args &A, cudaStream_t st) { return back2::launch<back2::B2_PAR>(A, st); }

}  // namespace sgb
