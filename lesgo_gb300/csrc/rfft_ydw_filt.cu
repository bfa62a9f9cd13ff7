// y pass, double-word transforms: filt_da (a unit of its own for the build's time).
#include "rfft_launch.cuh"
namespace lesgo {
template void ry_pass<df64, RY_FILT>(const RyArgs<df64, cplx<df64>, cplx<df64>>&, int, int, int, cudaStream_t);
}  // namespace lesgo
