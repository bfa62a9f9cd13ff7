// y pass, double-word transforms: 3/2 truncation (a unit of its own for the build's time).
#include "rfft_launch.cuh"
namespace lesgo {
template void ry_pass<df64, RY_UNPAD>(const RyArgs<df64, cplx<df64>, cplx<df64>>&, int, int, int, cudaStream_t);
}  // namespace lesgo
