// y pass, double-word transforms: 3/2 padding (a unit of its own for the build's time).
#include "rfft_launch.cuh"
namespace lesgo {
template void ry_pass<df64, RY_PAD>(const RyArgs<df64, cplx<df64>, cplx<df64>>&, int, int, int, cudaStream_t);
}  // namespace lesgo
