// y passes, float transforms.
#include "rfft_launch.cuh"
namespace lesgo {
template void ry_pass(RyKind, const RyArgs<float, cplx<float>, cplx<float>>&, int, int, int, cudaStream_t);
template void ry_spec(const RyArgs<float, cplx<float>, double2>&, int, int, int, cudaStream_t);
template void ry_phys(bool, const RyArgs<float, double2, cplx<float>>&, int, int, cudaStream_t);
}  // namespace lesgo
