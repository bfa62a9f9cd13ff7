// y passes, double transforms.
#include "rfft_launch.cuh"
namespace lesgo {
template void ry_pass(RyKind, const RyArgs<double, cplx<double>, cplx<double>>&, int, int, int, cudaStream_t);
template void ry_spec(const RyArgs<double, cplx<double>, double2>&, int, int, int, cudaStream_t);
template void ry_phys(bool, const RyArgs<double, double2, cplx<double>>&, int, int, cudaStream_t);
}  // namespace lesgo
