// y passes, float transforms.
#include "rfft_launch.cuh"
namespace lesgo {
#define X(k) template void ry_pass<float, k>(const RyArgs<float, cplx<float>, cplx<float>>&, int, int, int, cudaStream_t);
X(RY_FILT) X(RY_DIV) X(RY_PAD) X(RY_VPAD) X(RY_UNPAD) X(RY_TEST1) X(RY_TEST2)
#undef X
template void ry_spec(const RyArgs<float, cplx<float>, double2>&, int, int, int, cudaStream_t);
template void ry_phys(bool, const RyArgs<float, double2, cplx<float>>&, int, int, cudaStream_t);
}  // namespace lesgo
