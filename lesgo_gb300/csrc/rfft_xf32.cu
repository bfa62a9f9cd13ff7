// Forward x passes, float transforms.
#include "rfft_launch.cuh"
namespace lesgo {
template void rx_fwd(const RxGeom<float>&, const SrcFields<float, 1>&, cplx<float>*, cudaStream_t);
template void rx_fwd(const RxGeom<float>&, const SrcFields<float, 2>&, cplx<float>*, cudaStream_t);
template void rx_fwd(const RxGeom<float>&, const SrcFields<float, 3>&, cplx<float>*, cudaStream_t);
template void rx_fwd(const RxGeom<float>&, const SrcFields<float, 5>&, cplx<float>*, cudaStream_t);
template void rx_fwd(const RxGeom<float>&, const SrcVort<float, false>&, cplx<float>*, cudaStream_t);
template void rx_fwd(const RxGeom<float>&, const SrcVort<float, true>&, cplx<float>*, cudaStream_t);
template void rx_fwd21(const RxGeom<float>&, const SrcLagrange<float>&, cplx<float>*, cudaStream_t);
}  // namespace lesgo
