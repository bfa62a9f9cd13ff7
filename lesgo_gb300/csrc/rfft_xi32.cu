// Inverse x passes, float transforms.
#include "rfft_launch.cuh"
namespace lesgo {
template void rx_inv(const RxGeom<float>&, const cplx<float>*, const DstFields<float, 1>&, cudaStream_t);
template void rx_inv(const RxGeom<float>&, const cplx<float>*, const DstFields<float, 2>&, cudaStream_t);
template void rx_inv(const RxGeom<float>&, const cplx<float>*, const DstFields<float, 3>&, cudaStream_t);
template void rx_inv(const RxGeom<float>&, const cplx<float>*, const DstFields<float, 9>&, cudaStream_t);
template void rx_inv(const RxGeom<float>&, const cplx<float>*, const DstDiv<float, 1>&, cudaStream_t);
template void rx_inv(const RxGeom<float>&, const cplx<float>*, const DstDiv<float, 2>&, cudaStream_t);
template void rx_inv(const RxGeom<float>&, const cplx<float>*, const DstDiv<float, 3>&, cudaStream_t);
template void rx_inv(const RxGeom<float>&, const cplx<float>*, const DstConvec<float, false>&, cudaStream_t);
template void rx_inv(const RxGeom<float>&, const cplx<float>*, const DstConvec<float, true>&, cudaStream_t);
template void rx_inv(const RxGeom<float>&, const cplx<float>*, const DstPress<float, false>&, cudaStream_t);
template void rx_inv(const RxGeom<float>&, const cplx<float>*, const DstPress<float, true>&, cudaStream_t);
template void rx_inv42(const RxGeom<float>&, const cplx<float>*, const DstLagrange<float>&, cudaStream_t);
}  // namespace lesgo
