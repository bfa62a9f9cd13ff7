// Inverse x passes, double transforms.
#include "rfft_launch.cuh"
namespace lesgo {
template void rx_inv(const RxGeom<double>&, const cplx<double>*, const DstFields<double, 1>&, cudaStream_t);
template void rx_inv(const RxGeom<double>&, const cplx<double>*, const DstFields<double, 2>&, cudaStream_t);
template void rx_inv(const RxGeom<double>&, const cplx<double>*, const DstFields<double, 3>&, cudaStream_t);
template void rx_inv(const RxGeom<double>&, const cplx<double>*, const DstFields<double, 9>&, cudaStream_t);
template void rx_inv(const RxGeom<double>&, const cplx<double>*, const DstDiv<double, 1>&, cudaStream_t);
template void rx_inv(const RxGeom<double>&, const cplx<double>*, const DstDiv<double, 2>&, cudaStream_t);
template void rx_inv(const RxGeom<double>&, const cplx<double>*, const DstDiv<double, 3>&, cudaStream_t);
template void rx_inv(const RxGeom<double>&, const cplx<double>*, const DstConvec<double, false>&, cudaStream_t);
template void rx_inv(const RxGeom<double>&, const cplx<double>*, const DstConvec<double, true>&, cudaStream_t);
template void rx_inv(const RxGeom<double>&, const cplx<double>*, const DstPress<double, false>&, cudaStream_t);
template void rx_inv(const RxGeom<double>&, const cplx<double>*, const DstPress<double, true>&, cudaStream_t);
template void rx_inv42(const RxGeom<double>&, const cplx<double>*, const DstLagrange<double>&, cudaStream_t);
}  // namespace lesgo
