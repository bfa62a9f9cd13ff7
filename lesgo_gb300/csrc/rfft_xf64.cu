// Forward x passes, double transforms.
#include "rfft_launch.cuh"
namespace lesgo {
template void rx_fwd(const RxGeom<double>&, const SrcFields<double, 1>&, cplx<double>*, cudaStream_t);
template void rx_fwd(const RxGeom<double>&, const SrcFields<double, 2>&, cplx<double>*, cudaStream_t);
template void rx_fwd(const RxGeom<double>&, const SrcFields<double, 3>&, cplx<double>*, cudaStream_t);
template void rx_fwd(const RxGeom<double>&, const SrcFields<double, 5>&, cplx<double>*, cudaStream_t);
template void rx_fwd(const RxGeom<double>&, const SrcVort<double, false>&, cplx<double>*, cudaStream_t);
template void rx_fwd(const RxGeom<double>&, const SrcVort<double, true>&, cplx<double>*, cudaStream_t);
template void rx_fwd21(const RxGeom<double>&, const SrcLagrange<double>&, cplx<double>*, cudaStream_t);
}  // namespace lesgo
