// The convective 3/2-grid rows, float transforms.
#include "rfft_launch.cuh"
namespace lesgo {
template void rx_rows(RxRowsGeom<float>, int, int, const cplx<float>*, cplx<float>*, float, cudaStream_t);
}  // namespace lesgo
