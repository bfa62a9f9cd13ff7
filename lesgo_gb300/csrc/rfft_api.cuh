// Launchers of the register-transform passes (rfft_pass.cuh, rfft_rows.cuh),
// defined in rfft_launch.cuh and instantiated in translation units of their
// own.  The length must be one of the lists of rfft_pass.cuh.
#pragma once
#include "rfft_pass.cuh"
#include "rfft_rows.cuh"

namespace lesgo {

template <typename A, class Src> void rx_fwd(const RxGeom<A>& g, const Src& src, cplx<A>* out, cudaStream_t st);
template <typename A, class Dst> void rx_inv(const RxGeom<A>& g, const cplx<A>* in, const Dst& dst, cudaStream_t st);
template <typename A> void rx_fwd21(const RxGeom<A>& g, const SrcLagrange<A>& src, cplx<A>* out, cudaStream_t st);
template <typename A> void rx_inv42(const RxGeom<A>& g, const cplx<A>* in, const DstLagrange<A>& dst, cudaStream_t st);

enum RyKind { RY_FILT, RY_DIV, RY_PAD, RY_VPAD, RY_UNPAD, RY_TEST1, RY_TEST2 };
// The double-word form has the four kinds that gain by it (128^3, us against
// the run-time radix stages): filt_da 93 (150), divergence 107 (191), pad 161
// (226), unpad 91 (114).  With two filters, the forward modes kept for both,
// registers leave too few warps (852 against 624), the pressure's passes
// gain nothing (55 against 59, 53 against 51), and RY_VPAD's code alone would
// be several hundred KB.
template <typename A> constexpr bool kRyKind(RyKind k) {
  return !std::is_same<A, df64>::value || k == RY_FILT || k == RY_DIV || k == RY_PAD || k == RY_UNPAD;
}
// ny rows (the small grid's count) of nf fields, nlev planes
template <typename A, RyKind KIND>
void ry_pass(const RyArgs<A, cplx<A>, cplx<A>>& a, int ny, int nlev, int nf, cudaStream_t st);
template <typename A>
void ry_spec(const RyArgs<A, cplx<A>, double2>& a, int ny, int nlev, int nf, cudaStream_t st);
template <typename A>
void ry_phys(bool grad, const RyArgs<A, double2, cplx<A>>& a, int ny, int nlev, cudaStream_t st);

// g.cz, the levels per block, is set here from the launch's waves
template <typename A>
void rx_rows(RxRowsGeom<A> g, int H, int ninst, const cplx<A>* in, cplx<A>* out, A c, cudaStream_t st);

}  // namespace lesgo
