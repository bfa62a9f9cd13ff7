// Definitions of rfft_api.cuh's launchers (included by the translation units
// that instantiate them).
#pragma once
#include "launch_util.hpp"
#include "rfft_api.cuh"

namespace lesgo {

template <typename A, class Src> void rx_fwd(const RxGeom<A>& g, const Src& src, cplx<A>* out, cudaStream_t st) {
  with_rx(g.N, [&](auto len) {
    constexpr int R1 = decltype(len)::R1, R2 = decltype(len)::R2, L = rx_lines<R1, R2>();
    k_rx_fwd<A, R1, R2, Src><<<dim3((g.nrows + L - 1) / L, g.nf), L * cmax(R1, R2), 0, st>>>(g, src, out);
  });
}
template <typename A, class Dst> void rx_inv(const RxGeom<A>& g, const cplx<A>* in, const Dst& dst, cudaStream_t st) {
  with_rx(g.N, [&](auto len) {
    constexpr int R1 = decltype(len)::R1, R2 = decltype(len)::R2, L = rx_lines<R1, R2>();
    k_rx_inv<A, R1, R2, Dst><<<dim3((g.nrows + L - 1) / L, g.nf), L * cmax(R1, R2), 0, st>>>(g, in, dst);
  });
}

template <typename KF> static void smem_for(KF kern, size_t bytes) {
  if (bytes > 48 * 1024) raise_smem_limit(reinterpret_cast<const void*>(kern), bytes);
}

template <typename A> void rx_fwd21(const RxGeom<A>& g, const SrcLagrange<A>& src, cplx<A>* out, cudaStream_t st) {
  with_rx(g.N, [&](auto len) {
    constexpr int R1 = decltype(len)::R1, R2 = decltype(len)::R2;
    constexpr size_t smem = 21 * (cmax(R1 * odd_up(R2), R1 * R2 + 1) | 1) * sizeof(cplx<A>);
    auto kern = k_rx_fwd21<A, R1, R2, SrcLagrange<A>>;
    smem_for(kern, smem);
    kern<<<g.nrows, 21 * cmax(R1, R2), smem, st>>>(g, src, out);
  });
}
template <typename A> void rx_inv42(const RxGeom<A>& g, const cplx<A>* in, const DstLagrange<A>& dst, cudaStream_t st) {
  with_rx(g.N, [&](auto len) {
    constexpr int R1 = decltype(len)::R1, R2 = decltype(len)::R2;
    constexpr size_t smem = 42 * (cmax(R1 * odd_up(R2), R1 * R2) | 1) * sizeof(cplx<A>);
    auto kern = k_rx_inv42<A, R1, R2, DstLagrange<A>>;
    smem_for(kern, smem);
    kern<<<g.nrows, 21 * cmax(R1, R2), smem, st>>>(g, in, dst);
  });
}

template <typename A, RyKind KIND>
void ry_pass(const RyArgs<A, cplx<A>, cplx<A>>& a, int ny, int nlev, int nf, cudaStream_t st) {
  with_ry(ny, [&](auto len) {
    constexpr int R1 = decltype(len)::R1, R2 = decltype(len)::R2, S2 = 3 * R2 / 2;
    constexpr size_t e = ry_elems<R1, R2>(), eb = ry_elems<R1, S2>();
    const dim3 grid((a.K + kYC - 1) / kYC, nlev, nf);
    auto go = [&](auto kern, int threads, size_t elems) {
      smem_for(kern, elems * sizeof(cplx<A>));
      kern<<<grid, threads, elems * sizeof(cplx<A>), st>>>(a);
    };
    constexpr int t1 = kYC * cmax(R1, R2), t2 = kYC * cmax(R1, S2);
    if constexpr (KIND == RY_FILT) go(k_ry_filt<A, R1, R2>, t1, 2 * e + kYC);
    if constexpr (KIND == RY_DIV) go(k_ry_div<A, R1, R2>, t1, 2 * e + R2 * kYC);
    if constexpr (KIND == RY_PAD) go(k_ry_pad<A, R1, R2>, t2, e + eb);
    if constexpr (KIND == RY_VPAD) go(k_ry_vpad<A, R1, R2>, t2, e + eb);
    if constexpr (KIND == RY_UNPAD) go(k_ry_unpad<A, R1, R2>, t2, e + eb);
    if constexpr (KIND == RY_TEST1) go(k_ry_test<A, R1, R2, false>, t1, 2 * e);
    if constexpr (KIND == RY_TEST2) go(k_ry_test<A, R1, R2, true>, t1, 2 * e);
  });
}
template <typename A>
void ry_spec(const RyArgs<A, cplx<A>, double2>& a, int ny, int nlev, int nf, cudaStream_t st) {
  with_ry(ny, [&](auto len) {
    constexpr int R1 = decltype(len)::R1, R2 = decltype(len)::R2;
    constexpr size_t smem = ry_elems<R1, R2>() * sizeof(cplx<A>);
    auto kern = k_ry_spec<A, R1, R2>;
    smem_for(kern, smem);
    kern<<<dim3((a.K + kYC - 1) / kYC, nlev, nf), kYC * cmax(R1, R2), smem, st>>>(a);
  });
}
template <typename A>
void ry_phys(bool grad, const RyArgs<A, double2, cplx<A>>& a, int ny, int nlev, cudaStream_t st) {
  with_ry(ny, [&](auto len) {
    constexpr int R1 = decltype(len)::R1, R2 = decltype(len)::R2;
    constexpr size_t e = ry_elems<R1, R2>() * sizeof(cplx<A>);
    const dim3 grid((a.K + kYC - 1) / kYC, nlev);
    auto go = [&](auto kern, size_t smem) {
      smem_for(kern, smem);
      kern<<<grid, kYC * cmax(R1, R2), smem, st>>>(a);
    };
    if (grad) go(k_ry_phys<A, R1, R2, true>, 2 * e);
    else go(k_ry_phys<A, R1, R2, false>, e);
  });
}

template <typename A>
void rx_rows(RxRowsGeom<A> g, int H, int ninst, const cplx<A>* in, cplx<A>* out, A c, cudaStream_t st) {
  with_rxb(H, [&](auto len) {
    constexpr int R1 = decltype(len)::R1, R2 = decltype(len)::R2, L = rows_lines<A, R1, R2>();
    constexpr size_t smem = (L * rows_per_row<R1, R2>() + rows_besides<R1, R2>()) * sizeof(cplx<A>);
    constexpr int threads = L * R1;
    auto kern = k_rx_rows<A, R1, R2>;
    smem_for(kern, smem);
    // Levels per block: a block marches its chunk and about one level more
    // (two and three fields of the levels around it), so the launch takes
    // about (waves) x (chunk + 1) level times.
    int per_sm = 0, nsm = 0, dev = 0;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem));
    const long long tiles = (long long)((g.ny2 + L - 1) / L) * ninst;
    const long long slots = std::max(1LL, (long long)per_sm * nsm);
    int best = 1;
    long long best_t = -1;
    for (int n = 1; n <= g.nz; ++n) {
      const long long t = ((tiles * n + slots - 1) / slots) * ((g.nz + n - 1) / n + 1);
      if (best_t < 0 || t < best_t) { best_t = t; best = n; }
    }
    g.cz = (g.nz + best - 1) / best;
    kern<<<dim3((unsigned)((g.ny2 + L - 1) / L), (unsigned)((g.nz + g.cz - 1) / g.cz), (unsigned)ninst), threads, smem, st>>>(
        g, in, out, c);
  });
}

}  // namespace lesgo
