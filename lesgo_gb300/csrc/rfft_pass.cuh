// The batched x and y passes of the step on transforms held in registers
// (rfft_core.cuh), for the lengths of the lists below; fft_core.cuh's passes
// serve every other length.  Layouts are fft_core.cuh's: spectra are
// [field][line of planes][jy][kx], fields the reference's planes.
//
// A listed length always takes these passes: they were faster at every size
// measured.  One 128^3 instance, mixed form, us per launch against the
// run-time radix stages (and the time of the unique bytes at the copy
// bandwidth):
//   filt_da      x 14.3 (20.5; 7.5), y 22.9 (45.6; 15), x inverse 37 (50; 22)
//   divstress    x 19.8 (30.8; 12.5), y 20.0 (55.4; 10), x inverse 18.6 (36; 11)
//   convec       y pad with the vorticity 34.5 (x 36.3 and y 69.8; 15),
//                y unpad 19 (37; 9), x inverse with AB2 38.5 (43.3; 26)
//   pressure     x 14.5 (20.9; 7.5), y 17.1 (27.5; 11), y inverse 14.1 (22.6; 6),
//                x inverse with projection 28.5 (31.3; 15)
//   Lagrangian   x 86 (131; 38), y 84 (244; 79), x inverse 144 (303; 69)
// and one 48^3 instance 5.0 against 6.6 us for a pass of one wave: the
// stages' barriers (one per radix stage) were its latency.  In FP64, which
// the FP64 pipe bounds: 128^3 37.8 -> 33.2 ms for five steps, 32^3 3.9 -> 3.05
// ms for ten.
#pragma once
#include "rfft_core.cuh"
#include "stages.cuh"

namespace lesgo {

// Lengths and their factors.  x: complex length nx/2; R2 is even, so the
// real-transform split pairs mode k < N/2 with N - k.  y: ny = R1 R2 with R2
// even and ny2 = 3 ny / 2 = R1 (3 R2 / 2): padding to the 3/2 grid and
// truncation from it then only relabel the R2 or 3 R2 / 2 values that a
// thread holds.  xb: complex length 3 nx / 4 of the 3/2 grid's rows; R1 is a
// multiple of 3, so the padded modes are whole inputs of the first DFT, and
// R2 <= 9 keeps the products' operands of one thread in registers.
#define LESGO_RX_LENGTHS(X) \
  X(4, 4) X(3, 6) X(6, 4) X(8, 4) X(6, 6) X(8, 6) X(9, 6) X(8, 8) X(9, 8) X(12, 8) X(9, 12) X(16, 8)
#define LESGO_RY_LENGTHS(X) \
  X(6, 4) X(8, 4) X(6, 6) X(8, 6) X(9, 6) X(8, 8) X(9, 8) X(12, 8) X(9, 12) X(16, 8) X(12, 12) X(16, 12) X(18, 12) X(16, 16)
#define LESGO_RXB_LENGTHS(X) \
  X(6, 4) X(9, 3) X(6, 6) X(6, 8) X(9, 6) X(9, 8) X(9, 9) X(12, 8) X(18, 6) X(18, 8) X(18, 9) X(24, 8)

inline bool rx_factors(int n, int* r1, int* r2) {
#define X(a, b) if (n == (a) * (b)) { *r1 = a; *r2 = b; return true; }
  LESGO_RX_LENGTHS(X)
#undef X
  return false;
}
inline bool ry_factors(int n, int* r1, int* r2) {
#define X(a, b) if (n == (a) * (b)) { *r1 = a; *r2 = b; return true; }
  LESGO_RY_LENGTHS(X)
#undef X
  return false;
}
inline bool rxb_factors(int n, int* r1, int* r2) {
#define X(a, b) if (n == (a) * (b)) { *r1 = a; *r2 = b; return true; }
  LESGO_RXB_LENGTHS(X)
#undef X
  return false;
}
// Calls fn(Len<R1, R2>) for the listed length n.
template <class F> void with_rx(int n, F&& fn) {
#define X(a, b) if (n == (a) * (b)) { fn(Len<a, b>{}); return; }
  LESGO_RX_LENGTHS(X)
#undef X
}
template <class F> void with_ry(int n, F&& fn) {
#define X(a, b) if (n == (a) * (b)) { fn(Len<a, b>{}); return; }
  LESGO_RY_LENGTHS(X)
#undef X
}
template <class F> void with_rxb(int n, F&& fn) {
#define X(a, b) if (n == (a) * (b)) { fn(Len<a, b>{}); return; }
  LESGO_RXB_LENGTHS(X)
#undef X
}

// ---------------------------------------------------------------------------
// x passes
// ---------------------------------------------------------------------------
template <typename A>
struct RxGeom {
  int N;             // complex length nx/2 (= the modes kept)
  int nf;            // fields of the launch (blockIdx.y)
  int nrows;         // rows per field
  FastDiv fny;       // by the rows per level
  int nyrows;
  long long fs;      // complex elements between fields of the spectra
  int kz0, kz1;      // modes from which even / odd fields are zero and not read
  const cplx<A>* tw;   // tw[k1 * R2 + n2] = exp(-2 pi i k1 n2 / N)
  const cplx<A>* rtw;  // rtw[k] = exp(-2 pi i k / (2 N))
};

// p[f] without indexing the kernel's parameters at run time (which would
// copy them to local memory)
template <int NF, typename P> __device__ __forceinline__ P pick(P const (&p)[NF], int f) {
  P r = p[0];
#pragma unroll
  for (int i = 1; i < NF; ++i)
    if (f == i) r = p[i];
  return r;
}

// CNT pairs (x[2n], x[2n+1]) of field f, n = n0 + j * STEP, scaled.
template <int CNT, int STEP, typename R, int NF>
__device__ __forceinline__ void rx_load(const SrcFields<R, NF>& s, int f, int jy, int li, int n0, cplx<R>* v) {
  const int inst = s.im.inst(li), lv = li - inst * s.im.nli;
  const R* p = pick(s.p, f) + inst * s.im.istr + (long long)(s.lev0 + lv * s.levstride) * s.plane + (long long)jy * s.ld + 2 * n0;
  const R c = s.isc ? (R)(s.isc_mul * s.isc[inst * SC_N + s.isc_idx]) : s.scale;
#pragma unroll
  for (int j = 0; j < CNT; ++j) v[j] = *reinterpret_cast<const cplx<R>*>(p + 2 * STEP * j);
#pragma unroll
  for (int j = 0; j < CNT; ++j) v[j] = cscale(v[j], c);
}

// c * (h (A + A2) - B): the vorticity components are differences of two
// gradients, one of them averaged over two levels at the wall and the lid
template <int CNT, int STEP, typename R>
__device__ __forceinline__ void rx_diff(const R* a, const R* b, long long o, long long o2, bool avg, bool flip, R c,
                                        cplx<R>* v) {
  using C = cplx<R>;
  C x[CNT];
#pragma unroll
  for (int j = 0; j < CNT; ++j) v[j] = *reinterpret_cast<const C*>(a + o + 2 * STEP * j);
  if (avg) {
#pragma unroll
    for (int j = 0; j < CNT; ++j) {
      x[j] = *reinterpret_cast<const C*>(a + o2 + 2 * STEP * j);
      v[j] = cscale(cadd(v[j], x[j]), (R)0.5);
    }
  }
#pragma unroll
  for (int j = 0; j < CNT; ++j) x[j] = *reinterpret_cast<const C*>(b + 2 * STEP * j);
#pragma unroll
  for (int j = 0; j < CNT; ++j) v[j] = cscale(flip ? csub(x[j], v[j]) : csub(v[j], x[j]), c);
}

// convec.f90:71-168 (as SrcVort): fields u, v, w and the vorticity, or the
// three vorticity components alone.
template <int CNT, int STEP, typename R, bool VO>
__device__ __forceinline__ void rx_load(const SrcVort<R, VO>& s, int f, int jy, int li, int n0, cplx<R>* v) {
  const int inst = s.im.inst(li);
  const int k = li - inst * s.im.nli + 1;
  const long long o = inst * s.im.istr + (long long)k * s.plane + (long long)jy * s.ld + 2 * n0;
  const int q = VO ? f + 3 : f;
  if (q < 3 || (k == 1 && s.lbc == 0 && q < 5)) {
    const R* p = (q == 0 ? s.u : q == 1 ? s.v : s.w) + o;
#pragma unroll
    for (int j = 0; j < CNT; ++j) v[j] = q < 3 ? *reinterpret_cast<const cplx<R>*>(p + 2 * STEP * j) : czero<cplx<R>>();
#pragma unroll
    for (int j = 0; j < CNT; ++j) v[j] = cscale(v[j], s.c);
    return;
  }
  if (q == 5) {
    rx_diff<CNT, STEP, R>(s.dvdx, s.dudy + o, o, o, false, false, s.c, v);
    return;
  }
  // (dw/dy - dv/dz) or (du/dz - dw/dx), dw averaged at the wall and below
  // a lid with a wall condition, the z-derivative then one level down
  const bool wall = k == 1, lid = k == s.nz && s.ubc > 0;
  const long long oz = lid ? o - s.plane : o;
  const long long o2 = wall ? o + s.plane : o - s.plane;
  rx_diff<CNT, STEP, R>(q == 3 ? s.dwdy : s.dwdx, (q == 3 ? s.dvdz : s.dudz) + oz, o, o2, wall || lid, q == 4, s.c, v);
}

// Lines per block of the plain x passes: about 128 threads.  Small blocks
// keep the barriers cheap and fill the SMs at small grids.
template <int R1, int R2> __host__ __device__ constexpr int rx_lines() { return cmax(1, 128 / cmax(R1, R2)); }

// z[k1 + R1 k2] (thread k1 of a line) -> the modes of the real transform;
// without HALF their factor 1/2 is in the loader's scale:
//   X[k] = a - i w b, X[N-k] = conj(a + i w b), a = z_k + conj z_{N-k},
//   b = z_k - conj z_{N-k}, w = exp(-2 pi i k / 2N)
template <typename A, int R1, int R2, bool HALF>
__device__ __forceinline__ void rx_split_store(const cplx<A>* v, const cplx<A>* S, int k1, const cplx<A>* rtw,
                                               cplx<A>* out) {
  using T2 = cplx<A>;
  constexpr int N = R1 * R2;
  auto put = [&](int k, T2 x) { out[k] = HALF ? cscale(x, FftConst<A>::half()) : x; };
#pragma unroll
  for (int k2 = 0; k2 < R2 / 2; ++k2) {
    const int k = k1 + R1 * k2;
    const T2 zk = v[k2];
    const T2 zm = (k2 == 0 && k1 == 0) ? zk : S[N - k];
    const T2 a = cadd_conj(zk, zm), b = csub_conj(zk, zm);
    const T2 wb = cmul(b, ldt(rtw + k));
    put(k, mkc(a.x + wb.y, a.y - wb.x));
    if (k2 > 0 || k1 > 0) put(N - k, mkc(a.x - wb.y, -a.y - wb.x));
  }
  if (k1 == 0) out[N / 2] = HALF ? cconj(v[R2 / 2]) : mkc(v[R2 / 2].x + v[R2 / 2].x, -(v[R2 / 2].y + v[R2 / 2].y));
}

// Forward x pass.  Bound by HBM at large grids (reads a field, writes its
// nx/2 modes); three barriers per block.
template <typename A, int R1, int R2, class Src>
__global__ void __launch_bounds__(rx_lines<R1, R2>() * cmax(R1, R2))
k_rx_fwd(RxGeom<A> g, Src src, cplx<A>* __restrict__ out) {
  using T2 = cplx<A>;
  constexpr int N = R1 * R2, T = cmax(R1, R2), L = rx_lines<R1, R2>(), RP = odd_up(R2), LS = cmax(R1 * RP, N + 1);
  __shared__ T2 S[L * LS];
  const int f = blockIdx.y, row0 = blockIdx.x * L, id = threadIdx.x;
  T2 v[T];
  {
    const int l = id / R2, n2 = id - l * R2, row = row0 + l;
    if (l < L && row < g.nrows) {
      const int li = g.fny.div(row), jy = row - li * g.nyrows;
      rx_load<R1, R2>(src, f, jy, li, n2, v);
      Dft<T2, false, R1>::run(v);
      T2* s = S + l * LS + n2;
      s[0] = v[0];
#pragma unroll
      for (int k1 = 1; k1 < R1; ++k1) s[k1 * RP] = mul_tw<false>(v[k1], g.tw + k1 * R2 + n2);
    }
  }
  __syncthreads();
  const int l = id / R1, k1 = id - l * R1, row = row0 + l;
  const bool on = l < L && row < g.nrows;
  T2* s = S + l * LS;
  if (on) {
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) v[n2] = s[k1 * RP + n2];
    Dft<T2, false, R2>::run(v);
  }
  __syncthreads();
  if (on) {
#pragma unroll
    for (int k2 = R2 / 2; k2 < R2; ++k2) s[k1 + R1 * k2] = v[k2];
  }
  __syncthreads();
  if (on) rx_split_store<A, R1, R2, false>(v, s, k1, g.rtw, out + f * g.fs + (long long)row * N);
}

// The 21 Lagrangian quantities (SrcLagrange::load2 forms all of them at a
// point): one row per block, its 21 lines in shared memory.
template <typename A, int R1, int R2, class Src>
__global__ void __launch_bounds__(21 * cmax(R1, R2)) k_rx_fwd21(RxGeom<A> g, Src src, cplx<A>* __restrict__ out) {
  using T2 = cplx<A>;
  constexpr int N = R1 * R2, T = cmax(R1, R2), RP = odd_up(R2), LS = cmax(R1 * RP, N + 1) | 1, NF = 21;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T2* S = reinterpret_cast<T2*>(smem_raw);
  const int row = blockIdx.x, id = threadIdx.x;
  const int li = g.fny.div(row), jy = row - li * g.nyrows;
  for (int n = id; n < N; n += NF * T) {
    T2 q[NF];
    src.load2(n, jy, li, q);
#pragma unroll
    for (int f = 0; f < NF; ++f) S[f * LS + n] = q[f];
  }
  __syncthreads();
  T2 v[T];
  {
    const int l = id / R2, n2 = id - l * R2;
    T2* s = S + l * LS + n2;
    if (l < NF) {
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) v[n1] = s[n1 * R2];
      Dft<T2, false, R1>::run(v);
    }
    __syncthreads();
    if (l < NF) {
      s[0] = v[0];
#pragma unroll
      for (int k1 = 1; k1 < R1; ++k1) s[k1 * RP] = mul_tw<false>(v[k1], g.tw + k1 * R2 + n2);
    }
  }
  __syncthreads();
  const int l = id / R1, k1 = id - l * R1;
  T2* s = S + l * LS;
  if (l < NF) {
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) v[n2] = s[k1 * RP + n2];
    Dft<T2, false, R2>::run(v);
  }
  __syncthreads();
  if (l < NF) {
#pragma unroll
    for (int k2 = R2 / 2; k2 < R2; ++k2) s[k1 + R1 * k2] = v[k2];
  }
  __syncthreads();
  if (l < NF) rx_split_store<A, R1, R2, true>(v, s, k1, g.rtw, out + l * g.fs + (long long)row * N);
}

// Row epilogues: CNT pairs of field f at n = n0 + j * STEP.  Every load is
// issued before the first store (the arrays may alias for the compiler).
template <int CNT, int STEP, typename R, int NF>
__device__ __forceinline__ void rx_store(const DstFields<R, NF>& d, int f, int jy, int li, int n0, const cplx<R>* v) {
  const int inst = d.im.inst(li), lv = li - inst * d.im.nli;
  R* p = pick(d.p, f) + inst * d.im.istr + (long long)(d.lev0 + lv * d.levstride) * d.plane + (long long)jy * d.ld + 2 * n0;
#pragma unroll
  for (int j = 0; j < CNT; ++j) *reinterpret_cast<cplx<R>*>(p + 2 * STEP * j) = v[j];
}
template <int CNT, int STEP, typename R, int WHICH>
__device__ __forceinline__ void rx_store(const DstDiv<R, WHICH>& d, int f, int jy, int li, int n0, const cplx<R>* v) {
  using C = cplx<R>;
  const int inst = d.im.inst(li);
  const int k = li - inst * d.im.nli + 1;
  const long long q = inst * d.im.istr + (long long)k * d.plane + (long long)jy * d.ld + 2 * n0;
  const int w = WHICH == 2 ? 2 : f;   // divtx, divty, divtz
  if (w < 2 && k > d.nz - 1) return;
  R* o = (w == 0 ? d.divtx : w == 1 ? d.divty : d.divtz) + q;
  const R* t = (w == 0 ? d.txz : w == 1 ? d.tyz : d.tzz) + q;
  const bool der = w < 2 || (k >= 2 && k <= d.nz - 1);
  const R* hi = w < 2 ? t + d.plane : t;
  const R* lo = w < 2 ? t : t - d.plane;
  C a[CNT], b[CNT];
#pragma unroll
  for (int j = 0; j < CNT; ++j) {
    a[j] = der ? *reinterpret_cast<const C*>(hi + 2 * STEP * j) : czero<C>();
    b[j] = der ? *reinterpret_cast<const C*>(lo + 2 * STEP * j) : czero<C>();
  }
#pragma unroll
  for (int j = 0; j < CNT; ++j) *reinterpret_cast<C*>(o + 2 * STEP * j) = cadd(v[j], cscale(csub(a[j], b[j]), d.inv_dz));
}
template <int CNT, int STEP, typename R, bool FUSED>
__device__ __forceinline__ void rx_store(const DstConvec<R, FUSED>& d, int f, int jy, int li, int n0, const cplx<R>* v) {
  using C = cplx<R>;
  const int inst = d.im.inst(li);
  const int k = li - inst * d.im.nli + 1;
  const long long q = inst * d.im.istr + (long long)k * d.plane + (long long)jy * d.ld + 2 * n0;
  const bool in = k <= d.nz - 1;
  if (f < 2 && !in) return;
  R* rhs = (f == 0 ? d.RHSx : f == 1 ? d.RHSy : d.RHSz) + q;
  if (!FUSED) {
#pragma unroll
    for (int j = 0; j < CNT; ++j) *reinterpret_cast<C*>(rhs + 2 * STEP * j) = v[j];
    return;
  }
  const double* c = d.sc + inst * SC_N;
  const R dtr = (R)c[SC_DT], t1r = (R)c[SC_T1], t2r = (R)c[SC_T2];
  const bool euler = (d.iflags[inst] & IF_EULER) != 0;
  const R* dv = (f == 0 ? d.divtx : f == 1 ? d.divty : d.divtz) + q;
  const R* fa = (f == 0 ? d.fxa : f == 1 ? d.fya : d.fza) + q;
  R* rf = (f == 0 ? d.RHSxf : f == 1 ? d.RHSyf : d.RHSzf) + q;
  R* u = (f == 0 ? d.u : f == 1 ? d.v : d.w) + q;
  const R mp = (f < 2 && d.use_mpf) ? (R)(f == 0 ? d.mpfx : d.mpfy) : (R)0;
  C x[CNT], o[CNT], y[CNT];
#pragma unroll
  for (int j = 0; j < CNT; ++j) {
    x[j] = *reinterpret_cast<const C*>(dv + 2 * STEP * j);
    o[j] = *reinterpret_cast<const C*>(rhs + 2 * STEP * j);
    y[j] = *reinterpret_cast<const C*>(u + 2 * STEP * j);
  }
  const bool turb = d.turbines && in;
#pragma unroll
  for (int j = 0; j < CNT; ++j) {
    C n = mkc(-v[j].x - x[j].x, -v[j].y - x[j].y);
    if (f < 2 && d.use_mpf) n = mkc(n.x + mp, n.y + mp);
    if (turb) n = cadd(n, *reinterpret_cast<const C*>(fa + 2 * STEP * j));
    const C old = euler ? n : o[j];
    *reinterpret_cast<C*>(rf + 2 * STEP * j) = old;
    *reinterpret_cast<C*>(rhs + 2 * STEP * j) = n;
    *reinterpret_cast<C*>(u + 2 * STEP * j) =
        mkc(y[j].x + dtr * (t1r * n.x + t2r * old.x), y[j].y + dtr * (t1r * n.y + t2r * old.y));
  }
}
template <int CNT, int STEP, typename R, bool FUSED>
__device__ __forceinline__ void rx_store(const DstPress<R, FUSED>& d, int f, int jy, int li, int n0, const cplx<R>* v) {
  using C = cplx<R>;
  const int inst = d.im.inst(li);
  const int k = li - inst * d.im.nli + 1;
  const long long q = inst * d.im.istr + (long long)k * d.plane + (long long)jy * d.ld + 2 * n0;
  if (f == 0 || !FUSED) {
    R* p = (f == 0 ? d.p : f == 1 ? d.dpdx : d.dpdy) + q;
#pragma unroll
    for (int j = 0; j < CNT; ++j) *reinterpret_cast<C*>(p + 2 * STEP * j) = v[j];
    return;
  }
  const double* c = d.sc + inst * SC_N;
  const R dtr = (R)c[SC_DT], t1r = (R)c[SC_T1];
  R* rhs = (f == 1 ? d.RHSx : d.RHSy) + q;
  R* u = (f == 1 ? d.u : d.v) + q;
  C r[CNT], y[CNT];
#pragma unroll
  for (int j = 0; j < CNT; ++j) {
    r[j] = *reinterpret_cast<const C*>(rhs + 2 * STEP * j);
    y[j] = *reinterpret_cast<const C*>(u + 2 * STEP * j);
  }
#pragma unroll
  for (int j = 0; j < CNT; ++j) {
    *reinterpret_cast<C*>(rhs + 2 * STEP * j) = csub(r[j], v[j]);
    *reinterpret_cast<C*>(u + 2 * STEP * j) = mkc(y[j].x + dtr * (-t1r * v[j].x), y[j].y + dtr * (-t1r * v[j].y));
  }
}

// The modes of a real line -> z[k], thread n2's inputs k = n1 R2 + n2 of the
// inverse transform: z_k = (x_k + conj x_{N-k}) + i conj(w) (x_k - conj
// x_{N-k}).  Modes from kz on (K for all of them) are zero and not read.
template <typename A, int R1, int R2>
__device__ __forceinline__ void rx_merge_load(const cplx<A>* in, int kz, int n2, const cplx<A>* rtw, cplx<A>* v) {
  using T2 = cplx<A>;
  constexpr int N = R1 * R2;
  T2 m[R1];
#pragma unroll
  for (int n1 = 0; n1 < R1; ++n1) {
    const int k = n1 * R2 + n2, km = N - k;
    v[n1] = k < kz ? in[k] : czero<T2>();
    m[n1] = km < kz ? in[km] : czero<T2>();   // km = N: the Nyquist mode, zero
  }
#pragma unroll
  for (int n1 = 0; n1 < R1; ++n1) {
    const T2 a = cadd_conj(v[n1], m[n1]), b = csub_conj(v[n1], m[n1]);
    const T2 c = cmulconj(b, ldt(rtw + n1 * R2 + n2));
    v[n1] = mkc(a.x - c.y, a.y + c.x);
  }
}

// Inverse x pass with the row epilogue on registers: one barrier per block.
template <typename A, int R1, int R2, class Dst>
__global__ void __launch_bounds__(rx_lines<R1, R2>() * cmax(R1, R2))
k_rx_inv(RxGeom<A> g, const cplx<A>* __restrict__ in, Dst dst) {
  using T2 = cplx<A>;
  constexpr int N = R1 * R2, T = cmax(R1, R2), L = rx_lines<R1, R2>(), RP = odd_up(R2), LS = R1 * RP;
  __shared__ T2 S[L * LS];
  const int f = blockIdx.y, row0 = blockIdx.x * L, id = threadIdx.x;
  T2 v[T];
  {
    const int l = id / R2, n2 = id - l * R2, row = row0 + l;
    if (l < L && row < g.nrows) {
      rx_merge_load<A, R1, R2>(in + f * g.fs + (long long)row * N, N, n2, g.rtw, v);
      Dft<T2, true, R1>::run(v);
      T2* s = S + l * LS + n2;
      s[0] = v[0];
#pragma unroll
      for (int k1 = 1; k1 < R1; ++k1) s[k1 * RP] = mul_tw<true>(v[k1], g.tw + k1 * R2 + n2);
    }
  }
  __syncthreads();
  const int l = id / R1, k1 = id - l * R1, row = row0 + l;
  if (l < L && row < g.nrows) {
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) v[n2] = S[l * LS + k1 * RP + n2];
    Dft<T2, true, R2>::run(v);
    const int li = g.fny.div(row), jy = row - li * g.nyrows;
    rx_store<R2, R1>(dst, f, jy, li, k1, v);
  }
}

// The 42 test-filtered fields of one row and the pointwise Lagrangian model
// (DstLagrange reads all of them at a point): two rounds of 21 lines.
template <typename A, int R1, int R2, class Dst>
__global__ void __launch_bounds__(21 * cmax(R1, R2)) k_rx_inv42(RxGeom<A> g, const cplx<A>* __restrict__ in, Dst dst) {
  using T2 = cplx<A>;
  constexpr int N = R1 * R2, T = cmax(R1, R2), RP = odd_up(R2), LS = cmax(R1 * RP, N) | 1, NL = 21;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T2* S = reinterpret_cast<T2*>(smem_raw);
  const int row = blockIdx.x, id = threadIdx.x;
#pragma unroll 1
  for (int p = 0; p < 2; ++p) {
    T2 v[T];
    {
      const int l = id / R2, n2 = id - l * R2;
      if (l < NL) {
        rx_merge_load<A, R1, R2>(in + (2 * l + p) * g.fs + (long long)row * N, p ? g.kz1 : g.kz0, n2, g.rtw, v);
        Dft<T2, true, R1>::run(v);
        T2* s = S + (2 * l + p) * LS + n2;
        s[0] = v[0];
#pragma unroll
        for (int k1 = 1; k1 < R1; ++k1) s[k1 * RP] = mul_tw<true>(v[k1], g.tw + k1 * R2 + n2);
      }
    }
    __syncthreads();
    const int l = id / R1, k1 = id - l * R1;
    T2* s = S + (2 * l + p) * LS;
    if (l < NL) {
#pragma unroll
      for (int n2 = 0; n2 < R2; ++n2) v[n2] = s[k1 * RP + n2];
      Dft<T2, true, R2>::run(v);
    }
    __syncthreads();
    if (l < NL) {
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) s[k1 + R1 * k2] = v[k2];
    }
  }
  __syncthreads();
  const int li = g.fny.div(row), jy = row - li * g.nyrows;
  const A* Z = reinterpret_cast<const A*>(S);
  for (int i = id; i < 2 * N; i += NL * T) {
    typename Dst::Real vals[2 * NL];
#pragma unroll
    for (int f = 0; f < 2 * NL; ++f) vals[f] = Z[2 * f * LS + i];
    dst.store(jy, li, i, vals);
  }
}

// ---------------------------------------------------------------------------
// y passes: eight adjacent kx columns per block (64 or 128 contiguous bytes
// per row), max(R1, R2, 3 R2 / 2) threads per column.  The modes stay in the
// thread that holds them between the forward and the inverse transform, so
// the spectral operator costs no exchange: one barrier per transform.
// ---------------------------------------------------------------------------
constexpr int kYC = 8;   // columns per block

template <typename A, typename InT, typename OutT>
struct RyArgs {
  const InT* in;
  OutT* out;
  long long in_fs, out_fs;   // elements between fields
  int K, lh;
  int nli, in_inst_levels, in_lev0, in_levstride;
  FastDiv fnli;
  const cplx<A>* twn;   // of ny: twn[k1 * R2 + n2]
  const cplx<A>* twm;   // of 3 ny / 2: twm[k1 * S2 + n2]
  const A *kxw, *kyw, *G1, *G2;
  int zero1, zero2;          // first columns past the G1 / G2 cutoffs
  int ia[3], ib[3];          // k_ry_div: the input fields of each output
  A gs;                      // k_ry_test with one filter: factor of G1
  // k_ry_vpad: 1/dz, the bottom condition, its velocity, and the wall law's
  // constants per instance (wall_equilibrium)
  A inv_dz, ubot, lbc_scale;
  int lbc;
  const double* wall_i;
  __device__ __forceinline__ long long plane_in(int li) const {
    const int inst = fnli.div(li), lv = li - inst * nli;
    return (long long)inst * in_inst_levels + in_lev0 + lv * in_levstride;
  }
};

// Forward: thread t < R2 holds x[n1 R2 + t] in v[n1]; after it thread t < R1
// holds X[t + R1 k2] in v[k2].  W is free again after the next barrier.
template <typename T2, int R1, int R2>
__device__ __forceinline__ void ry_fwd(T2* v, T2* W, const T2* tw, int t, int c) {
  constexpr int RP = odd_up(R2);
  if (t < R2) {
    Dft<T2, false, R1>::run(v);
    T2* w = W + t * kYC + c;
    w[0] = v[0];
#pragma unroll
    for (int k1 = 1; k1 < R1; ++k1) w[k1 * RP * kYC] = mul_tw<false>(v[k1], tw + k1 * R2 + t);
  }
  __syncthreads();
  if (t < R1) {
    const T2* w = W + t * RP * kYC + c;
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) v[n2] = w[n2 * kYC];
    Dft<T2, false, R2>::run(v);
  }
}
// Inverse: thread t < R1 holds Y[t + R1 k2] in v[k2]; after it thread t < R2
// holds y[n1 R2 + t] in v[n1].
template <typename T2, int R1, int R2>
__device__ __forceinline__ void ry_inv(T2* v, T2* W, const T2* tw, int t, int c) {
  constexpr int RP = odd_up(R2);
  if (t < R1) {
    Dft<T2, true, R2>::run(v);
    T2* w = W + t * RP * kYC + c;
    w[0] = v[0];
#pragma unroll
    for (int n2 = 1; n2 < R2; ++n2) w[n2 * kYC] = mul_tw<true>(v[n2], tw + t * R2 + n2);
  }
  __syncthreads();
  if (t < R2) {
    const T2* w = W + t * kYC + c;
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) v[k1] = w[k1 * RP * kYC];
    Dft<T2, true, R1>::run(v);
  }
}
template <int R1, int R2> __host__ __device__ constexpr int ry_elems() { return R1 * odd_up(R2) * kYC; }

template <int CNT, typename T2>
__device__ __forceinline__ void ry_load(const T2* p, int step, bool live, T2* v) {
#pragma unroll
  for (int j = 0; j < CNT; ++j) v[j] = live ? p[j * step] : czero<T2>();
}
template <int CNT, typename T2>
__device__ __forceinline__ void ry_store(T2* p, int step, bool live, const T2* v) {
  if (!live) return;
#pragma unroll
  for (int j = 0; j < CNT; ++j) p[j * step] = v[j];
}
// the pressure's FP64 spectra to and from FP32 transforms
template <int CNT>
__device__ __forceinline__ void ry_load(const double2* p, int step, bool live, float2* v) {
  double2 d[CNT];
  bool odd = false;
#pragma unroll
  for (int j = 0; j < CNT; ++j) d[j] = live ? p[j * step] : make_double2(1.0, 1.0);
#pragma unroll
  for (int j = 0; j < CNT; ++j) v[j] = make_float2(narrow_fast(d[j].x, odd), narrow_fast(d[j].y, odd));
  if (odd) {
#pragma unroll
    for (int j = 0; j < CNT; ++j) v[j] = make_float2((float)d[j].x, (float)d[j].y);
  }
}
template <int CNT>
__device__ __forceinline__ void ry_store(double2* p, int step, bool live, const float2* v) {
  if (!live) return;
  double2 d[CNT];
  bool odd = false;
#pragma unroll
  for (int j = 0; j < CNT; ++j) d[j] = make_double2(widen_fast(v[j].x, odd), widen_fast(v[j].y, odd));
  if (odd) {
#pragma unroll
    for (int j = 0; j < CNT; ++j) d[j] = make_double2((double)v[j].x, (double)v[j].y);
  }
#pragma unroll
  for (int j = 0; j < CNT; ++j) p[j * step] = d[j];
}
// v[k2] *= i ky of row t + R1 k2 (zero in the Nyquist row of the table)
template <typename A, int R1, int R2>
__device__ __forceinline__ void ry_iky(const A* kyw, int t, cplx<A>* v) {
  if (t < R1) {
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) v[k2] = mul_ik(kyw[t + R1 * k2], v[k2]);
  }
}

#define LESGO_RY_HEAD(T)                                                             \
  using T2 = cplx<A>;                                                                \
  const int c = threadIdx.x & (kYC - 1), t = threadIdx.x / kYC;                      \
  const int kx = blockIdx.x * kYC + c, li = blockIdx.y, f = blockIdx.z;              \
  const bool live = kx < a.K;                                                        \
  const long long pin = a.plane_in(li);                                              \
  extern __shared__ __align__(16) unsigned char smem_raw[];                          \
  T2* W0 = reinterpret_cast<T2*>(smem_raw);                                          \
  (void)W0; (void)pin; (void)live; (void)f

// filt_da: x -> the filtered x, i kx of it, i ky of it (outputs 3 f, 3 f + 1,
// 3 f + 2).  The first two need no inverse transform: with the Nyquist row
// zeroed, forward and inverse along y give ny x(y) - (-1)^y X[ny/2].
template <typename A, int R1, int R2>
__global__ void __launch_bounds__(kYC * cmax(R1, R2)) k_ry_filt(RyArgs<A, cplx<A>, cplx<A>> a) {
  LESGO_RY_HEAD();
  constexpr int N = R1 * R2, E = ry_elems<R1, R2>();
  T2* W1 = W0 + E;
  T2* ny = W1 + E;
  const T2* src = a.in + f * a.in_fs + pin * N * a.K + t * a.K + kx;
  T2 v[cmax(R1, R2)];
  if (t < R2) ry_load<R1>(src, R2 * a.K, live, v);
  ry_fwd<T2, R1, R2>(v, W0, a.twn, t, c);
  if (t == 0) ny[c] = v[R2 / 2];
  ry_iky<A, R1, R2>(a.kyw, t, v);
  ry_inv<T2, R1, R2>(v, W1, a.twn, t, c);
  if (t < R2 && live) {
    T2* d = a.out + (3 * f) * a.out_fs + (long long)li * N * a.K + t * a.K + kx;
    ry_store<R1>(d + 2 * a.out_fs, R2 * a.K, true, v);
    const T2 s = (t & 1) ? mkc(-ny[c].x, -ny[c].y) : ny[c];
    const A k = a.kxw[kx], n = cvt<A>((float)N);
    ry_load<R1>(src, R2 * a.K, true, v);
#pragma unroll
    for (int j = 0; j < R1; ++j) {
      const T2 x = csub(cscale(v[j], n), s);
      d[j * R2 * a.K] = x;
      d[a.out_fs + j * R2 * a.K] = mul_ik(k, x);
    }
  }
}

// Stress divergence: output f = i kx p + i ky q of two input fields.  Only q
// is transformed; the i kx term is added after the inverse transform as
// above, with the Nyquist component of p summed directly.
template <typename A, int R1, int R2>
__global__ void __launch_bounds__(kYC * cmax(R1, R2)) k_ry_div(RyArgs<A, cplx<A>, cplx<A>> a) {
  LESGO_RY_HEAD();
  constexpr int N = R1 * R2, E = ry_elems<R1, R2>();
  T2* W1 = W0 + E;
  T2* sum = W1 + E;   // R2 partial sums per column
  const T2* pp = a.in + pick(a.ia, f) * a.in_fs + pin * N * a.K + t * a.K + kx;
  const T2* qq = a.in + pick(a.ib, f) * a.in_fs + pin * N * a.K + t * a.K + kx;
  T2 v[cmax(R1, R2)];
  if (t < R2) {
    ry_load<R1>(pp, R2 * a.K, live, v);
    T2 s = v[0];
#pragma unroll
    for (int j = 1; j < R1; ++j) s = cadd(s, v[j]);
    sum[t * kYC + c] = (t & 1) ? mkc(-s.x, -s.y) : s;
    ry_load<R1>(qq, R2 * a.K, live, v);
  }
  ry_fwd<T2, R1, R2>(v, W0, a.twn, t, c);
  ry_iky<A, R1, R2>(a.kyw, t, v);
  ry_inv<T2, R1, R2>(v, W1, a.twn, t, c);
  if (t < R2 && live) {
    T2 s = sum[c];
#pragma unroll
    for (int j = 1; j < R2; ++j) s = cadd(s, sum[j * kYC + c]);
    if (t & 1) s = mkc(-s.x, -s.y);
    const A k = a.kxw[kx], n = cvt<A>((float)N);
    T2* d = a.out + f * a.out_fs + (long long)li * N * a.K + t * a.K + kx;
    T2 x[R1];
    ry_load<R1>(pp, R2 * a.K, true, x);
#pragma unroll
    for (int j = 0; j < R1; ++j) {
      const T2 y = csub(cscale(x[j], n), s);
      d[j * R2 * a.K] = add_ik(v[j], k, y);
    }
  }
}

// The R2 modes of a thread of ny rows as the 3 R2 / 2 of 3 ny / 2 rows: the
// upper half moves up, the Nyquist row and the new ones are zero.
template <typename T2, int R2>
__device__ __forceinline__ void ry_relabel(T2* v, int t) {
#pragma unroll
  for (int j = R2 - 1; j >= R2 / 2; --j) v[j + R2 / 2] = v[j];
#pragma unroll
  for (int j = R2 / 2; j < R2; ++j) v[j] = czero<T2>();
  if (t == 0) v[R2] = czero<T2>();
}

// 3/2 padding: ny rows -> 3 ny / 2 rows (padd, fft.f90:43-72).
template <typename A, int R1, int R2>
__global__ void __launch_bounds__(kYC * cmax(R1, 3 * R2 / 2)) k_ry_pad(RyArgs<A, cplx<A>, cplx<A>> a) {
  LESGO_RY_HEAD();
  constexpr int N = R1 * R2, S2 = 3 * R2 / 2, M = R1 * S2;
  T2* W1 = W0 + ry_elems<R1, R2>();
  T2 v[cmax(R1, S2)];
  if (t < R2) ry_load<R1>(a.in + f * a.in_fs + pin * N * a.K + t * a.K + kx, R2 * a.K, live, v);
  ry_fwd<T2, R1, R2>(v, W0, a.twn, t, c);
  ry_relabel<T2, R2>(v, t);
  ry_inv<T2, R1, S2>(v, W1, a.twm, t, c);
  if (t < S2) ry_store<R1>(a.out + f * a.out_fs + (long long)li * M * a.K + t * a.K + kx, S2 * a.K, live, v);
}

// 3/2 padding of u, v, w and of the vorticity formed from their modes
// (convec.f90:71-168): o3 = i kx v - i ky u, and with the staggered
// differences o1 = i ky w - (v(k) - v(k-1)) / dz, o2 = (u(k) - u(k-1)) / dz -
// i kx w; at the bottom wall w is averaged over the first two levels and the
// wall's du/dz, dv/dz are multiples of u, v (less the wall's velocity), so
// they too stay in the modes.  The inputs are the x spectra of u, v, w alone:
// the gradients are not transformed again, and the convective term does not
// wait for them.  (Level nz's o1 and o2 are not used: no product reads them.)
// blockIdx.z: 0 -> u, w, o2; 1 -> v, o3, o1.
// 34.5 us at 128^3 in the mixed form (unique bytes 15) against 21 for the
// vorticity's own forward x pass and 35.6 for the padding of six spectra; the
// step, which no longer waits for the column sweep here, 507 -> 469 us.
template <typename A, int R1, int R2>
__global__ void __launch_bounds__(kYC * cmax(R1, 3 * R2 / 2)) k_ry_vpad(RyArgs<A, cplx<A>, cplx<A>> a) {
  LESGO_RY_HEAD();
  constexpr int N = R1 * R2, S2 = 3 * R2 / 2, M = R1 * S2;
  T2* W1 = W0 + ry_elems<R1, R2>();
  const int inst = a.fnli.div(li), k = li - inst * a.nli + 1;
  const bool wall = k == 1;
  const int step = R2 * a.K;
  const T2* src = a.in + pin * N * a.K + t * a.K + kx;
  const long long lev = (long long)N * a.K;
  T2* dst = a.out + (long long)li * M * a.K + t * a.K + kx;
  const A kxv = live ? a.kxw[kx] : (A)0;
  // the wall's gradient over velocity, and the velocity that its mean mode loses
  const A ws = a.lbc == 2 ? (A)a.wall_i[2 * inst + 1] : a.lbc_scale;
  const A wu = (wall && a.lbc == 1 && kx == 0 && t == 0) ? a.ubot : (A)0;
  T2 v[cmax(R1, S2)];
  auto fwd = [&](int q, int up) {   // modes of field q (0 u, 1 v, 2 w), `up` levels above this one
    if (t < R2) ry_load<R1>(src + q * a.in_fs + up * lev, step, live, v);
    ry_fwd<T2, R1, R2>(v, W0, a.twn, t, c);
  };
  auto put = [&](int o) {
    ry_relabel<T2, R2>(v, t);
    ry_inv<T2, R1, S2>(v, W1, a.twm, t, c);
    if (t < S2) ry_store<R1>(dst + o * a.out_fs, S2 * a.K, live, v);
  };
  // i kxv a + b, and i ky of mode (t, j) times a
  auto ikx = [&](T2 x) { return mkc(-kxv * x.y, kxv * x.x); };
  auto iky = [&](T2 x, int j) {
    const A w = t < R1 ? a.kyw[t + R1 * j] : (A)0;
    return mkc(-w * x.y, w * x.x);
  };
  const A h = FftConst<A>::half();
  T2 p[R2], r[R2];
  auto keep = [&](T2* x) {
#pragma unroll
    for (int j = 0; j < R2; ++j) x[j] = v[j];
  };
  if (f == 0) {
    fwd(0, 0);
    keep(p);   // u
    put(0);
    fwd(2, 0);
    keep(r);   // w
    put(2);
    fwd(wall ? 2 : 0, wall ? 1 : -1);   // w above, or u below
#pragma unroll
    for (int j = 0; j < R2; ++j) {
      if (!wall) v[j] = csub(cscale(csub(p[j], v[j]), a.inv_dz), ikx(r[j]));
      else if (a.lbc == 0) v[j] = czero<T2>();
      else v[j] = csub(cscale(mkc(j == 0 ? p[j].x - wu : p[j].x, p[j].y), ws), ikx(cscale(cadd(r[j], v[j]), h)));
    }
    put(4);
  } else {
    fwd(1, 0);
    keep(p);   // v
    put(1);
    fwd(0, 0);
#pragma unroll
    for (int j = 0; j < R2; ++j) v[j] = csub(ikx(p[j]), iky(v[j], j));
    put(5);
    fwd(wall ? 2 : 1, wall ? 1 : -1);   // w above, or v below
    keep(r);
    __syncthreads();   // two forward transforms in a row share W0
    fwd(2, 0);
#pragma unroll
    for (int j = 0; j < R2; ++j) {
      if (!wall) v[j] = csub(iky(v[j], j), cscale(csub(p[j], r[j]), a.inv_dz));
      else if (a.lbc == 0) v[j] = czero<T2>();
      else v[j] = csub(iky(cscale(cadd(v[j], r[j]), h), j), cscale(p[j], ws));
    }
    put(3);
  }
}

// Truncation: 3 ny / 2 rows -> ny rows (unpadd, fft.f90:75-99).
template <typename A, int R1, int R2>
__global__ void __launch_bounds__(kYC * cmax(R1, 3 * R2 / 2)) k_ry_unpad(RyArgs<A, cplx<A>, cplx<A>> a) {
  LESGO_RY_HEAD();
  constexpr int N = R1 * R2, S2 = 3 * R2 / 2, M = R1 * S2;
  T2* W1 = W0 + ry_elems<R1, S2>();
  T2 v[cmax(R1, S2)];
  if (t < S2) ry_load<R1>(a.in + f * a.in_fs + pin * M * a.K + t * a.K + kx, S2 * a.K, live, v);
  ry_fwd<T2, R1, S2>(v, W0, a.twm, t, c);
  if (t < R1) {
#pragma unroll
    for (int j = R2 / 2; j < R2; ++j) v[j] = v[j + R2 / 2];
    if (t == 0) v[R2 / 2] = czero<T2>();
  }
  ry_inv<T2, R1, R2>(v, W1, a.twn, t, c);
  if (t < R2) ry_store<R1>(a.out + f * a.out_fs + (long long)li * N * a.K + t * a.K + kx, R2 * a.K, live, v);
}

// Forward only, to FP64 spectra (the pressure's right-hand sides).
template <typename A, int R1, int R2>
__global__ void __launch_bounds__(kYC * cmax(R1, R2)) k_ry_spec(RyArgs<A, cplx<A>, double2> a) {
  LESGO_RY_HEAD();
  constexpr int N = R1 * R2;
  T2 v[cmax(R1, R2)];
  if (t < R2) ry_load<R1>(a.in + f * a.in_fs + pin * N * a.K + t * a.K + kx, R2 * a.K, live, v);
  ry_fwd<T2, R1, R2>(v, W0, a.twn, t, c);
  if (t < R1) {
    if (t == 0) v[R2 / 2] = czero<T2>();
    ry_store<R2>(a.out + f * a.out_fs + (long long)li * N * a.K + t * a.K + kx, R1 * a.K, live, v);
  }
}

// Inverse only: P -> p (GRAD: and i kx p, i ky p).
template <typename A, int R1, int R2, bool GRAD>
__global__ void __launch_bounds__(kYC * cmax(R1, R2)) k_ry_phys(RyArgs<A, double2, cplx<A>> a) {
  LESGO_RY_HEAD();
  constexpr int N = R1 * R2;
  const double2* src = a.in + f * a.in_fs + pin * N * a.K + t * a.K + kx;
  T2* d = a.out + f * a.out_fs + (long long)li * N * a.K + t * a.K + kx;
  T2 v[cmax(R1, R2)];
  if (t < R1) {
    ry_load<R2>(src, R1 * a.K, live, v);
    if (t == 0) v[R2 / 2] = czero<T2>();
  }
  ry_inv<T2, R1, R2>(v, W0, a.twn, t, c);
  if (t < R2 && live) {
    ry_store<R1>(d, R2 * a.K, true, v);
    if constexpr (GRAD) {
      const A k = a.kxw[kx];
#pragma unroll
      for (int j = 0; j < R1; ++j) d[a.out_fs + j * R2 * a.K] = mul_ik(k, v[j]);
    }
  }
  if constexpr (GRAD) {
    if (t < R1) ry_load<R2>(src, R1 * a.K, live, v);
    ry_iky<A, R1, R2>(a.kyw, t, v);
    ry_inv<T2, R1, R2>(v, W0 + ry_elems<R1, R2>(), a.twn, t, c);
    if (t < R2) ry_store<R1>(d + 2 * a.out_fs, R2 * a.K, live, v);
  }
}

// Test filters: x -> G1 x (and, BOTH, G2 x).  Columns past a cutoff are not
// written with BOTH (the consumer does not read them) and written as zeros
// without.
template <typename A, int R1, int R2, bool BOTH>
__global__ void __launch_bounds__(kYC * cmax(R1, R2)) k_ry_test(RyArgs<A, cplx<A>, cplx<A>> a) {
  LESGO_RY_HEAD();
  constexpr int N = R1 * R2, E = ry_elems<R1, R2>();
  const int kx0 = blockIdx.x * kYC;
  T2* d = a.out + (BOTH ? 2 * f : f) * a.out_fs + (long long)li * N * a.K + t * a.K + kx;
  T2 v[cmax(R1, R2)];
  if (kx0 >= a.zero1) {   // zero2 <= zero1
    if constexpr (!BOTH) {
      if (t < R2) {
#pragma unroll
        for (int j = 0; j < R1; ++j) v[j] = czero<T2>();
        ry_store<R1>(d, R2 * a.K, live, v);
      }
    }
    return;
  }
  if (t < R2) ry_load<R1>(a.in + f * a.in_fs + pin * N * a.K + t * a.K + kx, R2 * a.K, live, v);
  ry_fwd<T2, R1, R2>(v, W0, a.twn, t, c);
  T2 x[R2];
  auto times = [&](const A* G) {
    if (t < R1) {
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) {
        const A w = live ? G[(t + R1 * k2) * a.lh + kx] : FftConst<A>::zero();
        v[k2] = cscale(x[k2], BOTH ? w : w * a.gs);
      }
    }
  };
#pragma unroll
  for (int k2 = 0; k2 < R2; ++k2) x[k2] = v[k2];
  times(a.G1);
  ry_inv<T2, R1, R2>(v, W0 + E, a.twn, t, c);
  if (t < R2) ry_store<R1>(d, R2 * a.K, live, v);
  if constexpr (BOTH) {
    if (kx0 >= a.zero2) return;
    times(a.G2);
    ry_inv<T2, R1, R2>(v, W0, a.twn, t, c);
    if (t < R2) ry_store<R1>(d + a.out_fs, R2 * a.K, live, v);
  }
}

}  // namespace lesgo
