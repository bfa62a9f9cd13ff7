// The convective term's x-rows on the 3/2 grid (convec.f90:170-255) with the
// transforms in registers: what k_convec_rows does with run-time radix
// stages in shared memory.
//
// A block owns L rows of one instance and marches up a chunk of levels.  The
// thread (row, k1 < R1) gets the c2r results u, v, w, o1, o2, o3 of a level
// at its R2 pairs n = k1 + R1 j, forms the products in registers, and the
// r2c transforms of the products start from those same registers (their
// first step runs over j).  The products at level k need w, o1 and o2 of
// level k + 1, and u and v of level k - 1: carried from level to level are
// the two sums that level k + 1 completes (registers) and u, v (the thread's
// own places in shared memory: no barrier).
//
// The six fields are transformed three at a time and the three products
// together, so that one barrier serves three exchanges (four barriers a
// level) and the step with R2 threads per line is spread over all threads.
// The spectra of the next three fields come in by bulk copies under the
// arithmetic of the current ones.
//
// Bound by the latency of shared memory at about nine warps per SM (issue 39
// % active, ncu): each row holds 8 KB of exchange lines and copies.  Mixed
// form, us per launch against k_convec_rows (and the 9 spectra at the copy
// bandwidth): 128^3 70 (141; 17), 256x256x192 353 (841; 101), 6 x 108x72x30
// 68 (11), 48^3 16.5 (18.5; 1).  Slower where few blocks leave the longer
// chain of a level exposed, in a step that is shorter all the same: one
// instance of 64x16x32 17.4 (14.3), of 64x48x24 17.8 (15.1), their whole
// steps 95.6 us (152) and 82 (177).  Measured and dropped: one field per
// exchange with 12 barriers a level and the spectra read in place (95 us at
// 128^3, 855 us at 256x256x192).
#pragma once
#include "bulk_copy.cuh"
#include "rfft_core.cuh"

namespace lesgo {

template <typename A>
struct RxRowsGeom {
  int ny2, nz, cz;           // rows per level, levels 1..nz, levels per block
  long long in_fs, out_fs;   // complex elements between fields
  const cplx<A>* tw;         // tw[k1 * R2 + n2] of H = R1 R2 = 3 nx / 4
  const cplx<A>* rtw;        // rtw[k] = exp(-2 pi i k / (2 H))
  int* err;                  // set to 1 when a copy wait gives up
};

// pairs of real values: products and sums by component
template <typename T2> __device__ __forceinline__ T2 pmul(T2 a, T2 b) { return mkc(a.x * b.x, a.y * b.y); }
template <> __device__ __forceinline__ float2 pmul<float2>(float2 a, float2 b) { return __fmul2_rn(a, b); }
template <typename T2> __device__ __forceinline__ T2 pfma(T2 a, T2 b, T2 c) { return mkc(a.x * b.x + c.x, a.y * b.y + c.y); }
template <> __device__ __forceinline__ float2 pfma<float2>(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
template <typename T2> __device__ __forceinline__ T2 pneg(T2 a) { return mkc(-a.x, -a.y); }

// an exchanged line: R1 x R2 padded to an odd stride either way, or H values in order
template <int R1, int R2> __host__ __device__ constexpr int rows_ls() {
  return cmax(cmax(R1 * odd_up(R2), R2 * odd_up(R1)), R1 * R2 + 1);
}
// complex elements of a row: the copied spectra of three fields, two buffers
// of three exchanged lines, u and v; and of a block besides: the twiddles
// and the barrier
template <int R1, int R2> __host__ __device__ constexpr int rows_per_row() { return 6 * rows_ls<R1, R2>() + 4 * R1 * R2; }
template <int R1, int R2> __host__ __device__ constexpr int rows_besides() { return 3 * R1 * R2 + 2; }
// Rows per block: about 100 threads and a third of an SM's shared memory (at
// H = 96, eight rows and three blocks per SM 66 us against nine rows and two
// blocks 76 us, one 128^3 instance).
constexpr int kRowsBytes = 75000;
template <typename A, int R1, int R2> __host__ __device__ constexpr int rows_lines() {
  constexpr int fit = (kRowsBytes / (int)sizeof(cplx<A>) - rows_besides<R1, R2>()) / rows_per_row<R1, R2>();
  return cmax(1, fit < 112 / R1 ? fit : 112 / R1);
}

template <typename A, int R1, int R2>
__global__ void __launch_bounds__(rows_lines<A, R1, R2>() * R1, 3)
k_rx_rows(RxRowsGeom<A> g, const cplx<A>* __restrict__ in, cplx<A>* __restrict__ out, A c) {
  using T2 = cplx<A>;
  static_assert(R1 % 3 == 0, "the padded modes are whole inputs of the first DFT");
  constexpr int H = R1 * R2, K = 2 * H / 3, L = rows_lines<A, R1, R2>(), LS = rows_ls<R1, R2>();
  constexpr int RP = odd_up(R2), QP = odd_up(R1), NT = L * R1, U = 3 * L * R2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T2* stage = reinterpret_cast<T2*>(smem_raw);     // [3][L][K]
  T2* X0 = stage + 3 * L * K;           // [3][L][LS]
  T2* X1 = X0 + 3 * L * LS;
  T2* tw = X1 + 3 * L * LS;                        // [k1][n2]
  T2* twt = tw + H;                                // [n2][k1]: each step reads neighbouring entries across threads
  T2* rtw = twt + H;
  T2* uv = rtw + H + threadIdx.x;                  // this thread's u and v of the last level, [2][R2] of stride NT
  uint64_t* bar = reinterpret_cast<uint64_t*>(rtw + H + 2 * R2 * NT);
  const int id = threadIdx.x;
  const int row0 = blockIdx.x * L, inst = blockIdx.z;
  const int rows = min(L, g.ny2 - row0);
  const int k0 = 1 + blockIdx.y * g.cz, k1e = min(k0 + g.cz, g.nz + 1);   // levels k0 .. k1e-1
  const int lb = id / R1, kb = id - lb * R1;
  const bool onb = lb < rows;
  auto lrow = [&](int lev) { return ((long long)inst * g.nz + (lev - 1)) * g.ny2 + row0; };
  const int top = g.nz - 1;   // the last level with products
  const int first = k0 >= 2 && k0 <= top ? k0 - 1 : k0, last = min(k1e, top);

  // Fields of triple t at a level, three bits each (7: not needed there):
  // o1, v, o2, then u, w, o3; below the chunk u and v only, above it w, o1
  // and o2 only.
  auto fields = [&](int k, int t) {
    const bool below = k < k0, above = k >= k1e;
    if (t == 0) return below ? 0717 : above ? 0473 : 0413;
    return below ? 0770 : above ? 0727 : 0520;
  };
  // thread 0: bulk copies of a triple's rows (rows x K modes per field,
  // contiguous) behind the barrier
  auto prefetch = [&](int k, int t) {
    if (id != 0 || k > last) return;
    const int m = fields(k, t);
    const unsigned bytes = (unsigned)(rows * K * sizeof(T2));
    int n = 0;
    for (int i = 0; i < 3; ++i) n += ((m >> (3 * i)) & 7) != 7;
    mbar_arrive_expect_tx(bar, bytes * n);
    for (int i = 0; i < 3; ++i) {
      const int f = (m >> (3 * i)) & 7;
      if (f != 7) bulk_g2s(stage + i * L * K, in + f * g.in_fs + lrow(k) * K, bytes, bar);
    }
  };
  if (id == 0) {
    mbar_init(bar, 1);
    mbar_init_fence();
  }
  for (int n = id; n < H; n += NT) {
    const int q = n / R2;
    tw[n] = g.tw[n];
    twt[(n - q * R2) * R1 + q] = g.tw[n];
    rtw[n] = g.rtw[n];
  }
  __syncthreads();
  unsigned phase = 0;
  if (first <= last) prefetch(first, 0);

  // Step A of a triple's c2r: lines -> X.  Ends with the barrier; false when
  // the copy wait gave up (in every thread).
  auto step_a = [&](int k, int t, T2* X) -> bool {
    const bool ok = mbar_wait(bar, phase & 1);
    ++phase;
    const int m = fields(k, t);
#pragma unroll 1
    for (int u = id; u < U; u += NT) {
      const int i = u / (L * R2), r = u - i * (L * R2), la = r / R2, na = r - la * R2;
      if (((m >> (3 * i)) & 7) == 7 || la >= rows) continue;
      const T2* src = stage + (i * L + la) * K + na;
      const T2* srm = stage + (i * L + la) * K + (H - na);
      T2 z[R1];
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) {
        // z_k = (x_k + conj x_{H-k}) + i conj(w) (x_k - conj x_{H-k}), k = n1 R2 + na
        const T2 w = rtw[n1 * R2 + na];
        if (n1 < R1 / 3) {
          const T2 x = src[n1 * R2], y = cmulconj(x, w);
          z[n1] = mkc(x.x - y.y, x.y + y.x);
        } else {
          const T2 x = n1 < 2 * R1 / 3 ? src[n1 * R2] : czero<T2>();
          const T2 xm = (n1 > R1 / 3 || na > 0) ? srm[-n1 * R2] : czero<T2>();
          const T2 a = cadd_conj(x, xm), y = cmulconj(csub_conj(x, xm), w);
          z[n1] = mkc(a.x - y.y, a.y + y.x);
        }
      }
      Dft<T2, true, R1>::run(z);
      T2* s = X + (i * L + la) * LS + na;
      s[0] = z[0];
#pragma unroll
      for (int q = 1; q < R1; ++q) s[q * RP] = cmulconj(z[q], tw[q * R2 + na]);
    }
    return !__syncthreads_or(!ok);
  };
  // Step B: this thread's R2 pairs of the triple's field i
  auto step_b = [&](int i, const T2* X, T2* v) {
    const T2* s = X + (i * L + lb) * LS + kb * RP;
#pragma unroll
    for (int j = 0; j < R2; ++j) v[j] = s[j];
    Dft<T2, true, R2>::run(v);
  };
  // r2c of up to three lines (bit i of `on`: line i from v_i, into field i at
  // level lev_i)
  auto put = [&](int i, T2* v) {
    if (!onb) return;
    Dft<T2, false, R2>::run(v);
    T2* s = X0 + (i * L + lb) * LS + kb;
    s[0] = v[0];
#pragma unroll
    for (int q = 1; q < R2; ++q) s[q * QP] = cmul(v[q], twt[q * R1 + kb]);
  };
  auto finish = [&](int on, int lev01, int lev2) {
    __syncthreads();
#pragma unroll 1
    for (int u = id; u < U; u += NT) {
      const int i = u / (L * R2), r = u - i * (L * R2), la = r / R2, na = r - la * R2;
      if (!((on >> i) & 1) || la >= rows) continue;
      const T2* s = X0 + (i * L + la) * LS + na * QP;
      T2 z[R1];
#pragma unroll
      for (int n = 0; n < R1; ++n) z[n] = s[n];
      Dft<T2, false, R1>::run(z);   // mode na + R2 p
      T2* y = X1 + (i * L + la) * LS + na;
#pragma unroll
      for (int p = 0; p < R1; ++p) y[R2 * p] = z[p];
    }
    __syncthreads();
    const A h = FftConst<A>::half() * c;
#pragma unroll 4
    for (int u = id; u < 3 * L * K; u += NT) {
      const int i = u / (L * K), r = u - i * (L * K), la = r / K, k = r - la * K;
      if (!((on >> i) & 1) || la >= rows) continue;
      const T2* y = X1 + (i * L + la) * LS;
      const T2 zk = y[k], zm = k == 0 ? zk : y[H - k];
      const T2 a = cadd_conj(zk, zm), w = cmul(csub_conj(zk, zm), rtw[k]);
      out[i * g.out_fs + lrow(i < 2 ? lev01 : lev2) * K + r] = cscale(mkc(a.x + w.y, a.y - w.x), h);
    }
  };

  const T2 hh = mkc(FftConst<A>::half(), FftConst<A>::half());
  bool ok = true;
  T2 cx[R2], cy[R2];   // the products x and y of the last level, without the next level's part
#pragma unroll 1
  for (int k = first; k <= last; ++k) {
    const bool below = k < k0, above = k >= k1e;
    T2 o1[R2], o2[R2], cz[R2], v[R2];
    ok = step_a(k, 0, X0);
    if (!ok) break;
    prefetch(k, 1);
    if (onb) {
      if (!below) {
        step_b(0, X0, o1);
        step_b(2, X0, o2);
      }
      if (!above) {
        step_b(1, X0, v);
#pragma unroll
        for (int j = 0; j < R2; ++j) {
          T2& vm = uv[(R2 + j) * NT];
          if (!below) cz[j] = k > 1 ? pmul(cadd(v[j], vm), o1[j]) : czero<T2>();
          vm = v[j];
        }
      }
    }
    ok = step_a(k, 1, X1);
    if (!ok) break;
    prefetch(k + 1, 0);
    if (onb) {
      if (!above) {
        step_b(0, X1, v);
#pragma unroll
        for (int j = 0; j < R2; ++j) {
          T2& um = uv[j * NT];
          if (!below && k > 1) cz[j] = pmul(hh, pfma(pneg(cadd(v[j], um)), o2[j], cz[j]));
          um = v[j];
        }
      }
      if (!below) {
        step_b(1, X1, v);
#pragma unroll
        for (int j = 0; j < R2; ++j) {
          const T2 h = pmul(hh, v[j]);
          const T2 p = pmul(h, o2[j]), q = pneg(pmul(h, o1[j]));   // w o2 / 2, -w o1 / 2
          o1[j] = cadd(cx[j], p);   // the products of level k - 1
          o2[j] = cadd(cy[j], q);
          cx[j] = k > 1 ? p : czero<T2>();
          cy[j] = k > 1 ? q : czero<T2>();
        }
        if (!above) {
          step_b(2, X1, v);
#pragma unroll
          for (int j = 0; j < R2; ++j) {
            cx[j] = pfma(pneg(uv[(R2 + j) * NT]), v[j], cx[j]);
            cy[j] = pfma(uv[j * NT], v[j], cy[j]);
          }
        }
      }
    }
    if (below) continue;
    const int on = (k > k0 ? 3 : 0) | (above ? 0 : 4);
    if (on & 3) {
      put(0, o1);
      put(1, o2);
    }
    if (on & 4) put(2, cz);
    finish(on, k - 1, k);
    if (!above && k == top) {
      // the last level with products waits for none
      put(0, cx);
      put(1, cy);
      finish(3, k, k);
    }
  }
  if (!ok) {
    // a copy wait gave up (every thread left the loop there): record it and
    // give the copies in flight another bounded wait before leaving
    if (id == 0) atomicExch(g.err, 1);
    mbar_wait(bar, (phase - 1) & 1);
    return;
  }
  // no product at the lid level
  if (k1e > g.nz) {
    const long long o = lrow(g.nz) * K;
    for (int f = 0; f < 3; ++f)
      for (int n = id; n < rows * K; n += NT) out[f * g.out_fs + o + n] = czero<T2>();
  }
}

}  // namespace lesgo
