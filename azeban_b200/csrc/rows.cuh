// Plain real <-> complex transforms along the contiguous axis (FFT<Dim>).  Two
// real lines share one complex transform, line a in the real part, line b in the
// imaginary part.
//
// c2r: the stages, places, twiddles and radices are those of k_zline's inverse in 2-D
// with one component (zline.cuh): the first stage reads the half spectra, the last one
// writes the lines, and lanes run along the lines in both.  256^3 x 3 FP64: 169 us
// against 249 us when lines were staged in shared memory on the way in and out (124 us
// for the bytes alone at the copy bandwidth).  Two stages of larger radices (8.24, 16.16,
// 16.24) are slower or the same: whole backward transforms (us, two stages -> these)
// 192^3 x3 FP64 265 -> 244, 256^3 x3 FP64 469 -> 478, 384^3 x3 FP64 1865 -> 1678, FP32 868
// -> 849; two fields of 256^2 in FP64 12.2 -> 9.9.
// r2c keeps the earlier form.  In this structure it takes 130 us instead of 196 there
// and adds in another order, which moves single modes of a 256^3 Taylor-Green vortex's
// spectrum, beside those that hold its energy, by up to 1.3e-12 of the root mean square
// of the others; the tolerance of that transform in perf/cases.py leaves no room for it.
//
// Reference: src/azeban/cuda/operations/cufft.cpp:133-149.
#pragma once

#include "fft_core.cuh"
#include "zline.cuh"

namespace azb {

struct RealRowArgs {
  const void* in;
  void* out;
  const void* tw;
  long long nlines;
  long long in_line, out_line;  // in elements of the respective type
};

template <typename T, int L> struct RowShape {
  using P = ZPlan<T, L, 2>;
  static constexpr int CB = int(sizeof(cvec<T>));
  static constexpr int S = L / P::RM;
  static constexpr int NLP = S >= 128 ? 1 : 128 / S;  // line pairs of a CTA
  static constexpr int NT = (NLP * S + 31) / 32 * 32;
  static constexpr int ROW = P::RM | 1;
  static constexpr int PP = S * ROW;
  static constexpr int NTW = (P::RM - 1) * S + (P::R2 - 1) * P::R1;
  static constexpr size_t BYTES = size_t(NTW + NLP * PP) * CB;
};

template <typename Sh, typename C> __device__ __forceinline__ void row_twiddles(C* twm, C* tw2, const C* tw) {
  using P = typename Sh::P;
  constexpr int S = Sh::S, NT = Sh::NT;
  for (int i = threadIdx.x; i < (P::RM - 1) * S; i += NT) twm[i] = tw[(i / S + 1) * (i % S)];
  if constexpr (P::R2 > 1)
    for (int i = threadIdx.x; i < (P::R2 - 1) * P::R1; i += NT) tw2[i] = tw[(i / P::R1 + 1) * (i % P::R1) * P::RM];
}

// c2r: lines of L/2+1 complex -> L real.  grid = ceil(nlines / (2 NLP)).
template <typename T, int L> __global__ void __launch_bounds__(RowShape<T, L>::NT) k_rows_c2r(RealRowArgs a) {
  using C = cvec<T>;
  using Sh = RowShape<T, L>;
  using P = typename Sh::P;
  constexpr int R1 = P::R1, R2 = P::R2, RM = P::RM, S = Sh::S, O = L / R1, ROW = Sh::ROW;
  extern __shared__ __align__(16) unsigned char az_smem[];
  C* twm = reinterpret_cast<C*>(az_smem);
  C* tw2 = twm + (RM - 1) * S;
  C* w = twm + Sh::NTW;
  const long long line0 = (long long)blockIdx.x * 2 * Sh::NLP;
  const long long nl = a.nlines - line0;  // lines of this CTA that exist, if fewer than 2 NLP
  const int npairs = nl >= 2 * Sh::NLP ? Sh::NLP : int((nl + 1) / 2);
  const C* in = reinterpret_cast<const C*>(a.in) + line0 * a.in_line;
  T* out = reinterpret_cast<T*>(a.out) + line0 * a.out_line;
  row_twiddles<Sh>(twm, tw2, reinterpret_cast<const C*>(a.tw));
  // radix R1 over k1, from the half spectra; the imaginary parts of bins 0 and
  // L/2 are dropped, as a c2r does
#pragma unroll 1
  for (int idx = threadIdx.x; idx < npairs * O; idx += Sh::NT) {
    const int p = idx / O, o = idx - p * O;
    const bool two = 2 * p + 1 < nl;
    const C* la = in + 2LL * p * a.in_line;
    const C* lb = la + a.in_line;
    C v[R1];
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) {
      const int m = k1 * O + o;
      const bool lo = m <= L / 2;
      const int k = lo ? m : L - m;
      C x = la[k];
      C y = two ? lb[k] : cmk<C>(T(0), T(0));
      if (m == 0 || 2 * m == L) {
        x.y = T(0);
        y.y = T(0);
      }
      v[k1] = lo ? cmk<C>(x.x - y.y, x.y + y.x) : cmk<C>(x.x + y.y, y.x - x.y);
    }
    DFT<R1, +1, C>::run(v);
    const int k2 = o / RM, k3 = o - k2 * RM;
    C* dst = w + p * Sh::PP + R1 * k2 * ROW + k3;
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) dst[n1 * ROW] = v[n1];
  }
  __syncthreads();
  if constexpr (R2 > 1) {
#pragma unroll 1
    for (int idx = threadIdx.x; idx < npairs * R1 * RM; idx += Sh::NT) {
      const int p = idx / (R1 * RM), r = idx - p * (R1 * RM), n1 = r / RM;
      C* at = w + p * Sh::PP + n1 * ROW + (r - n1 * RM);
      C v[R2];
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) {
        v[k2] = at[k2 * R1 * ROW];
        if (k2 > 0) v[k2] = cmulc(v[k2], tw2[(k2 - 1) * R1 + n1]);
      }
      DFT<R2, +1, C>::run(v);
#pragma unroll
      for (int n2 = 0; n2 < R2; ++n2) at[n2 * R1 * ROW] = v[n2];
    }
    __syncthreads();
  }
  const int p = threadIdx.x / S, s = threadIdx.x - p * S;
  if (p >= npairs) return;
  C v[RM];
#pragma unroll
  for (int k = 0; k < RM; ++k) {
    v[k] = w[p * Sh::PP + s * ROW + k];
    if (k > 0) v[k] = cmulc(v[k], twm[(k - 1) * S + s]);
  }
  DFT<RM, +1, C>::run(v);
  T* oa = out + 2LL * p * a.out_line + s;
#pragma unroll
  for (int n = 0; n < RM; ++n) oa[S * n] = v[n].x;
  if (2 * p + 1 < nl) {
    T* ob = oa + a.out_line;
#pragma unroll
    for (int n = 0; n < RM; ++n) ob[S * n] = v[n].y;
  }
}

// r2c: lines of L real -> L/2+1 complex.  grid = ceil(nlines / (2 NLP)).
template <typename T, int L, int NLP, int V>
__global__ void __launch_bounds__(NLP * Plan<L, V>::TPL) k_rows_r2c(RealRowArgs a) {
  using C = cvec<T>;
  using P = Plan<L, V>;
  constexpr int SROW = NLP + 1;
  constexpr int NT = NLP * P::TPL;
  constexpr int LH = L / 2 + 1;
  extern __shared__ __align__(16) unsigned char az_smem[];
  C* tw = reinterpret_cast<C*>(az_smem);
  C* sm = tw + L;
  T* smr = reinterpret_cast<T*>(sm);
  const int tid = threadIdx.x;
  const long long line0 = (long long)blockIdx.x * 2 * NLP;
  const T* in = reinterpret_cast<const T*>(a.in);
  C* out = reinterpret_cast<C*>(a.out);
  load_twiddles<C, L>(tw, reinterpret_cast<const C*>(a.tw));
  for (int idx = tid; idx < 2 * NLP * L; idx += NT) {
    const int m = idx % L;
    const int ln = idx / L;
    const long long line = line0 + ln;
    const T x = line < a.nlines ? in[line * a.in_line + m] : T(0);
    smr[2 * (m * SROW + ln / 2) + (ln & 1)] = x;
  }
  __syncthreads();
  {
    const int col = tid % NLP;
    const int tl = tid / NLP;
    fft_columns<C, -1, L, SROW, true, P>(
        sm, tw, col, tl, [&](int m) { return sm[m * SROW + col]; },
        [&](int m, C v) { sm[m * SROW + col] = v; });
  }
  __syncthreads();
  for (int idx = tid; idx < NLP * LH; idx += NT) {
    const int k = idx % LH;
    const int p = idx / LH;
    const C fk = sm[k * SROW + p];
    const C fm = sm[((L - k) % L) * SROW + p];
    const long long la = line0 + 2 * p;
    if (la < a.nlines)
      out[la * a.out_line + k] = cmk<C>(T(0.5) * (fk.x + fm.x), T(0.5) * (fk.y - fm.y));
    if (la + 1 < a.nlines)
      out[(la + 1) * a.out_line + k] = cmk<C>(T(0.5) * (fk.y + fm.y), T(-0.5) * (fk.x - fm.x));
  }
}

}  // namespace azb
