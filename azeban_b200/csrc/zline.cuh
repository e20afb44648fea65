// Contiguous-axis pass of the right-hand side: for each pair of lines the
// inverse real transform of the DIM velocity components, the CFL maximum, the
// products B = u (x) u, the forward real transform of the products, and the
// separation of the pair's two real spectra into bins [0, nh).
//
// A pair's two lines share one complex transform per component (line a in the
// real part, line b in the imaginary part), so neither inherits the other
// component's rounding.  With L = R1 R2 RM (R2 = 1 for two-stage lengths) the
// inverse runs radix R1, R2, RM and the forward RM, R2, R1.  The inverse's last
// stage and the forward's first stage work on the same rows
// n = s + (L/RM) n3, n3 in [0, RM), of every component, so one thread does both
// with the products between them in registers: the velocities and the products
// never pass through shared memory.  The forward's last stage takes butterflies
// j and L/R1 - j together, whose outputs are each other's mirror bins, so the
// separation is in registers too and the bins go straight to global memory.
//
// Every stage but the first reads and writes the same shared-memory places (the
// digits of an element's place are k-digits before a stage and n-digits after
// it), so an exchange costs one barrier and a stage may take any number of
// butterflies per thread.  Place of digits (d1, d2, d3), d3 < RM, of component
// q of a pair: (d1 + R1 d2) * row + d3 * (components) + q with an odd row: lanes
// run over (d3, q), a contiguous run, in the outer stages and over rows in the
// middle one, and neither has bank conflicts.
//
// The twiddles between the middle stage and its neighbours are W_L^(d3 s) in
// both directions; they are kept by thread order in shared memory.
//
// What bounds it: issue and the latency of 12 to 18 resident warps per SM; it
// executes some 250 instructions per row of a line pair, of which 200 are FP32
// arithmetic.  Against the earlier form, whose velocities and products went
// through shared memory (67 shared accesses per row of a pair instead of 25; us,
// before -> after): 512^3 FP32 5700 -> 4160, 64^3 x15 FP32 138 -> 91, 128^3 FP64 157 -> 122;
// 2-D 128^2 x256 FP32 63 -> 45, 512^2 x64 252 -> 209, 1024^2 FP64 98 -> 40.
//
// Reference: the inverse transform, max_norm and computeB of
// IncompressibleEuler::dudt (include/azeban/equations/incompressible_euler.hpp
// :103-120, :168-228, incompressible_euler_functions.hpp:26-45) and the
// forward transform that follows (src/azeban/cuda/operations/cufft.cpp:133-149).
#pragma once

#include <type_traits>

#include "bulk.cuh"
#include "fft_core.cuh"

namespace azb {

// L = R1 * R2 * RM, for 3-D and for 2-D solves.  RM is what a thread can hold of
// every component (DIM RM complex values and one product's RM); L / R1 is even
// (the separation pairs butterflies j and L/R1 - j).  A larger RM makes the
// outer stages fewer or smaller, a smaller one leaves registers for more
// resident warps, which the pass is short of.  Measured on 2.4e8 padded points
// (FP32, 3-D; us): 192 as 16.12 1603, 24.8 1751, 12.2.8 2146, 8.3.8 2133; 256 (N = 150)
// as 8.4.8 2180, 4.8.8 2291, 16.16 2444, 16.2.8 2668, 32.8 3417 (2379 with registers for
// 12 warps: a first stage of radix 32 off the 3/2 rule needs more than 128); 768 as
// 12.8.8 4148; with one product fewer 384 as 32.12 1558, 24.16 1852, 8.6.8 1808, 48.8
// 2348; 768 as 12.8.8 3631, 8.6.16 4860, 16.4.12 4052.  In FP64 (6e7 points; one product
// fewer): 384 as 12.8.4 868, 8.8.6 890, 8.6.8 992; 192 as 12.4.4 836, 24.8 882.  In 2-D a
// thread holds two components, so RM is larger (one product fewer): FP32 384 as 24.16
// 810, 32.12 995; 192 as 12.16 815, 16.12 885; FP64 384 as 8.6.8 474, 12.8.4 525.
template <typename T, int L, int DIM> struct ZPlan;
#define AZB_ZPLAN(Tv, Lv, A3, B3, M3, A2, B2, M2)              \
  template <> struct ZPlan<Tv, Lv, 3> {                        \
    static constexpr int R1 = A3, R2 = B3, RM = M3;            \
    static_assert(A3 * B3 * M3 == Lv && (Lv / A3) % 2 == 0);   \
  };                                                           \
  template <> struct ZPlan<Tv, Lv, 2> {                        \
    static constexpr int R1 = A2, R2 = B2, RM = M2;            \
    static_assert(A2 * B2 * M2 == Lv && (Lv / A2) % 2 == 0);   \
  };
AZB_ZPLAN(float, 4, 2, 1, 2, 2, 1, 2)
AZB_ZPLAN(float, 6, 3, 1, 2, 3, 1, 2)
AZB_ZPLAN(float, 8, 2, 1, 4, 2, 1, 4)
AZB_ZPLAN(float, 12, 3, 1, 4, 3, 1, 4)
AZB_ZPLAN(float, 16, 4, 1, 4, 4, 1, 4)
AZB_ZPLAN(float, 24, 6, 1, 4, 6, 1, 4)
AZB_ZPLAN(float, 32, 4, 1, 8, 4, 1, 8)
AZB_ZPLAN(float, 48, 6, 1, 8, 6, 1, 8)
AZB_ZPLAN(float, 64, 8, 1, 8, 8, 1, 8)
AZB_ZPLAN(float, 96, 12, 1, 8, 12, 1, 8)
AZB_ZPLAN(float, 128, 16, 1, 8, 8, 1, 16)
AZB_ZPLAN(float, 192, 16, 1, 12, 12, 1, 16)
AZB_ZPLAN(float, 256, 8, 4, 8, 16, 1, 16)
AZB_ZPLAN(float, 384, 32, 1, 12, 24, 1, 16)
AZB_ZPLAN(float, 512, 8, 8, 8, 32, 1, 16)
AZB_ZPLAN(float, 768, 12, 8, 8, 12, 8, 8)
AZB_ZPLAN(float, 1024, 16, 8, 8, 16, 8, 8)
AZB_ZPLAN(float, 1536, 12, 16, 8, 12, 16, 8)
AZB_ZPLAN(double, 4, 2, 1, 2, 2, 1, 2)
AZB_ZPLAN(double, 6, 3, 1, 2, 3, 1, 2)
AZB_ZPLAN(double, 8, 2, 1, 4, 2, 1, 4)
AZB_ZPLAN(double, 12, 3, 1, 4, 3, 1, 4)
AZB_ZPLAN(double, 16, 4, 1, 4, 4, 1, 4)
AZB_ZPLAN(double, 24, 6, 1, 4, 6, 1, 4)
AZB_ZPLAN(double, 32, 8, 1, 4, 8, 1, 4)
AZB_ZPLAN(double, 48, 6, 1, 8, 6, 1, 8)
AZB_ZPLAN(double, 64, 8, 1, 8, 8, 1, 8)
AZB_ZPLAN(double, 96, 12, 1, 8, 12, 1, 8)
AZB_ZPLAN(double, 128, 8, 4, 4, 16, 1, 8)
AZB_ZPLAN(double, 192, 12, 4, 4, 6, 4, 8)
AZB_ZPLAN(double, 256, 8, 8, 4, 8, 4, 8)
AZB_ZPLAN(double, 384, 12, 8, 4, 8, 6, 8)
AZB_ZPLAN(double, 512, 8, 16, 4, 8, 8, 8)
AZB_ZPLAN(double, 768, 12, 16, 4, 8, 12, 8)
AZB_ZPLAN(double, 1024, 16, 16, 4, 8, 16, 8)
AZB_ZPLAN(double, 1536, 16, 24, 4, 12, 16, 8)
#undef AZB_ZPLAN

struct ZArgs {
  const void* in;   // lines of nh x DIM complex, component innermost, in_line apart
  void* out;        // lines of nh x NB complex, component innermost, out_line apart
  const void* tw;
  long long nlines;  // lines per member (even)
  int nh;            // spectral bins per line
  int nmem;          // members
  int in_line, out_line;  // line strides (elements; multiples of 2 lines' 16 bytes)
  long long in_mem, out_mem;  // member strides (elements)
  double norm;       // 1 / (N^{d/2} M^{d/2})
  Ctrl* ctrl;
  int wait_polls;    // limit of the wait for the chunk's bulk copy (kWaitPolls)
  int pdl;           // to launch_pass: may be a programmatic dependent; to the kernel: is one
};

// Product c of the velocities u: 11, 12, 22 in 2-D; 11, 21, 22, 31, 32, 33 in 3-D
// (include/azeban/equations/incompressible_euler_functions.hpp:26-45).
template <int DIM, int c, typename T> __device__ __forceinline__ T product(const T (&u)[DIM]) {
  constexpr int i = c == 0 ? 0 : c < 3 ? 1 : 2;
  return u[i] * u[c - i * (i + 1) / 2];
}

// Shared memory of one CTA: the mbarrier, the middle stage's twiddles
// [RM-1][L/RM], the outer twiddles [R2-1][R1], then the work area.  The
// velocity rows start at its front, the chunk's input sits at its end, and the
// product rows (written when the input and the velocities are dead) take all of it.
template <typename T, int L, int NLP, int DIM> struct ZLineShape {
  using P = ZPlan<T, L, DIM>;
  static constexpr int CB = int(sizeof(cvec<T>));
  static constexpr int NB = products(DIM);
  static constexpr int S = L / P::RM;       // rows (middle-stage butterflies) of a pair
  static constexpr int SV = (P::RM * DIM) | 1;
  static constexpr int SP = (P::RM * NB) | 1;
  static constexpr int VP = S * SV, PP = S * SP;  // elements per pair
  static constexpr int NT = (NLP * S + 31) / 32 * 32;
  // Register cap: 12 resident warps per SM (168 registers) for the large middle
  // radices, which need them, 18 for the long FP32 lines of 2-D solves (L = 768 1220 us,
  // with 15 warps 1294), 15 (128 registers) for the others.
  static constexpr int WARPS = P::RM * CB > 64 ? 12 : DIM == 2 && CB == 8 && S >= 96 ? 18 : 15;
  static constexpr int NTW = (P::RM - 1) * S + (P::R2 - 1) * P::R1;
  static constexpr int OFF_TW = 16;
  static constexpr int OFF_W = (OFF_TW + NTW * CB + 15) / 16 * 16;
  // resident CTAs by registers and by the product rows' shared memory
  static constexpr int FIT = 228 * 1024 / (OFF_W + NLP * PP * CB + 1024);
  static constexpr int MINB = FIT < 2 || NT >= WARPS * 32 ? 1 : FIT < WARPS * 32 / NT ? FIT : WARPS * 32 / NT;
  static constexpr int V_END = (NLP * VP * CB + 15) / 16 * 16;  // bytes
  static __host__ __device__ int in_off(int in_line) {  // bytes from OFF_W to the input
    const int at_end = NLP * (PP * CB - 2 * in_line * CB) / 16 * 16;
    return at_end > V_END ? at_end : V_END;
  }
  static __host__ __device__ long long smem_bytes(int in_line) {
    const long long in_end = in_off(in_line) + 2LL * NLP * in_line * CB;
    const long long p_end = (long long)NLP * PP * CB;
    return OFF_W + (in_end > p_end ? in_end : p_end);
  }
};

// Running max of |x| that keeps a NaN once met.
struct AbsMax32 {
  float v = 0.0f;
  __device__ __forceinline__ void add(float a, float b) {
    asm("max.NaN.f32 %0, %0, %1, %2;" : "+f"(v) : "f"(fabsf(a)), "f"(fabsf(b)));
  }
  __device__ __forceinline__ unsigned bits() const { return __float_as_uint(v); }
};
struct AbsMax64 {
  unsigned long long v = 0;
  __device__ __forceinline__ void add(double a, double b) {
    const unsigned long long x = AbsBits<double>::of(a), y = AbsBits<double>::of(b);
    v = x > v ? x : v;
    v = y > v ? y : v;
  }
  __device__ __forceinline__ unsigned long long bits() const { return v; }
};
template <typename T> struct AbsMaxOf;
template <> struct AbsMaxOf<float> { using type = AbsMax32; };
template <> struct AbsMaxOf<double> { using type = AbsMax64; };

// Bits k1 whose rows k1 L/R1 + o, all o, are zero under the 3/2 rule.
template <int L, int R1, bool STD> __host__ __device__ constexpr unsigned long long zero_rows() {
  unsigned long long z = 0;
  if (STD)
    for (int k1 = 0; k1 < R1; ++k1)
      if (k1 * (L / R1) >= L / 3 + 1 && (k1 + 1) * (L / R1) - 1 <= L - (L / 3 + 1)) z |= 1ull << k1;
  return z;
}

// STD: nh == L/3 + 1 (the 3/2 rule), known at compile time, so the zero rows
// of the first stage and the dropped bins of the last one fold.
template <typename T, int L, int NLP, int DIM, bool STD>
__global__ void __launch_bounds__(ZLineShape<T, L, NLP, DIM>::NT, ZLineShape<T, L, NLP, DIM>::MINB)
    k_zline(ZArgs a) {
  using C = cvec<T>;
  using P = ZPlan<T, L, DIM>;
  using Z = ZLineShape<T, L, NLP, DIM>;
  constexpr int R1 = P::R1, R2 = P::R2, RM = P::RM;
  constexpr int NB = Z::NB, S = Z::S, SV = Z::SV, SP = Z::SP, NT = Z::NT;
  extern __shared__ __align__(16) unsigned char az_smem[];
  unsigned long long* bar = reinterpret_cast<unsigned long long*>(az_smem);
  C* twm = reinterpret_cast<C*>(az_smem + Z::OFF_TW);
  C* tw2 = twm + (RM - 1) * S;
  C* w = reinterpret_cast<C*>(az_smem + Z::OFF_W);
  const int member = blockIdx.y;
  Ctrl* ctrl = a.ctrl + member;
  if (a.pdl) pdl_enter();
  if (ctrl->skip) return;
  const int tid = threadIdx.x;
  const int nh = STD ? L / 3 + 1 : a.nh;
  const int in_line = a.in_line;
  const int out_line = a.out_line;
  const long long line0 = (long long)blockIdx.x * 2 * NLP;
  // Line pairs of this chunk that exist (nlines is even, so a pair is whole).
  const int npairs = int((a.nlines - line0) / 2 < NLP ? (a.nlines - line0) / 2 : NLP);
  const C* cin = reinterpret_cast<const C*>(az_smem + Z::OFF_W + Z::in_off(in_line));

  // Elected thread: one bulk copy of the chunk's lines into shared memory.
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_fence_init();
    const unsigned bytes = unsigned(2 * npairs * in_line * Z::CB);
    mbar_expect_tx(&bar[0], bytes);
    bulk_load(az_smem + Z::OFF_W + Z::in_off(in_line),
              reinterpret_cast<const C*>(a.in) + member * a.in_mem + line0 * in_line, bytes, &bar[0]);
  }
  {
    const C* tw = reinterpret_cast<const C*>(a.tw);
    for (int i = tid; i < (RM - 1) * S; i += NT) twm[i] = tw[(i / S + 1) * (i % S)];
    if constexpr (R2 > 1)
      for (int i = tid; i < (R2 - 1) * R1; i += NT) tw2[i] = tw[(i / R1 + 1) * (i % R1) * RM];
  }
  __syncthreads();
  const bool ok = mbar_wait_bounded(&bar[0], 0u, a.wait_polls);
  if (__syncthreads_or(!ok)) {
    // The wait ran out: flag it (bit 1 of the member's error word), and let
    // one thread wait, bounded, for the copy to land before the CTA exits,
    // so no bulk copy is still writing into shared memory the SM may hand to
    // the next CTA.  The CTA's shared memory stays allocated until its last
    // thread exits.
    if (tid == 0) {
      atomicOr(&ctrl->err, 2);
      mbar_wait_bounded(&bar[0], 0u, kWaitPolls);
    }
    return;
  }

  // 1. Inverse, radix R1 over k1 for each o = (k2, k3), from the half spectra:
  //    bin k < nh gives row k (X + iY) and row L - k (conj X + i conj Y); rows
  //    [nh, L - nh] are zero.  The imaginary parts of bin 0 and bin L/2 are
  //    dropped, as a c2r does.
  {
    constexpr int O = L / R1;
    constexpr int TA = O * DIM;
#pragma unroll 1
    for (int idx = tid; idx < npairs * TA; idx += NT) {
      const int p = idx / TA;
      const int r = idx - p * TA;
      const int o = r / DIM;
      const int q = r - o * DIM;
      const C* la = cin + 2 * p * in_line + q;
      const C* lb = la + in_line;
      // rows of this k1 that are certainly bins, certainly mirrors, or neither
      constexpr int H = L / 3 + 1;
      C v[R1];
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) {
        const int m = k1 * O + o;
        const bool all_lo = STD && (k1 + 1) * O <= H, no_lo = STD && k1 * O >= H;
        const bool all_hi = STD && k1 * O > L - H, no_hi = STD && (k1 + 1) * O - 1 <= L - H;
        const bool lo = all_lo || (!no_lo && m < nh);
        const bool hi = !lo && (all_hi || (!no_hi && m > L - nh));
        C x = cmk<C>(T(0), T(0)), y = x;
        const int k = lo ? m : L - m;
        if (lo || hi) {
          x = la[k * DIM];
          y = lb[k * DIM];
        }
        if ((k1 == 0 && o == 0) || (!STD && 2 * m == L)) {
          x.y = T(0);
          y.y = T(0);
        }
        v[k1] = lo ? cmk<C>(x.x - y.y, x.y + y.x) : cmk<C>(x.x + y.y, y.x - x.y);
      }
      DFTZ<R1, +1, C, zero_rows<L, R1, STD>()>::run(v);
      const int k2 = o / RM, k3 = o - k2 * RM;
      C* dst = w + p * Z::VP + R1 * k2 * SV + k3 * DIM + q;
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) dst[n1 * SV] = v[n1];
    }
  }
  __syncthreads();
  // Radix R2 over k2 for each (n1, k3), in place.
  if constexpr (R2 > 1) {
    constexpr int TB = R1 * RM * DIM;
#pragma unroll 1
    for (int idx = tid; idx < npairs * TB; idx += NT) {
      const int p = idx / TB;
      const int r = idx - p * TB;
      const int n1 = r / (RM * DIM);
      C* at = w + p * Z::VP + n1 * SV + (r - n1 * (RM * DIM));
      C v[R2];
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) {
        v[k2] = at[k2 * R1 * SV];
        if (k2 > 0) v[k2] = cmulc(v[k2], tw2[(k2 - 1) * R1 + n1]);
      }
      DFT<R2, +1, C>::run(v);
#pragma unroll
      for (int n2 = 0; n2 < R2; ++n2) at[n2 * R1 * SV] = v[n2];
    }
    __syncthreads();
  }

  // 2. Inverse radix RM of every component, the CFL maximum (unscaled), the
  //    scaling by 1/(N^{d/2} M^{d/2}), the products and their forward radix RM.
  typename AbsMaxOf<T>::type vmax;
  {
    const int p = tid / S;
    const int s = tid - p * S;
    const bool active = p < npairs;
    C u[DIM][RM], tws[RM];
    if (active) {
      const C* src = w + p * Z::VP + s * SV;
#pragma unroll
      for (int k = 0; k < RM; ++k) {
        if (k > 0) tws[k] = twm[(k - 1) * S + s];
#pragma unroll
        for (int q = 0; q < DIM; ++q) u[q][k] = src[k * DIM + q];
      }
    }
    __syncthreads();  // the products overwrite the velocity rows
    if (active) {
      // the products also take the separation's factor 1/2
      const T norm = T(a.norm * 0.70710678118654752440);
#pragma unroll
      for (int q = 0; q < DIM; ++q) {
#pragma unroll
        for (int k = 1; k < RM; ++k) u[q][k] = cmulc(u[q][k], tws[k]);
        DFT<RM, +1, C>::run(u[q]);
#pragma unroll
        for (int n = 0; n < RM; ++n) {
          vmax.add(u[q][n].x, u[q][n].y);
          u[q][n] = cscale(u[q][n], norm);
        }
      }
      C* dst = w + p * Z::PP + s * SP;
      auto one = [&](auto cc) {
        constexpr int c = decltype(cc)::value;
        C t[RM];
#pragma unroll
        for (int n = 0; n < RM; ++n) {
          T x[DIM], y[DIM];
#pragma unroll
          for (int q = 0; q < DIM; ++q) {
            x[q] = u[q][n].x;
            y[q] = u[q][n].y;
          }
          t[n] = cmk<C>(product<DIM, c>(x), product<DIM, c>(y));
        }
        DFT<RM, -1, C>::run(t);
#pragma unroll
        for (int m = 0; m < RM; ++m) dst[m * NB + c] = m > 0 ? cmul(t[m], tws[m]) : t[0];
      };
      one(std::integral_constant<int, 0>{});
      one(std::integral_constant<int, 1>{});
      one(std::integral_constant<int, 2>{});
      if constexpr (DIM == 3) {
        one(std::integral_constant<int, 3>{});
        one(std::integral_constant<int, 4>{});
        one(std::integral_constant<int, 5>{});
      }
    }
  }
  __syncthreads();

  // 3. Forward: radix R2 over n2 for each (n1, m3), in place.
  if constexpr (R2 > 1) {
    constexpr int TB = R1 * RM * NB;
#pragma unroll 1
    for (int idx = tid; idx < npairs * TB; idx += NT) {
      const int p = idx / TB;
      const int r = idx - p * TB;
      const int n1 = r / (RM * NB);
      C* at = w + p * Z::PP + n1 * SP + (r - n1 * (RM * NB));
      C v[R2];
#pragma unroll
      for (int n2 = 0; n2 < R2; ++n2) v[n2] = at[n2 * R1 * SP];
      DFT<R2, -1, C>::run(v);
#pragma unroll
      for (int m2 = 0; m2 < R2; ++m2) {
        if (m2 > 0) v[m2] = cmul(v[m2], tw2[(m2 - 1) * R1 + n1]);
        at[m2 * R1 * SP] = v[m2];
      }
    }
    __syncthreads();
  }

  // 4. Radix R1 over n1 of butterflies j and J - j (J = L/R1; 0 with J/2),
  //    whose bins j + J m and J - j + J (R1 - 1 - m) mirror each other; the
  //    separation of lines a and b; bins [0, nh) to global memory.  Lanes run
  //    over the components, then j: contiguous runs of a line.
  {
    constexpr int J = L / R1;
    constexpr int TC = (J / 2) * NB;
    C* out = reinterpret_cast<C*>(a.out) + member * a.out_mem + line0 * out_line;
#pragma unroll 1
    for (int idx = tid; idx < npairs * TC; idx += NT) {
      const int p = idx / TC;
      const int r = idx - p * TC;
      const int ja = r / NB;
      const int c = r - ja * NB;
      const int jb = ja == 0 ? J / 2 : J - ja;
      C f[R1], g[R1];
      {
        const C* base = w + p * Z::PP + c;
        const C* sa = base + R1 * (ja / RM) * SP + (ja % RM) * NB;
        const C* sb = base + R1 * (jb / RM) * SP + (jb % RM) * NB;
#pragma unroll
        for (int n = 0; n < R1; ++n) {
          f[n] = sa[n * SP];
          g[n] = sb[n * SP];
        }
      }
      DFT<R1, -1, C>::run(f);
      DFT<R1, -1, C>::run(g);
      C* oa = out + 2LL * p * out_line + c;
      C* ob = oa + out_line;
      // bin k, its value x and its mirror's y
      auto put = [&](int k, const C& x, const C& y) {
        oa[k * NB] = cmk<C>(x.x + y.x, x.y - y.y);
        ob[k * NB] = cmk<C>(x.y + y.y, y.x - x.x);
      };
      if (ja != 0) {
#pragma unroll
        for (int m = 0; m < R1; ++m) {
          if (STD && J * m >= L / 3 + 1) break;
          if (ja + J * m < nh) put(ja + J * m, f[m], g[R1 - 1 - m]);
          if (jb + J * m < nh) put(jb + J * m, g[m], f[R1 - 1 - m]);
        }
      } else {
#pragma unroll
        for (int m = 0; m < R1; ++m) {
          if (STD && J * m >= L / 3 + 1) break;
          if (J * m < nh) put(J * m, f[m], f[(R1 - m) % R1]);
          if (J / 2 + J * m < nh) put(J / 2 + J * m, g[m], g[R1 - 1 - m]);
        }
      }
    }
  }

  // CFL reduction: warp, then block, then one atomic per CTA.  A non-finite
  // value sets the error bit; the maximum then records infinity.
  using AB = AbsBits<T>;
  typename AB::U vbits = vmax.bits();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const typename AB::U other = __shfl_xor_sync(0xffffffffu, vbits, o);
    vbits = other > vbits ? other : vbits;
  }
  __shared__ typename AB::U red[NT / 32];
  if ((tid & 31) == 0) red[tid >> 5] = vbits;
  __syncthreads();
  if (tid == 0) {
    typename AB::U m = 0;
#pragma unroll
    for (int i = 0; i < NT / 32; ++i) m = red[i] > m ? red[i] : m;
    if (m >= AB::kInfBits) {
      atomicOr(&ctrl->err, 1);
      m = AB::kInfBits;
    }
    AB::to_ctrl(ctrl, m);
  }
}

}  // namespace azb
