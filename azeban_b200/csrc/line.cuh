// Passes along a strided axis on tiles of columns, in two or three stages with
// in-place exchanges: the padding inverse and the truncating forward passes of the
// right-hand side and the last pass of a 2-D one (with the projection, the
// viscosity and the SSP-RK3 stage).
//
// L = RA RM RB (RM = 1 for two-stage lengths).  Input row n = (L/RA) nA + RB nM +
// nB, output row k = kA + RA kM + RA RM kB; the stages run over nA, nM, nB.  The
// place of digits (dA, dM, dB) of a column is (dA + RA dM) * STR + dB * COLS + col:
// a stage reads and writes the same places (n-digits before it, k-digits after),
// so an exchange costs one barrier and a thread may take any number of a stage's
// butterflies, one after the other.  The first stage reads global memory (padding
// map applied, rows that are zero for every thread known at compile time), the
// last one writes it.  Twiddles are kept in shared memory in the order the
// threads read them: before the last stage W_L^(nB s), s = kA + RA kM, before the
// middle one W_(RA RM)^(nM kA).
//
// Against the earlier form (k_cols: every thread keeps its elements through all
// stages, two barriers per exchange) a thread holds one butterfly at a time, which
// leaves registers for radices up to 32, two stages up to L = 1024 and more
// loads in flight.  Measured (us, before -> after): 512^3 FP32 inverse y 1622 ->
// 1336, forward y 2992 -> 2642; 128^3 FP64 54 -> 42 and 81 -> 71; 2-D last pass 128^2
// x256 FP32 54 -> 43.
#pragma once

#include "euler_kernels.cuh"

namespace azb {

template <typename T, int L, int A, int M, int B> struct LinePlan {
  static constexpr int RA = A, RM = M, RB = B;
  static constexpr int S = L / B;   // last-stage butterflies of a column
  static constexpr int O = L / A;   // first-stage butterflies of a column
  static constexpr int NTW = (B - 1) * S + (M - 1) * A;
  static_assert(A * M * B == L);
};

// Elements from one butterfly row (dA, dM) to the next: lanes of the last stage
// run over `run` consecutive groups of `lanes` elements, then over rows, so a row
// is offset by what the run leaves of a 128-byte wavefront.
constexpr int line_stride(int row, int run, int cb) {
  const int q = 128 / cb;
  if (run >= q) return row;
  while (row % q != run % q) ++row;
  return row;
}

// The twiddles of a CTA, fetched before the first stage's loads and put into
// shared memory after it, so the two global round trips overlap.
template <typename P, int NT, typename C> struct LineTwiddles {
  static constexpr int K = (P::NTW + NT - 1) / NT;
  C t[K > 0 ? K : 1];
  __device__ __forceinline__ void fetch(const C* tw) {
    constexpr int NS = (P::RB - 1) * P::S;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const int i = threadIdx.x + j * NT, m = i - NS;
      if (i < P::NTW) t[j] = tw[i < NS ? (i / P::S + 1) * (i % P::S) : (m / P::RA + 1) * (m % P::RA) * P::RB];
    }
  }
  __device__ __forceinline__ void put(C* tws) const {
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const int i = threadIdx.x + j * NT;
      if (i < P::NTW) tws[i] = t[j];
    }
  }
};

template <int SGN, typename C> __device__ __forceinline__ C twid(C v, C w) {
  return SGN < 0 ? cmul(v, w) : cmulc(v, w);
}

// Bits nA whose rows nA O + o are zero for every o, under the padding map of the
// 3/2 rule.
template <int L, int RA> __host__ __device__ constexpr unsigned long long pad_zero_rows() {
  unsigned long long z = 0;
  const int n = 2 * L / 3, O = L / RA;
  for (int a = 0; a < RA; ++a)
    if (a * O >= n / 2 + 1 && (a + 1) * O - 1 < n / 2 + 1 + L - n) z |= 1ull << a;
  return z;
}

// First stage of one butterfly o of one column; `dst` is the column's place 0.
template <typename P, int SGN, unsigned long long Z, int STR, int COLS, typename C, typename Load>
__device__ __forceinline__ void line_first(C* dst, int o, Load&& load) {
  C v[P::RA];
#pragma unroll
  for (int a = 0; a < P::RA; ++a) v[a] = ((Z >> a) & 1ull) ? cmk<C>(0, 0) : load(a * P::O + o);
  DFTZ<P::RA, SGN, C, Z>::run(v);
  const int m = o / P::RB, b = o - m * P::RB;
  C* at = dst + P::RA * m * STR + b * COLS;
#pragma unroll
  for (int a = 0; a < P::RA; ++a) at[a * STR] = v[a];
}

// Middle stage, in place, of all columns of the tile.
template <typename P, int SGN, int STR, int COLS, int NT, typename C>
__device__ __forceinline__ void line_middle(C* sm, const C* twm) {
  if constexpr (P::RM > 1) {
    __syncthreads();
    constexpr int ROW = P::RB * COLS;
#pragma unroll 1
    for (int idx = threadIdx.x; idx < P::RA * ROW; idx += NT) {
      const int a = idx / ROW;
      C* at = sm + a * STR + (idx - a * ROW);
      C v[P::RM];
#pragma unroll
      for (int m = 0; m < P::RM; ++m) {
        v[m] = at[m * P::RA * STR];
        if (m > 0) v[m] = twid<SGN>(v[m], twm[(m - 1) * P::RA + a]);
      }
      DFT<P::RM, SGN, C>::run(v);
#pragma unroll
      for (int m = 0; m < P::RM; ++m) at[m * P::RA * STR] = v[m];
    }
  }
}

// Padded row k of butterfly row s and digit kB -> retained row of an axis of n
// rows, or -1; KEEP_ALL / DROP_ALL decide it at compile time where they can.
template <int L, int S, bool STD> struct Retained {
  static constexpr int N = 2 * L / 3;
  static __host__ __device__ constexpr bool dropped(int b) {  // every s
    return STD && b * S > N / 2 && (b + 1) * S - 1 < L - N / 2 + 1;
  }
  static __host__ __device__ constexpr bool low(int b) { return STD && (b + 1) * S - 1 <= N / 2; }
  static __host__ __device__ constexpr bool high(int b) { return STD && b * S >= L - N / 2 + 1; }
  static __device__ __forceinline__ int row(int s, int b, int n) {
    const int k = s + S * b;
    if (low(b)) return k;
    if (high(b)) return k - (L - N);
    const int nn = STD ? N : n;
    if (k <= nn / 2) return k;
    if (k >= L - nn / 2 + 1) return k - (L - nn);
    return -1;
  }
};

template <typename T, typename P, int NC> struct ColShape {
  static constexpr int CB = int(sizeof(cvec<T>));
  static constexpr int STR = line_stride(P::RB * NC, NC, CB);
  static constexpr size_t BYTES = size_t(P::NTW + P::S * STR) * CB;
};

// Padding inverse (MODE COL_PAD, SGN +1) or truncating forward (COL_TRUNC, -1)
// transforms of the columns of a tile.  grid = (ntile * nouter, 1, nmembers).
// STD: the unpadded length is 2L/3 (the 3/2 rule), known at compile time.
template <typename T, int L, typename P, int NC, int NT, int MINB, int SGN, int MODE, bool STD>
__global__ void __launch_bounds__(NT, MINB) k_columns(ColArgs a) {
  using C = cvec<T>;
  using Sh = ColShape<T, P, NC>;
  constexpr int STR = Sh::STR;
  static_assert(NT % NC == 0);
  extern __shared__ __align__(16) unsigned char az_smem[];
  C* tws = reinterpret_cast<C*>(az_smem);
  C* twm = tws + (P::RB - 1) * P::S;
  C* sm = tws + P::NTW;
  if (!pass_enter(a)) return;
  const int member = blockIdx.z;
  const int outer = blockIdx.x / a.ntile;
  const int tile = blockIdx.x - outer * a.ntile;
  const int col = threadIdx.x % NC;
  const int t0 = threadIdx.x / NC;
  const long long p = (long long)tile * NC + col;
  bool valid = p < a.ninner;
  long long pin;
  if (a.grp > 0) {
    const long long g = p / a.grp;
    const int q = int(p - g * a.grp);
    valid = valid && q < a.grp_valid;
    pin = g * a.in_grp + (a.in_ci == 1 ? q : (q % a.in_ci) * a.in_comp + q / a.in_ci);
  } else {
    pin = a.in_ci == 1 ? p : (p % a.in_ci) * a.in_comp + p / a.in_ci;
  }
  const C* in = reinterpret_cast<const C*>(a.in) + member * a.in_mem + outer * a.in_outer + pin;
  C* out = reinterpret_cast<C*>(a.out) + member * a.out_mem + outer * a.out_outer + p;
  const int n = STD ? 2 * L / 3 : a.n_short;
  // Row offsets fit 32 bits (the launcher checks L * stride < 2^31).
  const int in_row = int(a.in_row);
  const int out_row = int(a.out_row);
  constexpr unsigned long long Z = MODE == COL_PAD && STD ? pad_zero_rows<L, P::RA>() : 0ull;
  using Rt = Retained<L, P::S, STD && MODE == COL_TRUNC>;
  LineTwiddles<P, NT, C> twiddles;
  twiddles.fetch(reinterpret_cast<const C*>(a.tw));
#pragma unroll 1
  for (int o = t0; o < P::O; o += NT / NC) {
    line_first<P, SGN, Z, STR, NC>(sm + col, o, [&](int m) -> C {
      const int src = MODE == COL_PAD ? pad_src_row(m, n, L) : m;
      if (!valid || src < 0) return cmk<C>(T(0), T(0));
      return in[src * in_row];
    });
  }
  twiddles.put(tws);
  line_middle<P, SGN, STR, NC, NT>(sm, twm);
  __syncthreads();
#pragma unroll 1
  for (int s = t0; s < P::S; s += NT / NC) {
    C v[P::RB];
#pragma unroll
    for (int b = 0; b < P::RB; ++b) {
      v[b] = sm[s * STR + b * NC + col];
      if (b > 0) v[b] = twid<SGN>(v[b], tws[(b - 1) * P::S + s]);
    }
    DFT<P::RB, SGN, C>::run(v);
    if (valid) {
#pragma unroll
      for (int b = 0; b < P::RB; ++b) {
        if (MODE == COL_TRUNC) {
          if (Rt::dropped(b)) continue;
          const int dst = Rt::row(s, b, n);
          if (Rt::low(b) || Rt::high(b) || dst >= 0) out[dst * out_row] = v[b];
        } else {
          out[(s + P::S * b) * out_row] = v[b];
        }
      }
    }
  }
}

template <typename T, typename P, int NCM> struct Epi2Shape {
  static constexpr int CB = int(sizeof(cvec<T>));
  static constexpr int NB = 2;
  static constexpr int COLS = NB * NCM;
  static constexpr int W = 16 / CB;  // components a thread of the last stage reads at once
  static constexpr int STR = line_stride(P::RB * COLS, W * NCM, CB);
  static constexpr int TW = (P::NTW + W - 1) / W * W;
  static constexpr size_t BYTES = size_t(TW + P::S * STR) * CB;
  // Place of component c of mode pl in a row: groups of the W components that a thread
  // reads at once, the modes of a group contiguous (the last stage's lanes).
  static __host__ __device__ constexpr int place(int c, int pl) { return c / W * (W * NCM) + pl * W + c % W; }
};

// Last pass of a 2-D right-hand side: forward along x of B11 - B22 and B12 (a
// transform fewer; the projection meets them as this difference alone, with one factor,
// so rounding has the same weights as with both.  It is taken here, on values already
// transformed along y: in a shear flow u_x(y) the rounding of u_x^2 is the same on every
// line x = const and has no part in kx != 0, but that of u_x^2 - u_y^2 is another on each,
// and a product pass that took it put a 128^2 FP32 double shear layer 2.9e-5 off FP64
// instead of 5e-6), kept at the N retained rows, then per mode dudt = |k| = 0 ? 0 : -L +
// nu(|k|) u_hat with L the projected divergence (incompressible_euler.hpp:230-347,
// incompressible_euler_functions.hpp:47-112), which in 2-D is
//   L_x = i ky q / k^2, L_y = -i kx q / k^2,
//   q = kx ky (B11 - B22) + (ky^2 - kx^2) B12,
// then the stage combination as in k_fwd_epilogue.  A thread of the last stage
// holds both components of its butterfly, so the transform's outputs stay in
// registers.  grid = (ntile, nmembers).
template <typename T, int L, typename P, int NCM, int NT, int MINB, bool STD>
__global__ void __launch_bounds__(NT, MINB) k_epilogue2d(EpiArgs a) {
  using C = cvec<T>;
  using Sh = Epi2Shape<T, P, NCM>;
  constexpr int NB = Sh::NB, STR = Sh::STR, COLS = Sh::COLS, W = Sh::W;
  extern __shared__ __align__(16) unsigned char az_smem[];
  C* tws = reinterpret_cast<C*>(az_smem);
  C* twm = tws + (P::RB - 1) * P::S;
  C* sm = tws + Sh::TW;
  if (a.pdl) pdl_enter();
  const int member = blockIdx.y;
  if (a.ctrl != nullptr && a.ctrl[member].skip) return;
  __shared__ double step_dt;
  const int tile = blockIdx.x;
  const int N = STD ? 2 * L / 3 : a.N;
  const int B_row = int(a.B_row);  // L * B_row < 2^31, checked by the launcher
  LineTwiddles<P, NT, C> twiddles;
  twiddles.fetch(reinterpret_cast<const C*>(a.tw));
  const C* B = reinterpret_cast<const C*>(a.B) + member * a.B_mem + (long long)tile * (3 * NCM);
  const int left = int(a.ninner) - tile * NCM;  // modes of this tile that exist
  // lanes over the modes, then the butterflies; the component is the same for a warp
#pragma unroll 1
  for (int idx = threadIdx.x; idx < P::O * COLS; idx += NT) {
    const int c = idx / (P::O * NCM), r = idx - c * (P::O * NCM);
    const int o = r / NCM, pl = r - o * NCM;
    const C* b = B + 3 * pl;
    C* at = sm + Sh::place(c, pl);
    const bool valid = pl < left;
    if (c == 0) {
      line_first<P, -1, 0ull, STR, COLS>(at, o, [&](int m) -> C {
        return valid ? vsub(b[m * B_row], b[m * B_row + 2]) : cmk<C>(T(0), T(0));
      });
    } else {
      line_first<P, -1, 0ull, STR, COLS>(at, o, [&](int m) -> C {
        return valid ? b[m * B_row + 1] : cmk<C>(T(0), T(0));
      });
    }
  }
  twiddles.put(tws);
  if (threadIdx.x == 0) step_dt = epilogue_dt<T>(a, member);
  line_middle<P, -1, STR, COLS, NT>(sm, twm);
  __syncthreads();

  const T dt = T(step_dt);
  const T twopi = T(2 * 3.14159265358979323846);
  const C* u = reinterpret_cast<const C*>(a.u) + member * a.u_mem;
  const C* u0 = reinterpret_cast<const C*>(a.u0) + member * a.u_mem;
  C* out = reinterpret_cast<C*>(a.out) + member * a.u_mem;
  const StateLayout lu = a.lu, lu0 = a.lu0, lout = a.lout;  // offsets < 2^31, checked by the launcher
  const T inv_k0sq = T(1.0 / (a.visc.k0 * a.visc.k0));
  // the stage combination as uniform coefficients, as in k_fwd_epilogue
  const bool use_u = a.mode != MODE_DUDT;
  const bool need_u0 = a.mode == MODE_RK2 || a.mode == MODE_RK3;
  const T dd = use_u ? dt : T(1);
  const T ct = a.mode == MODE_RK2 ? T(0.25) : a.mode == MODE_RK3 ? T(2.0 / 3.0) : T(1);
  using Rt = Retained<L, P::S, STD>;
#pragma unroll 1
  for (int idx = threadIdx.x; idx < P::S * NCM; idx += NT) {
    const int s = idx / NCM, pl = idx - s * NCM;
    const int p = tile * NCM + pl;
    if (pl >= left) continue;
    C v[NB][P::RB];
#pragma unroll
    for (int b = 0; b < P::RB; ++b) {
      const C w = b > 0 ? tws[(b - 1) * P::S + s] : cmk<C>(T(1), T(0));
#pragma unroll
      for (int g = 0; g < NB; g += W) {
        const C* src = sm + s * STR + b * COLS + Sh::place(g, pl);
        if constexpr (W == 2) {
          const float4 q = *reinterpret_cast<const float4*>(src);
          v[g][b] = cmk<C>(q.x, q.y);
          v[g + 1][b] = cmk<C>(q.z, q.w);
        } else {
          v[g][b] = *src;
        }
#pragma unroll
        for (int i = 0; i < W; ++i)
          if (b > 0) v[g + i][b] = cmul(v[g + i][b], w);
      }
    }
#pragma unroll
    for (int g = 0; g < NB; ++g) DFT<P::RB, -1, C>::run(v[g]);
    const T k2 = T(p), kv2 = twopi * k2;  // whole wavenumber, and 2 pi times it
    // The state values of the rows first: out may be u or u0, so no load could be moved
    // over an earlier row's store.  Half of the rows at a time where no row is known to be
    // dropped and all values would take more registers than there are (L = 256 FP32
    // spilled 492 bytes, FP64 some 260 at every length; 22 solves with N = 150 and M = 256
    // 96 -> 89 us a step, 40 FP64 ones with N = 106 and M = 192 117 -> 110).
    constexpr int HB = STD || P::RB * Sh::CB <= 64 ? P::RB : P::RB / 2;
    static_assert(P::RB % HB == 0);
#pragma unroll
    for (int b0 = 0; b0 < P::RB; b0 += HB) {
      C uc[HB][2], wc[HB][2];
#pragma unroll
      for (int b = 0; b < HB; ++b) {
        if (Rt::dropped(b0 + b)) continue;
        const int i = Rt::row(s, b0 + b, N);
        if (!(Rt::low(b0 + b) || Rt::high(b0 + b)) && i < 0) continue;
        const int ou = i * lu.row + p * lu.ps, ow = i * lu0.row + p * lu0.ps;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uc[b][c] = u[c * lu.comp + ou];
          wc[b][c] = need_u0 ? u0[c * lu0.comp + ow] : cmk<C>(T(0), T(0));
        }
      }
#pragma unroll
      for (int b = 0; b < HB; ++b) {
        if (Rt::dropped(b0 + b)) continue;
        const int i = Rt::row(s, b0 + b, N);
        if (!(Rt::low(b0 + b) || Rt::high(b0 + b)) && i < 0) continue;
        const int oo = i * lout.row + p * lout.ps;
        const T k1 = T(i >= N / 2 + 1 ? i - N : i), kv1 = twopi * k1;
        const T n2 = k1 * k1 + k2 * k2;
        const bool zero = n2 == T(0);
        const T inv = twopi / n2;
        const T e0 = k1 * k2, e1 = k2 * k2 - k1 * k1;
        const C v0 = v[0][b0 + b], v1 = v[1][b0 + b];
        const C q = cmk<C>((e0 * v0.x + e1 * v1.x) * inv, (e0 * v0.y + e1 * v1.y) * inv);
        const C Lh[2] = {cmk<C>(k2 * q.x, k2 * q.y), cmk<C>(-k1 * q.x, -k1 * q.y)};  // L / i
        const T nu = visc_from_k2<T>(a.visc, kv1 * kv1 + kv2 * kv2, inv_k0sq);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const C x = uc[b][c], w = wc[b][c];
          const C d = zero ? cmk<C>(T(0), T(0)) : cmk<C>(Lh[c].y + nu * x.x, nu * x.y - Lh[c].x);
          const C t = use_u ? cmk<C>(x.x + dd * d.x, x.y + dd * d.y) : d;
          out[c * lout.comp + oo] = cmk<C>(fma(ct, t.x - w.x, w.x), fma(ct, t.y - w.y, w.y));
        }
      }
    }
  }
}

}  // namespace azb
