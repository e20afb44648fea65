// Fused transform passes of the spectral-viscosity incompressible Euler
// right-hand side.
//
// One 3-D right-hand side (reference: IncompressibleEuler::dudt,
// include/azeban/equations/incompressible_euler.hpp:103-120) runs as five
// passes, each one HBM read and one HBM write of the live array.  The
// intermediates keep the component index innermost, so a tile of consecutive
// columns is one contiguous run per row in every pass:
//   1 k_columns<PAD>    inverse along x: u_hat [3][N][N][Nh] -> A1 [M][N][Nh][3]
//                       (copy_to_padded along x fused into the loads)
//   2 k_columns<PAD>    inverse along y: A1 -> A2 [M][M][Nh][3]
//   3 k_zline           along z: c2r, max|u|, B = u (x) u, r2c, keep k < Nh:
//                       A2 -> B1 [M][M][Nh][6]
//   4 k_columns<TRUNC>  forward along y, keep the N retained rows: B1 -> B2 [M][N][Nh][6]
//   5 k_fwd_epilogue    forward along x, keep retained rows, then computeDudt
//                       (Leray projection of i k.B, spectral viscosity)
//                       and the SSP-RK3 stage combination: B2 + u -> out
// 2-D uses passes 1 (along x), 3 (along y) and a last pass k_epilogue2d, with A1
// [M][Nh][2] and B1 [M][Nh][3].  k_columns and k_epilogue2d are in line.cuh, k_zline
// in zline.cuh; 3-D solves with M = 384 have k_cols and k_zfused (zfused.cuh) in their
// place (kRegisterColumns).
#pragma once

#include "az_types.h"
#include "fft_core.cuh"

namespace azb {

enum ColMode : int { COL_PLAIN = 0, COL_PAD = 1, COL_TRUNC = 2 };

// Padded row m -> source row of an axis of unpadded length n, or -1 for a
// zero (copy_to_padded_functions.hpp:36-51 in the reference; the Nyquist
// index n/2 stays on the positive side).
__device__ __forceinline__ int pad_src_row(int m, int n, int L) {
  if (m < n / 2 + 1) return m;
  if (m < n / 2 + 1 + L - n) return -1;
  return m - (L - n);
}

// Padded row m -> retained row of the unpadded axis, or -1 if dropped
// (inverse of i_B = i >= n/2+1 ? L - n + i : i, incompressible_euler.hpp:294-299).
__device__ __forceinline__ int retained_row(int m, int n, int L) {
  if (m <= n / 2) return m;
  if (m >= L - n / 2 + 1) return m - (L - n);
  return -1;
}

struct ColArgs {
  const void* in;
  void* out;
  const void* tw;
  long long ninner;  // contiguous columns per slab
  int ntile;         // ceil(ninner / NC)
  int n_short;       // unpadded length (input rows for PAD, output rows for TRUNC)
  long long in_row, out_row;
  long long in_outer, out_outer;
  long long in_comp, out_comp;
  long long in_mem, out_mem;
  Ctrl* ctrl;     // optional: per-member skip flags
  int clear_max;  // nonzero: the first pass; reset the member's CFL accumulator
  int begin;      // StepBegin, with its max_dt
  double max_dt;
  int pdl;        // to launch_pass: may be a programmatic dependent; to the kernel: is one
  int in_ci;      // input component interleave: column p reads component p % in_ci
                  // at in_comp stride, position p / in_ci (1: plain columns)
  // Grouped columns (grp > 0): column p is entry q = p % grp of group
  // g = p / grp; entries q >= grp_valid are padding (not read, not written),
  // and the input of entry q sits at g * in_grp + (q / in_ci or q).
  int grp, grp_valid;
  long long in_grp;
};

// Entry of a column pass: false if the member (blockIdx.z) is to be skipped.
// The values that other blocks read here (time, t_end) are not written here.
__device__ __forceinline__ bool pass_enter(const ColArgs& a) {
  if (a.pdl) pdl_enter();
  if (a.ctrl == nullptr) return true;
  Ctrl* c = a.ctrl + blockIdx.z;
  const bool skip = a.begin == BEGIN_NONE ? c->skip != 0 : a.begin == BEGIN_SIM ? !(c->time < c->t_end) : false;
  if (a.clear_max && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
    // The CFL accumulator is read only after the product pass of this
    // right-hand side, which runs after this kernel.
    if (!skip) {
      c->umax64 = 0ull;
      c->umax32 = 0u;
    }
    if (a.begin != BEGIN_NONE) {
      c->skip = skip ? 1 : 0;
      if (!skip) c->max_dt = a.begin == BEGIN_SIM ? fmin(c->t_end - c->time, a.max_dt) : a.max_dt;
      if (a.begin == BEGIN_HOST) c->err = 0;
    }
  }
  return !skip;
}

// Batched column transforms along a strided axis.  grid = (ntile * nouter,
// ncomp, nmembers); block = NC * L/E threads.
// STD: the unpadded length is 2L/3 (the 3/2 rule, a.n_short == 2L/3), known at
// compile time, so the padding and truncation maps fold: rows whose fate does
// not depend on the thread's row offset are kept, zeroed or dropped without a
// test.
template <typename T, int L, int NC, int S, int MODE, int V, bool STD = false>
__global__ void __launch_bounds__(NC * Plan<L, V>::TPL) k_cols(ColArgs a) {
  using C = cvec<T>;
  using P = Plan<L, V>;
  extern __shared__ __align__(16) unsigned char az_smem[];
  C* tw = reinterpret_cast<C*>(az_smem);
  C* sm = tw + L;
  const int member = blockIdx.z;
  if (!pass_enter(a)) return;
  const int tile = blockIdx.x % a.ntile;
  const int outer = blockIdx.x / a.ntile;
  const int comp = blockIdx.y;
  const int col = threadIdx.x % NC;
  const int tl = threadIdx.x / NC;
  const long long p = (long long)tile * NC + col;
  bool valid = p < a.ninner;
  long long pin;
  if (a.grp > 0) {
    const long long g = p / a.grp;
    const int q = int(p - g * a.grp);
    valid = valid && q < a.grp_valid;
    pin = g * a.in_grp + (a.in_ci == 1 ? comp * a.in_comp + q : (q % a.in_ci) * a.in_comp + q / a.in_ci);
  } else {
    pin = a.in_ci == 1 ? comp * a.in_comp + p : (p % a.in_ci) * a.in_comp + p / a.in_ci;
  }
  const C* in = reinterpret_cast<const C*>(a.in) + member * a.in_mem + outer * a.in_outer + pin;
  C* out = reinterpret_cast<C*>(a.out) + member * a.out_mem + comp * a.out_comp +
           outer * a.out_outer + p;
  const int n = STD ? 2 * L / 3 : a.n_short;
  // Row offsets fit 32 bits (the launcher checks L * stride < 2^31).
  const int in_row = int(a.in_row);
  const int out_row = int(a.out_row);
  auto load = [&](int m) -> C {
    int src = m;
    if constexpr (MODE == COL_PAD) src = pad_src_row(m, n, L);
    if (!valid || src < 0) return cmk<C>(T(0), T(0));
    return in[src * in_row];
  };
  auto store = [&](int m, C v) {
    int dst = m;
    if constexpr (MODE == COL_TRUNC) dst = retained_row(m, n, L);
    if (valid && dst >= 0) out[dst * out_row] = v;
  };
  // The first-stage loads go out before the twiddle table is fetched, so the
  // two global round trips overlap.
  C v[P::E];
  fft_load<C, L, P>(v, tl, load);
  load_twiddles<C, L>(tw, reinterpret_cast<const C*>(a.tw));
  __syncthreads();
  fft_run<C, S, L, NC, false, P>(sm, v, tw, col, tl, store);
}

// Layout of one member's state: element (component c, retained row i, mode
// p) at c * comp + i * row + p * ps.  Planar, the reference's [d][N]..[Nh]:
// comp = N^{d-1} Nh, row = N^{d-2} Nh, ps = 1.  Component innermost,
// [N]..[Nh][d] (the stepper's stage buffers): comp = 1, row = d N^{d-2} Nh,
// ps = d, so a tile's few modes are d times more contiguous bytes per row.
struct StateLayout {
  int comp, row, ps;
};

struct EpiArgs {
  const void* B;  // [M][modes][NB], component innermost
  const void* u;
  const void* u0;
  void* out;
  const void* tw;
  long long ninner;  // modes per retained row: N*Nh (3-D) or Nh (2-D)
  int ntile;
  int N, nh;
  long long B_row, B_mem;
  StateLayout lu, lu0, lout;  // layouts of u, u0 and out
  long long u_mem;
  int mode;
  Visc visc;
  Ctrl* ctrl;
  double C, Md;  // MODE_RK1: dt = min(C / (N u_max), max_dt), u_max = max / M^d, is set here
  int end_step;  // the last pass of a step inside simulate_until: time += dt
  int pdl;       // to launch_pass: may be a programmatic dependent; to the kernel: is one
  // > 0: B's modes are grouped, nh per group with a group stride of b_grp
  // elements (the padded rows of B2 [M][N][b_grp]); 0: contiguous modes.
  long long b_grp;
};

// nu(|k|) of the reference's viscosity laws
// (include/azeban/equations/spectral_viscosity.hpp:27-123), evaluated from
// |k|^2: SmoothCutoff1D takes (|k|/k0)^2 = |k|^2 / k0^2 and Quadratic
// (|k|/2 pi)^2 = |k|^2 / (2 pi)^2, so neither needs the square root.  Step1D
// compares |k| > k0 as the reference does, on the square root.
template <typename T> __device__ __forceinline__ T visc_from_k2(const Visc& v, T absk2, T inv_k0sq) {
  switch (v.type) {
    case VISC_SMOOTH_CUTOFF: {
      const T k2 = absk2 * inv_k0sq;
      const T k4 = k2 * k2;
      const T k8 = k4 * k4;
      const T k16 = k8 * k8;
      const T k18 = k16 * k2;
      const T q = T(1) - exp(-k18);
      const T pk = (v.s == 1.0) ? absk2 : T(pow(absk2, T(v.s)));
      return -T(v.eps) * pk * q;
    }
    case VISC_STEP: {
      const T k = sqrt(absk2);
      const T q = k > T(v.k0) ? T(1) : T(0);
      const T pk = (v.s == 1.0) ? k * k : T(pow(k, T(2 * v.s)));
      return -T(v.eps) * pk * q;
    }
    case VISC_QUADRATIC: {
      const T kn2 = absk2 * T(1.0 / (4 * 3.14159265358979323846 * 3.14159265358979323846));
      return -T(v.eps) * fmax(T(0), kn2 - T(v.N));
    }
    default:
      return T(0);
  }
}

// The step size of a member, by one thread of each block: the first stage takes
// it from the CFL maximum (incompressible_euler.hpp:116-124), the first block
// keeps it for the later stages and, at the step's end, moves the clock
// (simulation.cpp:100).  What the other blocks read is not written here.
template <typename T> __device__ __forceinline__ double epilogue_dt(const EpiArgs& a, int member) {
  if (a.mode == MODE_DUDT || a.ctrl == nullptr) return 0.0;
  Ctrl* c = a.ctrl + member;
  if (a.mode != MODE_RK1) {
    const double dt = c->dt;
    if (a.end_step && blockIdx.x == 0) {
      c->time += dt;
      c->nsteps += 1;
    }
    return dt;
  }
  const double m = sizeof(T) == 4 ? (double)__uint_as_float(c->umax32) : __longlong_as_double((long long)c->umax64);
  const double u_max = m / a.Md;
  const double dt = fmin(a.C / ((double)a.N * u_max), c->max_dt);
  if (blockIdx.x == 0) c->dt = dt;
  return dt;
}

// Forward transform along x of the six product components, kept at the N
// retained rows, then per mode: L = (I - k k^T/|k|^2)(i k.B_hat),
// dudt = |k| = 0 ? 0 : -L + nu(|k|) u_hat (incompressible_euler.hpp:230-347,
// incompressible_euler_functions.hpp:47-112), then the stage combination:
//   MODE_DUDT: out = dudt
//   MODE_RK1:  out = u + dt dudt                      (ssp_rk3.hpp:55)
//   MODE_RK2:  out = 3/4 u0 + 1/4 (u + dt dudt)       (ssp_rk3.hpp:57-58)
//   MODE_RK3:  out = 2/3 (u + dt dudt) + 1/3 u0       (ssp_rk3.hpp:60-61)
// grid = (ntile, nmembers); block = NB * NCM * L/E.
// FP32 std plans of up to 384 threads: two resident CTAs per SM.
template <typename T, int L, int NCM, int V> struct EpiMinBlocks {
  static constexpr int value =
      (sizeof(T) == 4 && V == 0 && products(3) * NCM * Plan<L, V>::TPL <= 384) ? 2 : 1;
};

// STD: N == 2L/3 (the 3/2 rule), known at compile time, so the retained-row
// map and the per-mode row loops fold.
template <typename T, int L, int NCM, int V, bool STD>
__global__ void __launch_bounds__(products(3) * NCM * Plan<L, V>::TPL,
                                  EpiMinBlocks<T, L, NCM, V>::value)
    k_fwd_epilogue(EpiArgs a) {
  using C = cvec<T>;
  using P = Plan<L, V>;
  constexpr int DIM = 3;
  constexpr int NB = products(DIM);
  constexpr int NC = NB * NCM;
  constexpr int SROW = NC;
  constexpr int TPL = P::TPL;
  constexpr int NT = NC * TPL;
  extern __shared__ __align__(16) unsigned char az_smem[];
  C* tw = reinterpret_cast<C*>(az_smem);
  C* sm = tw + L;
  const int member = blockIdx.y;
  if (a.pdl) pdl_enter();
  if (a.ctrl != nullptr && a.ctrl[member].skip) return;
  const int tid = threadIdx.x;
  const int tile = blockIdx.x;
  __shared__ double step_dt;
  const int N = STD ? 2 * L / 3 : a.N;
  {
    // column col = (mode pl, component c) with c fastest: one contiguous run
    const int col = tid % NC;
    const int tl = tid / NC;
    const int pl = col / NB;
    const long long p = (long long)tile * NCM + pl;
    const bool valid = p < a.ninner;
    long long bcol;
    if (a.b_grp > 0) {
      const long long g = p / a.nh;
      bcol = g * a.b_grp + (p - g * a.nh) * NB + (col - pl * NB);
    } else {
      bcol = (long long)tile * NC + col;
    }
    const C* Bp = reinterpret_cast<const C*>(a.B) + member * a.B_mem + bcol;
    const int B_row = int(a.B_row);  // L * B_row < 2^31, checked by the launcher
    // First-stage loads before the twiddle table, as in k_cols.
    C v[P::E];
    fft_load<C, L, P>(v, tl, [&](int m) -> C { return valid ? Bp[m * B_row] : cmk<C>(T(0), T(0)); });
    load_twiddles<C, L>(tw, reinterpret_cast<const C*>(a.tw));
    if (tid == 0) step_dt = epilogue_dt<T>(a, member);  // behind the loads in flight
    __syncthreads();
    fft_run<C, -1, L, SROW, true, P>(sm, v, tw, col, tl, [&](int m, C x) {
      const int i = retained_row(m, N, L);
      if (i >= 0) sm[i * SROW + col] = x;
    });
  }
  __syncthreads();

  const T dt = T(step_dt);
  const T twopi = T(2 * 3.14159265358979323846);
  const C* u = reinterpret_cast<const C*>(a.u) + member * a.u_mem;
  const C* u0 = reinterpret_cast<const C*>(a.u0) + member * a.u_mem;
  C* out = reinterpret_cast<C*>(a.out) + member * a.u_mem;
  const StateLayout lu = a.lu, lu0 = a.lu0, lout = a.lout;  // offsets < 2^31, checked by the launcher
  const T inv_k0sq = T(1.0 / (a.visc.k0 * a.visc.k0));
  // The stage combination as a uniform coefficient instead of per-element
  // branches: t = u + dt d (d itself for MODE_DUDT), r = ct t + (1 - ct) u0,
  // evaluated as u0 + ct (t - u0) (u0 = 0 and ct = 1 for MODE_DUDT and
  // MODE_RK1).  The weights then sum to exactly one in either precision: with
  // the FP32 weights 2/3 and 1/3 the sum is 1 + 3e-8, which scales the state
  // by that factor at every step.  t - u0 is exact while t and u0 lie within a
  // factor of two (Sterbenz), so the form rounds once, in the fma.
  const bool use_u = a.mode != MODE_DUDT;
  const T dd = use_u ? dt : T(1);
  const T ct = a.mode == MODE_RK2 ? T(0.25) : a.mode == MODE_RK3 ? T(2.0 / 3.0) : T(1);
  // NT is a multiple of NCM, so a thread keeps one mode column pl (and its
  // second and third wavenumbers) and walks the retained rows i.
  const int pl = tid % NCM;
  const int p = tile * NCM + pl;
  if (p >= a.ninner) return;
  const int j = p / a.nh;
  const int kk = p - j * a.nh;
  const T k2 = twopi * T(j >= N / 2 + 1 ? j - N : j);
  const T k3 = twopi * T(kk);
  // Rows of this thread: i = tid / NCM + it * ISTEP.  For the first MAXIT
  // rows (all of them when N <= 2L/3 + 1, the 3/2 padding) its state values
  // (u, and u0 for the RK2/RK3 combinations) are loaded first, so their
  // latencies overlap; further rows load as they go.
  constexpr int ISTEP = NT / NCM;
  constexpr int MAXIT = (2 * L / 3 + 1 + ISTEP - 1) / ISTEP;
  const int i0 = tid / NCM;
  const bool need_u0 = a.mode == MODE_RK2 || a.mode == MODE_RK3;
  C uv[MAXIT][DIM], wv[MAXIT][DIM];
#pragma unroll
  for (int it = 0; it < MAXIT; ++it) {
    const int i = i0 + it * ISTEP;
    if (i < N) {
      const int ou = i * lu.row + p * lu.ps, ow = i * lu0.row + p * lu0.ps;
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        uv[it][c] = u[c * lu.comp + ou];
        wv[it][c] = need_u0 ? u0[c * lu0.comp + ow] : cmk<C>(T(0), T(0));
      }
    }
  }
  auto process = [&](int i, const C (&uc_)[DIM], const C (&wc_)[DIM]) {
    const int oo = i * lout.row + p * lout.ps;
    const int i_ = i >= N / 2 + 1 ? i - N : i;
    const T k1 = twopi * T(i_);
    C Bv[NB];
    if constexpr (sizeof(C) == 8) {
      // 16-byte reads: with rows of NB * NCM elements a quarter-warp's reads
      // fall on distinct bank groups
      const float4* b4 = reinterpret_cast<const float4*>(sm + i * SROW + pl * NB);
#pragma unroll
      for (int c = 0; c < NB / 2; ++c) {
        const float4 q = b4[c];
        Bv[2 * c] = cmk<C>(q.x, q.y);
        Bv[2 * c + 1] = cmk<C>(q.z, q.w);
      }
    } else {
#pragma unroll
      for (int c = 0; c < NB; ++c) Bv[c] = sm[i * SROW + pl * NB + c];
    }
    // b = i k.B (force = 0), then L = b - k (k.b) / |k|^2
    C Lh[DIM];
    T absk2;
    absk2 = k1 * k1 + k2 * k2 + k3 * k3;
    // B order: 0 B11, 1 B21, 2 B22, 3 B31, 4 B32, 5 B33
    const C b1 = cmk<C>(-k1 * Bv[0].y - k2 * Bv[1].y - k3 * Bv[3].y,
                        k1 * Bv[0].x + k2 * Bv[1].x + k3 * Bv[3].x);
    const C b2 = cmk<C>(-k1 * Bv[1].y - k2 * Bv[2].y - k3 * Bv[4].y,
                        k1 * Bv[1].x + k2 * Bv[2].x + k3 * Bv[4].x);
    const C b3 = cmk<C>(-k1 * Bv[3].y - k2 * Bv[4].y - k3 * Bv[5].y,
                        k1 * Bv[3].x + k2 * Bv[4].x + k3 * Bv[5].x);
    const T inv = T(1) / absk2;
    const C sk = cmk<C>((k1 * b1.x + k2 * b2.x + k3 * b3.x) * inv, (k1 * b1.y + k2 * b2.y + k3 * b3.y) * inv);
    Lh[0] = cmk<C>(b1.x - k1 * sk.x, b1.y - k1 * sk.y);
    Lh[1] = cmk<C>(b2.x - k2 * sk.x, b2.y - k2 * sk.y);
    Lh[2] = cmk<C>(b3.x - k3 * sk.x, b3.y - k3 * sk.y);
    const T nu = visc_from_k2<T>(a.visc, absk2, inv_k0sq);
    const bool zero = absk2 == T(0);
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      const C uc = uc_[c];
      const C d = zero ? cmk<C>(T(0), T(0)) : cmk<C>(-Lh[c].x + nu * uc.x, -Lh[c].y + nu * uc.y);
      const C t = use_u ? cmk<C>(uc.x + dd * d.x, uc.y + dd * d.y) : d;
      const C w = wc_[c];
      out[c * lout.comp + oo] = cmk<C>(fma(ct, t.x - w.x, w.x), fma(ct, t.y - w.y, w.y));
    }
  };
#pragma unroll
  for (int it = 0; it < MAXIT; ++it) {
    const int i = i0 + it * ISTEP;
    if (i < N) process(i, uv[it], wv[it]);
  }
  for (int i = i0 + MAXIT * ISTEP; i < N; i += ISTEP) {
    const int ou = i * lu.row + p * lu.ps, ow = i * lu0.row + p * lu0.ps;
    C uc[DIM], wc[DIM];
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      uc[c] = u[c * lu.comp + ou];
      wc[c] = need_u0 ? u0[c * lu0.comp + ow] : cmk<C>(T(0), T(0));
    }
    process(i, uc, wc);
  }
}

}  // namespace azb
