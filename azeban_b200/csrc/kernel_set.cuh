// Launchers for every pass kernel of one (precision, transform length L).
// Each instantiation unit (inst_<prec>_<L>.cu) compiles one KernelSet, so the
// build parallelises over lengths.
#pragma once

#include <cuda_runtime.h>

#include "euler_kernels.cuh"
#include "line.cuh"
#include "rows.cuh"
#include "zfused.cuh"
#include "zline.cuh"

namespace azb {

// KernelSet::cols takes the plain kinds and, where reg3 is set, COLK_PAD_INV and
// COLK_TRUNC_FWD; else those are KernelSet::columns', with COLK_PAD_STATE, the padding
// pass that reads the state.
enum ColKind : int { COLK_PAD_INV = 0, COLK_PLAIN_INV = 1, COLK_TRUNC_FWD = 2, COLK_PLAIN_FWD = 3, COLK_PAD_STATE = 4 };

// v: plan variant (0 std, 1 wide; see Plan<L, V>).  The launchers pick the tile
// of a launch and set the ntile of its arguments.
struct KernelSet {
  int L;
  int precision;  // 0 FP64, 1 FP32
  bool reg3;      // 3-D solves take cols and the product pass k_zfused (kRegisterColumns)
  cudaError_t (*cols)(int v, int kind, const ColArgs&, long long nouter, unsigned ncomp, unsigned nmem, cudaStream_t);
  cudaError_t (*product)(int dim, const ZArgs&, cudaStream_t);
  // kinds COLK_PAD_INV, COLK_PAD_STATE and COLK_TRUNC_FWD
  cudaError_t (*columns)(int kind, const ColArgs&, long long nouter, unsigned nmem, cudaStream_t);
  // last pass of a 3-D and of a 2-D right-hand side
  cudaError_t (*epilogue3)(int v, const EpiArgs&, unsigned nmem, cudaStream_t);
  cudaError_t (*epilogue2)(const EpiArgs&, unsigned nmem, cudaStream_t);
  cudaError_t (*c2r)(const RealRowArgs&, cudaStream_t);
  cudaError_t (*r2c)(int v, const RealRowArgs&, cudaStream_t);
};

// Lengths whose 3-D passes keep a column in the registers of a few threads (k_cols,
// k_zfused) instead of k_columns and k_zline.  At 384 the latter are faster under the
// 3/2 rule (a step of four 256^3 FP32 members 16400 us against 17500, of one in FP64 8280
// against 9370; with N = 214 4810 against 4120 in FP32, 6780 against 8080 in FP64) and as
// far from FP64, 3.1e-6 and 8e-15 in the 2-norm of a Taylor-Green step without its leading
// modes.  But they add in another order, and single modes beside the leading ones move by
// up to 1.2e-3 (FP32) and 6e-12 (FP64) of the root mean square of the others (either form
// is half as far from FP64 there), which the tolerance of the 256^3 vortex solves in
// perf/cases.py does not allow.
template <int L> inline constexpr bool kRegisterColumns = L == 384;

constexpr int kpow2floor(int x) {
  int p = 1;
  while (p * 2 <= x) p *= 2;
  return p;
}
constexpr int kclamp(int x, int lo, int hi) { return x < lo ? lo : (x > hi ? hi : x); }

template <typename T, int L, int V> struct Tiles {
  static constexpr int CB = int(sizeof(cvec<T>));
  static constexpr int NC = kclamp(kpow2floor(49152 / (L * CB)), 2, 32);
  // FP32 at L = 768: twice the budget, 4 modes per CTA (one CTA per SM;
  // measured 2.95 ms against 3.67 ms with 2 modes at 512^3).
  static constexpr int NCM3 = kclamp(kpow2floor(((CB == 8 && L == 768) ? 163840 : 81920) / (L * 6 * CB)), 1, 16);
  // few modes for launches that would leave SMs without a CTA
  static constexpr int NCM3_NARROW = NCM3 < 2 ? NCM3 : 2;
};

// Line pairs per CTA of the product pass.  Wide: about 96 threads (one
// middle-stage butterfly each), 128 for the plans with RM = 12 (measured best of 1 to
// 12 pairs; L = 768 FP32 with one pair and with two: 3-D 4148 and 4557 us, 2-D 1220 and
// 1267, off the 3/2 rule 1436 and 2037).  Narrow, taken when the wide chunks would not
// give every SM its CTAs: one warp, or one pair where that is half a warp or more (two
// of them take turns in the outer stages: a step of one 2-D N = 150
// M = 256 FP32 solve 79 us with two pairs, 70 with one).
template <typename T, int L, int DIM> struct ZLineTile {
  static constexpr int S = L / ZPlan<T, L, DIM>::RM;
  static constexpr int WIDE = S >= 96 ? 1 : ZPlan<T, L, DIM>::RM == 12 ? 128 / S : 96 / S;
  static constexpr int NARROW = S >= 16 ? 1 : 32 / S;
};

// Radix plans and tiles of the passes of line.cuh: columns (modes) of a tile,
// threads, and the resident CTAs the register cap is set for.  A CTA's tile is
// 128 bytes of a row where its work area stays below some 60 KB: loads in flight
// need room in the L1 cache beside it (L = 384, 16 columns, 256 threads: three
// CTAs per SM 583 us, four 749 us).  Each row: column passes, then the 2-D last
// pass.  Measured (us; 2.4e8 points in FP32, 6e7 in FP64, the three stages of a
// step averaged).  Columns: 96 as 12.8 by 16 columns 590, by 32 659; 192 as 16.12
// 632, 12.16 760, 24.8 656; 768 as 32.24 1350, 12.8.8 1554, 16.6.8 1634; FP64 192
// as 16.12 279, 24.8 303, 8.4.6 339.  32 in FP32 by 32 columns: a step of 915 3-D solves
// with N = 18 1590, by 16 1909; shorter lengths and FP64 are slower by twice the columns.
// Last pass, 2-D: 192 x256 as 24.8 42.8, 16.12 44.4 (16 modes 46.3); 384 x192 as 48.8
// 115, 24.16 131; 768 x64 as 12.8.8 by 8 modes 194, by 4 221; FP64 192 as 8.3.8 475, 24.8
// 499, 1536 x1 as 16.12.8 by 2 modes 29, 12.16.8 by 1 38.
template <typename T, int L> struct PadTile;
template <typename T, int L> struct Epi2Tile;
#define AZB_LINE(Tv, Lv, A, M, B, NC_, NT_, MINB_, A2, M2, B2, NCM_, NT2, MINB2) \
  template <> struct PadTile<Tv, Lv> {                                          \
    using P = LinePlan<Tv, Lv, A, M, B>;                                        \
    static constexpr int NC = NC_, NT = NT_, MINB = MINB_;                      \
  };                                                                            \
  template <> struct Epi2Tile<Tv, Lv> {                                         \
    using P = LinePlan<Tv, Lv, A2, M2, B2>;                                     \
    static constexpr int NCM = NCM_, NT = NT2, MINB = MINB2;                    \
  };
AZB_LINE(float, 4, 2, 1, 2, 16, 32, 8, 2, 1, 2, 8, 32, 8)
AZB_LINE(float, 6, 3, 1, 2, 16, 32, 8, 3, 1, 2, 8, 32, 8)
AZB_LINE(float, 8, 4, 1, 2, 16, 64, 8, 4, 1, 2, 8, 32, 8)
AZB_LINE(float, 12, 4, 1, 3, 16, 64, 8, 4, 1, 3, 8, 32, 8)
AZB_LINE(float, 16, 4, 1, 4, 16, 64, 8, 4, 1, 4, 8, 64, 8)
AZB_LINE(float, 24, 6, 1, 4, 16, 64, 8, 6, 1, 4, 8, 64, 8)
AZB_LINE(float, 32, 8, 1, 4, 32, 128, 6, 8, 1, 4, 8, 64, 8)
AZB_LINE(float, 48, 8, 1, 6, 16, 128, 6, 8, 1, 6, 8, 64, 8)
AZB_LINE(float, 64, 8, 1, 8, 16, 128, 6, 8, 1, 8, 8, 128, 4)
AZB_LINE(float, 96, 12, 1, 8, 16, 128, 6, 12, 1, 8, 8, 96, 6)
AZB_LINE(float, 128, 16, 1, 8, 16, 128, 6, 16, 1, 8, 8, 128, 4)
AZB_LINE(float, 192, 16, 1, 12, 16, 128, 6, 24, 1, 8, 8, 128, 4)
AZB_LINE(float, 256, 16, 1, 16, 16, 256, 3, 16, 1, 16, 8, 128, 4)
AZB_LINE(float, 384, 24, 1, 16, 16, 256, 3, 48, 1, 8, 8, 192, 2)
AZB_LINE(float, 512, 32, 1, 16, 8, 128, 4, 32, 1, 16, 4, 128, 3)
AZB_LINE(float, 768, 32, 1, 24, 8, 192, 3, 12, 8, 8, 8, 384, 1)
AZB_LINE(float, 1024, 32, 1, 32, 8, 256, 2, 16, 8, 8, 4, 256, 2)
AZB_LINE(float, 1536, 16, 4, 24, 4, 128, 3, 16, 12, 8, 2, 192, 3)
AZB_LINE(double, 4, 2, 1, 2, 8, 32, 8, 2, 1, 2, 4, 32, 8)
AZB_LINE(double, 6, 3, 1, 2, 8, 32, 8, 3, 1, 2, 4, 32, 8)
AZB_LINE(double, 8, 4, 1, 2, 8, 32, 8, 4, 1, 2, 4, 32, 8)
AZB_LINE(double, 12, 4, 1, 3, 8, 32, 8, 4, 1, 3, 4, 32, 8)
AZB_LINE(double, 16, 4, 1, 4, 8, 32, 8, 4, 1, 4, 4, 32, 8)
AZB_LINE(double, 24, 6, 1, 4, 8, 64, 8, 6, 1, 4, 4, 32, 8)
AZB_LINE(double, 32, 8, 1, 4, 8, 64, 8, 8, 1, 4, 4, 64, 8)
AZB_LINE(double, 48, 8, 1, 6, 8, 64, 8, 8, 1, 6, 4, 64, 6)
AZB_LINE(double, 64, 8, 1, 8, 8, 64, 8, 8, 1, 8, 4, 64, 6)
AZB_LINE(double, 96, 12, 1, 8, 8, 96, 6, 12, 1, 8, 4, 64, 6)
AZB_LINE(double, 128, 16, 1, 8, 8, 128, 4, 16, 1, 8, 4, 64, 6)
AZB_LINE(double, 192, 16, 1, 12, 8, 128, 4, 8, 3, 8, 4, 96, 4)
AZB_LINE(double, 256, 16, 1, 16, 8, 128, 4, 8, 4, 8, 4, 128, 3)
AZB_LINE(double, 384, 24, 1, 16, 8, 128, 3, 8, 6, 8, 4, 192, 2)
AZB_LINE(double, 512, 32, 1, 16, 4, 128, 3, 8, 8, 8, 2, 128, 3)
AZB_LINE(double, 768, 32, 1, 24, 4, 128, 3, 12, 8, 8, 2, 192, 2)
AZB_LINE(double, 1024, 16, 4, 16, 4, 256, 2, 16, 8, 8, 1, 128, 3)
AZB_LINE(double, 1536, 16, 12, 8, 2, 256, 2, 16, 12, 8, 2, 384, 1)
#undef AZB_LINE

// Tiles of 32 bytes of a row, for launches whose ordinary tiles would leave some
// of the 148 SMs without a CTA.
inline bool idle_sms(long long ctas) { return ctas < 148; }
// (One FP64 2-D solve with M = 512: radices 8.8.8 instead of 32.16 here and 16.8.4
// instead of 8.8.8 in the last pass, 66 us a step instead of 72.)
template <typename T, int L> struct PadNarrowPlan { using P = typename PadTile<T, L>::P; };
template <> struct PadNarrowPlan<double, 512> { using P = LinePlan<double, 512, 8, 8, 8>; };
template <typename T, int L> struct PadTileNarrow {
  using P = typename PadNarrowPlan<T, L>::P;
  static constexpr int NC = 32 / int(sizeof(cvec<T>));
  static constexpr int NT = kclamp((NC * (P::O > P::S ? P::O : P::S) + 31) / 32 * 32, 32, 256);
  static constexpr int MINB = 1;
};
// The last pass of 2-D solves takes them for launches of at most one ordinary tile for
// two SMs (10 FP32 solves with N = 214 and M = 384, 140 ordinary tiles: 113 us a step with
// narrow ones, 89 without), and with radices that leave a thread of the last stage eight
// or four rows instead of sixteen or eight (one FP32 solve: N = 150, M = 256 70 -> 60; N =
// 298, M = 512 90 -> 72; in FP64 M = 512 see PadNarrowPlan).
template <typename T, int L> struct Epi2NarrowPlan { using P = typename Epi2Tile<T, L>::P; };
template <> struct Epi2NarrowPlan<float, 256> { using P = LinePlan<float, 256, 32, 1, 8>; };
template <> struct Epi2NarrowPlan<float, 512> { using P = LinePlan<float, 512, 8, 8, 8>; };
template <> struct Epi2NarrowPlan<double, 512> { using P = LinePlan<double, 512, 16, 8, 4>; };
template <typename T, int L> struct Epi2TileNarrow {
  using P = typename Epi2NarrowPlan<T, L>::P;
  static constexpr int NCM = 16 / int(sizeof(cvec<T>));
  static constexpr int NT = kclamp((NCM * (2 * P::O > P::S ? 2 * P::O : P::S) + 31) / 32 * 32, 32, 256);
  static constexpr int MINB = 1;
};
// First pass of a 3-D right-hand side in FP32 at L = 768: it reads the state in
// runs of a tile's columns, rows a plane apart, so 16 columns (128 bytes).
template <typename T, int L> struct PadStateTile : PadTile<T, L> {};
template <> struct PadStateTile<float, 768> {
  using P = LinePlan<float, 768, 32, 1, 24>;
  static constexpr int NC = 16, NT = 192, MINB = 2;
};

// Allows a kernel `bytes` of dynamic shared memory.  The 48 KB that need no asking count
// its static shared memory too (the last pass at L = 512 in FP64 takes 48 KB and a step
// size beside them).
template <typename K> inline cudaError_t set_smem(K kernel, size_t bytes) {
  cudaFuncAttributes f;
  const cudaError_t ce = cudaFuncGetAttributes(&f, kernel);
  if (ce != cudaSuccess || f.sharedSizeBytes + bytes <= 48 * 1024) return ce;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
}

// Launches a pass kernel.  a.pdl on entry: it may start before the kernel in front of
// it on the stream has ended (it waits for that itself, pdl_enter); done for launches of
// at most one CTA for every two of the 148 SMs, and a.pdl then tells the kernel whether
// it was.  The CTAs of an early start go where room is first, several to an SM beside
// idle ones, and to SMs still split between shared memory and L1 for the kernel in
// front: steps (us; limit of 74 CTAs, 148, 296, none early) 2-D M = 768 FP32 58, 65, 65,
// 58; M = 512 N = 298 FP32 90, 94, 123, 90; M = 48 N = 32 FP64 35, 35, 35, 37; 3-D
// M = 48 N = 26 FP64 74, 74, 88, 74; all launches early: a 512^3 FP32 step 43500 instead of
// 34700.
template <typename K, typename A, typename... R>
inline cudaError_t launch_pass(K k, dim3 g, int nt, size_t smem, cudaStream_t st, A a, const R&... rest) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = g;
  cfg.blockDim = dim3(unsigned(nt));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  a.pdl = a.pdl && (long long)g.x * g.y * g.z <= 148 / 2 ? 1 : 0;
  cfg.numAttrs = unsigned(a.pdl);
  return cudaLaunchKernelEx(&cfg, k, a, rest...);
}

template <typename T, int L, int V> struct LaunchV {
  using C = cvec<T>;
  using TS = Tiles<T, L, V>;
  static constexpr int TPL = Plan<L, V>::TPL;

  template <int S, int MODE, bool STD, int NC>
  static cudaError_t col_run(ColArgs a, long long nouter, unsigned ncomp, unsigned nmem, cudaStream_t st) {
    const size_t smem = size_t(L + L * NC) * sizeof(C);
    auto k = k_cols<T, L, NC, S, MODE, V, STD>;
    static const cudaError_t attr = set_smem(k, smem);
    if (attr != cudaSuccess) return attr;
    a.ntile = int((a.ninner + NC - 1) / NC);
    const long long gx = a.ntile * nouter;
    if (gx <= 0 || gx > 0x7fffffffLL || nmem > 65535) return cudaErrorInvalidValue;
    return launch_pass(k, dim3(unsigned(gx), ncomp, nmem), NC * TPL, smem, st, a);
  }

  // The padding and truncating passes of the 3/2 rule (n == 2L/3) take the
  // form with the maps folded at compile time.
  template <int S, int MODE, int NC>
  static cudaError_t col_std(const ColArgs& a, long long nouter, unsigned ncomp, unsigned nmem, cudaStream_t st) {
    if constexpr (MODE != COL_PLAIN && L % 3 == 0) {
      if (3LL * a.n_short == 2LL * L) return col_run<S, MODE, true, NC>(a, nouter, ncomp, nmem, st);
    }
    return col_run<S, MODE, false, NC>(a, nouter, ncomp, nmem, st);
  }

  static cudaError_t cols(int kind, const ColArgs& a, long long nouter, unsigned ncomp, unsigned nmem,
                          cudaStream_t st) {
    // The column kernels index rows with 32-bit offsets.
    const long long lim = 0x7fffffffLL;
    if ((long long)L * a.in_row >= lim || (long long)L * a.out_row >= lim) return cudaErrorInvalidValue;
    constexpr int NC = TS::NC;
    switch (kind) {
      case COLK_PAD_INV:
        if constexpr (kRegisterColumns<L>) return col_std<+1, COL_PAD, NC>(a, nouter, ncomp, nmem, st);
        else return cudaErrorInvalidValue;
      case COLK_PLAIN_INV: return col_std<+1, COL_PLAIN, NC>(a, nouter, ncomp, nmem, st);
      case COLK_TRUNC_FWD:
        if constexpr (kRegisterColumns<L>) return col_std<-1, COL_TRUNC, NC>(a, nouter, ncomp, nmem, st);
        else return cudaErrorInvalidValue;
      case COLK_PLAIN_FWD: return col_std<-1, COL_PLAIN, NC>(a, nouter, ncomp, nmem, st);
      default: return cudaErrorInvalidValue;
    }
  }

  template <int NCM, bool STD> static cudaError_t epi_run(EpiArgs a, unsigned nmem, cudaStream_t st) {
    constexpr int NB = products(3);
    const size_t smem = size_t(L + L * NB * NCM) * sizeof(C);
    auto k = k_fwd_epilogue<T, L, NCM, V, STD>;
    static const cudaError_t attr = set_smem(k, smem);
    if (attr != cudaSuccess) return attr;
    a.ntile = int((a.ninner + NCM - 1) / NCM);
    if (nmem > 65535) return cudaErrorInvalidValue;
    return launch_pass(k, dim3(unsigned(a.ntile), nmem), NB * NCM * TPL, smem, st, a);
  }

  template <int NCM> static cudaError_t epi_std(const EpiArgs& a, unsigned nmem, cudaStream_t st) {
    if constexpr (L % 3 == 0) {
      if (3LL * a.N == 2LL * L) return epi_run<NCM, true>(a, nmem, st);
    }
    return epi_run<NCM, false>(a, nmem, st);
  }

  static cudaError_t epi(const EpiArgs& a, unsigned nmem, cudaStream_t st) {
    // 32-bit offsets: rows of B and one member's state.
    const long long lim = 0x7fffffffLL;
    if ((long long)L * a.B_row >= lim) return cudaErrorInvalidValue;
    for (const StateLayout& l : {a.lu, a.lu0, a.lout})
      if (2LL * l.comp + (long long)(a.N - 1) * l.row + (a.ninner - 1) * l.ps >= lim) return cudaErrorInvalidValue;
    if constexpr (TS::NCM3_NARROW < TS::NCM3) {
      if (idle_sms((a.ninner + TS::NCM3 - 1) / TS::NCM3 * nmem)) return epi_std<TS::NCM3_NARROW>(a, nmem, st);
    }
    return epi_std<TS::NCM3>(a, nmem, st);
  }
};

// Real <-> complex lines of FFT<Dim>; v: plan variant of r2c.
template <typename T, int L> struct LaunchRows {
  static cudaError_t c2r(const RealRowArgs& a, cudaStream_t st) {
    using Sh = RowShape<T, L>;
    static const cudaError_t attr = set_smem(k_rows_c2r<T, L>, Sh::BYTES);
    if (attr != cudaSuccess) return attr;
    const long long gx = (a.nlines + 2 * Sh::NLP - 1) / (2 * Sh::NLP);
    if (gx > 0x7fffffffLL) return cudaErrorInvalidValue;
    k_rows_c2r<T, L><<<unsigned(gx), Sh::NT, Sh::BYTES, st>>>(a);
    return cudaGetLastError();
  }
  template <int V> static cudaError_t r2c_(const RealRowArgs& a, cudaStream_t st) {
    constexpr int NLP = kclamp(kpow2floor(49152 / (L * int(sizeof(cvec<T>)))), 1, 64);
    constexpr size_t smem = size_t(L + L * (NLP + 1)) * sizeof(cvec<T>);
    auto k = k_rows_r2c<T, L, NLP, V>;
    static const cudaError_t attr = set_smem(k, smem);
    if (attr != cudaSuccess) return attr;
    const long long gx = (a.nlines + 2 * NLP - 1) / (2 * NLP);
    if (gx > 0x7fffffffLL) return cudaErrorInvalidValue;
    k<<<unsigned(gx), NLP * Plan<L, V>::TPL, smem, st>>>(a);
    return cudaGetLastError();
  }
  static cudaError_t r2c(int v, const RealRowArgs& a, cudaStream_t st) { return v ? r2c_<1>(a, st) : r2c_<0>(a, st); }
};

// The product pass (one plan per length).
template <typename T, int L> struct LaunchZ {
  template <int DIM, int NLP, bool STD>
  static cudaError_t run(const ZArgs& a, cudaStream_t st) {
    using Z = ZLineShape<T, L, NLP, DIM>;
    if (a.in_line < a.nh * DIM || a.out_line < a.nh * Z::NB) return cudaErrorInvalidValue;
    // The bulk copy needs a 16-byte aligned chunk of whole line pairs.
    if ((reinterpret_cast<uintptr_t>(a.in) & 15) != 0 || (2LL * a.in_line * Z::CB) % 16 != 0 ||
        (a.in_mem * Z::CB) % 16 != 0 || (a.nlines & 1) != 0)
      return cudaErrorInvalidValue;
    auto k = k_zline<T, L, NLP, DIM, STD>;
    // The limit for the longest lines (rows padded to 128 bytes), raised once.
    constexpr long long kLimit = 227 * 1024 - 512;  // leaves the kernel its static shared memory
    static const cudaError_t attr = [&] {
      const long long most = Z::smem_bytes(DIM * (L / 2 + 1) + 16);
      return set_smem(k, size_t(most < kLimit ? most : kLimit));
    }();
    if (attr != cudaSuccess) return attr;
    const long long smem = Z::smem_bytes(a.in_line);
    if (smem > kLimit) return cudaErrorInvalidValue;
    const long long chunks = (a.nlines + 2 * NLP - 1) / (2 * NLP);
    if (chunks == 0 || a.nmem == 0) return cudaSuccess;
    if (chunks > 0x7fffffffLL || a.nmem > 65535) return cudaErrorInvalidValue;
    return launch_pass(k, dim3(unsigned(chunks), unsigned(a.nmem)), Z::NT, size_t(smem), st, a);
  }
  template <int DIM, int NLP> static cudaError_t run(const ZArgs& a, cudaStream_t st) {
    if constexpr (L % 3 == 0) {
      if (a.nh == L / 3 + 1) return run<DIM, NLP, true>(a, st);
    }
    return run<DIM, NLP, false>(a, st);
  }
  template <int DIM> static cudaError_t run(const ZArgs& a, cudaStream_t st) {
    using Z = ZLineTile<T, L, DIM>;
    if constexpr (Z::NARROW < Z::WIDE) {
      if ((a.nlines + 2 * Z::WIDE - 1) / (2 * Z::WIDE) * a.nmem < 3 * 148) return run<DIM, Z::NARROW>(a, st);
    }
    return run<DIM, Z::WIDE>(a, st);
  }
  // k_zfused: the forward transforms on the wide plan, the inverse on the std
  // plan, four line pairs per CTA in FP32 and two in FP64 (some 80 KB).
  template <bool STD> static cudaError_t run_fused(const ZArgs& a, cudaStream_t st) {
    constexpr int NLP = sizeof(T) == 4 ? 4 : 2;
    using Z = ZFShape<T, L, NLP, 1, 0>;
    if (a.in_line < a.nh * 3 || a.out_line < a.nh * Z::NB) return cudaErrorInvalidValue;
    // Each pair's bulk copy needs 16-byte aligned source, destination and size.
    if ((reinterpret_cast<uintptr_t>(a.in) & 15) != 0 || (2LL * a.in_line * Z::CB) % 16 != 0 ||
        (a.in_mem * Z::CB) % 16 != 0 || (a.nlines & 1) != 0)
      return cudaErrorInvalidValue;
    auto k = k_zfused<T, L, NLP, 1, 0, STD>;
    const int pstride = zfused_pair_stride(a.in_line, Z::CB, NLP, 3, Z::CS, Z::NINV);
    const long long smem = Z::smem_bytes(pstride);
    static const cudaError_t attr = set_smem(k, 227 * 1024 - 512);
    if (attr != cudaSuccess) return attr;
    if (smem > 227 * 1024 - 512) return cudaErrorInvalidValue;
    const long long chunks = (a.nlines + 2 * NLP - 1) / (2 * NLP);
    if (chunks == 0 || a.nmem == 0) return cudaSuccess;
    if (chunks > 0x7fffffffLL || a.nmem > 65535) return cudaErrorInvalidValue;
    return launch_pass(k, dim3(unsigned(chunks), unsigned(a.nmem)), Z::NT, size_t(smem), st, a, pstride);
  }
  static cudaError_t product(int dim, const ZArgs& a, cudaStream_t st) {
    if (dim == 2) return run<2>(a, st);
    if (dim != 3) return cudaErrorInvalidValue;
    if constexpr (kRegisterColumns<L>)
      return a.nh == L / 3 + 1 ? run_fused<true>(a, st) : run_fused<false>(a, st);
    else
      return run<3>(a, st);
  }
};

// The passes of line.cuh.
template <typename T, int L> struct LaunchLine {
  template <typename Tile, int MODE, bool STD>
  static cudaError_t col_run(ColArgs a, long long nouter, unsigned nmem, cudaStream_t st) {
    const size_t smem = ColShape<T, typename Tile::P, Tile::NC>::BYTES;
    auto k = k_columns<T, L, typename Tile::P, Tile::NC, Tile::NT, Tile::MINB, MODE == COL_PAD ? +1 : -1, MODE, STD>;
    static const cudaError_t attr = set_smem(k, smem);
    if (attr != cudaSuccess) return attr;
    a.ntile = int((a.ninner + Tile::NC - 1) / Tile::NC);
    const long long gx = a.ntile * nouter;
    if (gx <= 0 || gx > 0x7fffffffLL || nmem > 65535) return cudaErrorInvalidValue;
    return launch_pass(k, dim3(unsigned(gx), 1, nmem), Tile::NT, smem, st, a);
  }
  template <typename Tile, int MODE>
  static cudaError_t col_std(const ColArgs& a, long long nouter, unsigned nmem, cudaStream_t st) {
    if constexpr (L % 3 == 0) {
      if (3LL * a.n_short == 2LL * L) return col_run<Tile, MODE, true>(a, nouter, nmem, st);
    }
    return col_run<Tile, MODE, false>(a, nouter, nmem, st);
  }
  template <typename Tile, int MODE>
  static cudaError_t col_tile(const ColArgs& a, long long nouter, unsigned nmem, cudaStream_t st) {
    using Narrow = PadTileNarrow<T, L>;
    if constexpr (Narrow::NC < Tile::NC) {
      if (idle_sms((a.ninner + Tile::NC - 1) / Tile::NC * nouter * nmem))
        return col_std<Narrow, MODE>(a, nouter, nmem, st);
    }
    return col_std<Tile, MODE>(a, nouter, nmem, st);
  }
  static cudaError_t columns(int kind, const ColArgs& a, long long nouter, unsigned nmem, cudaStream_t st) {
    const long long lim = 0x7fffffffLL;  // 32-bit row offsets
    if ((long long)L * a.in_row >= lim || (long long)L * a.out_row >= lim) return cudaErrorInvalidValue;
    if (kind == COLK_PAD_STATE) return col_tile<PadStateTile<T, L>, COL_PAD>(a, nouter, nmem, st);
    if (kind == COLK_PAD_INV) return col_tile<PadTile<T, L>, COL_PAD>(a, nouter, nmem, st);
    if (kind == COLK_TRUNC_FWD) return col_tile<PadTile<T, L>, COL_TRUNC>(a, nouter, nmem, st);
    return cudaErrorInvalidValue;
  }

  template <typename Tile, bool STD>
  static cudaError_t epi_run(EpiArgs a, unsigned nmem, cudaStream_t st) {
    const size_t smem = Epi2Shape<T, typename Tile::P, Tile::NCM>::BYTES;
    auto k = k_epilogue2d<T, L, typename Tile::P, Tile::NCM, Tile::NT, Tile::MINB, STD>;
    static const cudaError_t attr = set_smem(k, smem);
    if (attr != cudaSuccess) return attr;
    a.ntile = int((a.ninner + Tile::NCM - 1) / Tile::NCM);
    if (nmem > 65535) return cudaErrorInvalidValue;
    return launch_pass(k, dim3(unsigned(a.ntile), nmem), Tile::NT, smem, st, a);
  }
  template <typename Tile> static cudaError_t epi_std(const EpiArgs& a, unsigned nmem, cudaStream_t st) {
    if constexpr (L % 3 == 0) {
      if (3LL * a.N == 2LL * L) return epi_run<Tile, true>(a, nmem, st);
    }
    return epi_run<Tile, false>(a, nmem, st);
  }
  static cudaError_t epilogue2(const EpiArgs& a, unsigned nmem, cudaStream_t st) {
    using Tile = Epi2Tile<T, L>;
    using Narrow = Epi2TileNarrow<T, L>;
    // 32-bit offsets: rows of B and one member's state.
    const long long lim = 0x7fffffffLL;
    if ((long long)L * a.B_row >= lim) return cudaErrorInvalidValue;
    for (const StateLayout& l : {a.lu, a.lu0, a.lout})
      if (l.comp + (long long)(a.N - 1) * l.row + (a.ninner - 1) * l.ps >= lim) return cudaErrorInvalidValue;
    if constexpr (Narrow::NCM < Tile::NCM) {
      if ((a.ninner + Tile::NCM - 1) / Tile::NCM * nmem <= 148 / 2) return epi_std<Narrow>(a, nmem, st);
    }
    return epi_std<Tile>(a, nmem, st);
  }
};

template <typename T, int L> struct Launch {
  static cudaError_t cols(int v, int kind, const ColArgs& a, long long nouter, unsigned ncomp, unsigned nmem,
                          cudaStream_t st) {
    return (v & 1) ? LaunchV<T, L, 1>::cols(kind, a, nouter, ncomp, nmem, st)
                   : LaunchV<T, L, 0>::cols(kind, a, nouter, ncomp, nmem, st);
  }
  static cudaError_t epilogue3(int v, const EpiArgs& a, unsigned nmem, cudaStream_t st) {
    return v ? LaunchV<T, L, 1>::epi(a, nmem, st) : LaunchV<T, L, 0>::epi(a, nmem, st);
  }
  static const KernelSet* get() {
    static const KernelSet ks = {L,
                                 sizeof(T) == 8 ? 0 : 1,
                                 kRegisterColumns<L>,
                                 &cols,
                                 &LaunchZ<T, L>::product,
                                 &LaunchLine<T, L>::columns,
                                 &epilogue3,
                                 &LaunchLine<T, L>::epilogue2,
                                 &LaunchRows<T, L>::c2r,
                                 &LaunchRows<T, L>::r2c};
    return &ks;
  }
};

}  // namespace azb

#define AZB_INSTANTIATE(TYPE, TAG, LEN)                              \
  namespace azb {                                                    \
  const KernelSet* kernel_set_##TAG##_##LEN() { return Launch<TYPE, LEN>::get(); } \
  }
