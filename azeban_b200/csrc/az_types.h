// Plain-old-data types shared by the CUDA kernels and the host runtime.
#pragma once

#include <cstdint>

namespace azb {

// Per-solve control block, resident in device memory.  Holds the CFL maximum
// of the current right-hand side, the step size and the solve's own clock, so
// a whole SSP-RK3 step runs without a host round trip.
struct alignas(64) Ctrl {
  unsigned long long umax64;  // max |u_i| over the padded grid, FP64 bits
  unsigned int umax32;        // the same, FP32 bits (FP32-bulk solves)
  int skip;                   // 1: this solve is finished, kernels return at once
  double dt;                  // step size of the current SSP-RK3 step
  double time;                // the solve's clock (Simulation::time_)
  double t_end;               // target of simulate_until
  double max_dt;              // min(t_end - time, viscous cap) of this step
  long long nsteps;           // completed steps
  int err;                    // bit 0: non-finite value met in the CFL reduction;
                              // bit 1: a bounded wait on a bulk copy ran out
  int pad_;
};

enum ViscType : int { VISC_NONE = 0, VISC_SMOOTH_CUTOFF = 1, VISC_STEP = 2, VISC_QUADRATIC = 3 };

// Viscosity parameters as the reference's factory leaves them
// (eps already divided by N^{2s-1}, k0 = m0 N^theta).
struct Visc {
  int type;
  int pad_;
  double eps;
  double s;
  double k0;
  long long N;
};

// Products of velocities that a right-hand side transforms: the entries of u (x) u on and
// below its diagonal.  (A multiple of the identity adds only a gradient, which the
// projection removes, so five would do in 3-D, 11 - 33, 21, 22 - 33, 31, 32, and 1.1 times
// as fast.  But the rounding of a large u_z^2 then enters equations that 33 itself, which
// meets nothing but k_z, has no part in: two crossing shear layers with u_x / u_z = 0.01
// were off FP64 by 2.4e-5 instead of 1e-6 in FP32, a jet along z with a hundredth of its
// velocity across it by 2e-5 instead of 3e-7, the same flows along x not at all.)
constexpr int products(int dim) { return dim * (dim + 1) / 2; }

enum Mode : int { MODE_DUDT = 0, MODE_RK1 = 1, MODE_RK2 = 2, MODE_RK3 = 3 };

// What the first pass of a right-hand side does to the control blocks on its
// way: nothing, the start of a step inside simulate_until (max_dt = min(t_end -
// time, cap), src/azeban/simulation.cpp:91-95; a finished solve is marked skip),
// or of a call with a given max_dt.  (One launch less than a kernel of its own;
// these kernels took 1.5 us each beside passes of 4 to 9 us on small solves.)
enum StepBegin : int { BEGIN_NONE = 0, BEGIN_SIM = 1, BEGIN_HOST = 2 };

}  // namespace azb
